"""The bracket search of the radial integrals (bracket_near), compiled for the host: the interval of
numpy's search on logarithmic, linear and uneven grids, whatever the guess, in few reads of the grid
-- two for a right guess, 2 log2(d) + 4 for one d intervals off."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    out = tmp_path_factory.mktemp("bracket") / "bracket"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "fjmodels_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "host_bracket.cpp"), "-o", str(out)], check=True)
    return out


@pytest.mark.parametrize("nr", [2, 3, 4, 17, 80, 601, 4096])
@pytest.mark.parametrize("kind", ["log", "linear", "uneven"])
def test_interval_and_reads(exe, nr, kind):
    g = np.random.default_rng(nr)
    ar = {"log": np.geomspace(1e-3, 300.0, nr), "linear": np.linspace(0.01, 100.0, nr),
          "uneven": np.cumsum(np.exp(g.uniform(-8, 2, nr)))}[kind]
    x = np.concatenate([ar[:-1], np.nextafter(ar[1:], 0), ar[0] + (ar[-1] - ar[0]) * g.uniform(0, 1, 200)])
    want = np.searchsorted(ar, x, side="right") - 1
    want[x >= ar[-1]] = nr - 2
    logs = ((np.log(x) - np.log(ar[0])) * (nr - 1) / (np.log(ar[-1]) - np.log(ar[0]))).astype(int)
    xs, guesses, wants = [], [], []
    for gu in (logs, want, want - 1, want + 1, np.zeros_like(want), np.full_like(want, nr), g.integers(0, nr, len(x))):
        xs.append(x), guesses.append(np.clip(gu, 0, nr - 2)), wants.append(want)
    xs, guesses, wants = map(np.concatenate, (xs, guesses, wants))
    text = f"{nr}\n" + " ".join(map(repr, ar.tolist())) + f"\n{len(xs)}\n" + "\n".join(
        f"{a!r} {b}" for a, b in zip(xs.tolist(), guesses.tolist()))
    r = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True)
    got = np.array([line.split() for line in r.stdout.splitlines()], dtype=int)
    assert np.array_equal(got[:, 0], wants)
    d = np.abs(guesses - wants)
    assert np.all(got[:, 1] <= np.where(d == 0, 2, 2 * np.log2(np.maximum(d, 1)) + 4))
