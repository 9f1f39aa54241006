"""The mixed form's evaluator as the kernels run it -- tables of differences and quadratic corrections,
the multipole loop unrolled -- has the bits of the form without them, at positions inside and beyond
the grid, on its nodes, in its quadratic part and beside the grid point; and is the FP64 potential's
difference to FP32 rounding."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import fjmodels_gb300 as F
from oracle import oracle as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    out = tmp_path_factory.mktemp("evaluator") / "evaluator"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "fjmodels_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "host_evaluator.cpp"), "-o", str(out)], check=True)
    return out


@pytest.mark.parametrize("nr,npl", [(11, 1), (12, 2), (24, 3), (40, 5), (80, 7), (33, 8), (60, 9), (40, 24)])
def test_tables_and_unrolled_loop(exe, nr, npl):
    ar = F.log_grid(0.01, 100.0, nr)
    phil = O.compute_phil(ar, F.guess_rhl(ar, 48, npl, "Hernquist", q=0.8), cumulative=True)[0]
    g = np.random.default_rng(nr)
    n = 600
    r = np.exp(g.uniform(np.log(0.01), np.log(100.0), n))
    c = g.uniform(0.02, 0.98, n)
    s = np.exp(g.uniform(np.log(0.004), np.log(300.0), n))
    s[::4] = r[::4] * (1 + 0.02 * g.standard_normal(len(r[::4])))  # beside the point
    s[1::6] = ar[g.integers(0, nr, len(s[1::6]))]
    s[2::6] = np.exp(g.uniform(np.log(ar[0]), np.log(ar[min(10, nr - 1)]), len(s[2::6])))
    d = g.uniform(0.02, 0.98, n)
    pos = np.stack([r * np.sqrt(1 - c * c), r * c, s * np.sqrt(1 - d * d), s * d], 1)
    text = f"{nr} {npl}\n" + "\n".join(map(repr, [*ar.tolist(), *phil.ravel().tolist()])) + f"\n{n}\n" + "\n".join(
        " ".join(map(repr, p)) for p in pos.tolist())
    out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout.splitlines()
    rows = [line.split() for line in out]
    assert len(rows) == n
    assert all(a == b == c for a, b, c, _, _ in rows)
    got, ref = np.array([[float(x[3]), float(x[4])] for x in rows]).T
    scale = np.abs(phil[0, 0])
    assert np.max(np.abs(got - ref)) < 1e-5 * scale  # the sum of 2 npoly + 2 FP32 roundings of values up to |Phi(0)|
