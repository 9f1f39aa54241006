"""The moments when the device refuses their workspace (2.2 GB of node records for a large mixed
launch, 0.2 GB of the blocks' scratch in FP64): smaller slices and fewer blocks, the same bits,
and no error left behind.  A cudaMalloc in front of the
library's refuses everything above a limit, with the runtime's own answer to an absurd size."""
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
#include <stdlib.h>
int cudaMalloc(void **p, size_t n)
{
    static int (*real)(void **, size_t);
    if (!real) real = (int (*)(void **, size_t))dlsym(RTLD_NEXT, "cudaMalloc");
    const char *max = getenv("MALLOC_MAX");
    return real(p, max && n > strtoull(max, 0, 10) ? (size_t)1 << 60 : n);
}
extern int cudaGetDeviceCount(int *);
int needs_the_runtime(void) { int n; return cudaGetDeviceCount(&n); }
"""

RUN = r"""
import os, sys
import numpy as np, torch
import fjmodels_gb300 as F
from fjmodels_gb300 import _abi as A
from oracle import oracle as O
dev = lambda a: torch.tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda")
ar = F.log_grid(0.01, 100.0, 24)
phil, Pr, Pr2 = O.compute_phil(ar, F.guess_rhl(ar, 16, 4, "Hernquist", q=0.8))
E, D, _ = F.tabulate_delta(ar, phil, Pr, Pr2)
g = np.random.default_rng(1)
r, c = np.exp(g.uniform(np.log(0.02), np.log(30.0), 150)), g.uniform(0.05, 0.95, 150)
pts = dev(np.stack([r * np.sqrt(1 - c * c), r * c], 1))  # 150 points of 22^3 nodes: 190 MB of records
rules = [F.Rule(*F.tanh_sinh_rule(22), precision=p) for p in (A.FJ_PREC_MIXED, A.FJ_PREC_FP64)]
df = F.DFParams("Hernquist", chi=1.0)
outs = [[], []]
for limit in (None, 48 << 20):
    ctx = F.Context(0)
    pot, delta = ctx.potential(*map(dev, (ar, phil, Pr, Pr2))), ctx.delta(dev(E), dev(D))
    if limit:
        os.environ["MALLOC_MAX"] = str(limit)
    for _ in range(3):
        for o, rule in zip(outs, rules):
            o.append(torch.zeros((6, 150), dtype=torch.float64, device="cuda"))
            ctx.moments_points(pot, delta, df, rule, pts, o[-1])
    few = torch.zeros((6, 2), dtype=torch.float64, device="cuda")
    for rule in rules:
        ctx.moments_points(pot, delta, df, rule, pts[:2].contiguous(), few)  # nothing of the refusal is left
    ctx.close()
torch.cuda.synchronize()
assert all(torch.equal(x, o[0]) for o in outs for x in o)
print("same")
"""


def test_refused_workspace(tmp_path):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    src, lib = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "lib64")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(lib), str(src), f"-L{cuda}", f"-Wl,-rpath,{cuda}", "-lcudart",
                    "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(lib), PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", RUN], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stderr[-2000:]
