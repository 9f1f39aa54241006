"""The kernels' QAGS bookkeeping (GroupQags of fj_group_qags.cuh, the source the GPU compiles), on the
CPU: FP64 against the oracle's QAGS (result and QUADPACK class), FP32 against the one-thread FP32 form
bit for bit, on smooth, kinked, singular, oscillating and noisy integrands, with the tolerances of the
momentum integrals, the radial integrals and tighter ones; and a list that runs full."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from oracle import oracle as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
F64, F32 = C.CFUNCTYPE(C.c_double, C.c_double), C.CFUNCTYPE(C.c_float, C.c_float)

CASES = {
    "smooth": (lambda x: np.sin(x) ** 2, 0.0, np.pi),
    "kinks": (lambda x: abs(np.sin(5 * x)) + abs(x - 0.3) ** 0.5, 0.0, 2.0),
    "root ends": (lambda x: np.sqrt(max(0.0, x * (1 - x))) * np.sin(x), 0.0, 1.0),
    "cut": (lambda x: np.sqrt(max(0.0, np.cos(3 * x))) * np.sin(x), 0.0, np.pi / 2),
    "log": (lambda x: np.log(x), 0.0, 1.0),
    "inverse root": (lambda x: 1.0 / np.sqrt(x), 0.0, 1.0),
    "strong pole": (lambda x: x ** -0.95, 0.0, 1.0),
    "peak": (lambda x: 1.0 / (1e-8 + (x - 0.377) ** 2), 0.0, 1.0),
    "oscillating": (lambda x: np.sin(300 * x * x), 0.0, 2.0),
    "step": (lambda x: 1.0 if x > 0.123456 else 0.0, 0.0, 1.0),
    "zero": (lambda x: 0.0, 0.0, 1.0),
    "cancelling": (lambda x: (x - 0.5) ** 3 * abs(x - 0.1), 0.0, 1.0),
    "noise": (lambda x: 1e-3 * np.sin(1e5 * x) + x, 0.0, 1.0),
}
TOLS = [(1e-5, 1e-3), (1e-4, 1e-3), (1e-9, 1e-7), (8e-4, 8e-3)]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    so = tmp_path_factory.mktemp("qags") / "qags.so"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "fjmodels_gb300", "csrc"), os.path.join(ROOT, "tests", "host_group_qags.cpp"),
                    "-o", str(so)], check=True)
    L = C.CDLL(str(so))
    L.group64.argtypes = [F64, C.c_int] + [C.c_double] * 4 + [C.POINTER(C.c_double), C.POINTER(C.c_int)]
    for fn in (L.group32, L.one_thread32):
        fn.argtypes, fn.restype = [F32] + [C.c_float] * 4 + [C.POINTER(C.c_int)], C.c_float
    return L


@pytest.mark.parametrize("tol", TOLS, ids=str)
@pytest.mark.parametrize("name", CASES)
def test_fp64_against_the_oracle(lib, name, tol):
    f, a, b = CASES[name]
    r, full = C.c_double(), C.c_int()
    ier = lib.group64(F64(f), 21, a, b, *tol, C.byref(r), C.byref(full))
    ref, _, ref_ier = O.qags(f, a, b, *tol)
    assert ier >= 0, "an interval's number in the tree is not its own"
    if full.value:  # the oracle's list holds 1000 intervals
        assert ref_ier != 0 or abs(r.value - ref) <= 10 * max(tol[0], tol[1] * abs(ref))
        return
    assert ier == ref_ier
    assert abs(r.value - ref) <= 1e-12 * abs(ref)


def test_fp64_15_points(lib):
    """the rule of the external integrals, on the transformed half line (the oracle's QAGIU)"""
    for f, a in ((lambda x: x ** -3.0, 0.7), (lambda x: np.exp(-x) * abs(np.sin(x)), 0.1), (lambda x: 1 / (1 + x * x), 5.0)):
        g = lambda t: f(a + (1 - t) / t) / t / t  # noqa: E731
        r, full = C.c_double(), C.c_int()
        ier = lib.group64(F64(g), 15, 0.0, 1.0, 1e-4, 1e-3, C.byref(r), C.byref(full))
        ref, _, ref_ier = O.qagiu(f, a)
        assert ier == ref_ier and not full.value
        assert abs(r.value - ref) <= 1e-12 * abs(ref)


@pytest.mark.parametrize("tol", TOLS, ids=str)
@pytest.mark.parametrize("name", CASES)
def test_fp32_against_one_thread(lib, name, tol):
    f, a, b = CASES[name]
    full = [C.c_int(), C.c_int()]
    got = lib.group32(F32(f), a, b, *tol, C.byref(full[0]))
    ref = lib.one_thread32(F32(f), a, b, *tol, C.byref(full[1]))
    assert np.float32(got).tobytes() == np.float32(ref).tobytes()
    assert full[0].value == full[1].value


def test_a_list_runs_full(lib):
    f = F32(lambda x: np.sin(4000 * x * x))
    full = C.c_int()
    lib.group32(f, 0.0, 3.0, 1e-9, 1e-7, C.byref(full))
    assert full.value == 1
    r, full64 = C.c_double(), C.c_int()
    lib.group64(F64(lambda x: np.sin(4000 * x * x)), 21, 0.0, 12.0, 1e-12, 1e-12, C.byref(r), C.byref(full64))
    assert full64.value == 1 and np.isfinite(r.value)
