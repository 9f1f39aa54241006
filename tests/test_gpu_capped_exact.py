"""The mixed form's FP64 pass over capped nodes, node by node: a build of the library in which every
bound node goes through it.  Its actions (fj_set_action_output) are those of the FP64 solver to FP32
rounding (2^-24, and the parity tests' 1e-9 between two FP64 solves), its moments the plain FP64 form's
to 1e-9.  Tables staged in shared memory and read from device memory; the list of left nodes as it
is, and too short, so that most nodes are solved item by item; a batch of both models."""
import concurrent.futures as cf
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fjmodels_gb300 as F  # noqa: E402
from fjmodels_gb300 import _abi as A  # noqa: E402
from fjmodels_gb300 import build as B  # noqa: E402
from oracle import oracle as O  # noqa: E402
from tests.helpers import rel  # noqa: E402

pytestmark = pytest.mark.gpu
TOL = 1e-9
NQ, NPTS = 10, 9


def dev(a):
    return torch.tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda")


@pytest.fixture(scope="module")
def libs(tmp_path_factory):
    """the library with every bound node left to the FP64 pass, with the list as it is and of 100 entries"""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    B.build(force=not all(os.path.exists(os.path.join(B.BUILD, s.replace(".cu", ".o"))) for s in B.SOURCES))
    d = tmp_path_factory.mktemp("capped")

    def obj(src, define):
        out = str(d / (src + ".o"))
        subprocess.run([B.nvcc(), *B.ARCH, *B.FLAGS, *B.SOURCES[src], define, "-c", os.path.join(B.CSRC, src), "-o", out],
                       check=True)
        return out

    with cf.ThreadPoolExecutor(2) as ex:
        new = dict(zip(("fj_moments_mixed.cu", "fj_api.cu"),
                       ex.map(obj, ("fj_moments_mixed.cu", "fj_api.cu"), ("-DFJ_MIXED_LEAVE_ALL=1", "-DFJ_DEFER_LIST=100"))))
    out = []
    for name, replaced in (("list", ["fj_moments_mixed.cu"]), ("short", ["fj_moments_mixed.cu", "fj_api.cu"])):
        path = str(d / f"lib{name}.so")
        objs = [new[s] if s in replaced else os.path.join(B.BUILD, s.replace(".cu", ".o")) for s in B.SOURCES]
        subprocess.run([B.nvcc(), *B.ARCH, "-shared", "-o", path, *objs, "-lcudart", "-lpthread"], check=True)
        lib = C.CDLL(path)
        for fn, (args, res) in A.SIGNATURES.items():
            getattr(lib, fn).argtypes, getattr(lib, fn).restype = args, res
        out.append(lib)
    return out


def _model(nr, npl):
    ar = F.log_grid(0.01, 100.0, nr)
    tabs = O.compute_phil(ar, F.guess_rhl(ar, 24, npl, "Hernquist", q=0.8), cumulative=True)
    E, D, _ = F.tabulate_delta(ar, *tabs)
    g = np.random.default_rng(nr)
    r, c = np.exp(g.uniform(np.log(0.03), np.log(30.0), NPTS)), g.uniform(0.05, 0.95, NPTS)
    return ar, tabs, (E, D), np.stack([r * np.sqrt(1 - c * c), r * c], 1)


def _device(ctx, model):
    ar, tabs, table, _ = model
    return ctx.potential(*map(dev, (ar, *tabs))), ctx.delta(*map(dev, table))


@pytest.mark.parametrize("which", [0, 1], ids=["list", "short list"])
@pytest.mark.parametrize("nr,npl", [(24, 4), (200, 9)], ids=["staged", "device memory"])
def test_every_node(libs, monkeypatch, which, nr, npl):
    model = _model(nr, npl)
    x, w = F.tanh_sinh_rule(NQ)
    df, pts = F.DFParams("Hernquist", chi=1.0), model[3]
    plain = F.Context(0)
    pot, delta = _device(plain, model)
    want = torch.zeros((6, NPTS), dtype=torch.float64, device="cuda")
    bound = plain.moments_points(pot, delta, df, F.Rule(x, w), dev(pts), want).bound
    # the nodes' velocities, as the moments form them
    far = np.array([[10 * model[0][-1]] * 2])
    out = torch.zeros((NPTS + 1, 3), dtype=torch.float64, device="cuda")
    plain.potential_eval(pot, dev(np.concatenate([pts, far])), out)
    phi = out.cpu().numpy()[:, 0]
    Ve = np.sqrt(-2 * (phi[:-1] - phi[-1]))
    V = 1e-6 + Ve[:, None, None] * np.stack(np.meshgrid(x, x, x, indexing="ij"), -1).reshape(1, NQ ** 3, 3)
    every = np.concatenate([np.broadcast_to(pts[:, None, :], (NPTS, NQ ** 3, 2)), V], -1)
    ref = torch.zeros((NPTS * NQ ** 3, 2), dtype=torch.float64, device="cuda")
    plain.uvOrb_actions(pot, delta, dev(every.reshape(-1, 5)), ref)
    torch.cuda.synchronize()
    ref = ref.cpu().numpy()
    plain.close()

    monkeypatch.setattr(A, "_lib", libs[which])
    ctx = F.Context(0)
    jout = torch.zeros((NPTS, NQ ** 3, 2), dtype=torch.float32, device="cuda")
    got = torch.zeros_like(want)
    ctx.set_action_output(jout)
    st = ctx.moments_points(pot, delta, df, F.Rule(x, w, precision=A.FJ_PREC_MIXED), dev(pts), got)
    torch.cuda.synchronize()
    ctx.close()
    assert st.resolved64 == st.bound == bound and st.failures == 0
    J = jout.cpu().numpy().reshape(-1, 2).astype(np.float64)
    assert np.array_equal(np.isnan(J[:, 0]), ref[:, 0] == -1)
    on = ref[:, 0] != -1
    scale = np.maximum(np.abs(ref[on]), 1e-6 * np.abs(ref[on]).sum(1, keepdims=True))
    assert np.max(np.abs(J[on] - ref[on]) / scale) < 2.0 ** -24 + TOL
    a, b = got.cpu().numpy(), want.cpu().numpy()
    for q in (0, 2, 3, 4):
        assert rel(a[q], b[q]) < TOL, q


def test_batch(libs, monkeypatch):
    """a staged model and one in device memory in one launch, nodes beyond the list in both"""
    rules = [F.Rule(*F.tanh_sinh_rule(8), precision=p) for p in (A.FJ_PREC_FP64, A.FJ_PREC_MIXED)]
    df, models = F.DFParams("Hernquist", chi=0.5), [_model(24, 4), _model(200, 9)]
    outs = []
    for rule, lib in ((rules[0], A._lib), (rules[1], libs[0]), (rules[1], libs[1])):
        monkeypatch.setattr(A, "_lib", lib)
        ctx = F.Context(0)
        items = [(*_device(ctx, m), df, ng, torch.zeros((6, len(m[0]), ng), dtype=torch.float64, device="cuda"))
                 for m, ng in zip(models, (2, 1))]
        st = ctx.moments_batch(items, rule)
        torch.cuda.synchronize()
        outs.append([it[4].cpu().numpy() for it in items])
        ctx.close()
        assert rule is rules[0] or st.resolved64 == st.bound > 100
    for o in outs[1:]:
        for a, b in zip(o, outs[0]):
            for q in (0, 2, 3, 4):
                assert rel(a[q], b[q]) < TOL, q
