"""One context used from several streams without a synchronisation in between: its calls share work
counters, orbit records and partial sums, so each waits for the one before it whatever its stream."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fjmodels_gb300 as F  # noqa: E402
from fjmodels_gb300 import _abi as A  # noqa: E402
from oracle import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda")


def _inputs(ctx, n, seed):
    ar = F.log_grid(0.01, 100.0, 40)
    phil, Pr, Pr2 = O.compute_phil(ar, F.guess_rhl(ar, 16, 5, "Hernquist", q=0.8), cumulative=True)
    E, D = np.linspace(phil[0, 0] * 0.99, phil[-1, 0] * 1.01, 30), np.linspace(0.04, 0.4, 30)
    g = np.random.default_rng(seed)
    r, c = np.exp(g.uniform(np.log(0.05), np.log(30.0), n)), g.uniform(0.05, 0.95, n)
    v = g.standard_normal((n, 3)) * (0.4 / np.sqrt(1 + r))[:, None]
    pts = dev(np.concatenate([np.stack([r * np.sqrt(1 - c * c), r * c], 1), v], 1))
    return ctx.potential(*map(dev, (ar, phil, Pr, Pr2))), ctx.delta(dev(E), dev(D)), pts


def _out(n):
    return torch.zeros((n, 2), dtype=torch.float64, device="cuda")


def test_action_calls_on_two_streams(ctx):
    cases = [_inputs(ctx, n, n) for n in (20_001, 700, 9_000, 64)]
    want = [_out(len(c[2])) for c in cases]
    for c, o in zip(cases, want):
        ctx.uvOrb_actions(*c, o)
        torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(4):
        got = [_out(len(c[2])) for c in cases]
        torch.cuda.synchronize()
        for i, (c, o) in enumerate(zip(cases, got)):
            with torch.cuda.stream(streams[i % 2]):
                ctx.uvOrb_actions(*c, o)
        torch.cuda.synchronize()
        for g, w in zip(got, want):
            assert torch.equal(g, w)


@pytest.mark.parametrize("precision", [A.FJ_PREC_FP64, A.FJ_PREC_MIXED])
def test_moments_and_actions_on_two_streams(ctx, precision):
    """fj_moments_points without stats returns with its work queued."""
    pot, delta, pts = _inputs(ctx, 4_000, 5)
    df, rule = F.DFParams("Hernquist"), F.Rule(*F.tanh_sinh_rule(8), precision=precision)
    Rz = [pts[:40, :2].contiguous(), pts[40:64, :2].contiguous()]

    def moments(i, out):
        ctx._on_torch_stream()
        ctx._check(ctx.lib.fj_moments_points(ctx.h, pot.c, delta.c, df.c, rule.c, Rz[i].data_ptr(), len(Rz[i]),
                                             out.data_ptr(), None), "fj_moments_points")

    def outs():
        return [torch.zeros((6, len(r)), dtype=torch.float64, device="cuda") for r in Rz] + [_out(len(pts))]

    def run(got, streams):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                moments(i, got[i]) if i < 2 else ctx.uvOrb_actions(pot, delta, pts, got[2])
            if len(set(streams)) == 1:
                torch.cuda.synchronize()
        torch.cuda.synchronize()

    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    want = outs()
    torch.cuda.synchronize()
    run(want, [a, a, a])
    for _ in range(3):
        got = outs()
        torch.cuda.synchronize()
        run(got, [a, b, a])
        for g, w in zip(got, want):
            assert torch.equal(g, w)
