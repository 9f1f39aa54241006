"""The mixed form's two kernels at the sizes where they can go wrong: multipole counts with an
unrolled loop (3 to 8) and without one, velocity rules whose nodes fill part of an item, every
build and item size, launches worked off in slices."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fjmodels_gb300 as F  # noqa: E402
from fjmodels_gb300 import _abi as A  # noqa: E402
from oracle import oracle as O  # noqa: E402
from tests.helpers import rel  # noqa: E402

pytestmark = pytest.mark.gpu
MIXED_TOL = 1e-4  # the mixed form's gate on the density and the dispersions
ORDER_TOL = 1e-12  # the same node values, summed in another order


def dev(a):
    return torch.tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda")


def _model(ctx, nr, npl):
    ar = F.log_grid(1e-3, 300.0, nr)
    phil, Pr, Pr2 = O.compute_phil(ar, F.guess_rhl(ar, 24, npl, "NFW", q=0.8))
    E, D, _ = F.tabulate_delta(ar, phil, Pr, Pr2)
    return ctx.potential(*map(dev, (ar, phil, Pr, Pr2))), ctx.delta(dev(E), dev(D))


def _points(n, seed):
    g = np.random.default_rng(seed)
    r, c = np.exp(g.uniform(np.log(2e-3), np.log(100.0), n)), g.uniform(0.05, 0.95, n)
    return dev(np.stack([r * np.sqrt(1 - c * c), r * c], 1))


def _moments(ctx, model, rule, pts):
    out = torch.zeros((6, len(pts)), dtype=torch.float64, device="cuda")
    ctx.moments_points(*model, F.DFParams("NFW", chi=1.0, k=0.5), rule, pts, out)
    torch.cuda.synchronize()
    return out


@pytest.fixture
def config(ctx):
    before = ctx.mixed_config()
    yield ctx.set_mixed_config
    ctx.set_mixed_config(*before)


@pytest.mark.parametrize("npl", [1, 2, 3, 8, 9])
def test_multipole_counts_vs_plain(ctx, npl):
    model, pts = _model(ctx, 40, npl), _points(7, npl)
    x, w = F.tanh_sinh_rule(22)
    a = _moments(ctx, model, F.Rule(x, w, precision=A.FJ_PREC_MIXED), pts).cpu().numpy()
    b = _moments(ctx, model, F.Rule(x, w), pts).cpu().numpy()
    for q in (0, 2, 3, 4):
        assert rel(a[q], b[q]) < MIXED_TOL, q


@pytest.mark.parametrize("nq", [5, 6, 11])  # 125, 216 and 1331 nodes per point
@pytest.mark.parametrize("npl", [2, 5])
def test_builds_and_item_sizes_agree(ctx, config, npl, nq):
    model, pts = _model(ctx, 24, npl), _points(9, nq)
    g = np.random.default_rng(nq)
    x = np.sort(g.uniform(-0.95, 0.95, nq))
    rule = F.Rule(x, np.full(nq, 2.0 / nq), precision=A.FJ_PREC_MIXED)
    config(7, 1024)
    ref = _moments(ctx, model, rule, pts)
    scale = ref.abs().amax(dim=1, keepdim=True)
    for chunk in (128, 129, 1000, 8192):
        first = None
        for variant in range(8):
            config(variant, chunk)
            out = _moments(ctx, model, rule, pts)
            first = out if first is None else first
            assert torch.equal(out, first), (variant, chunk)
        assert bool(((first - ref).abs() <= ORDER_TOL * scale).all()), chunk


def test_slices_of_a_large_launch(ctx, config):
    """1 991 points (21.2 M nodes) take two slices; the same points in three calls take one each."""
    config(7, 1024)
    model, pts = _model(ctx, 24, 4), _points(1991, 3)
    x, w = F.tanh_sinh_rule(22)
    rule = F.Rule(x, w, precision=A.FJ_PREC_MIXED)
    whole = _moments(ctx, model, rule, pts)
    parts = torch.cat([_moments(ctx, model, rule, p) for p in (pts[:700], pts[700:1500], pts[1500:])], dim=1)
    assert torch.equal(whole, parts)
