"""The capped nodes' FP64 pass of the mixed form (two warps per node, bracket walks of 32
positions at once) at models whose tables are staged in shared memory and ones read from global
memory: the moments against the plain FP64 form, and the same bits in every launch shape."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fjmodels_gb300 as F  # noqa: E402
from fjmodels_gb300 import _abi as A  # noqa: E402
from oracle import oracle as O  # noqa: E402
from tests.helpers import rel  # noqa: E402

pytestmark = pytest.mark.gpu
MIXED_TOL = 1e-4  # the mixed form's gate on the density and the dispersions


def dev(a):
    return torch.tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda")


@pytest.mark.parametrize("nr,npl,kind", [(80, 7, "NFW"), (200, 9, "NFW"), (40, 1, "Hernquist")])
def test_capped_nodes(ctx, nr, npl, kind):
    lo, hi = (1e-3, 300.0) if kind == "NFW" else (1e-2, 100.0)
    ar = F.log_grid(lo, hi, nr)
    phil, Pr, Pr2 = O.compute_phil(ar, F.guess_rhl(ar, 24, npl, kind, q=0.8))
    E, D, _ = F.tabulate_delta(ar, phil, Pr, Pr2)
    pot, delta = ctx.potential(*map(dev, (ar, phil, Pr, Pr2))), ctx.delta(dev(E), dev(D))
    g = np.random.default_rng(nr)
    r, c = np.exp(g.uniform(np.log(2 * lo), np.log(hi / 3), 48)), g.uniform(0.05, 0.95, 48)
    pts = dev(np.stack([r * np.sqrt(1 - c * c), r * c], 1))
    x, w = F.tanh_sinh_rule(22)
    df = F.DFParams(kind, chi=1.0, k=0.5)
    outs, resolved = [], []
    for rule, p in ((F.Rule(x, w), pts), (F.Rule(x, w, precision=A.FJ_PREC_MIXED), pts),
                    (F.Rule(x, w, precision=A.FJ_PREC_MIXED), pts.flip(0).contiguous())):
        out = torch.zeros((6, len(pts)), dtype=torch.float64, device="cuda")
        resolved.append(ctx.moments_points(pot, delta, df, rule, p, out).resolved64)
        torch.cuda.synchronize()
        outs.append(out)
    plain, mixed = outs[0].cpu().numpy(), outs[1].cpu().numpy()
    for q in (0, 2, 3, 4):
        assert rel(mixed[q], plain[q]) < MIXED_TOL, q
    assert torch.equal(outs[2].flip(1), outs[1])
    assert resolved[1] == resolved[2]
