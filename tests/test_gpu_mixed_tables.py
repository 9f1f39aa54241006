"""Mixed-form models whose tables do not fit a block's shared memory beside the node lists: moments
against the oracle at the mixed form's 1e-4; a small model launched together with a large one has
the bits of its own launch (the same tables, read elsewhere)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fjmodels_gb300 as F  # noqa: E402
from fjmodels_gb300 import _abi as A  # noqa: E402
from oracle import oracle as O  # noqa: E402
from tests.helpers import rel  # noqa: E402

pytestmark = pytest.mark.gpu
MIXED_TOL = 1e-4


def dev(a):
    return torch.tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda")


def _model(ctx, nr, npl, xq=O.XPT11, wq=O.XW11):
    ar = F.log_grid(0.01, 100.0, nr)
    phil, Pr, Pr2 = O.compute_phil(ar, F.guess_rhl(ar, 48, npl, "Hernquist", q=0.8), cumulative=True)
    E, D = np.linspace(phil[0, 0] * 0.99, phil[-1, 0] * 1.01, 30), np.linspace(0.04, 0.4, 30)
    m = O.Model(ar, phil, Pr, Pr2, E, D, 8, alpha=1.667, beta=5.0, xq=xq, wq=wq)
    return m, ar, ctx.potential(*map(dev, (ar, phil, Pr, Pr2))), ctx.delta(dev(E), dev(D))


@pytest.mark.parametrize("nr,npl", [(570, 24), (700, 24), (1200, 12), (2600, 5), (7000, 1)])
def test_large_mixed_models(ctx, nr, npl):
    x, w = F.tanh_sinh_rule(12)
    rule, df = F.Rule(x, w, precision=A.FJ_PREC_MIXED), F.DFParams("Hernquist")
    m, ar, pot, delta = _model(ctx, nr, npl, x, w)
    pts = np.array([[0.3, 0.2], [2.0, 1.5]])
    out = torch.zeros((6, 2), dtype=torch.float64, device="cuda")
    st = ctx.moments_points(pot, delta, df, rule, dev(pts), out)
    torch.cuda.synchronize()
    ref = np.array([m.rhofDF(R, z)[0] for R, z in pts])
    got = out.cpu().numpy().T
    assert st.failures == 0
    assert rel(got[:, [0, 2, 3, 4]], ref[:, [0, 2, 3, 4]]) < MIXED_TOL


def test_small_model_beside_a_large_one(ctx):
    """Both launched together, so the small one too goes through the kernels of large tables."""
    rule = F.Rule(*F.tanh_sinh_rule(6), precision=A.FJ_PREC_MIXED)
    df = F.DFParams("Hernquist", chi=1.0)
    items = []
    for nr, npl, ng in ((24, 5, 3), (1100, 24, 1)):
        _, _, pot, delta = _model(ctx, nr, npl)
        items.append((pot, delta, df, ng, torch.zeros((6, nr, ng), dtype=torch.float64, device="cuda")))
    ctx.moments_batch(items, rule)
    alone = torch.zeros_like(items[0][4])
    ctx.moments(*items[0][:3], rule, 3, alone)
    torch.cuda.synchronize()
    assert torch.equal(items[0][4], alone)
