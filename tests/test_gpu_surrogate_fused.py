"""The fused surrogate kernel against the separate passes at the sizes where its tiles and
node lists can go wrong: a velocity rule of four points, fewer bound nodes than a tile, a
remainder, several node ranges per point, a rule too long for the tabulated squares.  Both
evaluate the same network with the same BF16 rounding points, so the moments agree to the
summation order: 1e-12 of the density (and of the dispersions)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fjmodels_gb300 as F  # noqa: E402
from oracle import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,ng,npl,nq,chi", [(12, 1, 1, 4, 0.0), (11, 3, 2, 6, 1.0), (16, 2, 9, 14, 0.5),
                                              (12, 1, 4, 24, 1.0), (11, 1, 3, 66, 0.0)])
def test_fused_equals_separate_passes(ctx, nr, ng, npl, nq, chi):
    ar = F.log_grid(0.01, 100.0, nr)
    phil, Pr, Pr2 = O.compute_phil(ar, F.guess_rhl(ar, 8, npl, "Hernquist", q=0.8))
    dev = lambda a: torch.tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda")  # noqa: E731
    pot = ctx.potential(*map(dev, (ar, phil, Pr, Pr2)))
    df, rule = F.DFParams("Hernquist", chi=chi), F.Rule(*F.tanh_sinh_rule(nq))
    s = F.Surrogate(ctx, batch=1024, seed=5)
    p = s.params()
    p += 0.05 * np.random.default_rng(1).standard_normal(p.size) * (p != 0)  # activations over a wide range
    s.set_params(p)
    got = [torch.zeros((6, nr, ng), dtype=torch.float64, device="cuda") for _ in range(2)]
    for g, fused in zip(got, (True, False)):
        s.moments(pot, df, rule, ng, g, fused=fused)
    torch.cuda.synchronize()
    a, b = (g.cpu().numpy() for g in got)
    assert np.all(b[0] > 0)
    for q in (0, 2, 3, 4):
        assert np.max(np.abs(a[q] - b[q]) / np.abs(b[q])) < 1e-12, q
    s.close()
