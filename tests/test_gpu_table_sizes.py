"""The action batch at table sizes around the 48 KB of shared memory that need no opt-in, the static
part included, and far beyond: against the oracle at the parity tests' 1e-9."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fjmodels_gb300 as F  # noqa: E402
from oracle import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu
TOL = 1e-9


def dev(a):
    return torch.tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda")


def _model(ctx, nr, npl, xq=O.XPT11, wq=O.XW11):
    ar = F.log_grid(0.01, 100.0, nr)
    phil, Pr, Pr2 = O.compute_phil(ar, F.guess_rhl(ar, 48, npl, "Hernquist", q=0.8), cumulative=True)
    E, D = np.linspace(phil[0, 0] * 0.99, phil[-1, 0] * 1.01, 30), np.linspace(0.04, 0.4, 30)
    m = O.Model(ar, phil, Pr, Pr2, E, D, 8, alpha=1.667, beta=5.0, xq=xq, wq=wq)
    return m, ar, ctx.potential(*map(dev, (ar, phil, Pr, Pr2))), ctx.delta(dev(E), dev(D))


@pytest.mark.parametrize("nr,npl", [(100, 13), (150, 9), (190, 7), (54, 24), (96, 13), (110, 13), (700, 24)])
def test_actions_around_the_opt_in(ctx, nr, npl):
    m, ar, pot, delta = _model(ctx, nr, npl)
    g = np.random.default_rng(nr)
    r, c = np.exp(g.uniform(np.log(0.02), np.log(50.0), 33)), g.uniform(0.05, 0.95, 33)
    Rz = np.stack([r * np.sqrt(1 - c * c), r * c], 1)
    phi = np.array([m.phi(R, z) for R, z in Rz])
    pts = np.concatenate([Rz, g.standard_normal((33, 3)) * (0.4 * np.sqrt(-2 * phi))[:, None]], 1)
    out = torch.zeros((33, 2), dtype=torch.float64, device="cuda")
    ctx.uvOrb_actions(pot, delta, dev(pts), out)
    torch.cuda.synchronize()
    ref = np.array([m.actions(*p) if 0.5 * (p[2:] ** 2).sum() + f < 0 else (-1, -1) for p, f in zip(pts, phi)])
    scale = np.maximum(np.abs(ref), 1e-6 * np.abs(ref).sum(1, keepdims=True))
    assert np.max(np.abs(out.cpu().numpy() - ref) / scale) < TOL
