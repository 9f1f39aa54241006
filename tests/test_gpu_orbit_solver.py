"""The block-wide FP64 orbit solver and the potential's interpolation constants at the sizes
where they can go wrong, against the oracle at the parity tests' 1e-9: counts of points
around the group, warp, block and work-item sizes; radii on the nodes, inside and outside
the table; an uneven radial grid (the interval guess assumes a logarithmic one); tables too
large for shared memory; velocity rules whose nodes fill part of an item."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fjmodels_gb300 as F  # noqa: E402
from oracle import oracle as O  # noqa: E402
from tests.helpers import rel  # noqa: E402

pytestmark = pytest.mark.gpu
TOL = 1e-9


def dev(a):
    return torch.tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda")


def host(t):
    torch.cuda.synchronize()
    return t.cpu().numpy()


def _model(ctx, nr, npl, uneven=False, xq=O.XPT11, wq=O.XW11):
    ar = F.log_grid(0.01, 100.0, nr)
    if uneven:  # ratios of neighbours from 1.02 to 2, not monotonic
        f = np.cumsum(np.random.default_rng(5).uniform(0.02, 0.7, nr))
        ar = 0.01 * np.exp((f - f[0]) * np.log(1e4) / (f[-1] - f[0]))
    phil, Pr, Pr2 = O.compute_phil(ar, F.guess_rhl(ar, 16, npl, "Hernquist", q=0.8))
    E, D = np.linspace(phil[0, 0] * 0.99, phil[-1, 0] * 1.01, 30), np.linspace(0.04, 0.4, 30)
    m = O.Model(ar, phil, Pr, Pr2, E, D, 8, alpha=1.667, beta=5.0, xq=xq, wq=wq)
    return m, ar, ctx.potential(*map(dev, (ar, phil, Pr, Pr2))), ctx.delta(dev(E), dev(D))


def _points(ar, n, seed):  # every third radius on a node
    g = np.random.default_rng(seed)
    r = np.exp(g.uniform(np.log(ar[0] / 2), np.log(ar[-1] * 2), n))
    r[::3] = ar[g.integers(0, len(ar), len(r[::3]))]
    c = g.uniform(0.02, 0.98, n)
    return np.stack([r * np.sqrt(1 - c * c), r * c], 1), g


@pytest.mark.parametrize("n,nr,npl,uneven", [(1, 11, 1, False), (31, 20, 4, True), (33, 40, 5, False),
                                             (129, 24, 7, True), (257, 16, 3, False), (40, 700, 24, False)])
def test_actions_and_potential(ctx, n, nr, npl, uneven):
    m, ar, pot, delta = _model(ctx, nr, npl, uneven)
    Rz, g = _points(ar, n, n)
    out = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    ctx.potential_eval(pot, dev(Rz), out)
    ref = np.array([[m.phi(R, z), m.dR(R, z), m.dz(R, z)] for R, z in Rz])
    # derivatives on the scale |Phi| / r; the l = 46 sums amplify rounding by up to n^2
    err = np.abs(host(out) - ref) / np.abs(ref[:, :1])
    assert np.max(err[:, 0]) < 1e-12 and np.max(err[:, 1:] * np.hypot(*Rz.T)[:, None]) < 1e-10
    Rz = Rz[np.hypot(*Rz.T) >= ar[0]]  # inside the table's first radius an orbit sees no radial force
    phi = np.array([m.phi(R, z) for R, z in Rz])
    n = len(Rz)
    v = g.standard_normal((n, 3)) * (0.5 * np.sqrt(-2 * phi))[:, None]
    v[::7] *= 4  # some unbound
    pts = np.concatenate([Rz, v], 1)
    out = torch.zeros((n, 2), dtype=torch.float64, device="cuda")
    ctx.uvOrb_actions(pot, delta, dev(pts), out)
    ref = np.array([m.actions(*p) if 0.5 * (p[2:] ** 2).sum() + f < 0 else (-1, -1) for p, f in zip(pts, phi)])
    scale = np.maximum(np.abs(ref), 1e-6 * np.abs(ref).sum(1, keepdims=True))
    assert np.max(np.abs(host(out) - ref) / scale) < TOL


@pytest.mark.parametrize("n,nq", [(1, 4), (1, 10), (2, 12), (12, 8)])
def test_moment_items(ctx, n, nq):
    x, w = F.tanh_sinh_rule(nq)
    m, ar, pot, delta = _model(ctx, 20, 4, xq=x, wq=w)
    Rz, _ = _points(ar[2:-2], n, nq)
    out = torch.zeros((6, n), dtype=torch.float64, device="cuda")
    st = ctx.moments_points(pot, delta, F.DFParams("Hernquist"), F.Rule(x, w), dev(Rz), out)
    ref = np.array([m.rhofDF(R, z)[0] for R, z in Rz])
    got = host(out).T
    assert st.failures == 0
    assert rel(got[:, [0, 2, 3, 4]], ref[:, [0, 2, 3, 4]]) < TOL
