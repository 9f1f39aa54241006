"""The adaptive and cumulative Poisson kernels at the sizes where their launch shapes can go
wrong, against the oracle at the parity tests' 1e-9: one multipole, odd numbers of integrals,
grids beyond the tabulated powers and reciprocals, an uneven grid, a density whose external
integrals are tried again with doubled tolerances."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fjmodels_gb300 as F  # noqa: E402
from fjmodels_gb300 import _abi as A  # noqa: E402
from oracle import oracle as O  # noqa: E402
from tests.helpers import rel_rows  # noqa: E402

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda")


@pytest.mark.parametrize("cumulative", [False, True])
@pytest.mark.parametrize("nr,npl,uneven,model", [(2, 1, False, "Hernquist"), (11, 1, False, "NFW"),
                                                 (13, 3, True, "Hernquist"), (80, 7, False, "NFW"),
                                                 (900, 1, False, "Isochrone"), (2100, 1, False, "NFW")])
def test_poisson_launch_shapes(ctx, cumulative, nr, npl, uneven, model):
    ar = F.log_grid(1e-2, 100.0, nr)
    if uneven:
        f = np.cumsum(np.random.default_rng(3).uniform(0.05, 0.9, nr))
        ar = 0.01 * np.exp((f - f[0]) * np.log(1e4) / (f[-1] - f[0]))
    rhl = F.guess_rhl(ar, 16, npl, model, q=0.7)
    ref = O.compute_phil(ar, rhl, cumulative=cumulative)
    outs = [torch.zeros((nr, npl), dtype=torch.float64, device="cuda") for _ in range(3)]
    mode = ctx.poisson()
    ctx.set_poisson(A.FJ_POISSON_CUMULATIVE if cumulative else A.FJ_POISSON_QAGS)
    try:
        ctx.computePhil(dev(ar), dev(rhl), *outs)
    finally:
        ctx.set_poisson(mode)
    torch.cuda.synchronize()
    got = [o.cpu().numpy() for o in outs]
    assert rel_rows(got[0], ref[0]) < 1e-9 and rel_rows(got[1], ref[1]) < 1e-9
    scale = np.abs(4 * np.pi * rhl[:, :1]) + np.abs(ref[2][:, :1])  # Pr2's terms nearly cancel
    assert np.max(np.abs(got[2] - ref[2]) / scale) < 1e-8
