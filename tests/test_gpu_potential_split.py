"""The potential batch at the sizes where its split over blocks changes: the same bits as the point
alone has in a large batch."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fjmodels_gb300 as F  # noqa: E402
from oracle import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,npl", [(24, 4), (400, 9)])  # tables in shared and in device memory
def test_prefixes_of_a_large_batch(ctx, nr, npl):
    dev = lambda a: torch.tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda")  # noqa: E731
    ar = F.log_grid(0.01, 100.0, nr)
    tabs = O.compute_phil(ar, F.guess_rhl(ar, 24, npl, "Hernquist", q=0.8), cumulative=True)
    pot = ctx.potential(*map(dev, (ar, *tabs)))
    held = 2 * torch.cuda.get_device_properties(0).multi_processor_count  # blocks of 256 points
    N = 4 * held * 256 + 77
    g = np.random.default_rng(nr)
    r, c = np.exp(g.uniform(np.log(0.005), np.log(200.0), N)), g.uniform(-1, 1, N)
    Rz = dev(np.stack([r * np.sqrt(1 - c * c), r * c], 1))
    whole = torch.zeros((N, 3), dtype=torch.float64, device="cuda")
    ctx.potential_eval(pot, Rz, whole)
    for n in (1, 31, 32, 33, 32 * held, 32 * held + 1, 256 * held - 1, 256 * held, 256 * held + 1, 512 * held + 1):
        out = torch.full((n + 1, 3), 7.0, dtype=torch.float64, device="cuda")
        ctx.potential_eval(pot, Rz[:n], out)
        torch.cuda.synchronize()
        assert torch.equal(out[:n], whole[:n]) and bool((out[n] == 7.0).all()), n
