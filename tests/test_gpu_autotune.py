"""fj_autotune_mixed times the item sizes that it names: a launch of few sample points is not cut
below them, so its moments have the bits of the same points in a launch too large to be cut."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fjmodels_gb300 as F  # noqa: E402
from fjmodels_gb300 import _abi as A  # noqa: E402
from oracle import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


def test_autotune_times_the_sizes_it_names():
    dev = lambda a: torch.tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda")  # noqa: E731
    ctx = F.Context(0)
    ar = F.log_grid(0.01, 100.0, 24)
    phil, Pr, Pr2 = O.compute_phil(ar, F.guess_rhl(ar, 16, 4, "Hernquist", q=0.8))
    E, D, _ = F.tabulate_delta(ar, phil, Pr, Pr2)
    pot, delta = ctx.potential(*map(dev, (ar, phil, Pr, Pr2))), ctx.delta(dev(E), dev(D))
    df, rule = F.DFParams("Hernquist", chi=1.0), F.Rule(*F.tanh_sinh_rule(22), precision=A.FJ_PREC_MIXED)
    g = np.random.default_rng(2)
    r, c = np.exp(g.uniform(np.log(0.02), np.log(30.0), 12)), g.uniform(0.05, 0.95, 12)
    pts = dev(np.stack([r * np.sqrt(1 - c * c), r * c], 1))
    out, ms = torch.zeros((6, 12), dtype=torch.float64, device="cuda"), np.zeros(1)
    table = np.zeros((8, 3))
    import ctypes as C
    ctx._on_torch_stream()
    ctx._check(ctx.lib.fj_autotune_mixed(ctx.h, C.byref(pot.c), C.byref(delta.c), C.byref(df.c), C.byref(rule.c),
                                         C.c_void_p(pts.data_ptr()), 12, C.c_void_p(out.data_ptr()),
                                         ms.ctypes.data_as(A.DP), table.ctypes.data_as(A.DP)), "fj_autotune_mixed")
    assert np.all(table > 0) and ms[0] == table.min()
    kept = ctx.mixed_config()
    assert kept == (table.argmin() // 3, (1024, 2048, 4096)[table.argmin() % 3])
    # the last configuration timed: items of at most 4096 nodes; 840 points fill the GPU with them
    ctx.set_mixed_config(7, 4096)
    many = torch.zeros((6, 840), dtype=torch.float64, device="cuda")
    ctx.moments_points(pot, delta, df, rule, pts.repeat(70, 1), many)
    torch.cuda.synchronize()
    assert torch.equal(out, many[:, :12])
    ctx.close()
