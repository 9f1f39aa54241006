"""Host threads with a context each and models of different table sizes: a kernel's shared-memory
limit belongs to the process, so a call must not leave it below what another thread's launch needs."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fjmodels_gb300 as F  # noqa: E402
from fjmodels_gb300 import _abi as A  # noqa: E402
from oracle import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu
ROUNDS, CALLS = 40, 50


def dev(a):
    return torch.tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda")


@pytest.mark.parametrize("what", ["actions", "fp64", "mixed"])
def test_threads_with_different_table_sizes(what):
    rule = F.Rule(*F.tanh_sinh_rule(4), precision=A.FJ_PREC_MIXED if what == "mixed" else A.FJ_PREC_FP64)
    df = F.DFParams("Hernquist")
    jobs = []
    for nr, npl in ((400, 12), (130, 13)):  # 94 and 63 KB of FP64 tables, 80 and 34 KB of FP32 ones
        ar = F.log_grid(0.01, 100.0, nr)
        phil, Pr, Pr2 = O.compute_phil(ar, F.guess_rhl(ar, 24, npl, "Hernquist", q=0.8), cumulative=True)
        E, D = np.linspace(phil[0, 0] * 0.99, phil[-1, 0] * 1.01, 30), np.linspace(0.04, 0.4, 30)
        c = F.Context(0)
        pts = dev([[0.5, 0.3, 0.1, 0.3, 0.2], [1.5, 1.0, 0.2, 0.2, 0.1]])
        jobs.append((c, c.potential(*map(dev, (ar, phil, Pr, Pr2))), c.delta(dev(E), dev(D)), pts))

    def call(job, out):
        c, pot, delta, pts = job
        c.use_own_stream()
        if what == "actions":
            c._check(c.lib.fj_actions(c.h, pot.c, delta.c, pts.data_ptr(), 2, 0, out.data_ptr()), what)
        else:
            c._check(c.lib.fj_moments_points(c.h, pot.c, delta.c, df.c, rule.c, Rz.data_ptr(), 2, out.data_ptr(),
                                             None), what)

    Rz = dev([[0.5, 0.3], [1.5, 1.0]])
    shape = (2, 2) if what == "actions" else (6, 2)
    torch.cuda.synchronize()
    want = [torch.zeros(shape, dtype=torch.float64, device="cuda") for _ in jobs]
    for job, out in zip(jobs, want):
        call(job, out)
        job[0].sync()
    errors = []

    def work(i):
        out = torch.zeros(shape, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        try:
            for _ in range(ROUNDS):
                for _ in range(CALLS):  # queued one after the other
                    call(jobs[i], out)
                jobs[i][0].sync()
            if not torch.equal(out, want[i]):
                errors.append("wrong result")
        except Exception as e:  # reported by the test's thread
            errors.append(repr(e))

    pool = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    for job in jobs:
        job[0].close()
    assert not errors, errors[0]
