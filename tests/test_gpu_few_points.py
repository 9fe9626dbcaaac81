"""Few points: the Limber kernels spread a multipole's nodes and pairs over
several threads when there are fewer CTAs than SMs, and the sums keep their
order, so a point's results do not depend on how many are evaluated with it.
Tolerance: none in the mixed plan's tables (the same sums); the FP64 plan's
contraction sums a column in one order at any batch too."""
import numpy as np
import pytest

from cl2pt import lib, workloads


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("name,n", [("real_3x2pt_small", 90), ("real_3x2pt_small_limber", 90), ("real_3x2pt", 20),
                                    ("real_3x2pt_tatt_small", 60)])
def test_alone_and_in_a_batch(gpu_lib, name, n, precision):
    w = workloads.make(name)
    tabs, nus = workloads.points(w, n, seed=4)
    args, lin = workloads.stack(tabs), workloads.stack_lin(tabs)
    prec = lib.PREC_MIXED if precision == "mixed" else lib.PREC_FP64
    plan = lib.Plan(w.cfg, w.src, w.lens, w.base, prec, max_batch=n, linear_table=True)
    many = plan.eval_real(*args, nus, lnPL=lin)
    for i in (0, n // 2, n - 1):
        one = plan.eval_real(*[a[i:i + 1] for a in args], nus[i:i + 1], lnPL=lin[i:i + 1])
        assert np.array_equal(one[0], many[i]), (i, np.abs(one[0] - many[i]).max())
