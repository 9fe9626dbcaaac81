"""A plan that does not fit the device is an error of that call alone: the next
plan is made and evaluates as before."""
import numpy as np
import pytest

from cl2pt import lib, workloads


@pytest.mark.gpu
def test_plan_after_a_plan_that_did_not_fit(gpu_lib):
    w = workloads.make("real_3x2pt_small")
    tabs, nus = workloads.points(w, 2, seed=95)
    args = workloads.stack(tabs)
    plan = lib.Plan(w.cfg, w.src, w.lens, w.base, lib.PREC_MIXED, max_batch=2)
    ref = plan.eval_real(*args, nus)
    with pytest.raises(lib.CL2PTError):
        lib.Plan(w.cfg, w.src, w.lens, w.base, lib.PREC_MIXED, max_batch=10 ** 6)  # 320 GB of tables
    assert np.array_equal(plan.eval_real(*args, nus), ref)
    with pytest.raises(lib.CL2PTError):
        lib.Plan(w.cfg, w.src, w.lens, w.base, lib.PREC_MIXED, max_batch=10 ** 6)
    again = lib.Plan(w.cfg, w.src, w.lens, w.base, lib.PREC_MIXED, max_batch=2)
    assert np.array_equal(again.eval_real(*args, nus), ref)
