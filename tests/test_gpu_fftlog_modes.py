"""cl2pt_plan_set_fftlog_state: every mode is accepted and runs the same kernels,
so results are equal bit for bit; anything else is an argument error."""
import numpy as np
import pytest

from cl2pt import lib, workloads


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [lib.PREC_MIXED, lib.PREC_FP64])
def test_modes(gpu_lib, prec):
    w = workloads.make("real_3x2pt_small")
    tabs, nus = workloads.points(w, 3, seed=81)
    args = workloads.stack(tabs)
    plan = lib.Plan(w.cfg, w.src, w.lens, w.base, prec, max_batch=3)
    ref = plan.eval_real(*args, nus)
    modes = (lib.FFTLOG_STATE_AUTO, lib.FFTLOG_STATE_GLOBAL, lib.FFTLOG_STATE_SHARED)
    for m in modes:
        plan.set_fftlog_state(m)
        assert np.array_equal(plan.eval_real(*args, nus), ref)
    for bad in (min(modes) - 1, max(modes) + 1):
        with pytest.raises(lib.CL2PTError):
            plan.set_fftlog_state(bad)
    assert np.array_equal(plan.eval_real(*args, nus), ref)
