"""The shear adjoint sweep with up to a point per SM (one CTA of 1024 threads)
and with more (two of 512): a point's gradient does not depend on how many
points are evaluated with it.  The table gradient's atomics add in a
run-dependent order, as do those of the nuisances: FP64 sums of FP32 terms, so
1e-12 of the largest entry."""
import numpy as np
import pytest

from cl2pt import abi, lib, workloads


@pytest.mark.gpu
@pytest.mark.parametrize("hdi", [0, 1])
def test_either_side_of_the_sm_count(gpu_lib, hdi):
    w = workloads.make("real_3x2pt_small_limber")
    w.cfg.probes, w.cfg.high_def_integration, w.cfg.n_ell = abi.PROBE_XI, hdi, 77
    tabs, nus = workloads.points(w, 160, seed=97)
    args = workloads.stack(tabs)
    plan = lib.Plan(w.cfg, w.src, w.lens, w.base, lib.PREC_MIXED, max_batch=160)
    v = np.random.default_rng(98).normal(size=(160, plan.n_total))
    many = plan.vjp_real(*args, nus, v)
    for n in (1, 152):
        few = plan.vjp_real(*[a[:n] for a in args], nus[:n], v[:n])
        for a, b in zip(few[1:3], many[1:3]):
            assert np.abs(a - b[:n]).max() <= 1e-12 * np.abs(b).max()
