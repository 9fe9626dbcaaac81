"""Gradients of many points, and of fewer than the plan was made for.

The shear adjoint sweep with up to a point per SM (one CTA of 1024 threads) and
with more (two of 512): a point's gradient does not depend on how many points
are evaluated with it.  The table gradient's atomics add in a run-dependent
order, as do those of the nuisances: FP64 sums of FP32 terms, so 1e-12 of the
largest entry."""
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


@pytest.mark.gpu
def test_tatt_batch_of_several_fastpt_waves(gpu_lib):
    """The TATT tables' FAST-PT plan works in waves of 256 spectra, the plan in
    waves of 512 points: a gradient of 300 points is that of two batches of 150
    (2e-5 of the largest entry, as test_gpu_fpt_cell; with cotangents of one
    sign, since two runs of one plan differ by up to that where they cancel)."""
    w = workloads.make("real_3x2pt_tatt_small")
    w.cfg.n_ell, w.cfg.adopt_limber_gg = 33, 1
    tabs, nus = workloads.points(w, 300, seed=99)
    args = workloads.stack(tabs)
    plan = lib.Plan(w.cfg, w.src, w.lens, w.base, lib.PREC_FP64, max_batch=300)
    v = np.random.default_rng(100).uniform(0.5, 1.5, (300, plan.n_total))
    many = plan.vjp_real(*args, nus, v)
    for sl in (slice(0, 150), slice(150, 300)):
        half = plan.vjp_real(*[a[sl] for a in args], nus[sl], v[sl])
        assert np.array_equal(half[0], many[0][sl])
        for a, b in zip(half[1:3], many[1:3]):
            s = np.abs(a).max(axis=1, keepdims=True)
            assert (np.abs(a - b[sl]) <= 2e-5 * s).all()


@pytest.mark.gpu
@pytest.mark.parametrize("tatt,one_loop", [(True, 1), (True, 0), (False, 1)])
def test_batch_smaller_than_the_plan(gpu_lib, tatt, one_loop):
    """A plan for 12 points evaluates 12, then 5: the 5 have the gradient of a
    plan for 5, with nothing left of the larger batch (2e-5 of the largest entry
    as above; what was left was of its size)."""
    w = workloads.make("real_3x2pt_tatt_small")
    w.cfg.n_ell, w.cfg.adopt_limber_gg, w.cfg.one_loop_bias = 33, 1, one_loop
    if not tatt:
        w.cfg.ia_model = abi.IA_NLA
    tabs, nus = workloads.points(w, 12, seed=101)
    if not one_loop:
        for nu in nus:
            for q in range(w.cfg.n_lens):
                nu.gb[1][q] = nu.gb[2][q] = 0.0
    args = workloads.stack(tabs)
    big, small = (lib.Plan(w.cfg, w.src, w.lens, w.base, lib.PREC_FP64, max_batch=n) for n in (12, 5))
    v = np.random.default_rng(102).uniform(0.5, 1.5, (12, big.n_total))
    big.vjp_real(*args, nus, v)
    few = [a[7:] for a in args], nus[7:], v[7:]
    got, want = (p.vjp_real(*few[0], few[1], few[2]) for p in (big, small))
    for a, b in zip(got[1:3], want[1:3]):
        s = np.abs(b).max(axis=1, keepdims=True)
        assert (np.abs(a - b) <= 2e-5 * s).all()
