"""vjp_fourier where the Fourier vector is longer than the plan's real-space
vector (few angular bins, or one probe's bins only): the workspace is sized by
the real-space vector, so no part of it may be placed by the Fourier one.  The
angular bins do not enter the Fourier vector, so its gradient is that of a plan
with many; FP64 sums by atomics, hence 1e-10 of the largest entry, and the mixed
plan's FP32 sums in a run-dependent order, 1e-6 (as test_gpu_vjp_fourier)."""
import numpy as np
import pytest

from cl2pt import abi, lib, workloads


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [lib.PREC_MIXED, lib.PREC_FP64])
@pytest.mark.parametrize("probes", [7, abi.PROBE_WTHETA, abi.PROBE_XI])
def test_few_angular_bins(gpu_lib, prec, probes):
    ell = np.geomspace(20.0, 3000.0, 33)
    got = []
    for ntheta in (2, 30):
        w = workloads.make("real_3x2pt_small")
        w.cfg.ntheta, w.cfg.probes = ntheta, probes
        tabs, nus = workloads.points(w, 3, seed=91)
        om, h0, chi, G, lnP = workloads.stack(tabs)
        plan = lib.Plan(w.cfg, w.src, w.lens, w.base, prec, max_batch=3)
        assert (plan.n_total < plan.fourier_n_total(len(ell))) == (ntheta == 2)
        cot = np.random.default_rng(92).normal(size=(3, plan.fourier_n_total(len(ell))))
        got.append(plan.vjp_fourier(om, h0, chi, G, lnP, nus, ell, cot)[:3])
        plan.close()
    (da, la, na), (db, lb, nb) = got
    assert np.array_equal(da, db)
    tol = 1e-10 if prec == lib.PREC_FP64 else 1e-6
    for a, b in ((la, lb), (na, nb)):
        a, b = a.reshape(3, -1), b.reshape(3, -1)
        assert (np.abs(b).max(axis=1) > 0).all()
        assert (np.abs(a - b) <= tol * np.abs(b).max(axis=1, keepdims=True)).all()
