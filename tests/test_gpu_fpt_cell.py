"""The TATT / one-loop terms and their adjoint at the sizes where the work is
split: one point and several, multipole counts that end inside a chunk or a
tile, more nodes than one group of threads (high_def_integration 1), one
source bin.  The mixed plan takes the FAST-PT grid cell in two-float form; its
terms and gradients against the FP64 plan, whose cell is the reference's.
Tolerance: FP32 rounding of sums of ~1e2 terms, 2e-5 of the largest entry (the
FAST-PT adjoint amplifies the row cotangents' rounding by ~1e2)."""
import numpy as np
import pytest

from cl2pt import lib, workloads


@pytest.mark.gpu
@pytest.mark.parametrize("n,n_ell,ns,hdi", [(1, 200, 4, 0), (3, 77, 4, 0), (2, 33, 1, 0), (2, 130, 3, 1),
                                            (9, 101, 2, 0)])
def test_mixed_vs_fp64(gpu_lib, n, n_ell, ns, hdi):
    w = workloads.make("real_3x2pt_tatt_small")
    w.cfg.n_ell, w.cfg.n_source, w.cfg.high_def_integration = n_ell, ns, hdi
    w.src = np.ascontiguousarray(w.src[:, :ns + 1])
    tabs, nus = workloads.points(w, n, seed=41, bmag=True)
    om, h0, chi, G, lnP = workloads.stack(tabs)
    out = []
    for prec in (lib.PREC_MIXED, lib.PREC_FP64):
        plan = lib.Plan(w.cfg, w.src, w.lens, w.base, prec, max_batch=n)
        cot = np.random.default_rng(3).normal(size=(n, plan.n_total))
        out.append(plan.vjp_real(om, h0, chi, G, lnP, nus, cot))
        plan.close()
    for a, b in zip(*out):
        scale = np.abs(b).max(axis=1, keepdims=True)
        assert np.isfinite(a).all()
        assert (np.abs(a - b) <= 2e-5 * scale).all(), (np.abs(a - b) / scale).max()
