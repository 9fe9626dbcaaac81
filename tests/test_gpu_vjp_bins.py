"""TATT / one-loop gradients with as many source bins as the adjoint takes: the
row cotangents' kernels (k_vjpr_ss, k_vjpr_gs) at the bins where their shared
memory once refused a plan.  Nuisances against central
differences of the FP64 plan's forward at the framework's bar, 1e-4 relative
(the mixed plan's sums round to ~1e-6, the differences to ~1e-7); the table
gradient, whose differences the rounding of the TATT convolutions swamps,
against a plan with fewer bins at test_gpu_fpt_cell's bar, 2e-5 of the largest
entry (the direct convolutions' adjoint amplifies rounding: two runs of one
FP64 plan differ by 2.5e-8 of it)."""
import numpy as np
import pytest

from cl2pt import lib, synthetic, workloads
from test_gpu_vjp import H, clone, flat_index, nu_get, nu_set


def case(ns, hdi, n_ell=60, one_loop=1):
    w = workloads.make("real_3x2pt_tatt_small")
    w.cfg.n_source, w.cfg.high_def_integration, w.cfg.n_ell = ns, hdi, n_ell
    w.cfg.adopt_limber_gg, w.cfg.one_loop_bias = 1, one_loop
    w.src = synthetic.source_nz(ns)
    return w


@pytest.mark.gpu
@pytest.mark.parametrize("prec,ns,hdi", [(lib.PREC_FP64, 8, 0), (lib.PREC_FP64, 9, 0), (lib.PREC_FP64, 10, 0), (lib.PREC_FP64, 12, 0),
                                         (lib.PREC_MIXED, 14, 0), (lib.PREC_MIXED, 16, 0), (lib.PREC_MIXED, 13, 1),
                                         (lib.PREC_MIXED, 11, 2)])
def test_gradient_vs_forward_differences(gpu_lib, prec, ns, hdi):
    w = case(ns, hdi)
    tabs, nus = workloads.points(w, 2, seed=71)
    om, h0, chi, G, lnP = workloads.stack(workloads.one_table(tabs))
    plan = lib.Plan(w.cfg, w.src, w.lens, w.base, prec, max_batch=2)
    fwd = lib.Plan(w.cfg, w.src, w.lens, w.base, lib.PREC_FP64, max_batch=2)
    dv = fwd.eval_real(om, h0, chi, G, lnP, nus)
    # every spectrum weighs alike
    nt = w.cfg.ntheta
    rms = np.sqrt(np.mean(dv.reshape(2, -1, nt) ** 2, axis=2, keepdims=True))
    rng = np.random.default_rng(72)
    v = (rng.uniform(0.5, 1.5, dv.shape).reshape(rms.shape[0], -1, nt) / rms).reshape(dv.shape)
    _, lbar, nbar = plan.vjp_real(om, h0, chi, G, lnP, nus, v)
    sl = slice(1, 2)

    def f(nu, lp):
        return float(v[1] @ fwd.eval_real(om[sl], h0[sl], chi[sl], G[sl], lp, [nu])[0])

    for field, i, j in [("ia", 0, 0), ("ia", 1, 0), ("ia", 2, 0), ("gb", 0, 1), ("gb", 1, 2), ("src_dz", ns - 1, None)]:
        x0 = nu_get(nus[1], field, i, j)
        h = H * max(abs(x0), 0.1)
        d = []
        for sg in (1, -1):
            nu = clone(nus[1])
            nu_set(nu, field, i, j, x0 + sg * h)
            d.append(f(nu, lnP[sl]))
        fd = (d[0] - d[1]) / (2 * h)
        an = nbar[1, flat_index(field, i, j)]
        assert abs(an - fd) <= 1e-4 * abs(fd), (field, i, j, an, fd)
    # the table gradient of a cotangent on the last bins' spectra alone is that
    # of a plan with those bins
    m = 8 if prec == lib.PREC_FP64 else 10
    sub = case(m, hdi)
    sub.src = np.ascontiguousarray(w.src[:, [0] + list(range(ns + 1 - m, ns + 1))])
    few = lib.Plan(sub.cfg, sub.src, sub.lens, sub.base, prec, max_batch=2)
    npair = m * (m + 1) // 2
    va = rng.normal(size=(2, 2, npair, nt)) / rms.mean()
    vb = np.zeros((2, 2, ns * (ns + 1) // 2, nt))
    pair = [(i, j) for i in range(ns) for j in range(i, ns)]
    vb[:, :, [k for k, (i, j) in enumerate(pair) if i >= ns - m]] = va
    pad = lambda p, x: np.pad(x.reshape(2, -1), ((0, 0), (0, p.n_total - p.n_xi)))  # noqa: E731
    for nu in nus:
        for s in range(ns):
            nu.src_dz[s], nu.shear_m[s] = 0.01, 0.0
    a = plan.vjp_real(om, h0, chi, G, lnP, nus, pad(plan, vb))[1]
    b = few.vjp_real(om, h0, chi, G, lnP, nus, pad(few, va))[1]
    assert np.abs(a - b).max() <= 2e-5 * np.abs(b).max()


@pytest.mark.gpu
def test_one_loop_alone_needs_no_shear_rows(gpu_lib):
    """NLA with one-loop bias at 16 bins runs none of the TATT kernels."""
    w = case(16, 0)
    from cl2pt import abi
    w.cfg.ia_model, w.tatt = abi.IA_NLA, False
    tabs, nus = workloads.points(w, 1, seed=73)
    om, h0, chi, G, lnP = workloads.stack(workloads.one_table(tabs))
    plan = lib.Plan(w.cfg, w.src, w.lens, w.base, lib.PREC_MIXED, max_batch=1)
    for q in range(w.cfg.n_lens):
        nus[0].gb[1][q] = 0.3
    _, lbar, nbar = plan.vjp_real(om, h0, chi, G, lnP, nus, np.ones((1, plan.n_total)))
    assert np.isfinite(lbar).all() and np.abs(lbar).max() > 0
    assert np.abs(nbar[0, flat_index("gb", 1, 0)]) > 0
