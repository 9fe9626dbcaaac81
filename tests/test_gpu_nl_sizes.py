"""Radial grids whose FFTLog sizes are odd: the size rule (next 7-smooth number
of the padded grid, tried again once if odd) leaves 735, 1225, 1715, 2205, 3125
or 3675 points for the galaxy kernel (padded by 2 x 200) or the other two (2 x
500).  Against the oracle's C_cl_tomo at the framework's bar, and the adjoint
against central differences of the plan's forward in FP64 (1e-6, as
test_gpu_vjp) and against the FP64 plan in the mixed one (1e-4)."""
import numpy as np
import pytest

from cl2pt import lib, workloads
from test_gpu_real import REL, rel_err
from test_gpu_vjp import GRAD_REL, H, clone, flat_index, nu_get, nu_set

SIZES = [205, 214, 325, 690, 700, 805, 1170, 1300, 1770, 2080, 2610, 2680]


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [lib.PREC_MIXED, lib.PREC_FP64])
@pytest.mark.parametrize("nchi", SIZES)
def test_odd_sizes_vs_oracle(gpu_lib, oracle_built, prec, nchi):
    import oracle as O
    w = workloads.make("real_3x2pt_small")
    w.cfg.lmax_nolimber, w.cfg.nl_nchi = 40, nchi
    tabs, nus = workloads.points(w, 2, seed=33, bmag=True)
    plan = lib.Plan(w.cfg, w.src, w.lens, w.base, prec, max_batch=2, linear_table=True)
    om, h0, chi, G, lnP = workloads.stack(tabs)
    cl, conv = plan.cl_nonlimber(om, h0, chi, G, lnP, nus, lnPL=workloads.stack_lin(tabs))
    o = O.Oracle("orc")
    o.setup(w.cfg, w.src, w.lens)
    for i in range(2):
        o.set_point(tabs[i], nus[i])
        ocl, oconv = o.C_cl_tomo()
        assert np.array_equal(conv[i], oconv)
        assert rel_err(cl[i][:, 1:], ocl[:, 1:]) <= REL


@pytest.mark.gpu
@pytest.mark.parametrize("nchi", [325, 690, 1300])
def test_odd_sizes_gradient(gpu_lib, nchi):
    w = workloads.make("real_3x2pt_small")
    w.cfg.lmax_nolimber, w.cfg.nl_nchi = 40, nchi
    tabs, nus = workloads.points(w, 1, seed=34, bmag=True)
    om, h0, chi, G, lnP = workloads.stack(tabs)
    plans = [lib.Plan(w.cfg, w.src, w.lens, w.base, p, max_batch=1) for p in (lib.PREC_FP64, lib.PREC_MIXED)]
    v = np.zeros((1, plans[0].n_total))
    v[:, plans[0].n_xi + plans[0].n_gammat:] = np.random.default_rng(35).uniform(0.5, 1.5, (1, plans[0].n_w))
    (_, la, na), (_, lb, nb) = (p.vjp_real(om, h0, chi, G, lnP, nus, v) for p in plans)
    for i, j in ((0, 0), (0, 2), (4, 1)):
        x0 = nu_get(nus[0], "gb", i, j)
        h = H * max(abs(x0), 0.1)
        f = []
        for sg in (1, -1):
            nu = clone(nus[0])
            nu_set(nu, "gb", i, j, x0 + sg * h)
            f.append(float(v[0] @ plans[0].eval_real(om, h0, chi, G, lnP, [nu])[0]))
        fd, an = (f[0] - f[1]) / (2 * h), na[0, flat_index("gb", i, j)]
        assert abs(an - fd) <= GRAD_REL * abs(fd), (i, j, an, fd)
    assert np.abs(la - lb).max() <= 1e-4 * np.abs(la).max()
    assert (np.abs(na - nb) <= 1e-4 * np.abs(na).max()).all()
