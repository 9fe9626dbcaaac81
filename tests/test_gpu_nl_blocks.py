"""The FFTLog's multipole blocks (k_nl_cg, k_nl_block, k_nl_handover): ends of
a block of 16, odd counts, a single pair, magnification bias, several waves,
and plans whose phase and Gamma tables hold only a part of the multipoles at a
time.  Against the oracle's C_cl_tomo at the framework's bar (1e-4 relative;
the FP32 transforms measure below 1e-6)."""
import numpy as np
import pytest

from cl2pt import lib, workloads
from test_gpu_real import REL, rel_err


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [lib.PREC_MIXED, lib.PREC_FP64])
@pytest.mark.parametrize("lnl,nchi,bmag", [(2, 500, False), (15, 500, False), (17, 333, True), (48, 64, False),
                                           (151, 500, True), (40, 2048, False)])
def test_blocks_vs_oracle(gpu_lib, oracle_built, prec, lnl, nchi, bmag):
    import oracle as O
    w = workloads.make("real_3x2pt_small")
    w.cfg.lmax_nolimber, w.cfg.nl_nchi = lnl, nchi
    tabs, nus = workloads.points(w, 2, seed=31, bmag=bmag)
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
@pytest.mark.parametrize("prec", [lib.PREC_MIXED, lib.PREC_FP64])
def test_table_chunks(gpu_lib, prec):
    """A plan for 512 points at 2048 samples keeps 4 GB of phase and Gamma
    tables, a part of the 200 multipoles; one for 2 points keeps them all.
    The same blocks run either way, so the C_l and vectors are equal, and the
    FP64 plan's adjoint up to its atomics.  The mixed plan's slice adjoint
    sums up to ~200 terms a cell in FP32, warps racing within an instruction:
    200 x 2^-24 of the cell's terms at worst."""
    w = workloads.make("fourier_serving")
    tabs, nus = workloads.points(w, 2, seed=32)
    om, h0, chi, G, lnP = workloads.stack(tabs)
    cot = np.random.default_rng(1).normal(size=len(w.ell) * (55 + 100 + 10))
    got = []
    for n in (2, 512 if prec == lib.PREC_MIXED else 256):
        plan = lib.Plan(w.cfg, w.src, w.lens, w.base, prec, max_batch=n)
        cl, conv = plan.cl_nonlimber(om, h0, chi, G, lnP, nus)
        dv, lbar, nbar = plan.vjp_fourier(om, h0, chi, G, lnP, nus, w.ell, cot)
        got.append((cl, conv, dv, lbar, nbar))
        plan.close()
    a, b = got
    for x, y in zip(a[:3], b[:3]):
        assert np.array_equal(x, y)
    tol = 200 * 2.0 ** -24 if prec == lib.PREC_MIXED else 1e-10
    for x, y in zip(a[3:], b[3:]):
        assert np.abs(x - y).max() <= tol * np.abs(x).max()
