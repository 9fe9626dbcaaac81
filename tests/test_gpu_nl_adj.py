"""The FFTLog adjoint's slice terms (k_nl_adj, k_nl_adj_slice): a multipole
whose cotangent lies below the FP32 normal range is taken, or left out, by both
kernels alike.  The gradient is linear in the cotangent, so one scaled by s has
at most s times the entries: within a factor of 2 where the weights have bits
left, and where they are rounded to multiples of the smallest subnormal
(1.4e-45, some hundred multipoles) within 1e-40 of the unscaled ones.  A term
that a call reads without having written it is one of an earlier call, with
that call's weight: of the unscaled gradient's size."""
import numpy as np
import pytest

from cl2pt import lib, workloads


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [lib.PREC_MIXED, lib.PREC_FP64])
def test_tiny_cotangents(gpu_lib, prec):
    w = workloads.make("real_3x2pt_small")
    tabs, nus = workloads.points(w, 2, seed=61)
    om, h0, chi, G, lnP = workloads.stack(tabs)
    plan = lib.Plan(w.cfg, w.src, w.lens, w.base, prec, max_batch=2)
    v = np.zeros((2, plan.n_total))
    v[:, plan.n_xi + plan.n_gammat:] = np.random.default_rng(2).normal(size=(2, plan.n_w))
    big = np.abs(plan.vjp_real(om, h0, chi, G, lnP, nus, v)[1]).max()
    for e in range(36, 48):
        got = np.abs(plan.vjp_real(om, h0, chi, G, lnP, nus, v * 10.0 ** -e)[1]).max()
        assert got <= 2 * big * 10.0 ** -e + 1e-40 * big, (e, got, big)


@pytest.mark.gpu
def test_memory_of_the_first_gradient(gpu_lib):
    """The terms take 2 GB at most, however many lens bins and samples: a
    512-point plan's first gradient allocates at most that more at 2048 samples
    than at 64 (the other buffers do not depend on them; 64 MB for the
    allocator's granularity)."""
    import torch
    grown = []
    for nchi in (64, 2048):
        w = workloads.make("fourier_serving")
        w.cfg.nl_nchi = nchi
        tabs, nus = workloads.points(w, 1, seed=62)
        om, h0, chi, G, lnP = workloads.stack(tabs)
        plan = lib.Plan(w.cfg, w.src, w.lens, w.base, lib.PREC_MIXED, max_batch=512)
        plan.eval_fourier(om, h0, chi, G, lnP, nus, w.ell)
        free = torch.cuda.mem_get_info()[0]
        plan.vjp_fourier(om, h0, chi, G, lnP, nus, w.ell, np.ones((1, plan.fourier_n_total(len(w.ell)))))
        grown.append(free - torch.cuda.mem_get_info()[0])
        plan.close()
    print(grown)
    assert grown[1] - grown[0] <= (2 << 30) + (64 << 20), grown
