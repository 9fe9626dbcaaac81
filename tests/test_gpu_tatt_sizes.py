"""The TATT / one-loop terms at the sizes of test_gpu_fpt_cell (one point and
several, multipole counts that end inside a chunk or a tile, one source bin,
high_def_integration 1), each spectrum on its own scale.

Forward: both plans against the oracle, table by table and spectrum by spectrum,
at the framework's bar with the envelope that test_gpu_real states.  Gradient:
the mixed plan against the FP64 plan for a cotangent on one kind of spectrum at
a time, each nuisance on its own scale, 1e-4 of its largest entry (the mixed
plan's sums round to ~1e-6)."""
import numpy as np
import pytest

from cl2pt import abi, lib, workloads
from test_gpu_real import REL, blocks, run_case

SIZES = [(1, 200, 4, 0), (3, 77, 4, 0), (2, 33, 1, 0), (2, 130, 3, 1), (2, 101, 2, 0)]


def tweak(n_ell, ns, hdi):
    def f(w):
        w.cfg.n_ell, w.cfg.n_source, w.cfg.high_def_integration = n_ell, ns, hdi
        w.src = np.ascontiguousarray(w.src[:, :ns + 1])
    return f


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [lib.PREC_MIXED, lib.PREC_FP64])
@pytest.mark.parametrize("n,n_ell,ns,hdi", SIZES)
def test_forward_vs_oracle(gpu_lib, oracle_built, prec, n, n_ell, ns, hdi):
    worst, _ = run_case("real_3x2pt_tatt_small", n, prec, seed=41, tweak=tweak(n_ell, ns, hdi), bmag=True)
    for k, v in worst.items():
        assert v <= REL, (k, v, worst)


@pytest.mark.gpu
@pytest.mark.parametrize("n,n_ell,ns,hdi", SIZES)
def test_nuisance_gradient_by_spectrum(gpu_lib, n, n_ell, ns, hdi):
    w = workloads.make("real_3x2pt_tatt_small")
    tweak(n_ell, ns, hdi)(w)
    tabs, nus = workloads.points(w, n, seed=41, bmag=True)
    om, h0, chi, G, lnP = workloads.stack(tabs)
    plans = [lib.Plan(w.cfg, w.src, w.lens, w.base, p, max_batch=n) for p in (lib.PREC_MIXED, lib.PREC_FP64)]
    rng = np.random.default_rng(43)
    for name, part in blocks(plans[0], np.arange(plans[0].n_total)).items():
        cot = np.zeros((n, plans[0].n_total))
        cot[:, part] = rng.uniform(0.5, 1.5, (n, len(part)))
        a, b = (p.vjp_real(om, h0, chi, G, lnP, nus, cot)[2].reshape(n, 13, abi.MAX_BINS) for p in plans)
        scale = np.abs(b).max(axis=2, keepdims=True)
        assert (np.abs(a - b) <= 1e-4 * scale).all(), (name, (np.abs(a - b) / (scale + 1e-300)).max(axis=(0, 2)))
        assert scale.any()
