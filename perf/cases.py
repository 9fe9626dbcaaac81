"""The work that users of cl2pt have it do, as cases that can be timed.

A sampler holds one plan per analysis and hands it batches of parameter
points, each with its own distances, growth, P(k, z) table and nuisances:
one point per call from a Metropolis chain, tens from an ensemble sampler or
a set of HMC chains, hundreds to thousands from an emulator's training run
or a serving process.  FAST-PT is called on its own as well, for one
spectrum or for a batch.  The workloads are those of cl2pt.workloads.

    listed()              the cases
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   inputs on the GPU (host arrays where the call takes
                          host arrays) and the plan
    run(state)            one call through the public entry points
    work(case)            bytes and operations that the call cannot do without
    exact(case, seed)     the same outputs in 64 bits by plain numpy
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "cocoa-cosmolike-core_gb300"))

from cl2pt import abi, autograd, lib, workloads  # noqa: E402

MB = abi.MAX_BINS
NU = 13 * MB


def listed():
    return [
        # one step of a cosmic-shear chain: 15 spectra at 20 multipoles from
        # host arrays, the smallest call there is
        dict(name="shear_1", kind="fourier", workload="cosmic_shear_fourier", n=1, host=True, precision="mixed"),
        # one step of a 3x2pt chain from host arrays, with the linear and the
        # nonlinear table that a Boltzmann code hands over
        dict(name="real_1", kind="real", workload="real_3x2pt", n=1, host=True, two=True, precision="mixed"),
        # an ensemble sampler's walkers, inputs on the device
        dict(name="real_37", kind="real", workload="real_3x2pt", n=37, host=False, two=False, precision="mixed"),
        # a large batch (an emulator's training set, the benchmark's step)
        dict(name="real_512", kind="real", workload="real_3x2pt", n=512, host=False, two=False, precision="mixed"),
        # the plan that does every stage in FP64
        dict(name="real_fp64_24", kind="real", workload="real_3x2pt", n=24, host=False, two=False,
             precision="fp64"),
        # value and gradient for parallel HMC chains
        dict(name="grad_100", kind="grad", workload="real_3x2pt", n=100),
        # chi^2 and its gradient through the likelihood, host arrays, a few
        # chains, a reduced analysis with both tables
        dict(name="like_3", kind="like", workload="real_3x2pt_small", n=3),
        # TATT alignments and one-loop bias: forward, and value and gradient
        dict(name="tatt_30", kind="real", workload="real_3x2pt_tatt", n=30, host=False, two=False,
             precision="mixed"),
        dict(name="tatt_grad_16", kind="grad", workload="real_3x2pt_tatt", n=16),
        # a serving process: the Fourier vector with each walker's own scale
        # cuts, replayed as a graph
        dict(name="serving_4096", kind="serving", workload="fourier_serving", n=4096),
        # FAST-PT by itself: one spectrum on the reference's 1100-point grid
        # from host arrays, and a batch on 2048 points on the device
        dict(name="fastpt_1", kind="fastpt", n=1, nk=1100, host=True),
        dict(name="fastpt_512", kind="fastpt", n=512, nk=2048, host=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fourier", "real", "real", "real64", "grad", "like", "tatt", "tatt_grad", "serving",
                       "fastpt", "fastpt"])
    if kind == "fourier":
        return dict(kind="fourier", workload="cosmic_shear_fourier", n=_log_int(rng, 1, 512),
                    host=rng.random() < 0.5, precision=rng.choice(["mixed", "fp64"]))
    if kind == "real":
        host = rng.random() < 0.3
        return dict(kind="real", host=host, n=_log_int(rng, 1, 24 if host else 512), two=rng.random() < 0.4,
                    workload=rng.choice(["real_3x2pt", "real_3x2pt", "real_3x2pt_limber", "real_3x2pt_small",
                                         "real_3x2pt_small_nla"]), precision="mixed")
    if kind == "real64":
        return dict(kind="real", host=False, n=_log_int(rng, 1, 64), two=False, workload="real_3x2pt",
                    precision="fp64")
    if kind == "grad":
        return dict(kind="grad", workload=rng.choice(["real_3x2pt", "real_3x2pt_small"]), n=_log_int(rng, 1, 256))
    if kind == "like":
        return dict(kind="like", workload=rng.choice(["real_3x2pt_small", "real_3x2pt_small_limber"]),
                    n=_log_int(rng, 1, 24))
    if kind == "tatt":
        return dict(kind="real", workload=rng.choice(["real_3x2pt_tatt", "real_3x2pt_tatt_small"]),
                    n=_log_int(rng, 1, 128), host=False, two=False, precision="mixed")
    if kind == "tatt_grad":
        return dict(kind="grad", workload=rng.choice(["real_3x2pt_tatt", "real_3x2pt_tatt_small"]),
                    n=_log_int(rng, 1, 64))
    if kind == "serving":
        return dict(kind="serving", workload=rng.choice(["fourier_serving", "fourier_serving_small"]),
                    n=_log_int(rng, 64, 4096))
    host = rng.random() < 0.4
    return dict(kind="fastpt", host=host, n=_log_int(rng, 1, 16 if host else 512),
                nk=2 * rng.randint(300, 1024))


# ------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=None)
def _workload(name):
    return workloads.make(name)


@functools.lru_cache(maxsize=2)
def _plan(name, precision, cap, two):
    """The plan of one analysis, kept between batches as a sampler keeps it."""
    w = _workload(name)
    return lib.Plan(w.cfg, w.src, w.lens, w.base, lib.PREC_FP64 if precision == "fp64" else lib.PREC_MIXED,
                    max_batch=cap, linear_table=two)


def _cumulative(z, f):
    """Cumulative Simpson integral of f on the grid z, [n][len(z)]."""
    zm = 0.5 * (z[1:] + z[:-1])
    d = (z[1:] - z[:-1]) / 6.0 * (f(z[:-1]) + 4.0 * f(zm) + f(z[1:]))
    return torch.nn.functional.pad(torch.cumsum(d, 1), (1, 0))


def _points(w, n, seed, device):
    """n parameter points around the workload's base cosmology, every one
    with its own distances, growth, tables and nuisances (the ranges of
    workloads.points): tensors on `device`."""
    rng = np.random.default_rng(seed)
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64), device=device)  # noqa: E731
    om = t(rng.normal(0.3, 0.01, n))
    h0 = t(rng.normal(0.7, 0.01, n))
    m = om[:, None]
    z = t(w.base.chi_z)
    e2 = lambda x: m * (1.0 + x) ** 3 + (1.0 - m)  # noqa: E731
    chi = 2997.92458 * _cumulative(z, lambda x: e2(x) ** -0.5)
    growth = _cumulative(z, lambda x: -((m * (1.0 + x) ** 3 / e2(x)) ** 0.55) / (1.0 + x))
    G = torch.exp(growth) * (1.0 + z)
    tilt = 2.0 * t(rng.normal(0.0, 0.02, n))[:, None] + \
        t(rng.normal(0.0, 0.01, n))[:, None] * math.log(10.0) * t(w.base.log10k)
    table = lambda p: (t(p)[None] + tilt[:, :, None]).reshape(n, -1)  # noqa: E731
    ns, nl = w.cfg.n_source, w.cfg.n_lens
    nu = np.zeros((n, 13, MB))
    nu[:, 2] = 1.0
    nu[:, 0, :ns] = rng.normal(0.0, 0.02, (n, ns))
    nu[:, 1, :nl] = rng.normal(0.0, 0.005, (n, nl))
    nu[:, 3, :ns] = rng.normal(0.0, 0.01, (n, ns))
    nu[:, 4, :nl] = rng.uniform(1.2, 2.2, (n, nl))
    if w.tatt:
        eta = rng.uniform(-2.0, 2.0, n)
        nu[:, 10, 0], nu[:, 10, 1] = rng.uniform(-1.0, 1.0, n), eta
        nu[:, 11, 0], nu[:, 11, 1] = rng.uniform(-2.0, 2.0, n), eta
        nu[:, 12, 0] = rng.uniform(0.0, 2.0, n)
        nu[:, 5, :nl] = rng.uniform(-1.0, 1.0, (n, nl))
        nu[:, 6, :nl] = rng.uniform(-1.0, 1.0, (n, nl))
    if w.nla:
        nu[:, 10, 0], nu[:, 10, 1] = rng.uniform(0.3, 1.0, n), rng.uniform(-1.5, 1.5, n)
        nu[:, 2, :nl] = rng.uniform(0.9, 1.1, (n, nl))
    return dict(om=om, h0=h0, chi=chi.contiguous(), G=G.contiguous(), lnP=table(w.base.lnP).contiguous(),
                lnPL=table(w.base.lnPL), nu=t(nu.reshape(n, -1)))


def _host(d):
    h = {k: v.cpu().numpy() for k, v in d.items()}
    h["nus"] = [abi.Nuisance.from_buffer_copy(np.ascontiguousarray(r)) for r in h["nu"]]
    return h


_TABLES = ("om", "h0", "chi", "G", "lnP")


@functools.lru_cache(maxsize=2)
def _likelihood(name, n):
    """A data vector at the base point (rounded as in a file) and a
    correlated covariance of 5% errors."""
    w = _workload(name)
    plan = _plan(name, "mixed", n, True)
    nus = [abi.make_nuisance(b1=[1.6] * w.cfg.n_lens)]
    om, h0, chi, G, lnP = workloads.stack([w.base])
    d = plan.eval_real(om, h0, chi, G, lnP, nus, lnPL=workloads.stack_lin([w.base]))[0]
    d = np.array([float("%.6e" % v) for v in d])
    i = np.arange(len(d))
    s = 0.05 * np.abs(d) + 1e-3 * np.sqrt(np.mean(d ** 2))
    cov = np.exp(-np.abs(i[:, None] - i[None]) / 5.0) * s[:, None] * s[None]
    return plan.likelihood(d, np.linalg.inv(cov))


def _spectra(n, nk, seed):
    """Linear spectra k^ns / (1 + (k/k0)^2 L)^2 of the cold-dark-matter shape
    on nk log-spaced k in 1e-5..1e3 h/Mpc, each with its own amplitude, tilt
    and turnover."""
    rng = np.random.default_rng(seed)
    k = np.geomspace(workloads.FASTPT_KMIN, workloads.FASTPT_KMAX, nk)
    amp, ns, gam = rng.uniform(0.7, 1.3, (n, 1)), rng.uniform(0.92, 1.0, (n, 1)), rng.uniform(0.15, 0.28, (n, 1))
    q = k[None] / gam
    low = np.log(2.0 * math.e + 1.8 * q)
    return k, 3e6 * amp * k ** ns * (low / (low + (14.2 + 731.0 / (1.0 + 62.5 * q)) * q * q)) ** 2


@functools.lru_cache(maxsize=2)
def _fastpt(nk, n):
    k = np.geomspace(workloads.FASTPT_KMIN, workloads.FASTPT_KMAX, nk)
    return lib.FastPT.for_bias(k, max_spec=n), lib.FastPT.for_ia(k, max_spec=n)


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    if kind == "fastpt":
        _, P = _spectra(n, case["nk"], seed)
        bias, ia = _fastpt(case["nk"], n)
        s = dict(kind=kind, host=case["host"], bias=bias, ia=ia, P=P)
        if not case["host"]:
            s["P"] = torch.as_tensor(P, device="cuda")
            s["ob"] = torch.empty((n, 5, case["nk"]), dtype=torch.float64, device="cuda")
            s["oi"] = torch.empty((n, 10, case["nk"]), dtype=torch.float64, device="cuda")
        return s
    w = _workload(case["workload"])
    d = _points(w, n, seed, "cuda")
    s = dict(kind=kind, d=d, w=w, host=case.get("host", kind == "like"))
    if kind in ("fourier", "real"):
        two = case.get("two", False)
        s["plan"] = _plan(case["workload"], case["precision"], n, two)
        if s["host"]:
            s["d"] = _host(d)
            s["lnPL"] = s["d"]["lnPL"] if two else None
        else:
            s["lnPL"] = d["lnPL"] if two else None
            size = s["plan"].n_total if kind == "real" else s["plan"].fourier_n_total(len(w.ell))
            s["out"] = torch.empty((n, size), dtype=torch.float64, device="cuda")
    elif kind == "grad":
        s["plan"] = _plan(case["workload"], "mixed", n, False)
        s["cot"] = torch.as_tensor(np.random.default_rng(seed + 1).normal(size=(n, s["plan"].n_total)),
                                   device="cuda")
    elif kind == "like":
        s["plan"] = _plan(case["workload"], "mixed", n, True)
        s["like"] = _likelihood(case["workload"], n)
        s["d"] = _host(d)
    else:
        s["plan"] = _plan(case["workload"], "mixed", n, False)
        nell = len(w.ell)
        full = s["plan"].fourier_n_total(nell)
        # every batch holds walkers with 40% to 100% of the bins, in its own order
        keep = np.random.default_rng(seed + 1).permutation(np.linspace(0.4, 1.0, n))
        m = torch.as_tensor(np.maximum(1, np.round(keep * nell)), device="cuda")
        kept = (torch.arange(full, device="cuda") % nell)[None] < m[:, None]
        s["idx"] = torch.nonzero(kept)[:, 1].int()
        s["ptr"] = torch.nn.functional.pad(torch.cumsum(kept.sum(1), 0), (1, 0)).int()
        s["out"] = torch.empty(s["idx"].numel(), dtype=torch.float64, device="cuda")
        side = torch.cuda.Stream()
        torch.cuda.synchronize()
        s["graph"] = s["plan"].fourier_graph(*(d[k] for k in _TABLES), d["nu"], w.ell, s["out"], row_ptr=s["ptr"],
                                             idx=s["idx"], stream=side.cuda_stream)
        side.synchronize()
    return s


# --------------------------------------------------------------------- calls
def run(state):
    kind, host = state["kind"], state["host"]
    if kind == "fastpt":
        if host:
            return dict(bias=state["bias"].bias(state["P"]), ia=state["ia"].ia(state["P"]))
        stream = torch.cuda.current_stream().cuda_stream
        state["bias"].bias_device(state["P"], state["ob"], stream)
        state["ia"].ia_device(state["P"], state["oi"], stream)
        return dict(bias=state["ob"], ia=state["oi"])
    d, plan = state["d"], state["plan"]
    t = [d[k] for k in _TABLES]
    if kind == "like":
        chi2, lbar, nbar = plan.loglike_real(state["like"], *t, d["nus"], lnPL=d["lnPL"], grad=True)
        return dict(chi2=chi2, lnP=lbar, nu=nbar)
    if host:
        if kind == "real":
            return plan.eval_real(*t, d["nus"], lnPL=state["lnPL"])
        return plan.eval_fourier(*t, d["nus"], state["w"].ell)
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "real":
        plan.eval_real_device(*t, d["nu"], state["out"], lnPL=state["lnPL"], stream=stream)
        return state["out"]
    if kind == "fourier":
        plan.eval_fourier_device(*t, d["nu"], state["w"].ell, state["out"], stream=stream)
        return state["out"]
    if kind == "grad":
        dv, lbar, nbar = autograd.value_and_vjp(plan, *t, d["nu"], state["cot"])
        return dict(dv=dv, lnP=lbar, nu=nbar)
    state["graph"].launch(stream)
    return state["out"]


# ---------------------------------------------------------------------- work
def _fft(n):
    return 5.0 * n * math.log2(n)


def work(case):
    """Inputs read once and outputs written once; the operations of the
    quadratures, transforms and products as the method states them (30 per
    table walk, 2 per term of a product, 5 N log2 N per complex transform)."""
    n = case["n"]
    if case["kind"] == "fastpt":
        N = case["nk"] + 4000
        bias = 4.5 * _fft(2 * N) + 2.5 * _fft(2 * N) + 3.0 * _fft(N)
        ia = 26.0 * _fft(2 * N) + 8.0 * _fft(N)
        return dict(bytes=8.0 * case["nk"] * n * (1 + 5 + 1 + 10), flops=n * (bias + ia))
    w = _workload(case["workload"])
    c = w.cfg
    pss, pgs, pgg = abi.n_pairs(c)
    table = len(w.base.log10k) * len(w.base.pk_z)
    inputs = table * (2 if case.get("two") or case["kind"] == "like" else 1) + 2 * len(w.base.chi_z) + NU
    if case["kind"] in ("fourier", "serving"):
        K, nell = len(w.ell), len(w.ell)
        out = nell * (pss + (0 if c.probes == abi.PROBE_XI else pgs + pgg)) * (0.7 if case["kind"] == "serving" else 1)
        products = 0.0
    else:
        K = c.lmin_tab - 1 + c.n_ell
        out = c.ntheta * (2 * pss + pgs + pgg)
        products = 2.0 * K * out
    flops = K * 64.0 * (30 + 2 * pss)
    if c.probes != abi.PROBE_XI:
        flops += K * c.n_lens * 64.0 * (30 + 2 * c.n_source) + K * c.n_lens * 96.0 * 50
        if not c.adopt_limber_gg:  # half of the multipoles before the hand-over to Limber, two kernels each
            flops += c.n_lens * (0.5 * c.lmax_nolimber * 2 * (_fft(c.nl_nchi + 400) / 2 + 10 * c.nl_nchi))
    flops += products
    if w.tatt:
        flops += 35.0 * _fft(10240) + K * 64.0 * 10 * (pss + pgs)
    if case["kind"] in ("grad", "like"):
        return dict(bytes=8.0 * n * (2 * inputs + out), flops=3.0 * n * flops)
    return dict(bytes=8.0 * n * (inputs + out), flops=n * flops)


# --------------------------------------------------------------------- exact
def exact(case, seed):
    """The cosmic-shear spectra and the one-loop bias spectra in 64 bits.
    The 3x2pt vectors and gradients, with the FFTLog walk, the Legendre sums
    to l = 50000 and the quadratures of every pair, take minutes a batch in
    plain numpy, and the 184-term TATT tables as long: none for these."""
    if case["kind"] == "fastpt" and case["n"] * case["nk"] <= 1 << 20:
        return dict(bias=_bias_exact(*_spectra(case["n"], case["nk"], seed)), ia=None)
    if case["kind"] == "fourier":
        return _shear_exact(case, seed)
    return None


def _table_cell(x, v):
    return np.clip(np.searchsorted(x, v, side="right") - 1, 0, len(x) - 2)


def _natural_spline(x, y):
    """Second derivatives of the natural cubic spline through (x, y)."""
    n, h = len(x), np.diff(x)
    A = np.zeros((n, n))
    A[0, 0] = A[-1, -1] = 1.0
    i = np.arange(1, n - 1)
    A[i, i - 1], A[i, i], A[i, i + 1] = h[:-1], 2.0 * (h[:-1] + h[1:]), h[1:]
    r = np.zeros(n)
    r[1:-1] = 6.0 * (np.diff(y)[1:] / h[1:] - np.diff(y)[:-1] / h[:-1])
    return np.linalg.solve(A, r)


def _spline(x, y, m, v):
    i = _table_cell(x, v)
    h = x[i + 1] - x[i]
    a, b = (x[i + 1] - v) / h, (v - x[i]) / h
    s = a * y[i] + b * y[i + 1] + ((a ** 3 - a) * m[i] + (b ** 3 - b) * m[i + 1]) * h * h / 6.0
    return np.where((v < x[0]) | (v > x[-1]), 0.0, s)


def _shear_exact(case, seed):
    """C_ss by the Limber quadrature on Gauss-Legendre nodes in a, with the
    lens efficiencies from cumulative trapezoids of the shifted n(z)."""
    w = _workload(case["workload"])
    c, h = w.cfg, {k: v.cpu().numpy() for k, v in _points(w, case["n"], seed, "cuda").items()}
    ns, zraw, nz = c.n_source, w.src[:, 0], len(w.src)
    dzh = (zraw[-1] - zraw[0]) / (nz - 1)
    zlo, zhi = max(zraw[0], 1e-5), zraw[-1] + dzh
    dz = (zhi - zlo) / nz
    zc = zlo + (np.arange(nz) + 0.5) * dz
    hist = w.src[np.clip(np.floor((zc - zraw[0]) / dzh).astype(int), 0, nz - 1), 1:].T
    y = hist / (hist.sum(1, keepdims=True) * dz)
    m2 = [_natural_spline(zc, y[j]) for j in range(ns)]
    amin, amax = 1.0 / (zhi + 1.0), 0.999999
    per = 25 * (1 + abs(c.high_def_integration))
    af = np.linspace(amin, amax, per * (c.n_a - 1) + 1)
    da, dac = (amax - amin) / (len(af) - 1), (amax - amin) / (c.n_a - 1)
    xg, wg = np.polynomial.legendre.leggauss(64)
    b = 1.0 / (1.0 + max(zlo, 1e-6))
    a = 0.5 * (b + amin) + 0.5 * (b - amin) * xg
    wa = 0.5 * (b - amin) * wg
    z = 1.0 / a - 1.0
    ell = w.ell + 0.5
    pref = w.ell * (w.ell - 1.0) * (w.ell + 1.0) * (w.ell + 2.0) / ell ** 4
    cz, X, lk, pz = w.base.chi_z, h["chi"] / 2997.92458, w.base.log10k, w.base.pk_z
    pairs = abi.shear_pairs(ns)
    pss, pgs, pgg = abi.n_pairs(c)
    out = np.zeros((case["n"], len(ell) * (pss + pgs + pgg)))
    for p in range(case["n"]):
        x = X[p]
        fk, chif = np.interp(z, cz, x), np.interp(1.0 / af - 1.0, cz, x)
        j = _table_cell(cz, z)
        t = (z - cz[j]) / (cz[j + 1] - cz[j])
        up = (x[j + 2] - x[j]) / (cz[j + 2] - cz[j])
        lo = np.where(j > 0, j - 1, j)
        down = (x[j + 1] - x[lo]) / (cz[j + 1] - cz[lo])
        dchida = (down + t * (up - down)) / (a * a)
        W = np.empty((ns, len(a)))
        for s in range(ns):
            f = _spline(zc, y[s], m2[s], 1.0 / af - 1.0 - h["nu"][p, s]) / af ** 2
            cum = lambda g: np.concatenate([[0.0], np.cumsum(0.5 * da * (g[1:] + g[:-1]))])  # noqa: E731
            g = (cum(f) - chif * cum(f / chif))[::per]
            r = (a - amin) / dac
            i = np.clip(np.floor(r).astype(int), 0, c.n_a - 2)
            ga = np.where((a <= amin) | (a > 1.0 - dac), 0.0, g[i] + (r - i) * (g[i + 1] - g[i]))
            W[s] = 1.5 * h["om"][p] * fk / a * ga
        k = np.log10(ell[:, None] / fk[None] / 2997.92458)
        P = h["lnP"][p].reshape(len(lk), len(pz))
        ik, iz = _table_cell(lk, k), _table_cell(pz, z)[None]
        dx, dy = (k - lk[ik]) / (lk[ik + 1] - lk[ik]), ((z - pz[iz]) / (pz[iz + 1] - pz[iz]))
        lnp = (1 - dx) * ((1 - dy) * P[ik, iz] + dy * P[ik, iz + 1]) + \
            dx * ((1 - dy) * P[ik + 1, iz] + dy * P[ik + 1, iz + 1])
        core = np.exp(lnp) / 2997.92458 ** 3 * (wa * dchida / fk ** 2)[None] * pref[:, None]
        cal = 1.0 + h["nu"][p, 3 * MB:3 * MB + ns]
        for q, (s1, s2) in enumerate(pairs):
            out[p, q * len(ell):(q + 1) * len(ell)] = core @ (W[s1] * W[s2]) * cal[s1] * cal[s2]
    return out


def _next_size(n):
    """The next product of 2, 3, 5 and 7 that is at least n."""
    while True:
        r = n
        for p in (2, 3, 5, 7):
            while r % p == 0:
                r //= p
        if r == 1:
            return n
        n += 1


def _ln_gamma(z):
    """ln Gamma for complex z, Re z > -20: Stirling's series with Bernoulli
    numbers to 1/z^15 after 40 upward steps of the recurrence."""
    shift = np.zeros_like(z)
    for _ in range(40):
        shift = shift + np.log(z)
        z = z + 1.0
    s = (z - 0.5) * np.log(z) - z + 0.5 * math.log(2.0 * math.pi)
    for i, c in enumerate((1 / 12, -1 / 360, 1 / 1260, -1 / 1680, 1 / 1188, -691 / 360360, 1 / 156, -3617 / 122400)):
        s = s + c / z ** (2 * i + 1)
    return s - shift


def _bias_exact(k, P, npad=1500, nlow=500, nhigh=500, window=0.65):
    """P_d1d2, P_d2d2, P_d1s2, P_d2s2 and P_s2s2 by FAST-PT's J_abl sums:
    biased by k^2, log-extrapolated, padded, tapered, convolved in the
    Fourier index."""
    n, N0 = P.shape
    nu = -2.0
    N = _next_size(N0 + 2 * npad + nlow + nhigh)
    while N % 2:
        N = _next_size(N + 1)
    half, total, dl = N // 2, _next_size(2 * N + 1), math.log(k[1] / k[0])
    f = np.zeros((n, N))
    f[:, npad + nlow:npad + nlow + N0] = P * k ** -nu
    i = np.arange(-nlow, 0)
    f[:, npad:npad + nlow] = P[:, :1] * np.exp(i * np.log(P[:, 1:2] / P[:, :1])) * (k[0] * np.exp(i * dl)) ** -nu
    i = np.arange(N - npad - nhigh, N - npad) - (npad + nlow + N0)
    f[:, N - npad - nhigh:N - npad] = P[:, -1:] * np.exp(i * np.log(P[:, -1:] / P[:, -2:-1])) * \
        (k[-1] * np.exp(i * dl)) ** -nu
    cm = np.fft.rfft(f) / N
    cut = int(half * window)
    i = np.arange(cut + 1)
    taper = i / cut - np.sin(2.0 * np.pi * i / cut) / (2.0 * np.pi)
    cm[:, half - cut + i] *= taper
    cm[:, i] *= taper[cut - i]
    eta, tau = 2.0 * np.pi / dl / N * np.arange(half + 1), 2.0 * np.pi / dl / N * np.arange(N + 1)
    gm = lambda mu, q: np.exp(_ln_gamma((mu + 1 + q) / 2) - _ln_gamma((mu + 1 - q) / 2))  # noqa: E731
    spectra = {}

    def transform(alpha, l):
        if (alpha, l) not in spectra:
            up = cm * gm(l + 0.5, 1.5 + nu + alpha + 1j * eta)
            spectra[alpha, l] = np.fft.fft(np.concatenate([np.conj(up[:, :0:-1]), up], 1), total)
        return spectra[alpha, l]

    pw = -5 - 2 * int(nu)  # alpha + beta = 0 in every term
    zf = pw + 1 + 1j * tau
    fz = gm(0.5, zf - 0.5) * math.sqrt(math.pi) / 2.0 * np.exp(zf * math.log(2.0))
    terms = [(0, 0, 0, 34 / 21), (0, 2, 0, 8 / 21), (1, 1, 0, 2.0), (0, 0, 1, 2.0), (0, 0, 2, 16 / 315),
             (0, 2, 2, 508 / 441), (0, 4, 2, 32 / 245), (1, 1, 2, 8 / 15), (1, 3, 2, 4 / 5), (0, 2, 3, 4 / 3),
             (0, 0, 4, 8 / 45), (0, 2, 4, 16 / 63), (0, 4, 4, 16 / 35)]
    out = np.zeros((n, 5, N0))
    for row in range(5):
        acc = 0.0
        for alpha, l, o, coeff in terms:
            if o == row:
                acc = acc + (-1) ** l * coeff * transform(alpha, l) * transform(-alpha, l)
        conv = np.fft.ifft(acc)[:, N:2 * N + 1]
        conv[:, 0] = conv[:, 0].real
        v = conv * np.conj(fz) * np.exp(1j * tau * math.log(2.0))
        r = np.fft.irfft(v, 2 * N) * (2 * N)
        out[:, row] = r[:, 2 * (npad + nlow):2 * (npad + nlow + N0):2] * 2.0 ** (2 + 2 * nu) / np.pi ** 2 * k ** (-pw - 2.0)
    return out
