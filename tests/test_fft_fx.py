"""The fixed-point transforms (fft_fx.cuh).

CPU: the stages run on the host (the same functions that the kernels call)
against whole sums in extended precision.  Tolerance: the error of an FP64
transform grows with the stages, about log2(n) / 2 units of 2^-53 of the L2
norm, plus one unit for the result's own rounding to FP64.

GPU: J_abJ1J2Jk at padded sizes that take each radix, a generic prime stage,
the convolution form and the largest convolution, two equal terms sharing each
transform, against the oracle at the bar of the other FAST-PT tests.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "cocoa-cosmolike-core_gb300", "csrc")

SRC = r"""
#include "fft_fx.cuh"
#include <complex>
#include <cstring>
using namespace cl2pt::fx;
template <int R, bool D> void st(c64* z, const Desc& d, int s, const int4* tw, int sin, unsigned& top)
{
  for (int q = 0; q < d.n / R; q++) butterfly<R, D>(z, q, d.L[s], d.L[s] / R, d.n / d.L[s], d.m[s], tw, sin, top);
}
template <bool D> void stages(std::vector<c64>& z, const Desc& d, const int4* tw, unsigned top, float l1, int& K)
{
  for (int i = 0; i < d.nst; i++) {
    const int s = D ? i : d.nst - 1 - i, R = d.rad[s], m = d.L[s] / R, n = d.n;
    const int sin = room(top, R, l1);
    K -= sin;
    top = 0;
    switch (R) {
#define CASE(r) case r: st<r, D>(z.data(), d, s, tw, sin, top); break;
      CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7) CASE(8) CASE(9) CASE(10) CASE(12) CASE(14) CASE(15)
      default: {
        for (int j = 0; j < n; j++) z[j] = generic_pre<D>(z[j], j, m, R, n / d.L[s], d.m[s], d.r[s], tw, sin);
        std::vector<c64> y(n);
        for (int o = 0, p; o < n; o++) {
          const c64 v = generic_out<D>(z.data(), o, p, n, d.L[s], m, R, d.m[s], d.r[s], tw);
          y[p] = v;
          note(top, v);
        }
        z.swap(y);
      }
    }
  }
}
static unsigned long long bits(double v) { unsigned long long u; memcpy(&u, &v, 8); return u; }
static double dbl(unsigned long long u) { double v; memcpy(&v, &u, 8); return v; }
// T > 0: n points through the convolution of size T
extern "C" int run(int n, int T, int dif, const double* in, double* out)
{
  Desc d;
  if (!make_desc(T ? T : n, d, !T)) return -1;
  const std::vector<int4> tw = twiddles(d.n);
  const std::vector<int> rev = digit_reverse(d);
  std::vector<int4> w, b;
  int kb = 0;
  if (T) kb = chirp_tables(n, d, tw, w, b);
  double mx = 0;
  for (int i = 0; i < 2 * n; i++) mx = fmax(mx, fabs(in[i]));
  int K = 59 - ((int)(bits(mx) >> 52) - 1022);
  float l1 = 0;
  std::vector<c64> z(d.n, c64{0, 0});
  for (int p = 0; p < n; p++) {
    const int i = T || dif ? p : rev[p];
    z[p] = {to_fx(bits(in[2 * i]), K), to_fx(bits(in[2 * i + 1]), K)};
    l1 += (float)(llabs(z[p].x) >> 38) + (float)(llabs(z[p].y) >> 38) + 2.0f;
    if (T) z[p] = mulw(z[p], w[p]);
  }
  l1 = log2f(l1 * 1.001f) + 38.0f;
  const unsigned top = (1u << 27) - 1;
  if (T || dif) stages<true>(z, d, tw.data(), top, l1, K);
  else stages<false>(z, d, tw.data(), top, l1, K);
  if (T) {
    unsigned t = 0;
    for (int p = 0; p < d.n; p++) {
      const c64 a = mulw(z[p], b[p]);
      note(t, a);
      z[p] = {a.y, a.x};
    }
    stages<false>(z, d, tw.data(), t, 128.0f, K);
    K -= kb;
  }
  for (int p = 0; p < n; p++) {
    const int k = !T && dif ? rev[p] : p;
    const c64 a = T ? mulw(c64{z[p].y, z[p].x}, w[p]) : z[p];
    out[2 * k] = dbl(to_fp(a.x, K));
    out[2 * k + 1] = dbl(to_fp(a.y, K));
  }
  return d.nst;
}
typedef std::complex<long double> C;
static void dft(std::vector<C>& x)
{
  const int n = x.size();
  if (n == 1) return;
  int r = 2;
  while (n % r) r++;
  std::vector<std::vector<C>> s(r, std::vector<C>(n / r));
  for (int i = 0; i < n; i++) s[i % r][i / r] = x[i];
  for (auto& v : s) dft(v);
  std::vector<C> w(n);
  for (int j = 0; j < n; j++) w[j] = C(cosl(2 * 3.14159265358979323846264338L * j / n), -sinl(2 * 3.14159265358979323846264338L * j / n));
  for (int k = 0; k < n; k++) {
    x[k] = 0;
    for (int q = 0; q < r; q++) x[k] += s[q][k % (n / r)] * w[(long)q * k % n];
  }
}
// L2 distance of got from the transform of in, over its L2 norm
extern "C" double error(int n, const double* in, const double* got)
{
  std::vector<C> x(n);
  for (int i = 0; i < n; i++) x[i] = C(in[2 * i], in[2 * i + 1]);
  dft(x);
  long double e = 0, s = 0;
  for (int i = 0; i < n; i++) {
    e += std::norm(x[i] - C(got[2 * i], got[2 * i + 1]));
    s += std::norm(x[i]);
  }
  return (double)sqrtl(e / s);
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("fx")
    src, so = str(d / "fx.cu"), str(d / "fx.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run(["nvcc", "-O1", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I" + CSRC,
                    "-I" + os.path.join(ROOT, "include"), src, "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.error.restype = ctypes.c_double
    return lib


def signal(kind, n, rng):
    i = np.arange(n)
    if kind == "noise":
        return rng.standard_normal(n) + 1j * rng.standard_normal(n)
    if kind == "smooth":
        return np.exp(-(((i - n / 2) / (n / 14 + 1)) ** 2) / 2) * (1 + 0.1j * np.sin(i / 30.0))
    return np.exp(rng.uniform(-30, 30, n)) * (1 - 0.5j)  # 26 decades


@pytest.mark.parametrize("kind", ["noise", "smooth", "decades"])
@pytest.mark.parametrize("n,T", [(n, 0) for n in (2, 3, 4, 5, 6, 7, 8, 9, 10, 12, 14, 15, 16, 49, 90, 77, 286, 5100,
                                                    6048, 6144, 10206, 12150, 14406)] +
                         [(29, 60), (58, 120), (4654, 9375), (6044, 12096)])
def test_stages_on_the_host(host, n, T, kind):
    x = np.ascontiguousarray(signal(kind, n, np.random.default_rng(n)), np.complex128)
    tol = (1 + (2 if T else 1) * np.log2(n) / 2) * 2.0 ** -53
    P = ctypes.c_void_p
    for dif in (1,) if T else (1, 0):
        out = np.empty_like(x)
        assert host.run(n, T, dif, x.ctypes.data_as(P), out.ctypes.data_as(P)) > 0
        assert host.error(n, x.ctypes.data_as(P), out.ctypes.data_as(P)) <= tol


@pytest.mark.gpu
@pytest.mark.parametrize("N", [90, 96, 98, 144, 162, 160, 140, 46, 44, 58, 2018, 4654, 7200])
def test_padded_sizes_vs_oracle(gpu_lib, oracle_built, N):
    import oracle as O
    from cl2pt import lib
    from test_gpu_fastpt import REL, rel_rows
    npad, nx = N // 8, N // 16
    n0 = N - 2 * npad - 2 * nx
    x = np.geomspace(1e-2, 10.0, n0)
    P = 1e3 * x / (1 + (x / 0.05) ** 2) ** 1.3
    r = np.array([[0, 0, 0, 0, 0], [0, 0, 0, 0, 0], [1, -1, 2, 1, 1], [0, 0, 4, 2, 2], [0, 0, 4, 2, 2]])
    cfg = lib.fastpt_config()
    cfg.N_pad, cfg.N_extrap_low, cfg.N_extrap_high = npad, nx, nx
    got = lib.FastPT.jk(x, *r.T, cfg=cfg).J_abJ1J2Jk(P)[0]
    ref = O.Oracle("orc").J_abJ1J2Jk(x, P, *r.T, npad=npad, nlow=nx, nhigh=nx)
    assert rel_rows(got, ref) <= REL
    # equal terms in the two halves of a shared transform
    assert rel_rows(got[[0, 3]], got[[1, 4]]) <= REL
