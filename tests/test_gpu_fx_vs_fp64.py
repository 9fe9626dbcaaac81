"""The fixed-point transforms (fft_fx_dev.cuh) against the FP64 ones
(fft64.cuh) on the GPU, both against whole sums in extended precision: the
error of the fixed point is no larger, over all outputs (L2 norm) and over the
small ones alone (below 1e-6 and below 1e-10 of the largest), which an L2 norm
does not see.  That is the reason the FAST-PT transforms run in it, so the bound
is the FP64 form's own error, with half a unit of 2^-53 of the outputs' norm for
the results' rounding to FP64."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from test_fft_fx import CSRC, ROOT, signal

SRC = r"""
#include <complex>
#include "fft64.cuh"
#include "fft_fx_dev.cuh"
using namespace cl2pt;
__global__ void __launch_bounds__(512, 1) k_fx(fx::Desc d, const int4* tw, double2* x)
{
  extern __shared__ double2 b[];
  for (int i = threadIdx.x; i < d.n; i += blockDim.x) b[i] = x[i];
  __syncthreads();
  fx::dif<-1>(b, d, tw, false);
  for (int i = threadIdx.x; i < d.n; i += blockDim.x) x[i] = b[i];
}
__global__ void __launch_bounds__(512, 1) k_64(fft64::Desc d, const double2* tw, double2* x)
{
  extern __shared__ double2 b[];
  for (int i = threadIdx.x; i < d.n; i += blockDim.x) b[i] = x[i];
  __syncthreads();
  fft64::dif<-1>(b, d, tw);
  for (int i = threadIdx.x; i < d.n; i += blockDim.x) x[i] = b[i];
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
  for (int j = 0; j < n; j++)
    w[j] = C(cosl(2 * 3.14159265358979323846264338L * j / n), -sinl(2 * 3.14159265358979323846264338L * j / n));
  for (int k = 0; k < n; k++) {
    x[k] = 0;
    for (int q = 0; q < r; q++) x[k] += s[q][k % (n / r)] * w[(long)q * k % n];
  }
}
// err [2][3]: L2 error of (fixed point, FP64) over all outputs and those below
// 1e-6 and 1e-10 of the largest, in units of 2^-53 of the whole norm
extern "C" int run(int n, const double* in, double* err)
{
  fx::Desc d;
  if (!fx::make_desc(n, d, false)) return -1;
  fft64::Desc e{};
  e.n = n;
  int L = n;
  for (int r : {4, 2, 3, 5, 7})
    while (L % r == 0) {
      e.rad[e.nst] = r;
      e.L[e.nst++] = L;
      L /= r;
    }
  if (L != 1) return -2;
  const std::vector<int4> twx = fx::twiddles(n);
  std::vector<double2> tw(n), h(n);
  for (int j = 0; j < n; j++) tw[j] = make_double2(cos(-2.0 * M_PI * j / n), sin(-2.0 * M_PI * j / n));
  std::vector<C> x(n);
  for (int i = 0; i < n; i++) x[i] = C(in[2 * i], in[2 * i + 1]);
  dft(x);
  long double top = 0, all = 0;
  for (const C& v : x) {
    top = std::max(top, std::abs(v));
    all += std::norm(v);
  }
  const size_t sm = sizeof(double2) * n;
  void *t, *b;
  if (cudaMalloc(&t, sm) || cudaMalloc(&b, sm)) return -3;
  cudaFuncSetAttribute(k_fx, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  cudaFuncSetAttribute(k_64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  for (int f = 0; f < 2; f++) {
    cudaMemcpy(b, in, sm, cudaMemcpyHostToDevice);
    cudaMemcpy(t, f ? (const void*)tw.data() : (const void*)twx.data(), sm, cudaMemcpyHostToDevice);
    if (f) k_64<<<1, 512, sm>>>(e, (const double2*)t, (double2*)b);
    else k_fx<<<1, 512, sm>>>(d, (const int4*)t, (double2*)b);
    cudaMemcpy(h.data(), b, sm, cudaMemcpyDeviceToHost);
    long double s[3] = {0, 0, 0};
    for (int p = 0; p < n; p++) {
      int q = p, k = 0, m = 1;
      for (int i = 0; i < (f ? e.nst : d.nst); i++) {
        const int r = f ? e.rad[i] : d.rad[i], w = (f ? e.L[i] : d.L[i]) / r;
        k += q / w * m;
        q %= w;
        m *= r;
      }
      const long double v = std::norm(x[k] - C(h[p].x, h[p].y)), a = std::abs(x[k]) / top;
      s[0] += v;
      if (a < 1e-6L) s[1] += v;
      if (a < 1e-10L) s[2] += v;
    }
    for (int i = 0; i < 3; i++) err[3 * f + i] = (double)(sqrtl(s[i] / all) * 9007199254740992.0L);
  }
  cudaFree(t);
  cudaFree(b);
  return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def transforms(tmp_path_factory):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    d = tmp_path_factory.mktemp("fx64")
    src, so = str(d / "fx64.cu"), str(d / "fx64.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"), src, "-o", so], check=True)
    return ctypes.CDLL(so).run


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["noise", "smooth", "decades"])
@pytest.mark.parametrize("n", [5040, 6048, 6144, 10206, 12150, 14406])
def test_error_no_larger(transforms, n, kind):
    x = np.ascontiguousarray(signal(kind, n, np.random.default_rng(n)), np.complex128)
    err = np.zeros(6)
    P = ctypes.c_void_p
    assert transforms(n, x.ctypes.data_as(P), err.ctypes.data_as(P)) == 0
    print(n, kind, "units of 2^-53, all / below 1e-6 / below 1e-10: fixed point", err[:3], "FP64", err[3:])
    assert (err[:3] <= err[3:] + 0.5).all()
