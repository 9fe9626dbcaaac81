// fpt_dev.cuh -- device helpers shared by k_fastpt.cu and k_fastpt_vjp.cu.
#pragma once
#include "fastpt.h"
#include "fft_fx_dev.cuh"

namespace cl2pt {
namespace {

__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cmulc(double2 a, double2 b)  // a conj(b)
{
  return make_double2(fma(a.x, b.x, a.y * b.y), fma(a.y, b.x, -a.x * b.y));
}

// v 2^e by its exponent field (integer units; the rare rest by scalbn)
__device__ __forceinline__ double p2(double v, int e)
{
  const long long u = __double_as_longlong(v);
  const int x = (int)(u >> 52) & 0x7ff;
  if (x == 0 || x == 0x7ff || x + e <= 0 || x + e >= 0x7ff) return scalbn(v, e);
  return __longlong_as_double(u + ((long long)e << 52));
}
__device__ __forceinline__ double2 p2(double2 v, int e) { return make_double2(p2(v.x, e), p2(v.y, e)); }

// Packing balance.  Two sequences share one complex transform; the
// rounding of the larger lands on the smaller in proportion to their
// magnitudes, so the second is raised by the power of two that brings its
// largest entry to the first's (exact, undone after the split).
// hi_word: high words of magnitudes compare as integers
__device__ __forceinline__ unsigned mag(double2 a)
{
  return max((unsigned)__double2hiint(a.x) & 0x7fffffffu, (unsigned)__double2hiint(a.y) & 0x7fffffffu);
}
// the exponent from the CTA's largest a and b; red: 64 words of shared memory
__device__ __forceinline__ int balance(unsigned a, unsigned b, unsigned* red)
{
  a = __reduce_max_sync(0xffffffffu, a);
  b = __reduce_max_sync(0xffffffffu, b);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (l == 0) {
    red[w] = a;
    red[32 + w] = b;
  }
  __syncthreads();
  const int ea = (int)(__reduce_max_sync(0xffffffffu, l < nw ? red[l] : 0u) >> 20);
  const int eb = (int)(__reduce_max_sync(0xffffffffu, l < nw ? red[32 + l] : 0u) >> 20);
  return ea && eb && ea < 0x7ff && eb < 0x7ff ? ea - eb : 0;
}

// size-N transform of sbuf; frequency k of the result at posN[k]
template <int S> __device__ __forceinline__ int dft_n(double2* sbuf, const FPTDev& p, bool bal)
{
  return p.chirp.w ? fx::chirp<S>(sbuf, p.N, p.dT, p.twT, p.chirp, bal) : fx::dif<S>(sbuf, p.dN, p.twN, bal);
}

}  // namespace
}  // namespace cl2pt
