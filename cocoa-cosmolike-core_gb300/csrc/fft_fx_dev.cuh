// fft_fx_dev.cuh -- the CTA-wide transforms of fft_fx.cuh on an FP64 buffer
// in shared memory, converted in place on the way in and out.
#pragma once
#include "fft_fx.cuh"

namespace cl2pt {
namespace fx {

template <int R, bool DIF>
__device__ __noinline__ unsigned stage(c64* buf, int n, int L, int m, FastDiv md, const int4* __restrict__ tw, int sin)
{
  __builtin_assume(__isShared(buf));
  unsigned top = 0;
  const int tot = n / R, tstep = n / L;
  for (int q = threadIdx.x; q < tot; q += blockDim.x) butterfly<R, DIF>(buf, q, L, m, tstep, md, tw, sin, top);
  return top;
}

// n <= GENERIC_MAX_PER_THREAD * blockDim.x
template <bool DIF>
__device__ __noinline__ unsigned stage_generic(c64* buf, int n, int L, int m, int R, FastDiv md, FastDiv rd,
                                               const int4* __restrict__ tw, int sin)
{
  __builtin_assume(__isShared(buf));
  if (sin || !DIF) {
    for (int i = threadIdx.x; i < n; i += blockDim.x)
      buf[i] = generic_pre<DIF>(buf[i], i, m, R, n / L, md, rd, tw, sin);
    __syncthreads();
  }
  unsigned top = 0;
  c64 y[GENERIC_MAX_PER_THREAD];
#pragma unroll
  for (int c = 0; c < GENERIC_MAX_PER_THREAD; c++) {
    const int o = threadIdx.x + c * blockDim.x;
    int pos;
    if (o < n) {
      y[c] = generic_out<DIF>(buf, o, pos, n, L, m, R, md, rd, tw);
      note(top, y[c]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < GENERIC_MAX_PER_THREAD; c++) {
    const int o = threadIdx.x + c * blockDim.x;
    if (o < n) {
      const int q = quot(o, rd), k = o - q * R, b = quot(q, md);
      buf[b * L + q - b * m + k * m] = y[c];
    }
  }
  return top;
}

template <bool DIF>
__device__ __forceinline__ unsigned run_stage(c64* buf, const Desc& d, int s, const int4* tw, int sin)
{
  const int R = d.rad[s], n = d.n, L = d.L[s], m = L / R;
  switch (R) {
    case 2: return stage<2, DIF>(buf, n, L, m, d.m[s], tw, sin);
    case 3: return stage<3, DIF>(buf, n, L, m, d.m[s], tw, sin);
    case 4: return stage<4, DIF>(buf, n, L, m, d.m[s], tw, sin);
    case 5: return stage<5, DIF>(buf, n, L, m, d.m[s], tw, sin);
    case 6: return stage<6, DIF>(buf, n, L, m, d.m[s], tw, sin);
    case 7: return stage<7, DIF>(buf, n, L, m, d.m[s], tw, sin);
    case 8: return stage<8, DIF>(buf, n, L, m, d.m[s], tw, sin);
    case 9: return stage<9, DIF>(buf, n, L, m, d.m[s], tw, sin);
    case 10: return stage<10, DIF>(buf, n, L, m, d.m[s], tw, sin);
    case 12: return stage<12, DIF>(buf, n, L, m, d.m[s], tw, sin);
    case 14: return stage<14, DIF>(buf, n, L, m, d.m[s], tw, sin);
    case 15: return stage<15, DIF>(buf, n, L, m, d.m[s], tw, sin);
    default: return stage_generic<DIF>(buf, n, L, m, R, d.m[s], d.r[s], tw, sin);
  }
}

// A value's shared state between the conversions: scale 2^K, the union top
// of the high words, the L1 bound 2^l1, the exponent db that the imaginary
// parts were raised by
struct State {
  int K, db;
  unsigned top;
  float l1;
};

// union / sum over the CTA; returns after a __syncthreads()
__device__ __forceinline__ unsigned block_or(unsigned v, unsigned* red)
{
  v = __reduce_or_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  return __reduce_or_sync(0xffffffffu, lane < (int)(blockDim.x >> 5) ? red[lane] : 0u);
}

// the stages; red: two sets of 32 words, used in turn so that one barrier a
// stage serves the data and the reduction
template <bool DIF>
__device__ __forceinline__ void stages(c64* z, const Desc& d, const int4* tw, State& st, unsigned* red)
{
  for (int i = 0; i < d.nst; i++) {
    const int s = DIF ? i : d.nst - 1 - i;
    const int sin = room(st.top, d.rad[s], st.l1);
    st.K -= sin;
    st.top = block_or(run_stage<DIF>(z, d, s, tw, sin), red + 32 * (i & 1));
  }
}

// FP64 -> fixed point, times w (or none); the imaginary parts raised to the
// real ones' magnitude if bal.  False (buffer filled with NaN up to n, or
// zeros up to n) if an entry is not finite or all are zero.
__device__ __forceinline__ bool load(c64* z, int n, bool inv, bool bal, const int4* __restrict__ w, State& st,
                                     unsigned* red)
{
  ulonglong2* u = (ulonglong2*)z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  unsigned mx = 0, my = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const ulonglong2 v = u[i];
    mx = max(mx, (unsigned)(v.x >> 32) & 0x7fffffffu);
    my = max(my, (unsigned)(v.y >> 32) & 0x7fffffffu);
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  my = __reduce_max_sync(0xffffffffu, my);
  if (lane == 0) {
    red[warp] = mx;
    red[32 + warp] = my;
  }
  __syncthreads();
  mx = __reduce_max_sync(0xffffffffu, lane < nw ? red[lane] : 0u);
  my = __reduce_max_sync(0xffffffffu, lane < nw ? red[32 + lane] : 0u);
  const int ex = (int)(mx >> 20), ey = (int)(my >> 20);
  st.db = 0;
  if (ex == 0x7ff || ey == 0x7ff || (ex | ey) == 0) {
    const unsigned long long f = (ex | ey) ? 0x7ff8000000000000ull : 0ull;
    for (int i = threadIdx.x; i < n; i += blockDim.x) u[i] = make_ulonglong2(f, f);
    __syncthreads();
    return false;
  }
  if (bal && ex && ey) st.db = ex - ey;
  // parts below 2^(e - 1022), e the larger exponent: to 59 bits
  const int K = 59 - (max(ex, ey + st.db) - 1022);
  float l1 = 0.0f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const ulonglong2 v = u[i];
    c64 a = {to_fx(v.x, K), to_fx(v.y, K + st.db)};
    // (|x| + |y|) / 2^38 rounded up, the 21-bit parts to FP32 by their bits
    const unsigned ax = (unsigned)((a.x < 0 ? -a.x : a.x) >> 38), ay = (unsigned)((a.y < 0 ? -a.y : a.y) >> 38);
    l1 += (__uint_as_float(0x4B000000u + ax) - 8388607.0f) + (__uint_as_float(0x4B000000u + ay) - 8388607.0f);
    if (inv) a = {a.y, a.x};
    if (w) a = mulw(a, __ldg(w + i));
    z[i] = a;
  }
  for (int o = 16; o > 0; o >>= 1) l1 += __shfl_xor_sync(0xffffffffu, l1, o);
  __syncthreads();  // the maxima have been read
  if (lane == 0) red[warp] = __float_as_uint(l1);
  __syncthreads();
  l1 = 0.0f;
  for (int i = 0; i < nw; i++) l1 += __uint_as_float(red[i]);
  __syncthreads();
  st.K = K;
  st.top = (1u << 27) - 1u;
  st.l1 = log2f(l1 * 1.001f) + 38.0f;
  return true;
}

// fixed point, times w (or none) -> FP64
__device__ __forceinline__ void store(c64* z, int n, bool inv, const int4* __restrict__ w, int K)
{
  ulonglong2* u = (ulonglong2*)z;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    c64 a = z[i];
    if (w) a = mulw(a, __ldg(w + i));
    if (inv) a = {a.y, a.x};
    u[i] = make_ulonglong2(to_fp(a.x, K), to_fp(a.y, K));
  }
  __syncthreads();
}

// In-place transform of the FP64 buffer, sum_n x[n] exp(S 2 pi i n k / n).
// bal: the imaginary parts are raised by a power of two to the real ones'
// magnitude first (two real sequences packed in one, the larger one's
// rounding would swamp the smaller); its exponent is returned and stays in
// the result.  Caller synchronises before the call; returns after a
// __syncthreads().
template <int S, bool DIF>
__device__ int transform(double2* buf, const Desc& d, const int4* __restrict__ tw, bool bal)
{
  __shared__ unsigned red[64];
  c64* z = (c64*)buf;
  State st;
  if (!load(z, d.n, S > 0, bal, nullptr, st, red)) return 0;
  stages<DIF>(z, d, tw, st, red);
  store(z, d.n, S > 0, nullptr, st.K);
  return st.db;
}
template <int S> __device__ __forceinline__ int dif(double2* buf, const Desc& d, const int4* tw, bool bal)
{
  return transform<S, true>(buf, d, tw, bal);
}
template <int S> __device__ __forceinline__ int dit(double2* buf, const Desc& d, const int4* tw, bool bal)
{
  return transform<S, false>(buf, d, tw, bal);
}

// The same of n points through the convolution of size d.n >= 2 n - 1 (the
// buffer holds d.n), natural order in and out
template <int S>
__device__ int chirp(double2* buf, int n, const Desc& d, const int4* __restrict__ tw, const Chirp& c, bool bal)
{
  __shared__ unsigned red[64];
  c64* z = (c64*)buf;
  State st;
  if (!load(z, n, S > 0, bal, c.w, st, red)) return 0;
  for (int i = n + threadIdx.x; i < d.n; i += blockDim.x) z[i] = {0, 0};
  __syncthreads();
  stages<true>(z, d, tw, st, red);
  // times the chirp's transform; the inverse as the forward transform of
  // the exchanged parts
  unsigned top = 0;
  for (int i = threadIdx.x; i < d.n; i += blockDim.x) {
    const c64 a = mulw(z[i], __ldg(c.b + i));
    note(top, a);
    z[i] = {a.y, a.x};
  }
  __syncthreads();  // red: the last stage's union has been read
  st.top = block_or(top, red);
  __syncthreads();
  st.l1 = 128.0f;
  stages<false>(z, d, tw, st, red);
  for (int i = threadIdx.x; i < n; i += blockDim.x) z[i] = {z[i].y, z[i].x};
  store(z, n, S > 0, c.w, st.K - c.kb);
  return st.db;
}

}  // namespace fx
}  // namespace cl2pt
