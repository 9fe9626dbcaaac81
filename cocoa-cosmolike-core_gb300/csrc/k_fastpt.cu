// k_fastpt.cu -- batched FAST-PT convolutions (FP64 data).
//
// Kernels per wave of spectra, each CTA owning one in-place FFT buffer in
// shared memory:
//   k_fpt_input    one CTA per (pair of biases, spectrum): the padded,
//                  log-extrapolated spectrum (cfastpt/cfastpt.c:1066-1126,
//                  463-507) divided by x^nu of each bias, the two real
//                  sequences packed into one size-N transform and split.
//   k_fpt_forward  one CTA per (input pair, spectrum): the two padded
//                  Hermitian sequences x_u = out_b * G_u (cfastpt.c:1251-1290,
//                  620-650), centred at 0 and packed as x_u1 + i x_u2, one
//                  size-Ntot DIF; its real and imaginary parts are their
//                  real spectra R_u.
//   k_fpt_inverse  one CTA per (row pair, spectrum): sum_t c_t R_a R_b of
//                  each row (cfastpt.c:1300-1330), one size-Ntot DIT back to
//                  the lag domain, the two rows' Hermitian halves separated
//                  and multiplied by their final kernel (cfastpt.c:1340-1370,
//                  700-720).  Single-row groups finish here: the row is
//                  folded into a size-N Hermitian sequence whose inverse
//                  transform gives the even samples of the reference's size-2N
//                  c2r (cfastpt.c:1380-1415, 725-760), scaled by the k power.
//                  Multi-row groups store the products V for k_fpt_c2r.
//   k_fpt_c2r      one CTA per (group pair, spectrum): sums its rows' V,
//                  folds, transforms and scales as above.
//   The two fixed-kernel real convolutions of the TATT terms (pt_cfastpt.c:
//   681-866, utils_complex_cfastpt.c:235-318) are one more CTA per spectrum
//   of k_fpt_forward (transform and product) and of k_fpt_inverse (back): in
//   a kernel of their own (two FP64 transforms of 6144 points) they took
//   longer than those two together when there are few spectra.
#include <cuda_runtime.h>

#include "fpt_dev.cuh"

namespace cl2pt {

namespace {

__device__ __forceinline__ double qnan() { return __longlong_as_double(0x7ff8000000000000LL); }

__global__ void __launch_bounds__(FPT_THREADS, 1) k_fpt_input(FPTDev p, const double* __restrict__ fx)
{
  extern __shared__ double2 sbuf[];
  const int b1 = 2 * blockIdx.x, b2 = b1 + 1;
  const bool two = b2 < p.n_bias;
  const int s = blockIdx.y;
  const int N0 = p.N0;
  const int H1 = p.half + 1;
  const double* f = fx + (size_t)s * N0;
  double2* x1 = p.xin + ((size_t)s * p.n_bias + b1) * H1;
  double2* x2 = p.xin + ((size_t)s * p.n_bias + (two ? b2 : b1)) * H1;
  // extrapolation slopes; every thread evaluates the same checks, so the
  // early return below is uniform over the CTA
  bool bad = false;
  double sl = 1, lf0 = 0, dl = 0, sh = 1, lfN = 0, dh = 0;
  if (p.nlow) {
    const double f0 = f[0], f1 = f[1];
    if (f0 == 0.0 || f1 / f0 <= 0.0) {
      bad = true;
    } else {
      sl = f0 > 0 ? 1.0 : -1.0;
      lf0 = log(f0 * sl);
      dl = log(f1 / f0);
    }
  }
  if (p.nhigh) {
    const double f1 = f[N0 - 1], f2 = f[N0 - 2];
    if (f1 == 0.0 || f1 / f2 <= 0.0) {
      bad = true;
    } else {
      sh = f1 > 0 ? 1.0 : -1.0;
      lfN = log(f1 * sh);
      dh = log(f1 / f2);
    }
  }
  if (bad) {
    for (int k = threadIdx.x; k < H1; k += blockDim.x) {
      x1[k] = make_double2(qnan(), qnan());
      x2[k] = make_double2(qnan(), qnan());
    }
    if (threadIdx.x == 0) atomicOr(p.err, 1);
    return;
  }
  const int lo0 = p.npad, lo1 = p.npad + p.nlow;
  const int hi0 = p.N - p.npad - p.nhigh, hi1 = p.N - p.npad;
  const int jh0 = hi0 - p.off - N0;  // exponent offset of the first high point
  // the extrapolated points as products of two tables each: an FP64 exp is
  // some 40 operations, 2 (nlow / 32 + 32) of them against nlow
  double* tlo = (double*)(sbuf + p.N);
  double* thi = tlo + 2 * FPT_LO;
  for (int i = threadIdx.x; i < 2 * (FPT_LO + FPT_HI); i += blockDim.x) {
    const bool lo = i < 2 * FPT_LO;
    const int j = lo ? i : i - 2 * FPT_LO, half = lo ? FPT_LO : FPT_HI;
    const bool high = j >= half;
    const int t = high ? j - half : j, n = high ? p.nhigh : p.nlow;
    if (lo ? t < n : t * FPT_LO < n)
      (lo ? tlo : thi)[j] = lo ? exp((double)t * (high ? dh : dl))
                               : (high ? sh : sl) * exp((high ? lfN : lf0) + (double)(FPT_LO * t + (high ? jh0 : -p.nlow)) *
                                                                                 (high ? dh : dl));
  }
  __syncthreads();
  const double* d1 = p.rden + (size_t)b1 * p.N;
  const double* d2 = p.rden + (size_t)(two ? b2 : b1) * p.N;
  for (int n = threadIdx.x; n < p.N; n += blockDim.x) {
    double v = 0.0;
    if (n >= lo0 && n < lo1) {
      v = thi[(n - lo0) / FPT_LO] * tlo[(n - lo0) % FPT_LO];
    } else if (n >= p.off && n < p.off + N0) {
      v = f[n - p.off];
    } else if (n >= hi0 && n < hi1) {
      v = thi[FPT_HI + (n - hi0) / FPT_LO] * tlo[FPT_LO + (n - hi0) % FPT_LO];
    }
    sbuf[n] = make_double2(v * __ldg(d1 + n), two ? v * __ldg(d2 + n) : 0.0);
  }
  __syncthreads();
  const int db = dft_n<-1>(sbuf, p, two);
  for (int k = threadIdx.x; k < H1; k += blockDim.x) {
    const double2 zk = sbuf[p.posN[k]];
    if (!two) {
      x1[k] = zk;
    } else {
      // the transforms of two real sequences from their packed transform
      const double2 zm = sbuf[p.posN[k == 0 ? 0 : p.N - k]];
      x1[k] = p2(make_double2(zk.x + zm.x, zk.y - zm.y), -1);
      x2[k] = p2(make_double2(zk.y + zm.y, zm.x - zk.x), -1 - db);
    }
  }
}

// The direct convolutions of the TATT terms: the spectrum's transform times
// the kernels', and back
__device__ __forceinline__ void direct_forward(const FPTDirect& d, const double* __restrict__ f, double2* __restrict__ z,
                                               double2* sbuf)
{
  for (int n = threadIdx.x; n < d.M; n += blockDim.x) sbuf[n] = make_double2(n < d.N0 ? f[n] : 0.0, 0.0);
  __syncthreads();
  fft64::dif<-1>(sbuf, d.dM, d.twM);
  for (int q = threadIdx.x; q < d.M; q += blockDim.x) z[q] = cmul(sbuf[q], __ldg(d.F + q));
}
__device__ __forceinline__ void direct_inverse(const FPTDirect& d, const double* __restrict__ f,
                                               const double2* __restrict__ z, int s, double* __restrict__ out,
                                               double2* sbuf)
{
  for (int q = threadIdx.x; q < d.M; q += blockDim.x) sbuf[q] = z[q];
  __syncthreads();
  fft64::dit<1>(sbuf, d.dM, d.twM);
  double* o1 = out + ((size_t)s * d.n_out + d.slot1) * d.N0;
  double* o2 = out + ((size_t)s * d.n_out + d.slot2) * d.N0;
  for (int i = threadIdx.x; i < d.N0; i += blockDim.x) {
    const double2 g = sbuf[d.N0 - 1 + i];
    o1[i] = d.c1[i] * f[i] * g.x;
    o2[i] = d.c2[i] * f[i] * g.y;
  }
}

// What bounds it: the conversions and four integer stages of the transform
// (58 of 90 us a CTA at Ntot = 12150), then 7 FP64 operations per point at
// 1/64 of the FP32 rate (with an FP64 transform and phase: about 270 us).
__global__ void __launch_bounds__(FPT_THREADS, 1)
    k_fpt_forward(FPTDev p, FPTDirect d, const double* __restrict__ fx)
{
  extern __shared__ double2 sbuf[];
  __shared__ unsigned red[64];
  if (d.on && blockIdx.x == 0) {
    direct_forward(d, fx + (size_t)blockIdx.y * d.N0, d.z + (size_t)blockIdx.y * d.M, sbuf);
    return;
  }
  const int2 pr = p.fpair[blockIdx.x - d.on];
  const int s = blockIdx.y;
  const int H1 = p.half + 1, T = p.Ntot;
  const bool two = pr.y >= 0;
  const int u2 = two ? pr.y : pr.x;
  const int bb1 = p.in_bias ? p.in_bias[pr.x] : 0, bb2 = p.in_bias ? p.in_bias[u2] : 0;
  const double2* xs1 = p.xin + ((size_t)s * p.n_bias + bb1) * H1;
  const double2* xs2 = p.xin + ((size_t)s * p.n_bias + bb2) * H1;
  const double2* g1 = p.G + (size_t)pr.x * H1;
  const double2* g2 = p.G + (size_t)u2 * H1;
  // a = x_1 at i, b = x_2 at Ntot - i until the balance is known (both
  // places this thread's; entry 0 of a Hermitian sequence is real)
  unsigned m1 = 0, m2 = 0;
  for (int i = threadIdx.x; i < H1; i += blockDim.x) {
    const double2 a = cmul(xs1[i], __ldg(g1 + i));
    const double2 b = two ? cmul(xs2[i], __ldg(g2 + i)) : make_double2(0.0, 0.0);
    m1 = max(m1, mag(a));
    m2 = max(m2, mag(b));
    if (i == 0) {
      sbuf[0] = make_double2(a.x, b.x);
    } else {
      sbuf[i] = a;
      sbuf[T - i] = b;
    }
  }
  const int e = two ? balance(m1, m2, red) : 0;
  for (int i = threadIdx.x; i <= T / 2; i += blockDim.x) {
    if (i == 0) {
      const double2 z = sbuf[0];
      sbuf[0] = make_double2(z.x, p2(z.y, e));
    } else if (i < H1) {
      const double2 a = sbuf[i], b = p2(sbuf[T - i], e);
      sbuf[i] = make_double2(a.x - b.y, a.y + b.x);
      sbuf[T - i] = make_double2(a.x + b.y, b.x - a.y);
    } else {
      sbuf[i] = make_double2(0.0, 0.0);
      sbuf[T - i] = make_double2(0.0, 0.0);
    }
  }
  __syncthreads();
  fx::dif<-1>(sbuf, p.dT, p.twT, false);
  double* R1 = p.R + ((size_t)s * p.n_in + pr.x) * T;
  double* R2 = p.R + ((size_t)s * p.n_in + u2) * T;
  for (int q = threadIdx.x; q < T; q += blockDim.x) {
    const double2 r = sbuf[q];
    R1[q] = r.x;
    if (two) R2[q] = p2(r.y, -e);
  }
}

// the two rows' lag-domain values at m and Ntot - m -> twice their
// Hermitian halves (the factor is taken out with the output's scale)
__device__ __forceinline__ void split2(double2 z, double2 zc, double2& r1, double2& r2)
{
  r1 = make_double2(z.x + zc.x, z.y - zc.y);
  r2 = make_double2(z.y + zc.y, zc.x - z.x);
}

// Two groups' folded U on k = 0..N/2 -> the transform of U_1 + i U_2: U_1(k)
// at k and U_2(k) at N - k in sbuf (both real and sharing place k at 0 and
// N/2, where conj(U(N - k)) = U(k)), the larger magnitudes in m1 and m2, U_j
// = 2^ej times the value wanted.  Writes the even samples of the size-2N
// c2r, scaled by the k powers.
__device__ __forceinline__ void c2r_finish(const FPTDev& p, double2* sbuf, int s, int g1, int g2,
                                           double* __restrict__ out, unsigned m1, unsigned m2, int e1, int e2,
                                           unsigned* red)
{
  const int N = p.N, hN = N / 2, N0 = p.N0;
  const bool two = g2 >= 0;
  const int cs = two ? balance(m1, m2, red) : 0;
  for (int k = threadIdx.x; k <= hN; k += blockDim.x) {
    if (k == 0 || k == hN) {
      const double2 u = sbuf[k];
      sbuf[k] = make_double2(u.x, p2(u.y, cs));
    } else {
      const double2 u1 = sbuf[k], u2 = p2(sbuf[N - k], cs);
      sbuf[k] = make_double2(u1.x - u2.y, u1.y + u2.x);
      sbuf[N - k] = make_double2(u1.x + u2.y, u2.x - u1.y);
    }
  }
  __syncthreads();
  dft_n<1>(sbuf, p, false);
  double* o1 = out + ((size_t)s * p.n_out + p.grp_out[g1]) * N0;
  double* o2 = out + ((size_t)s * p.n_out + p.grp_out[two ? g2 : g1]) * N0;
  const double* k1 = p.kpow + (size_t)p.grp_kp[g1] * N0;
  const double* k2 = p.kpow + (size_t)p.grp_kp[two ? g2 : g1] * N0;
  for (int i = threadIdx.x; i < N0; i += blockDim.x) {
    const double2 v = sbuf[p.posN[i + p.off]];
    o1[i] = p2(v.x, -e1) * k1[i];
    if (two) o2[i] = p2(v.y, -e2 - cs) * k2[i];
  }
}

// sum_t c_t R_a R_b at q of terms t0 <= t < t1, factored (fastpt.h)
__device__ __forceinline__ double row_sum(const FPTDev& p, const double* __restrict__ Rs, int t0, int t1, int q)
{
  const int T = p.Ntot;
  double s = 0.0, g = 0.0;
  for (int t = t0; t < t1; t++) {
    const int a = __ldg(p.t_ua + t);
    g = fma(__ldg(p.t_c + t), Rs[(size_t)__ldg(p.t_ub + t) * T + q], g);
    if (a >= 0) {
      s = fma(Rs[(size_t)a * T + q], g, s);
      g = 0.0;
    }
  }
  return s;
}

template <bool FUSED>
__global__ void __launch_bounds__(FPT_THREADS, 1)
    k_fpt_inverse(FPTDev p, FPTDirect d, const double* __restrict__ fx, double* __restrict__ out)
{
  extern __shared__ double2 sbuf[];
  __shared__ unsigned red[64];
  if (d.on && blockIdx.x == 0) {
    direct_inverse(d, fx + (size_t)blockIdx.y * d.N0, d.z + (size_t)blockIdx.y * d.M, blockIdx.y, out, sbuf);
    return;
  }
  const int2 pr = p.ipair[blockIdx.x - d.on];
  const int s = blockIdx.y;
  const int T = p.Ntot, N = p.N;
  const double* Rs = p.R + (size_t)s * p.n_in * T;
  const int a0 = p.row_start[pr.x], a1 = p.row_start[pr.x + 1];
  const bool two = pr.y >= 0;
  const int b0 = two ? p.row_start[pr.y] : 0, b1 = two ? p.row_start[pr.y + 1] : 0;
  for (int q = threadIdx.x; q < T; q += blockDim.x)
    sbuf[q] = make_double2(row_sum(p, Rs, a0, a1, q), row_sum(p, Rs, b0, b1, q));
  __syncthreads();
  const int db = fx::dit<1>(sbuf, p.dT, p.twT, two);
  const double2* Ha = p.H + (size_t)p.row_p[pr.x] * (N + 1);
  const double2* Hb = p.H + (size_t)p.row_p[two ? pr.y : pr.x] * (N + 1);
  if (!FUSED) {
    // store V_j(m) = 2 r_j(m) H_j(m), m = 0..N, for the group kernel
    double2* V1 = p.V + ((size_t)s * p.n_row + pr.x) * (N + 1);
    double2* V2 = p.V + ((size_t)s * p.n_row + (two ? pr.y : pr.x)) * (N + 1);
    for (int m = threadIdx.x; m <= N; m += blockDim.x) {
      double2 r1, r2;
      split2(sbuf[m], sbuf[m == 0 ? 0 : T - m], r1, r2);
      V1[m] = cmul(r1, __ldg(Ha + m));
      if (two) V2[m] = p2(cmul(r2, __ldg(Hb + m)), -db);
    }
    return;
  }
  // c2r fold, in place: thread k owns positions k and N - k and reads
  // N - k, Ntot - k and Ntot - N + k, none of which another thread writes:
  // U_j(k) = V_j(k) + conj(V_j(N - k)), V_j = r_j H_j
  const int hN = N / 2;
  unsigned m1 = 0, m2 = 0;
  for (int k = threadIdx.x; k <= hN; k += blockDim.x) {
    double2 r1a, r2a, r1b, r2b, u1, u2 = make_double2(0.0, 0.0);
    split2(sbuf[N - k], sbuf[T - N + k], r1b, r2b);
    if (k == 0) {
      const double2 z0 = sbuf[0];
      u1 = make_double2(2.0 * z0.x * __ldg(Ha).x + cmul(r1b, __ldg(Ha + N)).x, 0.0);
      if (two) u2 = make_double2(2.0 * z0.y * __ldg(Hb).x + cmul(r2b, __ldg(Hb + N)).x, 0.0);
    } else {
      split2(sbuf[k], sbuf[T - k], r1a, r2a);
      const double2 v1k = cmul(r1a, __ldg(Ha + k)), v1m = cmul(r1b, __ldg(Ha + N - k));
      u1 = make_double2(v1k.x + v1m.x, v1k.y - v1m.y);
      if (two) {
        const double2 v2k = cmul(r2a, __ldg(Hb + k)), v2m = cmul(r2b, __ldg(Hb + N - k));
        u2 = make_double2(v2k.x + v2m.x, v2k.y - v2m.y);
      }
    }
    m1 = max(m1, mag(u1));
    m2 = max(m2, mag(u2));
    if (k == 0 || k == hN) {
      sbuf[k] = make_double2(u1.x, u2.x);
    } else {
      sbuf[k] = u1;
      sbuf[N - k] = u2;
    }
  }
  c2r_finish(p, sbuf, s, pr.x, two ? pr.y : -1, out, m1, m2, 1, 1 + db, red);
}

__global__ void __launch_bounds__(FPT_THREADS, 1) k_fpt_c2r(FPTDev p, double* __restrict__ out)
{
  extern __shared__ double2 sbuf[];
  __shared__ unsigned red[64];
  const int2 gp = p.gpair[blockIdx.x];
  const int s = blockIdx.y;
  const int N = p.N, hN = N / 2;
  const bool two = gp.y >= 0;
  const int r10 = p.grp_start[gp.x], r11 = p.grp_start[gp.x + 1];
  const int r20 = two ? p.grp_start[gp.y] : 0, r21 = two ? p.grp_start[gp.y + 1] : 0;
  const double2* Vs = p.V + (size_t)s * p.n_row * (N + 1);
  // U_g(k) = sum over the group's rows of V_j(k) + conj(V_j(N - k))
  auto fold = [&](int j0, int j1, int k) {
    double2 u = make_double2(0.0, 0.0);
    for (int j = j0; j < j1; j++) {
      const double2 a = Vs[(size_t)j * (N + 1) + k], b = Vs[(size_t)j * (N + 1) + N - k];
      u.x += a.x + b.x;
      u.y += a.y - b.y;
    }
    return u;
  };
  unsigned m1 = 0, m2 = 0;
  for (int k = threadIdx.x; k <= hN; k += blockDim.x) {
    double2 u1 = fold(r10, r11, k), u2 = fold(r20, r21, k);
    if (k == 0) u1.y = u2.y = 0.0;
    m1 = max(m1, mag(u1));
    m2 = max(m2, mag(u2));
    if (k == 0 || k == hN) {
      sbuf[k] = make_double2(u1.x, u2.x);
    } else {
      sbuf[k] = u1;
      sbuf[N - k] = u2;
    }
  }
  c2r_finish(p, sbuf, s, gp.x, two ? gp.y : -1, out, m1, m2, 1, 1, red);
}

__global__ void __launch_bounds__(FPT_THREADS, 1) k_fpt_kernel_fft(FPTDirect d, double2* __restrict__ F)
{
  extern __shared__ double2 sbuf[];
  for (int n = threadIdx.x; n < d.M; n += blockDim.x) sbuf[n] = F[n];
  __syncthreads();
  fft64::dif<-1>(sbuf, d.dM, d.twM);
  for (int n = threadIdx.x; n < d.M; n += blockDim.x) F[n] = sbuf[n];
}

}  // namespace

int fpt_smem_setup()
{
  const int mx = 232448 - 1024;  // 227 KB per CTA less the static reduction scratch
  const void* ks[] = {(const void*)k_fpt_input, (const void*)k_fpt_forward, (const void*)k_fpt_inverse<true>,
                      (const void*)k_fpt_inverse<false>, (const void*)k_fpt_c2r, (const void*)k_fpt_kernel_fft};
  for (const void* k : ks)
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, mx) != cudaSuccess) return -1;
  return 0;
}

void launch_fastpt(const FPTDev& p, const FPTDirect& d, const double* fx, int S, double* out, cudaStream_t st)
{
  const size_t smN = fpt_smem_n(p), smM = d.on ? (size_t)d.M * sizeof(double2) : 0;
  const size_t smT = fpt_smem_t(p) > smM ? fpt_smem_t(p) : smM;
  k_fpt_input<<<dim3((p.n_bias + 1) / 2, S), FPT_THREADS, fpt_smem_in(p), st>>>(p, fx);
  k_fpt_forward<<<dim3(p.n_fp + d.on, S), FPT_THREADS, smT, st>>>(p, d, fx);
  if (p.multi) {
    k_fpt_inverse<false><<<dim3(p.n_ip + d.on, S), FPT_THREADS, smT, st>>>(p, d, fx, out);
    k_fpt_c2r<<<dim3(p.n_gp, S), FPT_THREADS, smN, st>>>(p, out);
  } else {
    k_fpt_inverse<true><<<dim3(p.n_ip + d.on, S), FPT_THREADS, smT, st>>>(p, d, fx, out);
  }
}

void launch_fastpt_transforms(const FPTDev& p, const double* fx, int S, cudaStream_t st)
{
  k_fpt_input<<<dim3((p.n_bias + 1) / 2, S), FPT_THREADS, fpt_smem_in(p), st>>>(p, fx);
  k_fpt_forward<<<dim3(p.n_fp, S), FPT_THREADS, fpt_smem_t(p), st>>>(p, FPTDirect{}, fx);
}

void launch_fastpt_kernel_fft(const FPTDirect& d, double2* dev_f, cudaStream_t st)
{
  k_fpt_kernel_fft<<<1, FPT_THREADS, (size_t)d.M * sizeof(double2), st>>>(d, dev_f);
}

}  // namespace cl2pt
