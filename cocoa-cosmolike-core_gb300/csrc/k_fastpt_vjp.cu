// k_fastpt_vjp.cu -- adjoint (vector-Jacobian product) of the batched
// FAST-PT convolutions of k_fastpt.cu: given the cotangent of a program's
// outputs, the gradient with respect to the input spectra.
//
// The reference differentiates nothing; these kernels transpose the
// forward of J_abl (cfastpt/cfastpt.c:875-1430) and J_abJ1J2Jk (91-768) as
// the GPU program regroups them (fastpt.h).  Every stage is linear in the
// padded spectrum except two: the term products R_a R_b (bilinear) and the
// power-law extrapolation at both ends (cfastpt.c:1066-1126).  Backwards,
// per spectrum:
//   k_fptv_grp   per group g: the output cotangent times the k power on
//                the even samples of the size-2N grid; its size-N transform
//                gives the adjoint of the folded c2r input (2 X(m) inside,
//                X(0) at m = 0 and N, real there; X is stored).
//   k_fptv_row   per row j: 2 X_g(j) conj(H_j) is the adjoint of the row's lag
//                sequence, whose size-Ntot transform (real part) is the
//                adjoint of the row spectrum s_j at each DIF position.
//   k_fptv_in    per input u: R_bar_u = sum over the terms that use u of
//                c_t s_bar_row(t) R_other (the forward's transforms, still
//                in the program's scratch); one inverse transform back to the padded Hermitian sequence,
//                folded onto the biased spectrum's half-spectrum
//                (x_bar[i] = x_bar_u[half + i] conj(G_u[i]) +
//                conj(x_bar_u[half - i] G_u[i])).
//   Pairs of groups, rows and inputs share one complex transform each (the
//   real-sequence, Hermitian-part and J-symmetry splits noted at each
//   kernel).
//   k_fptv_bias  per bias: the inputs' half-spectra summed, one inverse
//                size-N transform (real part), times x^-nu.
//   k_fptv_out   per spectrum: the biases summed onto the input grid plus
//                the derivatives of the two log extrapolations
//                (v = f0 (f1/f0)^d: dv/df0 = (1 - d) v / f0, dv/df1 = d v / f1).
//   TATT plans: the adjoint of the two fixed-kernel real convolutions, the
//   pointwise factor plus a correlation with each kernel, is three more CTAs
//   per spectrum of k_fptv_row, summed in k_fptv_out (one CTA and kernel of
//   its own ran its six transforms in a row).
#include <cuda_runtime.h>

#include "fpt_dev.cuh"

namespace cl2pt {

namespace {

// per group pair: the output cotangents times the k power on the even
// samples of the size-2N grid (real, two groups packed as re + i im), one
// size-N transform, split into each group's D(m), m = 0..N
__global__ void __launch_bounds__(FPT_THREADS, 1)
    k_fptv_grp(FPTDev p, FPTAdj a, const double* __restrict__ obar)
{
  extern __shared__ double2 sbuf[];
  const int2 gp = a.grp_pair[blockIdx.x];
  const int s = blockIdx.y;
  const bool two = gp.y >= 0;
  const int N = p.N, N0 = p.N0, off = p.off;
  const double* o1 = obar + ((size_t)s * p.n_out + p.grp_out[gp.x]) * N0;
  const double* o2 = obar + ((size_t)s * p.n_out + p.grp_out[two ? gp.y : gp.x]) * N0;
  const double* k1 = p.kpow + (size_t)p.grp_kp[gp.x] * N0;
  const double* k2 = p.kpow + (size_t)p.grp_kp[two ? gp.y : gp.x] * N0;
  for (int n = threadIdx.x; n < N; n += blockDim.x) {
    double v1 = 0.0, v2 = 0.0;
    if (n >= off && n < off + N0) {
      v1 = o1[n - off] * k1[n - off];
      if (two) v2 = o2[n - off] * k2[n - off];
    }
    sbuf[n] = make_double2(v1, v2);
  }
  __syncthreads();
  const int db = dft_n<-1>(sbuf, p, two);
  double2* D1 = a.Dg + ((size_t)s * p.n_grp + gp.x) * (N + 1);
  double2* D2 = a.Dg + ((size_t)s * p.n_grp + (two ? gp.y : gp.x)) * (N + 1);
  // the transforms of the two real sequences, m and its mirror at once
  for (int m = threadIdx.x; m <= N / 2; m += blockDim.x) {
    const double2 z = sbuf[p.posN[m]], zc = sbuf[p.posN[m == 0 ? 0 : N - m]];
    const double2 x1 = p2(make_double2(z.x + zc.x, z.y - zc.y), -1);
    const double2 x2 = p2(make_double2(z.y + zc.y, zc.x - z.x), -1 - db);
    D1[m] = make_double2(x1.x, m == 0 ? 0.0 : x1.y);
    D1[N - m] = make_double2(x1.x, m == 0 ? 0.0 : -x1.y);
    if (two) {
      D2[m] = make_double2(x2.x, m == 0 ? 0.0 : x2.y);
      D2[N - m] = make_double2(x2.x, m == 0 ? 0.0 : -x2.y);
    }
  }
}

// out_1 = c1 f g1, out_2 = c2 f g2 with g = (f conv k1, f conv k2) at
// N0 - 1 + i (direct_inverse): f_bar = [o1 c1 g1 + o2 c2 g2] + [h1 corr k1] +
// [h2 corr k2], h_r[N0 - 1 + i] = o_r c_r f; one CTA a bracket (part 0, 1, 2)
__device__ __forceinline__ void direct_part(const FPTDirect& d, const FPTAdj& a, int part, int s,
                                            const double* __restrict__ fx, const double* __restrict__ obar,
                                            double2* sbuf)
{
  const int N0 = d.N0, M = d.M;
  const double* f = fx + (size_t)s * N0;
  const double* o1 = obar + ((size_t)s * d.n_out + d.slot1) * N0;
  const double* o2 = obar + ((size_t)s * d.n_out + d.slot2) * N0;
  double* fb = a.dbar + ((size_t)s * 3 + part) * N0;
  const double* o = part == 2 ? o2 : o1;
  const double* c = part == 2 ? d.c2 : d.c1;
  const double2* K = part == 0 ? d.F : part == 1 ? a.F1 : a.F2;
  for (int n = threadIdx.x; n < M; n += blockDim.x) {
    const int i = n - (N0 - 1);
    sbuf[n] = make_double2(part == 0 ? (n < N0 ? f[n] : 0.0) : (i >= 0 && i < N0) ? o[i] * c[i] * f[i] : 0.0, 0.0);
  }
  __syncthreads();
  fft64::dif<-1>(sbuf, d.dM, d.twM);
  for (int q = threadIdx.x; q < M; q += blockDim.x)
    sbuf[q] = part == 0 ? cmul(sbuf[q], __ldg(K + q)) : cmulc(sbuf[q], __ldg(K + q));
  __syncthreads();
  fft64::dit<1>(sbuf, d.dM, d.twM);
  for (int i = threadIdx.x; i < N0; i += blockDim.x) {
    if (part == 0) {
      const double2 g = sbuf[N0 - 1 + i];
      fb[i] = o1[i] * d.c1[i] * g.x + o2[i] * d.c2[i] * g.y;
    } else {
      fb[i] = sbuf[i].x;
    }
  }
}

// per row pair: r_bar_j = 2 X_g(j) conj(H_j) on m = 0..N (X_g(j) conj(H_j) at
// 0 and N).  The row spectrum's adjoint is Re FFT(r_bar_j) = FFT(h_j) with h_j
// the Hermitian part (r_bar_j[m] + conj(r_bar_j[-m])) / 2, whose transform is
// real: two rows'
// h packed as h_1 + i h_2 share one size-Ntot transform, whose real and
// imaginary parts are the two answers (r_bar_j lives on m <= N and its
// mirror on m >= Ntot - N, which do not overlap as Ntot > 2N)
__global__ void __launch_bounds__(FPT_THREADS, 1)
    k_fptv_row(FPTDev p, FPTDirect d, FPTAdj a, const double* __restrict__ fx, const double* __restrict__ obar)
{
  extern __shared__ double2 sbuf[];
  const int nd = 3 * d.on;
  if ((int)blockIdx.x < nd) {
    direct_part(d, a, blockIdx.x, blockIdx.y, fx, obar, sbuf);
    return;
  }
  const int2 rp = a.row_pair[blockIdx.x - nd];
  const int s = blockIdx.y;
  const bool two = rp.y >= 0;
  const int N = p.N, T = p.Ntot;
  const double2* D1 = a.Dg + ((size_t)s * p.n_grp + a.row_grp[rp.x]) * (N + 1);
  const double2* D2 = a.Dg + ((size_t)s * p.n_grp + a.row_grp[two ? rp.y : rp.x]) * (N + 1);
  const double2* H1 = p.H + (size_t)p.row_p[rp.x] * (N + 1);
  const double2* H2 = p.H + (size_t)p.row_p[two ? rp.y : rp.x] * (N + 1);
  __shared__ unsigned red[64];
  // h_1 at m, h_2 at Ntot - m until the balance is known (as k_fpt_forward)
  unsigned m1 = 0, m2 = 0;
  for (int m = threadIdx.x; m <= N; m += blockDim.x) {
    const int e = m == N ? -1 : 0;
    const double2 h1 = p2(cmulc(D1[m], __ldg(H1 + m)), e);
    const double2 h2 = two ? p2(cmulc(D2[m], __ldg(H2 + m)), e) : make_double2(0.0, 0.0);
    m1 = max(m1, mag(h1));
    m2 = max(m2, mag(h2));
    if (m == 0) {
      sbuf[0] = make_double2(h1.x, h2.x);
    } else {
      sbuf[m] = h1;
      sbuf[T - m] = h2;
    }
  }
  const int e = two ? balance(m1, m2, red) : 0;
  for (int m = threadIdx.x; m <= T / 2; m += blockDim.x) {
    if (m == 0) {
      const double2 z = sbuf[0];
      sbuf[0] = make_double2(z.x, p2(z.y, e));
    } else if (m <= N) {
      const double2 h1 = sbuf[m], h2 = p2(sbuf[T - m], e);
      sbuf[m] = make_double2(h1.x - h2.y, h1.y + h2.x);
      sbuf[T - m] = make_double2(h1.x + h2.y, h2.x - h1.y);
    } else {
      sbuf[m] = make_double2(0.0, 0.0);
      sbuf[T - m] = make_double2(0.0, 0.0);
    }
  }
  __syncthreads();
  fx::dif<-1>(sbuf, p.dT, p.twT, false);
  double* sb1 = a.sbar + ((size_t)s * p.n_row + rp.x) * T;
  double* sb2 = a.sbar + ((size_t)s * p.n_row + (two ? rp.y : rp.x)) * T;
  for (int q = threadIdx.x; q < T; q += blockDim.x) {
    const double2 z = sbuf[q];
    sb1[q] = z.x;
    if (two) sb2[q] = p2(z.y, -e);
  }
}

// per input pair: R_bar_u = sum over the terms that use u of c_t
// s_bar_row(t) R_other (factored, fastpt.h), the two inputs packed as
// re + i im, one inverse size-Ntot transform.  Each input's adjoint sequence
// y_u is Hermitian about 0 (as the forward's padded sequences are), so
// y_1 = (y + J y) / 2 and y_2 = (y - J y) / 2i with J y[n] = conj(y[-n]), and
// the fold onto the half-spectrum is x_bar[i] = (i ? 2 : 1) y_u[i] conj(G_u[i]).
__global__ void __launch_bounds__(FPT_THREADS, 1) k_fptv_in(FPTDev p, FPTAdj a)
{
  extern __shared__ double2 sbuf[];
  const int2 ip = a.in_pair[blockIdx.x];
  const int s = blockIdx.y;
  const bool two = ip.y >= 0;
  const int T = p.Ntot, h = p.half;
  const double* Rs = p.R + (size_t)s * p.n_in * T;
  const double* Sb = a.sbar + (size_t)s * p.n_row * T;
  auto sum = [&](int u, int q) {
    const bool br = __ldg(a.in_byrow + u) != 0;
    const double* K = br ? Sb : Rs;
    const double* V = br ? Rs : Sb;
    double c = 0.0, g = 0.0;
    const int e1 = __ldg(a.in_start + u + 1);
    for (int e = __ldg(a.in_start + u); e < e1; e++) {
      const int k = __ldg(a.in_key + e);
      g = fma(__ldg(a.in_c + e), V[(size_t)__ldg(a.in_val + e) * T + q], g);
      if (k >= 0) {
        c = fma(K[(size_t)k * T + q], g, c);
        g = 0.0;
      }
    }
    return c;
  };
  for (int q = threadIdx.x; q < T; q += blockDim.x) sbuf[q] = make_double2(sum(ip.x, q), two ? sum(ip.y, q) : 0.0);
  __syncthreads();
  const int db = fx::dit<1>(sbuf, p.dT, p.twT, two);
  const double2* G1 = p.G + (size_t)ip.x * (h + 1);
  const double2* G2 = p.G + (size_t)(two ? ip.y : ip.x) * (h + 1);
  double2* xb1 = a.xbar + ((size_t)s * p.n_in + ip.x) * (h + 1);
  double2* xb2 = a.xbar + ((size_t)s * p.n_in + (two ? ip.y : ip.x)) * (h + 1);
  for (int i = threadIdx.x; i <= h; i += blockDim.x) {
    const double2 y = sbuf[i], yc = sbuf[i == 0 ? 0 : T - i];
    const int e = i ? 0 : -1;
    xb1[i] = p2(cmulc(make_double2(y.x + yc.x, y.y - yc.y), __ldg(G1 + i)), e);
    if (two) xb2[i] = p2(cmulc(make_double2(y.y + yc.y, yc.x - y.x), __ldg(G2 + i)), e - db);
  }
}

__global__ void __launch_bounds__(FPT_THREADS, 1) k_fptv_bias(FPTDev p, FPTAdj a)
{
  extern __shared__ double2 sbuf[];
  const int b = blockIdx.x, s = blockIdx.y;
  const int N = p.N, h = p.half;
  const int e0 = a.bias_start[b], e1 = a.bias_start[b + 1];
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    double2 v = make_double2(0.0, 0.0);
    if (i <= h)
      for (int e = e0; e < e1; e++) {
        const double2 x = a.xbar[((size_t)s * p.n_in + a.bias_in[e]) * (h + 1) + i];
        v = make_double2(v.x + x.x, v.y + x.y);
      }
    sbuf[i] = v;
  }
  __syncthreads();
  dft_n<1>(sbuf, p, false);
  const double* rden = p.rden + (size_t)b * N;
  double* eb = a.ebar + ((size_t)s * p.n_bias + b) * N;
  for (int n = threadIdx.x; n < N; n += blockDim.x) eb[n] = sbuf[p.posN[n]].x * __ldg(rden + n);
}

__device__ __forceinline__ double block_sum(double v, double* red)
{
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  for (int i = 0; i < (int)(blockDim.x >> 5); i++) t += red[i];
  return t;
}

__global__ void __launch_bounds__(FPT_THREADS, 1)
    k_fptv_out(FPTDev p, FPTDirect d, FPTAdj a, const double* __restrict__ fx, double* __restrict__ fxbar)
{
  __shared__ double red[32];
  const int s = blockIdx.x;
  const int N = p.N, N0 = p.N0, off = p.off;
  const double* f = fx + (size_t)s * N0;
  double* fb = fxbar + (size_t)s * N0;
  const double* eb = a.ebar + (size_t)s * p.n_bias * N;
  for (int i = threadIdx.x; i < N0; i += blockDim.x) {
    double e = 0.0;
    for (int b = 0; b < p.n_bias; b++) e += eb[(size_t)b * N + off + i];
    fb[i] = e;
  }
  // the extrapolations (as k_fpt_input; a spectrum that failed its checks
  // has NaN outputs and its gradient is left as the interior part)
  const int lo0 = p.npad, lo1 = p.npad + p.nlow;
  const int hi0 = N - p.npad - p.nhigh, hi1 = N - p.npad;
  const int jh0 = hi0 - off - N0;
  double g0 = 0.0, g1 = 0.0, gN1 = 0.0, gN2 = 0.0;
  bool okl = false, okh = false;
  double sl = 1, lf0 = 0, dl = 0, sh = 1, lfN = 0, dh = 0;
  if (p.nlow) {
    const double f0 = f[0], f1 = f[1];
    okl = !(f0 == 0.0 || f1 / f0 <= 0.0);
    if (okl) {
      sl = f0 > 0 ? 1.0 : -1.0;
      lf0 = log(f0 * sl);
      dl = log(f1 / f0);
    }
  }
  if (p.nhigh) {
    const double f1 = f[N0 - 1], f2 = f[N0 - 2];
    okh = !(f1 == 0.0 || f1 / f2 <= 0.0);
    if (okh) {
      sh = f1 > 0 ? 1.0 : -1.0;
      lfN = log(f1 * sh);
      dh = log(f1 / f2);
    }
  }
  for (int n = threadIdx.x; n < N; n += blockDim.x) {
    double e = 0.0;
    if ((okl && n >= lo0 && n < lo1) || (okh && n >= hi0 && n < hi1))
      for (int b = 0; b < p.n_bias; b++) e += eb[(size_t)b * N + n];
    if (e == 0.0) continue;
    if (n < lo1) {
      const double x = (double)(n - lo1), v = sl * exp(lf0 + x * dl);
      g0 += e * (1.0 - x) * v / f[0];
      g1 += e * x * v / f[1];
    } else {
      const double x = (double)(n - hi0 + jh0), v = sh * exp(lfN + x * dh);
      gN1 += e * (1.0 + x) * v / f[N0 - 1];
      gN2 -= e * x * v / f[N0 - 2];
    }
  }
  g0 = block_sum(g0, red);
  g1 = block_sum(g1, red);
  gN1 = block_sum(gN1, red);
  gN2 = block_sum(gN2, red);
  __syncthreads();  // every thread's interior write is done
  if (threadIdx.x == 0) {
    fb[0] += g0;
    fb[1] += g1;
    fb[N0 - 1] += gN1;
    fb[N0 - 2] += gN2;
  }
  if (!d.on) return;
  __syncthreads();
  const double* db = a.dbar + (size_t)s * 3 * N0;
  for (int i = threadIdx.x; i < N0; i += blockDim.x) fb[i] = ((fb[i] + db[i]) + db[N0 + i]) + db[2 * N0 + i];
}

}  // namespace

int fptv_smem_setup()
{
  const int mx = 232448 - 1024;
  const void* ks[] = {(const void*)k_fptv_grp, (const void*)k_fptv_row, (const void*)k_fptv_in,
                      (const void*)k_fptv_bias};
  for (const void* k : ks)
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, mx) != cudaSuccess) return -1;
  return 0;
}

void launch_fastpt_vjp(const FPTDev& p, const FPTDirect& d, const FPTAdj& a, const double* fx, int S,
                       const double* obar, double* fxbar, cudaStream_t st)
{
  const size_t smN = fpt_smem_n(p), smT = fpt_smem_t(p), smM = d.on ? (size_t)d.M * sizeof(double2) : 0;
  k_fptv_grp<<<dim3(a.n_gpa, S), FPT_THREADS, smN, st>>>(p, a, obar);
  k_fptv_row<<<dim3(a.n_rpa + 3 * d.on, S), FPT_THREADS, smT > smM ? smT : smM, st>>>(p, d, a, fx, obar);
  k_fptv_in<<<dim3(a.n_ipa, S), FPT_THREADS, smT, st>>>(p, a);
  k_fptv_bias<<<dim3(p.n_bias, S), FPT_THREADS, smN, st>>>(p, a);
  k_fptv_out<<<S, FPT_THREADS, 0, st>>>(p, d, a, fx, fxbar);
}

}  // namespace cl2pt
