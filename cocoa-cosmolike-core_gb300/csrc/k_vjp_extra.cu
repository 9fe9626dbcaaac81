// k_vjp_extra.cu -- adjoint of the TATT intrinsic-alignment and one-loop
// galaxy-bias terms of the Limber integrands (the forward is k_extra.cu).
//
// The extra terms are linear in the FAST-PT table rows (functions of
// k = (l+1/2)/chi, read linearly in ln k, 0 off the grid) and polynomial in
// the node weights, so for given C_l adjoints each node needs the sums over
// l of (C_bar x row value); from those the node-weight adjoints follow in
// closed form:
//   k_vjpx_ss  C_ss EE/BB: per pair the five coefficient adjoints (A, B, C,
//              Dm, E of k_extra_ss), then u_bar (added to the NLA w_bar),
//              b_bar (W_S C1 b_TA D^2) and c_bar (W_S C2 D^2) per source bin;
//   k_vjpx_gs  C_gs: b_bar, c_bar, W_K_bar per source bin, the lens-weight
//              adjoints (added to L_bar of b1 and M_bar of bmag) and the b2,
//              bs2 gradients;
//   k_vjpx_gg  C_gg one-loop bias (node l, and integer l below LMAX_NOLIMBER
//              for the non-Limber hand-over): the b1, b2, bs2 gradients.
// CTAs over (point[, lens bin], part of the multipoles), one thread per node;
// per-(l, node) arithmetic in the plan's loop precision, chunks added up in FP64
// by atomics (their order, and with it the last FP64 digits, varies between
// runs); the gg cells, weights, rows and sums always FP64, as in the forward.
// The one-loop gate (any b2 != 0) is held fixed; the dependence of the FAST-PT
// rows on p_lin(k, z = 0) is k_vjp_fpt.cu's.
#include <algorithm>

#include "common.cuh"
#include "fpt_cell.cuh"
#include "kernels.cuh"

namespace cl2pt {

namespace {

constexpr int XLC = 32;  // multipoles per chunk

__device__ __forceinline__ double node_F(const Params& P, int pt, int idx, double* fK, double* D, double* a,
                                         double* H)
{
  const double* node = P.node + (size_t)pt * NF_COUNT * P.node_stride;
  *fK = node[(size_t)NF_FK * P.node_stride + idx];
  *D = node[(size_t)NF_D * P.node_stride + idx];
  *a = node[(size_t)NF_A * P.node_stride + idx];
  *H = node[(size_t)NF_H * P.node_stride + idx];
  return node[(size_t)NF_WT * P.node_stride + idx] * node[(size_t)NF_DCHIDA * P.node_stride + idx] / (*fK * *fK);
}

__device__ __forceinline__ double bsum(double v, double* red)
{
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < (int)((blockDim.x + 31) >> 5); i++) s += red[i];
  return s;
}

constexpr double LN10 = 2.302585092994045684;

// threads of a sum CTA: G groups of nn threads (a multiple of 32), each
// thread one node; the groups share the chunk's row values and take turns
// over its multipoles and tiles of four pairs
constexpr int XTP = 4;
static int x_threads(int nn) { return ((nn + 31) / 32) * 32; }
static int x_groups(int nn) { return x_threads(nn) >= 256 ? 1 : 256 / x_threads(nn); }

// ------------------------------------------------------------------ ss
// Coefficient sums cx [5][np][nn] over the multipoles, in chunks of XLC: FP32
// (the plan's loop precision) within a chunk, FP64 atomics across.  The
// chunks are spread over CTAs, so a few points fill the chip.  Bound by issue
// (8 row values and 8 broadcast cotangents per 28 multiply-adds).
// real_3x2pt_tatt, 16 points: one 64-thread CTA per point over all chunks
// took 5.3 ms, this takes under 0.2 ms.
template <typename T>
__global__ void __launch_bounds__(512) k_vjpx_ss(Params P, VJPParams V, int nnr, int G)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int pt = blockIdx.x, grp = threadIdx.x / nnr, p = threadIdx.x - grp * nnr;
  const int n = P.fpt_n, nn = P.n_ss, np = P.pss, K = P.nnode_ss, Kx = 2 * K;
  const int np4 = (np + XTP - 1) / XTP * XTP;
  T* cbE = (T*)smem_raw;                       // [XLC][np4] pref C_bar EE
  T* cbB = cbE + (size_t)np4 * XLC;            // [XLC][np4] pref C_bar BB
  T* rv = cbB + (size_t)np4 * XLC;             // [8][XLC][nn] row values of the chunk
  __shared__ typename FptPart<T>::type la[XLC];
  const double* src = P.fpt_ia + (size_t)pt * 8 * n;
  const bool act = p < nn;
  typename FptPart<T>::type bp = FptPart<T>::of_p(P, 0.0);
  if (act) bp = FptPart<T>::of_p(P, log(P.node[((size_t)pt * NF_COUNT + NF_FK) * P.node_stride + p]));
  const double* cb = V.cbar_ss + (size_t)pt * np * Kx;
  double* cx = V.cx_ss + (size_t)pt * 5 * np * nn;
  for (int L0 = blockIdx.y * XLC; L0 < K; L0 += gridDim.y * XLC) {
    const int nL = min(XLC, K - L0);
    __syncthreads();
    if (threadIdx.x < nL) la[threadIdx.x] = FptPart<T>::of_l(P, V.lfac_ss[2 * (L0 + threadIdx.x)] * LN10);
    for (int i = threadIdx.x; i < np4 * XLC; i += blockDim.x) {
      const int pr = i / XLC, l = i - pr * XLC;
      double e = 0, b = 0;
      if (l < nL && pr < np) {
        const double pref = V.lfac_ss[2 * (L0 + l) + 1];
        e = pref * cb[(size_t)pr * Kx + L0 + l];
        b = pref * cb[(size_t)pr * Kx + K + L0 + l];
      }
      cbE[l * np4 + pr] = round_to<T>(e);
      cbB[l * np4 + pr] = round_to<T>(b);
    }
    __syncthreads();
    if (act) {
      for (int l = grp; l < nL; l += G) {
        const FptCell<T> c = fpt_cell(P, la[l], bp);
        const int i1 = min(c.i + 1, n - 1);
        for (int r = 0; r < 8; r++) {
          const double* row = src + (size_t)r * n;
          T v = (T)0;
          if (c.in) {
            const T v0 = round_to<T>(row[c.i]);
            v = c.w * (round_to<T>(row[i1]) - v0) + v0;
          }
          rv[((size_t)r * XLC + l) * nn + p] = v;
        }
      }
    }
    __syncthreads();
    if (!act) continue;
    for (int pr0 = grp * XTP; pr0 < np; pr0 += G * XTP) {
      T a[XTP][5];
#pragma unroll
      for (int k = 0; k < XTP; k++)
#pragma unroll
        for (int m = 0; m < 5; m++) a[k][m] = (T)0;
      for (int l = 0; l < nL; l++) {
        const T* v = rv + (size_t)l * nn + p;
        const size_t st = (size_t)XLC * nn;
        T x[8];
#pragma unroll
        for (int r = 0; r < 8; r++) x[r] = v[r * st];
#pragma unroll
        for (int k = 0; k < XTP; k++) {
          const T e = cbE[l * np4 + pr0 + k], b = cbB[l * np4 + pr0 + k];
          a[k][0] += e * x[1];
          a[k][1] += e * x[2] + b * x[6];
          a[k][2] += e * x[3];
          a[k][3] += e * x[4] + b * x[7];
          a[k][4] += e * x[0] + b * x[5];
        }
      }
#pragma unroll
      for (int k = 0; k < XTP; k++) {
        if (pr0 + k >= np) break;
        const size_t o = (size_t)(pr0 + k) * nn + p, st = (size_t)np * nn;
#pragma unroll
        for (int m = 0; m < 5; m++) atomicAdd(&cx[o + m * st], (double)a[k][m]);
      }
    }
  }
}

// coefficient adjoints -> u_bar, b_bar, c_bar (k_extra_ss coefficients): one
// thread per (source bin, node) gathers the pairs of its bin
__global__ void __launch_bounds__(128) k_vjpx_ss_w(Params P, VJPParams V)
{
  const int pt = blockIdx.y, nn = P.n_ss, np = P.pss;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= P.ns * nn) return;
  const int s = t / nn, p = t - s * nn;
  double fK, D, a, H;
  const double F = node_F(P, pt, p, &fK, &D, &a, &H);
  const double D2 = D * D;
  const double* cx = V.cx_ss + (size_t)pt * 5 * np * nn;
  const double* u = P.wss + (size_t)pt * P.ns * nn;
  const double* bw = P.wss_b + (size_t)pt * P.ns * nn;
  const double* cw = P.wss_2 + (size_t)pt * P.ns * nn;
  double ub = 0, bb = 0, cb = 0;
  for (int pr = 0; pr < np; pr++) {
    const int i = P.z1[pr], j = P.z2[pr];
    if (i != s && j != s) continue;
    const size_t o = (size_t)pr * nn + p, st = (size_t)np * nn;
    const double A = cx[o] * F, B = cx[o + st] * F, C = cx[o + 2 * st] * F, Dm = cx[o + 3 * st] * F,
                 E = cx[o + 4 * st] * F;
    for (int h = 0; h < 2; h++) {
      if ((h ? j : i) != s) continue;
      const int o2 = h ? i : j;  // the pair's other bin
      const double uj = u[o2 * nn + p], bj = bw[o2 * nn + p], cj = cw[o2 * nn + p];
      ub += -A * bj * D2 + 5. * C * cj * D2;
      bb += -A * uj * D2 + B * bj - 5. * Dm * cj;
      cb += 5. * C * uj * D2 - 5. * Dm * bj + 25. * E * cj;
    }
  }
  const size_t o = ((size_t)pt * P.ns + s) * nn + p;
  V.wbar_ss[o] += ub;
  V.wbar_ssb[o] += bb;
  V.wbar_ss2[o] += cb;
}

// ------------------------------------------------------------------ gs
// Row sums cx_gs [nl][ns][7][nn] over the multipoles, as k_vjpx_ss: x0-x3, x6
// the l-free sums of taE, mix, d1d2, d1s2, d1p3, x4 and x5 those of taE and
// mix with l(l+1)/(l+1/2)^2.
constexpr int XGS = 7;
template <typename T>
__global__ void __launch_bounds__(512) k_vjpx_gs(Params P, VJPParams V, int nnr, int G)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int kk[CL2PT_MAXB], ss_[CL2PT_MAXB];
  __shared__ int npq;
  const int pt = blockIdx.x, q = blockIdx.y, grp = threadIdx.x / nnr, p = threadIdx.x - grp * nnr;
  const int n = P.fpt_n, nn = P.n_ss, K = P.nnode_g;
  if (threadIdx.x == 0) {
    int m = 0;
    for (int k = 0; k < P.pgs; k++)
      if (P.zl[k] == q) {
        kk[m] = k;
        ss_[m] = P.zs[k];
        m++;
      }
    npq = m;
  }
  __syncthreads();
  const int np = npq;
  if (np == 0) return;
  T* cb0 = (T*)smem_raw;                   // [np][XLC] pref2 C_bar
  T* cb1 = cb0 + (size_t)np * XLC;         // [np][XLC] pref2 pref C_bar
  T* rv = cb1 + (size_t)np * XLC;          // [5][XLC][nn] taE, mix, d1d2, d1s2, d1p3
  __shared__ typename FptPart<T>::type la[XLC];
  const double* src[5] = {P.tatt ? P.fpt_ia + ((size_t)pt * 8 + 1) * n : nullptr,
                          P.tatt ? P.fpt_ia + ((size_t)pt * 8 + 3) * n : nullptr,
                          P.one_loop ? P.fpt_b + ((size_t)pt * 5 + 0) * n : nullptr,
                          P.one_loop ? P.fpt_b + ((size_t)pt * 5 + 2) * n : nullptr,
                          P.one_loop ? P.fpt_d1p3 : nullptr};
  const bool act = p < nn;
  const int off = P.n_ss + q * P.n_ss;
  typename FptPart<T>::type bp = FptPart<T>::of_p(P, 0.0);
  if (act) bp = FptPart<T>::of_p(P, log(P.node[((size_t)pt * NF_COUNT + NF_FK) * P.node_stride + off + p]));
  const size_t b0 = (size_t)pt * P.nl + q;
  for (int L0 = blockIdx.z * XLC; L0 < K; L0 += gridDim.z * XLC) {
    const int nL = min(XLC, K - L0);
    __syncthreads();
    if (threadIdx.x < nL) la[threadIdx.x] = FptPart<T>::of_l(P, V.lfac_g[6 * (L0 + threadIdx.x)] * LN10);
    for (int i = threadIdx.x; i < np * XLC; i += blockDim.x) {
      const int m = i / XLC, l = i - m * XLC;
      double c0 = 0, c1 = 0;
      if (l < nL) {
        const double* fac = V.lfac_g + 6 * (L0 + l);
        const double cv = V.cbar_gs[((size_t)pt * P.pgs + kk[m]) * K + L0 + l] * fac[1];
        c0 = cv;
        c1 = cv * fac[2];
      }
      cb0[i] = round_to<T>(c0);
      cb1[i] = round_to<T>(c1);
    }
    __syncthreads();
    if (act) {
      for (int l = grp; l < nL; l += G) {
        const FptCell<T> c = fpt_cell(P, la[l], bp);
        const int i1 = min(c.i + 1, n - 1);
#pragma unroll
        for (int r = 0; r < 5; r++) {
          T v = (T)0;
          if (c.in && src[r]) {
            const T v0 = round_to<T>(src[r][c.i]);
            v = c.w * (round_to<T>(src[r][i1]) - v0) + v0;
          }
          rv[((size_t)r * XLC + l) * nn + p] = v;
        }
      }
    }
    __syncthreads();
    if (!act) continue;
    for (int m = grp; m < np; m += G) {
      T x0 = 0, x1 = 0, x2 = 0, x3 = 0, x4 = 0, x5 = 0, x6 = 0;
      for (int l = 0; l < nL; l++) {
        const T c0 = cb0[m * XLC + l], c1 = cb1[m * XLC + l];
        const T* v = rv + (size_t)l * nn + p;
        const size_t st = (size_t)XLC * nn;
        const T taE = v[0], mix = v[st], d1d2 = v[2 * st], d1s2 = v[3 * st], d1p3 = v[4 * st];
        x0 += c0 * taE;
        x1 += c0 * mix;
        x2 += c0 * d1d2;
        x3 += c0 * d1s2;
        x6 += c0 * d1p3;
        x4 += c1 * taE;
        x5 += c1 * mix;
      }
      double* cx = V.cx_gs + ((b0 * P.ns + ss_[m]) * XGS) * nn + p;
      const T x[XGS] = {x0, x1, x2, x3, x4, x5, x6};
#pragma unroll
      for (int r = 0; r < XGS; r++) atomicAdd(&cx[(size_t)r * nn], (double)x[r]);
    }
  }
}

// the row sums -> b_bar, c_bar, W_K_bar per source bin, the lens weights'
// adjoints and the b2, bs2, b3 gradients: one thread per node
__global__ void k_vjpx_gs_w(Params P, VJPParams V)
{
  __shared__ double red[32];
  const int pt = blockIdx.x, q = blockIdx.y, p = threadIdx.x, nn = P.n_ss;
  const bool act = p < nn;
  const int off = P.n_ss + q * P.n_ss;
  const size_t b0 = (size_t)pt * P.nl + q;
  double sb2 = 0, sbs2 = 0, sb3 = 0;
  if (act) {
    double fK, D, a, H;
    const double F = node_F(P, pt, off + p, &fK, &D, &a, &H), D2 = D * D;
    const double Lg = P.wgs_l[b0 * nn + p], Mg = P.wgs_m[b0 * nn + p];
    double g2 = 0, gs2 = 0, g3 = 0;
    if (P.one_loop) {
      g2 = P.wgs_1l[(b0 * 3 + 0) * nn + p];
      gs2 = P.wgs_1l[(b0 * 3 + 1) * nn + p];
      g3 = P.wgs_1l[(b0 * 3 + 2) * nn + p];
    }
    double Lbar = 0, Mbar = 0, g2bar = 0, gs2bar = 0, g3bar = 0;
    for (int k = 0; k < P.pgs; k++) {
      if (P.zl[k] != q) continue;
      const size_t o = (b0 * P.ns + P.zs[k]) * nn + p;
      const double* cx = V.cx_gs + ((b0 * P.ns + P.zs[k]) * XGS) * nn + p;
      double X[XGS];
#pragma unroll
      for (int r = 0; r < XGS; r++) X[r] = cx[(size_t)r * nn];
      if (P.tatt) {
        const double bw = P.wgs_b[o], cw = P.wgs_2[o];
        V.wbar_gsb[o] += -D2 * F * (Lg * X[0] + Mg * X[4]);
        V.wbar_gs2[o] += 5. * D2 * F * (Lg * X[1] + Mg * X[5]);
        Lbar += F * D2 * (-bw * X[0] + 5. * cw * X[1]);
        Mbar += F * D2 * (-bw * X[4] + 5. * cw * X[5]);
      }
      if (P.one_loop) {
        const double WK = P.wgs_k[o];
        V.wbar_gsk[o] += F * (g2 * X[2] + gs2 * X[3] + g3 * X[6]);
        g2bar += WK * F * X[2];
        gs2bar += WK * F * X[3];
        g3bar += WK * F * X[6];
      }
    }
    V.lbar_gs[(b0 * 2 + 0) * nn + p] += Lbar;
    V.lbar_gs[(b0 * 2 + 1) * nn + p] += Mbar;
    // g2 = 0.5 D^4 W_gal b2, gs2 = 0.5 D^4 W_gal bs2 (one-loop gate held)
    if (P.one_loop && V.one_loop_on[pt]) {
      const cl2pt_nuisance& nu = P.nu[pt];
      const double WGAL = nz_lens_d(P, 1. / a - 1., q, nu.lens_dz[q], nu.lens_stretch[q]) * H;
      sb2 = g2bar * 0.5 * D2 * D2 * WGAL;
      sbs2 = gs2bar * 0.5 * D2 * D2 * WGAL;
      sb3 = g3bar * 0.5 * D2 * D2 * WGAL;
    }
  }
  if (P.one_loop) {
    const double t2 = bsum(sb2, red);
    const double ts = bsum(sbs2, red);
    const double t3 = bsum(sb3, red);
    if (threadIdx.x == 0) {
      atomicAdd(&V.nu_bar[pt].gb[1][q], t2);
      atomicAdd(&V.nu_bar[pt].gb[2][q], ts);
      if (P.fpt_d1p3) atomicAdd(&V.nu_bar[pt].gb[3][q], t3);
    }
  }
}

// ------------------------------------------------------------------ gg
// The sums X_m(p) = sum_l C_bar row_m(k_lp) over the multipoles of a CTA's
// part, FP64 rows and sums.  The multipoles ascend, so a node's samples come
// in runs of one grid cell: a run's cotangents are summed with the weights of
// the cell's two ends, and the six rows read once per run.  Cell and weight in
// FP64 in both plans, as the rows and sums (the mixed plan's two-float cell
// takes 0.18 ms less at 16 points of real_3x2pt_tatt, and leaves the weight 24
// bits).  Bound by the FP64 pipe.
constexpr int XGG_L = 128, XGG_P = 128;  // multipoles and nodes per CTA
__global__ void __launch_bounds__(XGG_P) k_vjpx_gg(Params P, VJPParams V, int ntile)
{
  __shared__ double red[32];
  __shared__ double la[XGG_L], lcv[XGG_L], lcut[XGG_L];
  const int pt = blockIdx.x, q = blockIdx.y;
  const int lt = blockIdx.z / ntile, p = (blockIdx.z - lt * ntile) * blockDim.x + threadIdx.x;
  if (!V.one_loop_on[pt]) return;  // no gradient flows to the bias terms
  const int n = P.fpt_n, nn = P.n_gg, K = P.nnode_g, LNL = P.lmax_nolimber;
  const size_t b0 = (size_t)pt * P.nl + q;
  const int nL = K + (V.ggl_bar ? LNL : 0);
  const int L0 = lt * XGG_L, nLt = min(XGG_L, nL - L0);
  for (int i = threadIdx.x; i < nLt; i += blockDim.x) {
    const int L = L0 + i;
    const double* fac = L < K ? V.lfac_g + 6 * L : V.lfac_gi + 6 * (L - K);
    la[i] = fac[0] * LN10;
    lcut[i] = fac[5];
    lcv[i] = L < K ? V.cbar_gg[b0 * K + L] : V.ggl_bar[(b0 * LNL + (L - K)) * 2];
  }
  __syncthreads();
  const double* src = P.fpt_b + (size_t)pt * 5 * n;
  double g[4] = {0, 0, 0, 0};
  if (p < nn) {
    const int off = P.n_ss + P.nl * P.n_ss + q * nn;
    double fK, D, a, H;
    const double F = node_F(P, pt, off + p, &fK, &D, &a, &H);
    const double lnf = log(fK);
    const double chi_amin = P.chi_amin[pt];
    double X[6] = {0, 0, 0, 0, 0, 0};
    int run = -1;
    double s0 = 0.0, s1 = 0.0;  // a run's cotangent on the cell's two ends
    auto flush = [&]() {
      if (run < 0) return;
      const int i1 = min(run + 1, n - 1);
#pragma unroll
      for (int m = 0; m < 5; m++) X[m] += s0 * src[(size_t)m * n + run] + s1 * src[(size_t)m * n + i1];
      if (P.fpt_d1p3) X[5] += s0 * P.fpt_d1p3[run] + s1 * P.fpt_d1p3[i1];
    };
    for (int i = 0; i < nLt; i++) {
      const double cv = lcv[i];
      if (cv == 0.0 || fK * lcut[i] > chi_amin) continue;
      const FptCell<double> c = fpt_cell(P, la[i], lnf);
      if (!c.in) continue;
      if (c.i != run) {
        flush();
        run = c.i;
        s0 = s1 = 0.0;
      }
      s1 = fma(cv, c.w, s1);
      s0 = fma(-cv, c.w, s0 + cv);
    }
    flush();
    // wgg_1l = W_gal^2 D^4 (b1 b2, b2^2/4, b1 bs2, b2 bs2/2, bs2^2/4, b1 b3)
    const cl2pt_nuisance& nu = P.nu[pt];
    const double WGAL = nz_lens_d(P, 1. / a - 1., q, nu.lens_dz[q], nu.lens_stretch[q]) * H;
    const double c = WGAL * WGAL * D * D * D * D * F;
    const double b1 = nu.gb[0][q], b2 = nu.gb[1][q], bs2 = nu.gb[2][q];
    const double b3 = P.fpt_d1p3 ? nu.gb[3][q] : 0.0;
    g[0] = c * (X[0] * b2 + X[2] * bs2 + X[5] * b3);
    g[1] = c * (X[0] * b1 + X[1] * 0.5 * b2 + X[3] * 0.5 * bs2);
    g[2] = c * (X[2] * b1 + X[3] * 0.5 * b2 + X[4] * 0.5 * bs2);
    g[3] = P.fpt_d1p3 ? c * X[5] * b1 : 0.0;
  }
  for (int k = 0; k < 4; k++) {
    const double t = bsum(g[k], red);
    if (threadIdx.x == 0) atomicAdd(&V.nu_bar[pt].gb[k][q], t);
  }
}

// per-point one-loop gate: the reference adds the one-loop terms when any
// lens bin has b2 != 0
__global__ void k_vjpx_gate(Params P, VJPParams V)
{
  const int pt = blockIdx.x * blockDim.x + threadIdx.x;
  if (pt >= P.B) return;
  int on = 0;
  for (int i = 0; i < P.nl; i++) on |= (P.nu[pt].gb[1][i] != 0.0);
  V.one_loop_on[pt] = on;
}

template <typename T>
size_t xss_smem(const Params& P)
{
  return sizeof(T) * (8 * (size_t)XLC * P.n_ss + 2 * (size_t)(P.pss + XTP) * XLC) + 64;
}
template <typename T>
size_t xgs_smem(const Params& P)
{
  return sizeof(T) * (5 * (size_t)XLC * P.n_ss + 2 * (size_t)P.ns * XLC) + 64;
}

// CTAs over the chunks of `nchunk`, for about two per SM over `items` items
int x_split(int items, int nchunk)
{
  const int s = (2 * SM_COUNT + items - 1) / items;
  return s < 1 ? 1 : (s > nchunk ? nchunk : s);
}

template <typename T>
void launch_x(const Params& P, const VJPParams& V, int which, cudaStream_t s)
{
  const int nnr = x_threads(P.n_ss), G = x_groups(P.n_ss);
  if (which == 0) {
    const size_t sm = xss_smem<T>(P);
    cudaFuncSetAttribute(k_vjpx_ss<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    const int nc = (P.nnode_ss + XLC - 1) / XLC;
    k_vjpx_ss<T><<<dim3(P.B, x_split(P.B, nc)), nnr * G, sm, s>>>(P, V, nnr, G);
    k_vjpx_ss_w<<<dim3((P.ns * P.n_ss + 127) / 128, P.B), 128, 0, s>>>(P, V);
  } else {
    const size_t sm = xgs_smem<T>(P);
    cudaFuncSetAttribute(k_vjpx_gs<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    const int nc = (P.nnode_g + XLC - 1) / XLC;
    k_vjpx_gs<T><<<dim3(P.B, P.nl, x_split(P.B * P.nl, nc)), nnr * G, sm, s>>>(P, V, nnr, G);
    k_vjpx_gs_w<<<dim3(P.B, P.nl), nnr, 0, s>>>(P, V);
  }
}

}  // namespace

size_t vjp_extra_smem(const Params& P)
{
  if (P.prec == CL2PT_PREC_FP64) return std::max(xss_smem<double>(P), xgs_smem<double>(P));
  return std::max(xss_smem<float>(P), xgs_smem<float>(P));
}

// which: 0 ss, 1 gs, 2 gg; -1 the per-point gate
void launch_vjp_extra(const Params& P, const VJPParams& V, int which, cudaStream_t s)
{
  if (which < 0) {
    k_vjpx_gate<<<(P.B + 127) / 128, 128, 0, s>>>(P, V);
    return;
  }
  if (which == 2) {
    const int nL = P.nnode_g + (V.ggl_bar ? P.lmax_nolimber : 0);
    const int nt = std::min(x_threads(P.n_gg), XGG_P), ntile = (P.n_gg + nt - 1) / nt;
    const dim3 g(P.B, P.nl, (nL + XGG_L - 1) / XGG_L * ntile);
    k_vjpx_gg<<<g, nt, 0, s>>>(P, V, ntile);
    return;
  }
  if (P.prec == CL2PT_PREC_FP64) launch_x<double>(P, V, which, s);
  else launch_x<float>(P, V, which, s);
}

}  // namespace cl2pt
