// k_vjp_fpt.cu -- the FAST-PT tables' share of the 3x2pt adjoint: how the
// data vector depends on p_lin(k, z = 0) through the one-loop bias and TATT
// tables (the dependence k_vjp_extra.cu holds fixed).
//
//   k_vjpr_ss/gs/gg  the cotangent of every table row the TATT / one-loop
//                    Limber terms read (k_extra.cu): each (multipole, node)
//                    reads a row at k = (l + 1/2)/chi, linear in ln k
//                    between two grid points (fpti_row / fptb_row,
//                    cosmo2D.c:1411-1445), so the row adjoint is the sum over
//                    (l, node) of (C_l cotangent x integrand coefficient)
//                    scattered onto those two points.  One CTA per (point
//                    [, lens bin], part of the multipoles), shared-memory
//                    accumulators (FP32 in the mixed plan, FP64 in the FP64
//                    plan), flushed into FP64 with atomics.
//   k_vjpr_tables    the adjoint of the row assembly (k_fpt_tables): the
//                    TATT sums and the sigma_4 = P_d2d2(k_min) / 2
//                    subtractions (pt_cfastpt.c:170-176, cosmo2D.c:2560-2590).
//   (the FAST-PT adjoint of fastpt.cu then maps the table cotangents onto
//    p_lin on the FAST-PT grid)
//   k_vjpr_plin      the adjoint of p_lin(k, a = 1) on the FAST-PT grid
//                    (k_fpt_plin, cosmo3D.c:306-358): exp of a bilinear
//                    lnP in (log10 k, z), so each grid point adds
//                    p_lin x the cotangent x its corner weights to the
//                    linear table's cotangent.
#include <algorithm>

#include "common.cuh"
#include "fpt_cell.cuh"
#include "kernels.cuh"

namespace cl2pt {

namespace {

constexpr double LN10 = 2.302585092994045684;
constexpr int RT = 256;   // threads per CTA

// The row cotangents that a thread's multipoles, taken in ascending order at
// one node, put on the grid: they come in runs of one cell (two multipoles a
// cell on the usual axes), so a run's share of the cell's two ends is summed
// in registers and leaves with one atomic per end and row; a run that moves
// on by one cell keeps its upper end as the next lower one.  Accumulators A
// in shared memory over a CTA's multipoles, FP64 atomics across CTAs.
template <typename T, int NR, typename A>
struct RowRun {
  int i = -1;
  T lo[NR], hi[NR];
  __device__ __forceinline__ void put(A* acc, int n, int at, const T* v)
  {
#pragma unroll
    for (int r = 0; r < NR; r++)
      if (v[r] != (T)0) atomicAdd(acc + (size_t)r * n + at, (A)v[r]);
  }
  __device__ __forceinline__ void add(A* acc, int n, const FptCell<T>& c, const T* g)
  {
    if (c.i != i) {
      if (i >= 0) put(acc, n, i, lo);
      const bool next = c.i == i + 1;
      if (i >= 0 && !next && i + 1 < n) put(acc, n, i + 1, hi);
#pragma unroll
      for (int r = 0; r < NR; r++) {
        lo[r] = (next && i >= 0) ? hi[r] : (T)0;
        hi[r] = (T)0;
      }
      i = c.i;
    }
    const T w = c.w, u = (T)1 - w;
#pragma unroll
    for (int r = 0; r < NR; r++) {
      lo[r] += u * g[r];
      hi[r] += w * g[r];
    }
  }
  __device__ __forceinline__ void end(A* acc, int n)
  {
    if (i < 0) return;
    put(acc, n, i, lo);
    if (i + 1 < n) put(acc, n, i + 1, hi);
  }
};

__device__ __forceinline__ double node_F(const Params& P, int pt, int idx, double* fK, double* D)
{
  const double* node = P.node + (size_t)pt * NF_COUNT * P.node_stride;
  *fK = node[(size_t)NF_FK * P.node_stride + idx];
  *D = node[(size_t)NF_D * P.node_stride + idx];
  return node[(size_t)NF_WT * P.node_stride + idx] * node[(size_t)NF_DCHIDA * P.node_stride + idx] / (*fK * *fK);
}

template <typename A>
__device__ __forceinline__ void flush(double* dst, const A* acc, int m)
{
  for (int i = threadIdx.x; i < m; i += blockDim.x)
    if (acc[i] != (A)0) atomicAdd(dst + i, (double)acc[i]);
}

// ------------------------------------------------------------------ ss
// rows (k_extra_ss): EE += A r1 + B r2 + C r3 + Dm r4 + E r0,
// BB += B r6 + Dm r7 + E r5, both times l(l-1)(l+1)(l+2)/(l+1/2)^4.
// One CTA per (point, RSL multipoles): groups of nnr threads, one node each,
// take contiguous parts of them, four multipoles at a time over the pairs, so
// a coefficient is read once per four multipoles.  Bound by issue.
// real_3x2pt_tatt, 16 points: one CTA per point, with the cotangents
// converted per (multipole, node, pair), took 4.9 ms.
// The pair coefficients are read from global memory (through L2): staged in
// shared memory they take 5 pss n_ss entries, which refused 9 source bins in
// FP64, and save nothing (value and gradient at 16 points 9.89 ms staged, 9.88
// so; 200 points 48.7 and 48.4; FP64 at 8 bins, 64 points 92.8 and 92.7).
constexpr int RSL = 64, RLU = 4;
template <typename T>
__global__ void __launch_bounds__(512) k_vjpr_ss(Params P, VJPParams V, int nnr, int G)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int pt = blockIdx.x, grp = threadIdx.x / nnr, p = threadIdx.x - grp * nnr;
  const int n = P.fpt_n, nn = P.n_ss, np = P.pss, K = P.nnode_ss, Kx = 2 * K;
  typedef typename FptPart<T>::type Part;
  const int L0 = blockIdx.y * RSL, nL = min(RSL, K - L0);
  Part* la = (Part*)smem_raw;                  // [RSL]
  T* ce = (T*)(la + RSL);                      // [np][RSL] pref C_bar EE
  T* cbb = ce + (size_t)np * RSL;              // [np][RSL] pref C_bar BB
  T* acc = cbb + (size_t)np * RSL;             // [8][n]
  for (int i = threadIdx.x; i < 8 * n; i += blockDim.x) acc[i] = (T)0;
  const T* X = (const T*)P.ssx5 + (size_t)pt * 5 * np * nn;  // [5][np][nn]
  const double* cb = V.cbar_ss + (size_t)pt * np * Kx;
  for (int i = threadIdx.x; i < np * RSL; i += blockDim.x) {
    const int pr = i / RSL, l = i - pr * RSL;
    double e = 0, b = 0;
    if (l < nL) {
      const double pref = V.lfac_ss[2 * (L0 + l) + 1];
      e = pref * cb[(size_t)pr * Kx + L0 + l];
      b = pref * cb[(size_t)pr * Kx + K + L0 + l];
    }
    ce[i] = round_to<T>(e);
    cbb[i] = round_to<T>(b);
  }
  for (int i = threadIdx.x; i < nL; i += blockDim.x) la[i] = FptPart<T>::of_l(P, V.lfac_ss[2 * (L0 + i)] * LN10);
  __syncthreads();
  if (p < nn) {
    const Part bp = FptPart<T>::of_p(P, log(P.node[((size_t)pt * NF_COUNT + NF_FK) * P.node_stride + p]));
    const size_t st = (size_t)np * nn;
    const int per = RSL / G / RLU * RLU;  // multipoles of a group (G <= 8)
    RowRun<T, 8, T> run;
    for (int l = grp * per; l < min((grp + 1) * per, nL); l += RLU) {
      T g[RLU][8];
#pragma unroll
      for (int u = 0; u < RLU; u++)
#pragma unroll
        for (int r = 0; r < 8; r++) g[u][r] = (T)0;
      for (int pr = 0; pr < np; pr++) {
        const size_t o = (size_t)pr * nn + p;
        const T A = X[o], B = X[o + st], C = X[o + 2 * st], Dm = X[o + 3 * st], E = X[o + 4 * st];
#pragma unroll
        for (int u = 0; u < RLU; u++) {
          const T e = ce[pr * RSL + l + u], b = cbb[pr * RSL + l + u];
          g[u][1] += A * e;
          g[u][2] += B * e;
          g[u][3] += C * e;
          g[u][4] += Dm * e;
          g[u][0] += E * e;
          g[u][6] += B * b;
          g[u][7] += Dm * b;
          g[u][5] += E * b;
        }
      }
#pragma unroll
      for (int u = 0; u < RLU; u++) {
        if (l + u >= nL) break;
        const FptCell<T> c = fpt_cell(P, la[l + u], bp);
        if (c.in) run.add(acc, n, c, g[u]);
      }
    }
    run.end(acc, n);
  }
  __syncthreads();
  flush<T>(V.rbar_ia + (size_t)pt * 8 * n, acc, 8 * n);
}

// ------------------------------------------------------------------ gs
// rows (k_extra_gs): taE (TATT row 1) x (x0 + x4 pref), mix (row 3) x (x1 +
// x5 pref), d1d2 (bias row 0) x x2, d1s2 (bias row 2) x x3, all times
// sqrt((l-1)l(l+1)(l+2))/(l+1/2)^2; pref = l(l+1)/(l+1/2)^2.  As the ss rows,
// one CTA per (point, lens bin, RGL multipoles).
constexpr int RGL = 256;
template <typename T>
__global__ void __launch_bounds__(512) k_vjpr_gs(Params P, VJPParams V, int nnr, int G)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int kk[CL2PT_MAXB], ss_[CL2PT_MAXB];
  __shared__ int npq;
  const int pt = blockIdx.x, q = blockIdx.y, grp = threadIdx.x / nnr, p = threadIdx.x - grp * nnr;
  const int n = P.fpt_n, nn = P.n_ss, K = P.nnode_g;
  const int L0 = blockIdx.z * RGL, nL = min(RGL, K - L0);
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
  typedef typename FptPart<T>::type Part;
  Part* la = (Part*)smem_raw;                  // [RGL]
  T* X = (T*)(la + RGL);                       // [6][ns][nn] (a lens bin pairs with at most ns sources)
  T* c0 = X + 6 * (size_t)P.ns * nn;           // [ns][RGL] C_bar x its factor
  T* pf = c0 + (size_t)P.ns * RGL;             // [RGL] pref
  T* acc = pf + RGL;                           // [4][n]: taE, mix, d1d2, d1s2
  for (int i = threadIdx.x; i < 4 * n; i += blockDim.x) acc[i] = (T)0;
  __syncthreads();
  const int np = npq;
  if (np == 0) return;
  const int off = P.n_ss + q * P.n_ss;
  const size_t b0 = (size_t)pt * P.nl + q;
  const size_t st = (size_t)P.ns * nn;
  for (int idx = threadIdx.x; idx < nn * G; idx += blockDim.x) {
    // a node's coefficients of every G-th pair
    const int p2 = idx % nn, m0 = idx / nn;
    double fK, D;
    const double F = node_F(P, pt, off + p2, &fK, &D), D2 = D * D;
    const double Lg = P.wgs_l[b0 * nn + p2], Mg = P.wgs_m[b0 * nn + p2];
    const double f2 = P.one_loop ? P.wgs_1l[(b0 * 3 + 0) * nn + p2] : 0.0;
    const double f3 = P.one_loop ? P.wgs_1l[(b0 * 3 + 1) * nn + p2] : 0.0;
    for (int m = m0; m < np; m += G) {
      const size_t o = (b0 * P.ns + ss_[m]) * nn + p2;
      double x[6] = {0, 0, 0, 0, 0, 0};
      if (P.tatt) {
        const double b = P.wgs_b[o], c = P.wgs_2[o];
        x[0] = -b * D2 * Lg * F;
        x[1] = 5. * c * D2 * Lg * F;
        x[4] = -b * D2 * Mg * F;
        x[5] = 5. * c * D2 * Mg * F;
      }
      if (P.one_loop) {
        const double WK = P.wgs_k[o];
        x[2] = WK * f2 * F;
        x[3] = WK * f3 * F;
      }
#pragma unroll
      for (int r = 0; r < 6; r++) X[r * st + (size_t)m * nn + p2] = round_to<T>(x[r]);
    }
  }
  for (int i = threadIdx.x; i < np * RGL; i += blockDim.x) {
    const int m = i / RGL, l = i - m * RGL;
    double c = 0.0;
    if (l < nL) c = V.cbar_gs[((size_t)pt * P.pgs + kk[m]) * K + L0 + l] * V.lfac_g[6 * (L0 + l) + 1];
    c0[i] = round_to<T>(c);
  }
  for (int i = threadIdx.x; i < nL; i += blockDim.x) {
    la[i] = FptPart<T>::of_l(P, V.lfac_g[6 * (L0 + i)] * LN10);
    pf[i] = round_to<T>(V.lfac_g[6 * (L0 + i) + 2]);
  }
  __syncthreads();
  if (p < nn) {
    const Part bp = FptPart<T>::of_p(P, log(P.node[((size_t)pt * NF_COUNT + NF_FK) * P.node_stride + off + p]));
    const int per = RGL / G;
    RowRun<T, 4, T> run;
    for (int l = grp * per; l < min((grp + 1) * per, nL); l++) {
      const FptCell<T> c = fpt_cell(P, la[l], bp);
      if (!c.in) continue;
      T g[4] = {0, 0, 0, 0};
      for (int m = 0; m < np; m++) {
        const T e0 = c0[m * RGL + l], e1 = e0 * pf[l];
        const size_t o = (size_t)m * nn + p;
        g[0] += X[o] * e0 + X[4 * st + o] * e1;
        g[1] += X[st + o] * e0 + X[5 * st + o] * e1;
        g[2] += X[2 * st + o] * e0;
        g[3] += X[3 * st + o] * e0;
      }
      run.add(acc, n, c, g);
    }
    run.end(acc, n);
  }
  __syncthreads();
  if (P.tatt) {
    flush<T>(V.rbar_ia + ((size_t)pt * 8 + 1) * n, acc, n);
    flush<T>(V.rbar_ia + ((size_t)pt * 8 + 3) * n, acc + n, n);
  }
  if (P.one_loop) {
    flush<T>(V.rbar_b + ((size_t)pt * 5 + 0) * n, acc + 2 * n, n);
    flush<T>(V.rbar_b + ((size_t)pt * 5 + 2) * n, acc + 3 * n, n);
  }
}

// ------------------------------------------------------------------ gg
// rows (k_extra_gg, FP64 in both plans): bias rows m x W_gal^2 D^4 (...)_m
// at the C_l nodes and, below LMAX_NOLIMBER, at integer l (non-Limber
// hand-over); nodes past chi(a_min) give nothing.  The coefficients stay
// FP64; the accumulators are A (FP32 in the mixed plan).  The clustering rows
// weigh most in the table gradient and cancel in the FAST-PT adjoint, down
// to the rounding of these FP32 sums, which follows the order in which the
// warps' atomics meet: with the cell in the loop precision and the rows on
// CTAs of their own 1.48 ms became 0.30 (real_3x2pt_tatt, 16 points), but
// the largest gradient entries moved by twice what two runs differ by.
// Hence the FP64 cell and one CTA for the five rows.
// the table-row lookup of k_extra.cu: cell i and weight w, or out of range
struct RCell {
  int i;
  double w;
  bool in;
};
__device__ __forceinline__ RCell r_cell(const Params& P, double lnk)
{
  RCell c;
  c.in = !(lnk < P.fpt_lim0 || lnk > P.fpt_lim1);
  const double r = (lnk - P.fpt_lim0) / P.fpt_lim2;
  c.i = c.in ? (int)floor(r) : 0;
  c.w = r - c.i;
  if (c.i + 1 >= P.fpt_n) {
    c.i = P.fpt_n - 1;
    c.w = 0.0;
  }
  return c;
}

// scatter g onto row acc at cell c (the transpose of fpt_val); the
// accumulators are FP32 in the mixed plan (native shared-memory atomics)
// and FP64 in the FP64 plan
template <typename A>
__device__ __forceinline__ void r_scatter(A* acc, const RCell& c, A g, int n)
{
  if (c.i + 1 >= n) {
    atomicAdd(acc + c.i, g);
  } else {
    atomicAdd(acc + c.i, (A)(1.0 - c.w) * g);
    atomicAdd(acc + c.i + 1, (A)c.w * g);
  }
}

template <typename A>
__global__ void __launch_bounds__(RT) k_vjpr_gg(Params P, VJPParams V)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int pt = blockIdx.x, q = blockIdx.y;
  const int n = P.fpt_n, nn = P.n_gg, K = P.nnode_g, LNL = P.lmax_nolimber;
  double* X = (double*)smem_raw;     // [5][nn]
  double* nd = X + 5 * (size_t)nn;   // [2][nn]: ln chi, chi
  A* acc = (A*)(nd + 2 * (size_t)nn);  // [5][n]
  for (int i = threadIdx.x; i < 5 * n; i += blockDim.x) acc[i] = (A)0;
  const int off = P.n_ss + P.nl * P.n_ss + q * nn;
  const size_t b0 = (size_t)pt * P.nl + q;
  for (int idx = threadIdx.x; idx < 5 * nn; idx += blockDim.x) {
    const int m = idx / nn, p = idx - m * nn;
    double fK, D;
    const double F = node_F(P, pt, off + p, &fK, &D);
    X[m * nn + p] = P.wgg_1l[(b0 * 6 + m) * nn + p] * F;
    if (m == 0) {
      nd[p] = log(fK);
      nd[nn + p] = fK;
    }
  }
  __syncthreads();
  const double chi_amin = P.chi_amin[pt];
  const int nL = K + (V.ggl_bar ? LNL : 0);
  for (int w = threadIdx.x; w < nL * nn; w += blockDim.x) {
    const int L = w / nn, p = w - L * nn;
    const double* fac;
    double cv;
    if (L < K) {
      fac = V.lfac_g + 6 * L;
      cv = V.cbar_gg[b0 * K + L];
    } else {
      fac = V.lfac_gi + 6 * (L - K);
      cv = V.ggl_bar[(b0 * LNL + (L - K)) * 2];
    }
    if (cv == 0.0 || nd[nn + p] * fac[5] > chi_amin) continue;
    const RCell c = r_cell(P, fac[0] * LN10 - nd[p]);
    if (!c.in) continue;
#pragma unroll
    for (int m = 0; m < 5; m++) {
      const double g = X[m * nn + p] * cv;
      if (g != 0.0) r_scatter<A>(acc + (size_t)m * n, c, (A)g, n);
    }
  }
  __syncthreads();
  flush<A>(V.rbar_b + (size_t)pt * 5 * n, acc, 5 * n);
}

// ------------------------------------------------ row assembly adjoint
__global__ void __launch_bounds__(RT) k_vjpr_tables(Params P, VJPParams V)
{
  __shared__ double red[RT / 32];
  const int pt = blockIdx.x, n = P.fpt_n;
  if (P.tatt) {
    const double* r = V.rbar_ia + (size_t)pt * 8 * n;
    double* o = V.obar_fia + (size_t)pt * 10 * n;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      o[0 * n + i] = r[0 * n + i];
      o[1 * n + i] = r[5 * n + i];
      o[2 * n + i] = r[1 * n + i];
      o[3 * n + i] = r[1 * n + i];
      o[4 * n + i] = r[2 * n + i];
      o[5 * n + i] = r[6 * n + i];
      o[6 * n + i] = r[3 * n + i];
      o[7 * n + i] = r[3 * n + i];
      o[8 * n + i] = r[4 * n + i];
      o[9 * n + i] = r[7 * n + i];
    }
  }
  if (P.one_loop) {
    const double* r = V.rbar_b + (size_t)pt * 5 * n;
    double* o = V.obar_fb + (size_t)pt * 5 * n;
    double s4 = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      for (int m = 0; m < 5; m++) o[m * n + i] = r[m * n + i];
      s4 += -2. * r[1 * n + i] - 4. / 3. * r[3 * n + i] - 8. / 9. * r[4 * n + i];
    }
    for (int d = 16; d > 0; d >>= 1) s4 += __shfl_xor_sync(0xffffffffu, s4, d);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s4;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < RT / 32; w++) t += red[w];
      o[1 * n + 0] += 0.5 * t;  // sigma_4 = P_d2d2(k_min) / 2
    }
  }
}

// ------------------------------------------------ p_lin(k, a = 1) adjoint
__global__ void __launch_bounds__(RT) k_vjpr_plin(Params P, VJPParams V)
{
  const int pt = blockIdx.x, n = P.fpt_n;
  const double* tab = P.lnPL + (size_t)pt * P.pkl_nk * P.pkl_nz;
  double* bar = V.lnpl_bar;
  const double c3 = CL2PT_COVERH0 * CL2PT_COVERH0 * CL2PT_COVERH0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    double gb = 0.0;
    if (P.one_loop) gb += V.plinbar_b[(size_t)pt * n + i];
    if (P.tatt) gb += V.plinbar_ia[(size_t)pt * n + i];
    if (gb == 0.0) continue;
    const double k = exp(P.fpt_lim0 + i * P.fpt_lim2);
    const double log10k = log10(k / CL2PT_COVERH0), z = 0.0;
    const int a = bsearch_d(P.pkl_lk, P.pkl_nk, log10k);
    const int j = bsearch_d(P.pkl_z, P.pkl_nz, z);
    const double dx = (log10k - P.pkl_lk[a]) / (P.pkl_lk[a + 1] - P.pkl_lk[a]);
    const double dy = (z - P.pkl_z[j]) / (P.pkl_z[j + 1] - P.pkl_z[j]);
    const int nz = P.pkl_nz;
    const double v = (1 - dx) * (1 - dy) * tab[a * nz + j] + (1 - dx) * dy * tab[a * nz + j + 1] +
                     dx * (1 - dy) * tab[(a + 1) * nz + j] + dx * dy * tab[(a + 1) * nz + j + 1];
    const double g = gb * exp(v) / c3;
    const double w[4] = {(1 - dx) * (1 - dy), (1 - dx) * dy, dx * (1 - dy), dx * dy};
    const int idx[4] = {a * nz + j, a * nz + j + 1, (a + 1) * nz + j, (a + 1) * nz + j + 1};
#pragma unroll
    for (int c = 0; c < 4; c++)
      if (w[c] != 0.0) atomicAdd(bar + (size_t)pt * P.pkl_nk * nz + idx[c], g * w[c]);
  }
}

template <typename T>
size_t rss_smem(const Params& P)
{
  return sizeof(double) * RSL + sizeof(T) * (8 * (size_t)P.fpt_n + 2 * (size_t)P.pss * RSL);
}
template <typename T>
size_t rgs_smem(const Params& P)
{
  return sizeof(double) * RGL +
         sizeof(T) * (4 * (size_t)P.fpt_n + 6 * (size_t)P.ns * P.n_ss + (size_t)(P.ns + 1) * RGL);
}
template <typename A>
size_t rgg_smem(const Params& P)
{
  return sizeof(double) * 7 * (size_t)P.n_gg + sizeof(A) * 5 * (size_t)P.fpt_n + 16;
}

// threads per node group and groups of a CTA: 256 threads, or one group of
// as many as the nodes need
int r_threads(int nn) { return ((nn + 31) / 32) * 32; }
int r_groups(int nn) { return r_threads(nn) <= 64 ? 4 : r_threads(nn) <= 128 ? 2 : 1; }

template <typename T>
void launch_rows_t(const Params& P, const VJPParams& V, int which, cudaStream_t s)
{
  if (which == 0) {
    const int nnr = r_threads(P.n_ss), G = r_groups(P.n_ss);
    const size_t sm = rss_smem<T>(P);
    cudaFuncSetAttribute(k_vjpr_ss<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_vjpr_ss<T><<<dim3(P.B, (P.nnode_ss + RSL - 1) / RSL), nnr * G, sm, s>>>(P, V, nnr, G);
  } else if (which == 1) {
    const int nnr = r_threads(P.n_ss), G = r_groups(P.n_ss);
    const size_t sm = rgs_smem<T>(P);
    cudaFuncSetAttribute(k_vjpr_gs<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_vjpr_gs<T><<<dim3(P.B, P.nl, (P.nnode_g + RGL - 1) / RGL), nnr * G, sm, s>>>(P, V, nnr, G);
  } else {
    const size_t sm = rgg_smem<T>(P);
    cudaFuncSetAttribute(k_vjpr_gg<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_vjpr_gg<T><<<dim3(P.B, P.nl), RT, sm, s>>>(P, V);
  }
}

}  // namespace

// what the row kernels that this plan launches need
size_t vjp_fpt_smem(const Params& P)
{
  auto need = [&](auto t) {
    typedef decltype(t) T;
    size_t m = rgs_smem<T>(P);
    if (P.tatt) m = std::max(m, rss_smem<T>(P));
    if (P.one_loop) m = std::max(m, rgg_smem<T>(P));
    return m;
  };
  return P.prec == CL2PT_PREC_FP64 ? need(0.0) : need(0.0f);
}

void launch_vjp_fpt_rows(const Params& P, const VJPParams& V, int which, cudaStream_t s)
{
  if (!V.rbar_ia && !V.rbar_b) return;
  if (which == 2 && !P.one_loop) return;
  if (which == 0 && !P.tatt) return;
  if (P.prec == CL2PT_PREC_FP64) launch_rows_t<double>(P, V, which, s);
  else launch_rows_t<float>(P, V, which, s);
}

void launch_vjp_fpt_tables(const Params& P, const VJPParams& V, cudaStream_t s)
{
  k_vjpr_tables<<<P.B, RT, 0, s>>>(P, V);
}

void launch_vjp_fpt_plin(const Params& P, const VJPParams& V, cudaStream_t s)
{
  k_vjpr_plin<<<P.B, RT, 0, s>>>(P, V);
}

}  // namespace cl2pt
