// nonlimber.h -- constants of the non-Limber FFTLog stage.
#pragma once

#include <vector>

#include "common.cuh"
#include "kernels.cuh"

namespace cl2pt {

// One Stockham stage of a transform: radix R, sub-transform length Ns, R-th
// of the size NR = N / R, its twiddles at off of the size's table, and the divisor
// Ns as a multiply-high constant (j / Ns = (umulhi(j, m) + j) >> l for
// j < 2^31), so that the butterfly index needs no integer division (GB300
// builds those from conversions, which issue at the FP64 rate).
struct NLStage {
  int R, Ns, NR, off;
  unsigned m;
  int l;
};

struct NLParams {
  int N[3];         // transform sizes of the three radial kernels
  int pad[3];       // zero padding on each side (cosmo2D.c:4564-4577)
  double nu[3];     // power-law bias exponents
  int deriv[3];     // derivative orders of the Gamma-ratio kernels
  int fac[3][16];   // Stockham factors of N[j]
  int nfac[3];
  NLStage st[3][16];  // the stages of each transform
  const double* tw[3];  // stage by stage exp(+2 pi i r k / (Ns R)), [r - 1][k], as (re, im) pairs, FP64
  const void* twt[3];   // the same table in the multipole-loop precision
  int nmax;         // max N[j]
  int hstride;      // nmax / 2 + 1
  void* tout;       // [CTA][3][hstride] complex spectra (loop precision)
  size_t tout_stride;   // complex entries per CTA
  double* gdir;     // [point][3][ndirect][hstride] directly evaluated g_l (FP64 complex)
  // per point, shared by its lens bins (k_nl_slice, k_nl_cg): the geometry
  // record, the powers of x per radial sample (loop precision),
  // the phases and Gamma kernels of a chunk of lchunk multipoles
  // [lchunk][qs] (kernel j's N[j] / 2 + 1 entries from qoff[j]), the last
  // Gamma kernels of a chunk [2][qs]
  double* geom;     // [point][NL_GEOM]
  int* any_mag;     // [point] a lens bin has magnification bias
  void* xtab;       // [point][NL_XROWS][nchi]: (rc / x)^3, log10(rc / (x coverH0)), three powers of x
  void* ptab;       // [point][lchunk][nchi] p_lin(k, 1) at the chi samples (loop precision)
  void* ctab;
  void* gtabl;
  void* gcar;
  int qoff[3];
  int qs;
  int lchunk;       // multiple of 16
  // mixed plan, adjoint: the slice-adjoint terms of achunk multipoles (a
  // multiple of 16, at most lchunk) [point * bin][achunk][nchi] and their sums
  // between these chunks [point * bin][pkl_nk] (allocated with the first
  // adjoint)
  float* gadj;
  float* padj;
  int achunk;
  int* conv_blk;    // [point * bin] lowest converged block (NL_OPEN: none yet)
  // mixed plan: the slice's cells (head, tail, 1 / width, slope) [point]
  // [pkl_nk]; per plan, the FP32 axis, its cells at NL_LUT equally spaced
  // values, and 1 / width of the FP64 axis
  float4* pcell;
  const float* plkf;
  const unsigned short* lut;
  float lscale, lumax;
  const double* pinv;
  double* pslice;   // [point][pkl_nk] z = 0 slice of the linear table (k_nl_slice),
                    // read by all of a point's lens-bin CTAs
  float2* phase;    // mixed plan: [point][3][LNL] the phase increment
                    // theta = deta_j (ln(x0/xlast) - 2 pad_j dlnx + ln(k+1)),
                    // reduced to [-pi, pi] in FP64, as an FP32 head/tail
                    // (k_nl_slice); null in the FP64 plan
  int ndirect;      // multipoles evaluated directly per kernel
  int direct_every; // 1: restart the recurrence every 16-block (FP64 plan)
  // per-multipole constants of the loop, once per plan instead of per
  // thread: ln(k+1), log10(k+1) [LNL] and the c2r scales
  // sqrt(pi) / (4 N_j (k+1)^nu_j) [3][LNL]
  const double* lnk1;
  const double* l10k1;
  const double* sck;
  // FP32 copies for the mixed plan's loop: log10(k+1), the c2r scales and
  // nu_j - 1
  const float* l10k1f;
  const float* sckf;
  float nu1f[3];
  float nuf[3];     // nu_j in FP32 (the Gamma-ratio recurrence)
  // mixed plan: the Gamma part of g_l at l = 0, 1 tabulated in eta
  // (nl_gamma_tables), [3][2][gtab_m] (re, unwrapped im) pairs at
  // eta = (m - 3) / gtab_inv_h; null: direct evaluation (FP64 plan)
  const double* gtab;
  double gtab_inv_h;
  int gtab_m;
};

constexpr int NL_GEOM = 8;            // doubles per geometry record
constexpr int NL_XROWS = 5;           // rows of xtab per point
constexpr int NL_OPEN = 0x7fffffff;   // conv_blk: no converged block
__host__ __device__ constexpr int nl_lut_size(int nk) { return 2 * nk; }

// Host: the tables of NLParams::gtab for the kernels' nu and derivative
// orders, gtab_m entries of spacing 1 / inv_h from eta = -3 / inv_h.
void nl_gamma_tables(const NLParams& Q, double inv_h, int m, std::vector<double>& out);

void launch_nonlimber(const Params& P, const NLParams& Q, cudaStream_t s, int* launches,
                      const Hook& hk);
// the same in two parts: the kernel transforms and direct Gamma kernels
// (independent of the Limber tables, so they may run on another stream),
// then the multipole loop (reads the transforms, the direct kernels and the
// Limber C_gg tables)
void launch_nonlimber_prep(const Params& P, const NLParams& Q, cudaStream_t s, int* launches, const Hook& hk);
void launch_nonlimber_loop(const Params& P, const NLParams& Q, cudaStream_t s, int* launches, const Hook& hk);
// Adjoint of the FFTLog part (run after the forward wave): cbar [B][nl][LNL]
// = dL/dC_l below the hand-over multipole; adds into lnpl_bar [B][pkl_nk *
// pkl_nz] and nu_bar[pt].gb[0][q] (bias model 0).
void launch_nonlimber_vjp(const Params& P, const NLParams& Q, const double* cbar, double* lnpl_bar,
                          cl2pt_nuisance* nu_bar, cudaStream_t s, int* launches);

}  // namespace cl2pt
