// fastpt.h -- device-side description of a batched FAST-PT program.
//
// A program regroups the reference's term lists (J_abl: (alpha, beta, ell),
// cfastpt/cfastpt.c:875-1430; J_abJ1J2Jk: (alpha, beta, J1, J2, Jk),
// cfastpt.c:91-768) for the GPU:
//   biases b   the power-law biased copies of the padded spectrum, f / x^nu_b
//              (J_abl: nu; J_abJ1J2Jk: nu = -2 - alpha for every distinct
//              alpha or beta); each is transformed once per spectrum.
//   inputs u   distinct (bias, Gamma kernel) pairs; the padded Hermitian
//              sequence x_u[halfN + i] = out_b(u)[i] * G_u[i] with
//              G_u = window * g_m(...) / N is what one forward transform of
//              size Ntot sees.  Terms sharing a side share an input.
//   rows j     sums over terms of c_t * R_a(t) R_b(t) (the convolution's
//              spectrum) whose lag-domain result takes one final multiplier
//              H_j: conj(f_z(p + 1)) 2^{i tau} (J_abl) or conj(g_m(Jk + 1/2,
//              -1/2)) (J_abJ1J2Jk).
//   groups g   output spectra: the c2r of the sum of their rows' products,
//              times the k power kpow_g.  J_abl and the bias sums have one
//              row per group; the TATT groups have one row per Jk.
// Transforms are paired: a Hermitian sequence placed with its centre at 0
// (negative indices from Ntot down) has a real transform, so two inputs
// share one complex FFT; two rows' real spectra share one inverse FFT; two
// groups' real outputs share one size-N c2r; two biased real inputs share
// one size-N forward transform.
// Term sums are factored: the terms of a row that share an input are added
// up before that input multiplies them (t_ua is -1 on all but the last of
// such a run), one FP64 operation a term and one a run.
#pragma once
#include <cuda_runtime.h>

#include "fft64.cuh"
#include "fft_fx.cuh"

namespace cl2pt {

struct FPTDev {
  int N0, N, half, Ntot, npad, nlow, nhigh, off;  // off = npad + nlow
  int n_bias, n_in, n_fp, n_row, n_ip, n_grp, n_gp;
  fx::Desc dN, dT;
  const int4* twN;          // exp(-2 pi i j / N), j < N (fixed-point limbs)
  const int4* twT;          // exp(-2 pi i j / Ntot)
  fx::Chirp chirp;          // size N as a convolution of size Ntot (w null: directly, by dN)
  const int* posN;          // frequency k -> position in the size-N transform's output
  const double* rden;       // [n_bias][N] x_full^-nu_b on the padded grid (1 in the pads)
  const double2* G;         // [n_in][half + 1] window * g_m / N
  const int* in_bias;       // [n_in] bias of each input (null: all 0)
  const double2* H;         // [n_h][N + 1] final multiplier of each row class
  const double* kpow;       // [n_kp][N0] k power of each group class
  const int2* fpair;        // [n_fp] inputs (u1, u2 | -1)
  const int* t_ua;          // [terms] the run's shared input, at its last term; else -1
  const int* t_ub;          // [terms] the term's other input
  const double* t_c;        // [terms] coefficient * prefactor / Ntot
  const int* row_start;     // [n_row + 1] term range of each row
  const int* row_p;         // [n_row] H row of each row
  const int2* ipair;        // [n_ip] rows (j1, j2 | -1)
  const int* grp_start;     // [n_grp + 1] row range of each group (multi-row)
  const int* grp_kp;        // [n_grp] kpow row of each group
  const int* grp_out;       // [n_grp] output slot of each group
  const int2* gpair;        // [n_gp] groups (g1, g2 | -1)
  int n_out;                // output slots per spectrum
  bool multi;               // some group has several rows: V + c2r kernels
  double2* xin;             // scratch [S][n_bias][half + 1]
  double* R;                // scratch [S][n_in][Ntot]
  double2* V;               // scratch [S][n_row][N + 1] (multi-row programs)
  int* err;                 // bit 0: extrapolation sign failure
};

// The same program with FP64 transforms (k_fastpt64.cu): its own transforms,
// tables and term lists (each row's terms as given) under names of their own;
// the rest of it, and its scratch, in the base
struct FPT64 : FPTDev {
  fft64::Desc dN64, dT64;
  const double2* twN64;       // exp(-2 pi i j / N), j < N
  const double2* twT64;       // exp(-2 pi i j / Ntot)
  const double2* phT64;       // exp(-i pi N rev(p) / Ntot) at each DIF position p
  const int* posN64;          // frequency k -> DIF position, size N
  const double* den64;        // [n_bias][N] x_full^nu_b on the padded grid (1 in the pads)
  const int *t_ua64, *t_ub64; // [terms] inputs of the two sides
  const double* t_c64;
};

// direct real convolutions of the spectrum with two fixed kernels (the
// TATT delta-E2 and mix-B terms, pt_cfastpt.c:681-866)
struct FPTDirect {
  int N0, M, slot1, slot2, n_out;
  fft64::Desc dM;
  const double2* twM;       // exp(-2 pi i j / M)
  const double2* F;         // [M] FFT(f1) + i FFT(f2) at DIF positions
  const double* c1;         // [N0] output factors of the first kernel
  const double* c2;         // [N0] and of the second
  double2* z;               // scratch [S][M]: the product spectrum between k_fpt_forward and k_fpt_inverse
  int on;                   // 1: the program has them (extra CTAs of the program's kernels)
};

// Adjoint of a program (k_fastpt_vjp.cu): host-built term lists and the
// adjoint's scratch for one wave of spectra.
struct FPTAdj {
  const int* in_start;      // [n_in + 1] terms using each input (either side)
  const int* in_byrow;      // [n_in] 1: runs share a row, 0: the term's other input
  const int* in_key;        // the run's shared row / other input, at its last term; else -1
  const int* in_val;        // the term's other input / row
  const double* in_c;       // the term's coefficient (t_c; doubled for a square)
  const int* bias_start;    // [n_bias + 1] inputs of each bias
  const int* bias_in;
  const int2* grp_pair;     // [n_gpa] groups sharing one size-N transform (g1, g2 | -1)
  const int2* row_pair;     // [n_rpa] rows sharing one size-Ntot transform (j1, j2 | -1)
  const int2* in_pair;      // [n_ipa] inputs sharing one size-Ntot transform (u1, u2 | -1)
  int n_gpa, n_rpa, n_ipa;
  const int* row_grp;       // [n_row] group of each row
  double2* Dg;              // [S][n_grp][N + 1] X_g: half the adjoint of each group's folded c2r input
                            // (the whole of it at m = 0 and N)
  double* sbar;             // [S][n_row][Ntot] adjoint of each row spectrum (DIF order)
  double2* xbar;            // [S][n_in][half + 1] adjoint of each input's half-spectrum
  double* ebar;             // [S][n_bias][N] adjoint of the extrapolated spectrum, per bias
  const double2* F1;        // direct plans: DFT of each kernel (DIF order)
  const double2* F2;
  double* dbar;             // direct plans: [S][3][N0] parts of the direct convolutions' adjoint
};

constexpr int FPT_THREADS = 512;

// shared memory of the size-N and size-Ntot kernels; k_fpt_input's two
// extrapolation tables follow its N points
constexpr int FPT_LO = 32, FPT_HI = 256;  // x^(32 a + b) = hi[a] lo[b]
inline size_t fpt_smem_n(const FPTDev& p) { return (size_t)(p.chirp.w ? p.Ntot : p.N) * sizeof(double2); }
inline size_t fpt_smem_t(const FPTDev& p) { return (size_t)p.Ntot * sizeof(double2); }
inline size_t fpt_smem_in(const FPTDev& p)
{
  const size_t a = fpt_smem_n(p), b = (size_t)p.N * sizeof(double2) + 2 * (FPT_LO + FPT_HI) * sizeof(double);
  return a > b ? a : b;
}

int fpt_smem_setup();
// fx [S][N0] and out [S][n_out][N0] on device; d.on: and the direct
// convolutions
void launch_fastpt(const FPTDev& p, const FPTDirect& d, const double* fx, int S, double* out, cudaStream_t st);
// F = DIF of (f1 + i f2) zero-padded to M, in place on dev_f (M complex)
void launch_fastpt_kernel_fft(const FPTDirect& d, double2* dev_f, cudaStream_t st);
int fpt64_smem_setup();
void launch_fastpt64(const FPT64& p, const double* fx, int S, double* out, cudaStream_t st);
// the program's transforms p.R alone, for the adjoint
void launch_fastpt_transforms(const FPTDev& p, const double* fx, int S, cudaStream_t st);
// adjoint of launch_fastpt for spectra fx [S][N0] whose forward just ran
// (p.R holds its transforms): obar [S][n_out][N0] -> fxbar [S][N0]
// (overwritten)
int fptv_smem_setup();
void launch_fastpt_vjp(const FPTDev& p, const FPTDirect& d, const FPTAdj& a, const double* fx, int S,
                       const double* obar, double* fxbar, cudaStream_t st);

}  // namespace cl2pt
