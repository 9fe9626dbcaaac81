// k_nonlimber.cu -- non-Limber galaxy clustering C_l by FFTLog
// (C_cl_tomo + cfftlog_ells_p1/p2, cosmo2D.c:3995-4769), FP64.
//
// Per (point, lens bin): the three radial kernels f_j(chi) (galaxy bias, RSD,
// magnification) on the log-chi grid, their r2c transforms with the c-window
// taper (k_nl_forward); per point, the phases and Gamma-ratio kernels g_l of
// all multipoles (k_nl_gdirect, k_nl_cg: direct evaluation where the
// recurrence starts, the two-step recurrence after that).  Then, in blocks of
// 16 multipoles as the reference walks them (k_nl_block), for every l: each
// spectrum times its phase and g_l, one c2r transform per kernel in shared
// memory, F = F_0 + F_1 + bmag l(l+1) F_2 / y^2 and the integral of
// F^2 k^3 P_lin(k, z=0) over chi; at the end of a block the reference's 1%
// convergence test against the Limber C_l, whose first success hands the
// remaining multipoles to Limber (k_nl_handover).
//
// The FFT is a Stockham autosort transform (Govindaraju et al. 2008
// formulation) over the factors 4, 2, 3, 5, 7, one butterfly per thread per
// stage, ping-ponging two shared-memory buffers, with twiddles read from a
// per-size table.
#include <math.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "nonlimber.h"

namespace cl2pt {

// FP64 complex arithmetic, on the device and (for the plan's tables) the host
#define NL_HD __host__ __device__ __forceinline__
struct cd { double x, y; };
NL_HD cd cmk(double a, double b) { cd r; r.x = a; r.y = b; return r; }
NL_HD cd cadd(cd a, cd b) { return cmk(a.x + b.x, a.y + b.y); }
NL_HD cd csub(cd a, cd b) { return cmk(a.x - b.x, a.y - b.y); }
NL_HD cd cmul(cd a, cd b) { return cmk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
NL_HD cd cscale(cd a, double s) { return cmk(a.x * s, a.y * s); }
NL_HD cd cconj(cd a) { return cmk(a.x, -a.y); }
NL_HD cd cdivc(cd a, cd b)
{
  // Smith's algorithm
  if (fabs(b.x) >= fabs(b.y)) {
    const double r = b.y / b.x, d = b.x + b.y * r;
    return cmk((a.x + a.y * r) / d, (a.y - a.x * r) / d);
  }
  const double r = b.x / b.y, d = b.x * r + b.y;
  return cmk((a.x * r + a.y) / d, (a.y * r - a.x) / d);
}
NL_HD void sincos_hd(double a, double* s, double* c)
{
#ifdef __CUDA_ARCH__
  sincos(a, s, c);
#else
  *s = sin(a);
  *c = cos(a);
#endif
}
NL_HD cd clog_(cd a) { return cmk(log(hypot(a.x, a.y)), atan2(a.y, a.x)); }
NL_HD cd cexp_(cd a)
{
  const double m = exp(a.x);
  double s, c;
  sincos_hd(a.y, &s, &c);
  return cmk(m * c, m * s);
}
NL_HD cd csin_(cd a)
{
  double s, c;
  sincos_hd(a.x, &s, &c);
  return cmk(s * cosh(a.y), c * sinh(a.y));
}

// coefficients of the Lanczos sum, g = 7, n = 9 (the reference's ln Gamma)
NL_HD double lanczos_c(int w)
{
  switch (w) {
    case 0: return 0.99999999999980993227684700473478;
    case 1: return 676.520368121885098567009190444019;
    case 2: return -1259.13921672240287047156078755283;
    case 3: return 771.3234287776530788486528258894;
    case 4: return -176.61502916214059906584551354;
    case 5: return 12.507343278686904814458936853;
    case 6: return -0.13857109526572011689554707;
    case 7: return 9.984369578019570859563e-6;
    default: return 1.50563273514931155834e-7;
  }
}

// ln Gamma(a) for Re a >= 1/2, |a| >= 10: Stirling's series
// (Abramowitz & Stegun 6.1.40-41) to the B_16 term, remainder below 1e-17
// relative there; ~1/3 of the FP64 work of the Lanczos sum (one complex
// reciprocal instead of eight complex divisions, one complex log).
// Exponentiated only, so its branch of the imaginary part is immaterial.
NL_HD cd lngamma_stirling(cd a)
{
  const cd r = cdivc(cmk(1.0, 0.0), a);
  const cd r2 = cmul(r, r);
  // B_2n / (2n (2n - 1)), n = 1..8
  const double c1 = 1.0 / 12, c2 = -1.0 / 360, c3 = 1.0 / 1260, c4 = -1.0 / 1680, c5 = 1.0 / 1188,
               c6 = -691.0 / 360360, c7 = 1.0 / 156, c8 = -3617.0 / 122400;
  cd sr = cmk(c8, 0.0);
  sr = cadd(cmk(c7, 0.0), cmul(sr, r2));
  sr = cadd(cmk(c6, 0.0), cmul(sr, r2));
  sr = cadd(cmk(c5, 0.0), cmul(sr, r2));
  sr = cadd(cmk(c4, 0.0), cmul(sr, r2));
  sr = cadd(cmk(c3, 0.0), cmul(sr, r2));
  sr = cadd(cmk(c2, 0.0), cmul(sr, r2));
  sr = cadd(cmk(c1, 0.0), cmul(sr, r2));
  sr = cmul(sr, r);
  return cadd(csub(cmul(cmk(a.x - 0.5, a.y), clog_(a)), a), cmk(0.5 * log(2 * M_PI) + sr.x, sr.y));
}

// ln Gamma(1 + m) for Re m >= -1/2 (Lanczos g = 7, the reference's sum;
// Stirling's series for |1 + m| >= 10)
NL_HD cd lngamma_1p(cd m)
{
  if (hypot(m.x + 1.0, m.y) >= 10.0) return lngamma_stirling(cmk(m.x + 1.0, m.y));
  const double ln2pio2 = 0.5 * log(2 * M_PI);
  cd tmp = cmk(lanczos_c(0), 0.0);
#pragma unroll
  for (int w = 1; w < 9; w++) tmp = cadd(tmp, cdivc(cmk(lanczos_c(w), 0.0), cmk(m.x + w, m.y)));
  const cd t = cmk(m.x + 7.5, m.y);
  return cadd(csub(cadd(cmk(ln2pio2, 0.0), cmul(cmk(m.x + 0.5, m.y), clog_(t))), t), clog_(tmp));
}

// ln Gamma(a) with reflection for Re a < 1/2 (cosmo2D.c:4273-4294)
NL_HD cd lngamma_refl(cd a)
{
  if (a.x < 0.5) {
    // ln pi - ln sin(pi a) - ln Gamma(1 - a)
    const cd inner = lngamma_1p(cmk(-a.x, -a.y));
    const cd s = clog_(csin_(cscale(a, M_PI)));
    return csub(csub(cmk(log(M_PI), 0.0), s), inner);
  }
  return lngamma_1p(cmk(a.x - 1.0, a.y));
}

// g_l(z) for the three derivative orders (cosmo2D.c:4259-4430)
__device__ cd gl_direct(int deriv, double nu, double eta, int k)
{
  const double ln2 = log(2.);
  const cd z = cmk(nu, eta);
  if (deriv == 0) {
    const cd p1 = lngamma_refl(cscale(cmk(k + z.x, z.y), 0.5));
    const cd p2 = lngamma_refl(cscale(cmk(3 + k - z.x, -z.y), 0.5));
    return cexp_(cadd(cscale(z, ln2), csub(p1, p2)));
  }
  if (deriv == 1) {
    const cd p1 = lngamma_refl(cscale(cmk(k + z.x - 1., z.y), 0.5));
    const cd p2 = lngamma_refl(cscale(cmk(4 + k - z.x, -z.y), 0.5));
    const cd e = cexp_(cadd(cscale(cmk(z.x - 1, z.y), ln2), csub(p1, p2)));
    return cmul(cmk(-(z.x - 1), -z.y), e);
  }
  const cd p1 = lngamma_refl(cscale(cmk(k + z.x - 2, z.y), 0.5));
  const cd p2 = lngamma_refl(cscale(cmk(5 + k - z.x, -z.y), 0.5));
  const cd e = cexp_(cadd(cscale(cmk(z.x - 2, z.y), ln2), csub(p1, p2)));
  return cmul(cmul(cmk(z.x - 1, z.y), cmk(z.x - 2, z.y)), e);
}

constexpr int NL_NT = 256;

// complex arithmetic in the multipole loop's precision
template <typename T> struct ct { T x, y; };
template <typename T> __device__ __forceinline__ ct<T> tmk(T a, T b) { ct<T> r; r.x = a; r.y = b; return r; }
template <typename T> __device__ __forceinline__ ct<T> tmul(ct<T> a, ct<T> b)
{
  return tmk<T>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <typename T> __device__ __forceinline__ ct<T> tadd(ct<T> a, ct<T> b) { return tmk<T>(a.x + b.x, a.y + b.y); }
template <typename T> __device__ __forceinline__ ct<T> tdiv(ct<T> a, ct<T> b)
{
  if (fabs(b.x) >= fabs(b.y)) {
    const T r = b.y / b.x, d = b.x + b.y * r;
    return tmk<T>((a.x + a.y * r) / d, (a.y - a.x * r) / d);
  }
  const T r = b.x / b.y, d = b.x * r + b.y;
  return tmk<T>((a.x * r + a.y) / d, (a.y * r - a.x) / d);
}
template <typename T> __device__ __forceinline__ void tsincos(T a, T* s, T* c);
template <> __device__ __forceinline__ void tsincos<float>(float a, float* s, float* c) { __sincosf(a, s, c); }
template <> __device__ __forceinline__ void tsincos<double>(double a, double* s, double* c) { sincos(a, s, c); }
template <typename T> __device__ __forceinline__ T texp(T a);
template <> __device__ __forceinline__ float texp<float>(float a) { return expf(a); }
template <> __device__ __forceinline__ double texp<double>(double a) { return exp(a); }
template <typename T> __device__ __forceinline__ T tlog10(T a);
template <> __device__ __forceinline__ float tlog10<float>(float a) { return log10f(a); }
template <> __device__ __forceinline__ double tlog10<double>(double a) { return log10(a); }

// cos and sin of 2 pi e / R, e in [0, R), R = 3, 5, 7.  Not recursive: a
// recursive one is a call at run time, with FP64 arithmetic and a conversion
// per root, a third of k_nl_block's time.
template <int R>
__device__ constexpr double root_c(int e)
{
  if (e == 0) return 1.0;
  if (R == 3) return -0.5;
  if (R == 5) return (e == 1 || e == 4) ? 0.3090169943749474241023 : -0.8090169943749474241023;
  return (e == 1 || e == 6) ? 0.6234898018587335305250
         : (e == 2 || e == 5) ? -0.2225209339563144042889 : -0.9009688679024191262361;
}
template <int R>
__device__ constexpr double root_s(int e)
{
  if (e == 0) return 0.0;
  const int f = 2 * e > R ? R - e : e;
  const double v = R == 3   ? 0.8660254037844386467637
                   : R == 5 ? (f == 1 ? 0.9510565162951535721164 : 0.5877852522924731291687)
                            : (f == 1   ? 0.7818314824680298087084
                               : f == 2 ? 0.9749279121818236070181
                                        : 0.4338837391175581204758);
  return 2 * e > R ? -v : v;
}

// radix-R butterfly (R = 3, 5, 7) on v[0..R-1], SIGN the exponent's sign.
// FP32: output t is v_0 + v_1 w^t + v_2 w^2t + ... summed in that order,
// each term a complex product of one multiply and one fused multiply-add
// per part.  Outputs t and R - t meet conjugate roots, so the multiplies
// are formed once for both, and the roots are immediates (the FP32 roots of
// the twiddle table are these values and exactly conjugate).  Issue-bound:
// 88 instead of 120 instructions at R = 5, 28 instead of 36 at R = 3.
// FP64: sums and differences of v_r and v_{R-r} first, which halves the
// multiplies (the FP64 pipe bounds it).
template <typename T, int R, int SIGN>
__device__ __forceinline__ void dft_odd(ct<T>* v)
{
  ct<T> o[R];
  if constexpr (sizeof(T) == sizeof(float)) {
    o[0] = v[0];
#pragma unroll
    for (int r = 1; r < R; r++) o[0] = tadd(o[0], v[r]);
#pragma unroll
    for (int t = 1; t <= R / 2; t++) {
      ct<T> a = v[0], b = v[0];
#pragma unroll
      for (int r = 1; r < R; r++) {
        const float wr = (float)root_c<R>((r * t) % R), wi = SIGN * (float)root_s<R>((r * t) % R);
        const float m1 = __fmul_rn(v[r].y, wi), m2 = __fmul_rn(v[r].x, wi);
        a.x = __fadd_rn(a.x, __fmaf_rn(v[r].x, wr, -m1));
        a.y = __fadd_rn(a.y, __fmaf_rn(v[r].y, wr, m2));
        b.x = __fadd_rn(b.x, __fmaf_rn(v[r].x, wr, m1));
        b.y = __fadd_rn(b.y, __fmaf_rn(v[r].y, wr, -m2));
      }
      o[t] = a;
      o[R - t] = b;
    }
  } else {
    ct<T> p[R / 2 + 1], m[R / 2 + 1];
    o[0] = v[0];
#pragma unroll
    for (int r = 1; r <= R / 2; r++) {
      p[r] = tadd(v[r], v[R - r]);
      m[r] = tmk<T>(v[r].x - v[R - r].x, v[r].y - v[R - r].y);
      o[0] = tadd(o[0], p[r]);
    }
#pragma unroll
    for (int t = 1; t <= R / 2; t++) {
      ct<T> a = v[0], b = tmk<T>((T)0, (T)0);
#pragma unroll
      for (int r = 1; r <= R / 2; r++) {
        const double wr = root_c<R>((r * t) % R), wi = SIGN * root_s<R>((r * t) % R);
        a.x = fma(wr, p[r].x, a.x);
        a.y = fma(wr, p[r].y, a.y);
        b.x = fma(-wi, m[r].y, b.x);
        b.y = fma(wi, m[r].x, b.y);
      }
      o[t] = tadd(a, b);
      o[R - t] = tmk<T>(a.x - b.x, a.y - b.y);
    }
  }
#pragma unroll
  for (int t = 0; t < R; t++) v[t] = o[t];
}
template <typename T>
__device__ __forceinline__ void dft2(ct<T>* v)
{
  const ct<T> a = v[0], b = v[1];
  v[0] = tmk<T>(a.x + b.x, a.y + b.y);
  v[1] = tmk<T>(a.x - b.x, a.y - b.y);
}
template <typename T, int SIGN>
__device__ __forceinline__ void dft4(ct<T>* v)
{
  const ct<T> a = tmk<T>(v[0].x + v[2].x, v[0].y + v[2].y);
  const ct<T> b = tmk<T>(v[0].x - v[2].x, v[0].y - v[2].y);
  const ct<T> c = tmk<T>(v[1].x + v[3].x, v[1].y + v[3].y);
  ct<T> d = tmk<T>(v[1].x - v[3].x, v[1].y - v[3].y);
  // d * (SIGN i)
  d = (SIGN > 0) ? tmk<T>(-d.y, d.x) : tmk<T>(d.y, -d.x);
  v[0] = tmk<T>(a.x + c.x, a.y + c.y);
  v[2] = tmk<T>(a.x - c.x, a.y - c.y);
  v[1] = tmk<T>(b.x + d.x, b.y + d.y);
  v[3] = tmk<T>(b.x - d.x, b.y - d.y);
}

// One Stockham stage of radix R (compile-time, so the butterfly stays in
// registers): out[(j/Ns) Ns R + k + r Ns] = DFT_R over r of
// in[j + r N/R] w^(r k N / (Ns R)), k = j mod Ns; the twiddles lie in the order
// in which a warp reads them (a stride of r N / (Ns R) in one table of roots
// took a sector per lane).
template <typename T, int R, int SIGN>
__device__ __forceinline__ void stockham_stage(const ct<T>* __restrict__ in, ct<T>* __restrict__ out,
                                               const NLStage& S, const ct<T>* __restrict__ tw)
{
  const int NR = S.NR, Ns = S.Ns;
  const ct<T>* ts = tw + S.off;
  for (int j = threadIdx.x; j < NR; j += blockDim.x) {
    const int g = (int)((__umulhi((unsigned)j, S.m) + (unsigned)j) >> S.l);  // j / Ns
    const int k = j - g * Ns;
    ct<T> v[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
      ct<T> x = in[j + r * NR];
      if (r && k) {
        ct<T> t = ts[(r - 1) * Ns + k];
        if (SIGN < 0) t.y = -t.y;
        x = tmul(x, t);
      }
      v[r] = x;
    }
    if constexpr (R == 2) dft2(v);
    else if constexpr (R == 4) dft4<T, SIGN>(v);
    else dft_odd<T, R, SIGN>(v);
    const int dst = g * Ns * R + k;
#pragma unroll
    for (int r = 0; r < R; r++) out[dst + r * Ns] = v[r];
  }
}

// Stockham transform in the loop precision over the stages st[0..nf-1]
// (radices 4, 2, 3, 5, 7), ping-ponging in/out; returns the buffer holding
// the result.
template <typename T, int SIGN>
__device__ ct<T>* block_fft_t(ct<T>* in, ct<T>* out, const NLStage* st, int nf, const ct<T>* __restrict__ tw)
{
  for (int s = 0; s < nf; s++) {
    const NLStage& S = st[s];
    switch (S.R) {
      case 2: stockham_stage<T, 2, SIGN>(in, out, S, tw); break;
      case 3: stockham_stage<T, 3, SIGN>(in, out, S, tw); break;
      case 4: stockham_stage<T, 4, SIGN>(in, out, S, tw); break;
      case 5: stockham_stage<T, 5, SIGN>(in, out, S, tw); break;
      default: stockham_stage<T, 7, SIGN>(in, out, S, tw); break;
    }
    __syncthreads();
    ct<T>* t = in;
    in = out;
    out = t;
  }
  return in;
}

// Shared pieces of the three FFTLog kernels.
struct NLGeom {
  double rc, dlnchi, dlnx, x0, xlast;
};
__device__ __forceinline__ NLGeom nl_geom(const Params& P, int pt)
{
  const double* X = P.chi + (size_t)pt * P.chi_nz;
  NLGeom g;
  g.rc = CL2PT_COVERH0 / P.h0[pt];
  const double chi_min = chi_all_d(P.chi_z, X, P.chi_nz, 1. / (1.0 + 0.002)).chi * g.rc;
  const double chi_max = chi_all_d(P.chi_z, X, P.chi_nz, 1. / (1.0 + 4.0)).chi * g.rc;
  g.dlnchi = log(chi_max / chi_min) / ((double)P.nl_nchi - 1.0);
  g.x0 = chi_min;
  g.xlast = chi_min * exp(g.dlnchi * (P.nl_nchi - 1));
  g.dlnx = log((chi_min * exp(g.dlnchi)) / chi_min);
  return g;
}

// the same from the point's record (k_nl_slice)
__device__ __forceinline__ NLGeom nl_geom_rec(const NLParams& Q, int pt)
{
  const double* r = Q.geom + (size_t)pt * NL_GEOM;
  NLGeom g;
  g.rc = r[0];
  g.dlnchi = r[1];
  g.dlnx = r[2];
  g.x0 = r[3];
  g.xlast = r[4];
  return g;
}

// ---- 1. forward transforms (cfftlog_ells_p1, cosmo2D.c:4047-4130): one
// CTA per (point, lens bin) for the radial kernels j in [j0, j1): the
// per-sample factors (a(chi), H, D, n_lens, f, b1) are formed once into
// shared memory in FP64, then each kernel is filled, transformed and
// windowed (FP64; FP32 in the mixed plan, whose spectra are FP32).
// unit_b1: the galaxy kernel with b1 = 1 (the adjoint pass differentiates
// the linear-bias factor out of it; bias model 0 only).
template <typename T>
__global__ void __launch_bounds__(NL_NT) k_nl_forward(Params P, NLParams Q, int unit_b1, int j0, int j1)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int pt = blockIdx.x, q = blockIdx.y;
  const int tid = threadIdx.x;
  const cl2pt_nuisance& nu = P.nu[pt];
  const bool mag = nu.gb[4][q] != 0.0;  // the magnification kernel is read only with bmag != 0
  if (!mag && j1 > 2) j1 = 2;
  const int nchi = P.nl_nchi;
  const double* X = P.chi + (size_t)pt * P.chi_nz;
  const double* Gv = P.G + (size_t)pt * P.G_nz;
  const double g1 = G_at_d(P.G_z, Gv, P.G_nz, 0.0, nullptr);
  const double om = P.omega_m[pt];
  const NLGeom geo = nl_geom_rec(Q, pt);
  const double rc = geo.rc;
  cd* bufA = (cd*)smem_raw;
  cd* bufB = bufA + Q.nmax;
  // per sample: fx_j of the three kernels (0 outside the bin's z range)
  double* fx = (double*)(bufB + Q.nmax);  // [3][nchi]
  const double* glens = P.glens + ((size_t)pt * P.nl + q) * P.n_a;
  const double amin_lensg = 1.0 / (P.lens_zmax_all + 1.0);
  const double lnx0 = log(geo.x0);
  for (int m = tid; m < nchi; m += NL_NT) {
    double f0 = 0.0, f1 = 0.0, f2 = 0.0;
    const double xq = geo.x0 * exp(geo.dlnchi * m);
    const double chi = xq / rc;
    const double a = a_chi_d(P.chi_z, X, P.chi_nz, chi);
    const double z = 1. / a - 1.;
    if (!(z < P.lens_zmin[q] || z > P.lens_zmax[q])) {
      const double H = 1.0 / ((a * a) * chi_all_d(P.chi_z, X, P.chi_nz, a).dchida);
      const double D = growfac_d(P.G_z, Gv, P.G_nz, g1, a);
      const double pf = nz_lens_d(P, z, q, nu.lens_dz[q], nu.lens_stretch[q]);
      if (j0 <= 0 && 0 < j1) {
        double b1;
        if (unit_b1) {
          b1 = 1.0;
        } else switch (P.bias_model[0]) {
          case 0: b1 = nu.gb[0][q]; break;
          case 1: b1 = nu.gb[0][q] * ((1.0 + z) / (1. + P.zmean_lens[q])); break;
          case 3: b1 = nu.gb[0][0] / growfac_d(P.G_z, Gv, P.G_nz, g1, 1. / (z + 1.)); break;
          case 4: b1 = nu.gb[0][0] * pow(1 + z, nu.gb[0][1]); break;
          default: {
            const double zev = growfac_d(P.G_z, Gv, P.G_nz, g1, 1. / (z + 1.)) /
                               growfac_d(P.G_z, Gv, P.G_nz, g1,
                                         1. / (1. + 0.5 * (P.lens_zmin[q] + P.lens_zmax[q])));
            b1 = (nu.gb[0][q] - 1.) / zev + 1.;
          }
        }
        f0 = chi * pf * D * H * b1;
      }
      if (j0 <= 1 && 1 < j1) f1 = -chi * pf * D * H * f_growth_d(P.G_z, Gv, P.G_nz, z);
      if (j1 > 2) {
        // W_mag with the coarse g_lens table (interpol1d)
        const double amax = 0.999999;
        const double dac = (amax - amin_lensg) / ((double)P.n_a - 1.0);
        const double gl = (a < amin_lensg || a > 1.0 - dac) ? 0.0 : interpol1d_d(glens, P.n_a, amin_lensg, dac, a);
        const double WM = (1.5 * om * chi / a) * gl;
        f2 = (WM / chi / (rc * rc)) * D;
      }
    }
    // divided by x^nu_j = exp(nu_j ln x), ln x = ln x0 + m dlnchi
    const double lnx = lnx0 + geo.dlnchi * m;
    fx[m] = (f0 != 0.0) ? f0 / exp(Q.nu[0] * lnx) : 0.0;
    fx[nchi + m] = (f1 != 0.0) ? f1 / exp(Q.nu[1] * lnx) : 0.0;
    fx[2 * nchi + m] = (f2 != 0.0) ? f2 / exp(Q.nu[2] * lnx) : 0.0;
  }
  for (int j = j0; j < j1; j++) {
    const int N = Q.N[j];
    const int halfN = N / 2;
    const int kmax = (int)(halfN * 0.25);
    ct<T>* tout = (ct<T>*)Q.tout + ((size_t)pt * P.nl + q) * Q.tout_stride;
    __syncthreads();
    if constexpr (sizeof(T) == sizeof(float)) {
      // mixed plan: the transform and the window in FP32 (the spectra are
      // stored in FP32 and the multipole loop transforms in FP32), in the
      // FP64 buffer's space
      ct<float>* fa = (ct<float>*)bufA;
      ct<float>* fb = fa + Q.nmax;
      for (int i = tid; i < N; i += NL_NT) {
        const int qq = i - Q.pad[j];
        fa[i] = tmk<float>((qq >= 0 && qq < nchi) ? (float)fx[j * nchi + qq] : 0.0f, 0.0f);
      }
      __syncthreads();
      const ct<float>* r = block_fft_t<float, -1>(fa, fb, Q.st[j], Q.nfac[j], (const ct<float>*)Q.twt[j]);
      const float ikmax = 1.0f / (float)kmax;
      for (int i = tid; i <= halfN; i += NL_NT) {
        ct<float> v = r[i];
        const int k = halfN - i;  // window on the right side
        if (k <= kmax) {
          const float x = (float)k * ikmax;
          const float W = x - sinf(6.28318530717958647692f * x) * 0.159154943091895335769f;
          v = tmk<float>(v.x * W, v.y * W);
        }
        tout[j * Q.hstride + i] = tmk<T>(v.x, v.y);
      }
      continue;
    }
    for (int i = tid; i < N; i += NL_NT) {
      const int qq = i - Q.pad[j];
      bufA[i] = cmk((qq >= 0 && qq < nchi) ? fx[j * nchi + qq] : 0.0, 0.0);
    }
    __syncthreads();
    const cd* r = (const cd*)block_fft_t<double, -1>((ct<double>*)bufA, (ct<double>*)bufB, Q.st[j], Q.nfac[j],
                                                     (const ct<double>*)Q.tw[j]);
    for (int i = tid; i <= halfN; i += NL_NT) {
      cd v = r[i];
      const int k = halfN - i;  // window on the right side
      if (k <= kmax) {
        const double W = (double)k / kmax - sin(2. * M_PI * k / kmax) / (2. * M_PI);
        v = cscale(v, W);
      }
      tout[j * Q.hstride + i] = tmk<T>((T)v.x, (T)v.y);
    }
  }
}

// Gamma part of g_l for the mixed plan's table (NLParams::gtab):
// T(eta) = (z - d) ln 2 + ln Gamma(w + 1) - ln Gamma(v), z = nu + i eta,
// w = (l + z - d) / 2, v = (3 + d + l - z) / 2, d the derivative order, so
// that g_l = exp(T) poly_d(z) / w with poly_0 = 1, poly_1 = -(z - 1),
// poly_2 = (z - 1)(z - 2) -- the factors with zeros or poles near eta = 0
// stay outside the interpolated part.
NL_HD cd gl_gamma_part(int deriv, double nu, double eta, int l)
{
  const cd w1 = cmk(0.5 * (l + nu - deriv) + 1.0, 0.5 * eta);
  const cd v = cmk(0.5 * (3 + deriv + l - nu), -0.5 * eta);
  return csub(cadd(cscale(cmk(nu - deriv, eta), log(2.)), lngamma_refl(w1)), lngamma_refl(v));
}

void nl_gamma_tables(const NLParams& Q, double inv_h, int m, std::vector<double>& out)
{
  out.assign((size_t)3 * 2 * m * 2, 0.0);
  for (int j = 0; j < 3; j++)
    for (int l = 0; l < 2; l++) {
      double* o = out.data() + (size_t)(j * 2 + l) * m * 2;
      double prev = 0.0;
      for (int i = 0; i < m; i++) {
        const cd t = gl_gamma_part(Q.deriv[j], Q.nu[j], (i - 3) / inv_h, l);
        double im = t.y;
        // continuous imaginary part (steps of ~0.2 rad between entries)
        if (i) im += 2 * M_PI * nearbyint((prev - im) / (2 * M_PI));
        o[2 * i] = t.x;
        o[2 * i + 1] = im;
        prev = im;
      }
    }
}

// g_l at eta from the table tb = NLParams::gtab + (j, l): 6-point Lagrange
// interpolation of T in FP64, then exp(T) and the rational factor in FP32
// (the loop consumes g in FP32).  nu1 = nu - 1 in FP32.  false: eta beyond
// the table.
__device__ __forceinline__ bool gl_table(const NLParams& Q, const double* __restrict__ tb, int deriv, float nu1,
                                         int l, double eta, ct<float>* g)
{
  const double u = eta * Q.gtab_inv_h + 3.0;
  const int m = (int)u;
  if (m < 2 || m + 3 >= Q.gtab_m) return false;
  const double t = u - (double)m;
  const double e0 = t + 2.0, e1 = t + 1.0, e2 = t, e3 = t - 1.0, e4 = t - 2.0, e5 = t - 3.0;
  const double p01 = e0 * e1, p23 = e2 * e3, p45 = e4 * e5;
  // w_a = prod_{b != a} (t - b) / prod_{b != a} (a - b), nodes a = -2..3
  const double w[6] = {e1 * p23 * p45 * (-1.0 / 120.0), e0 * p23 * p45 * (1.0 / 24.0),
                       p01 * e3 * p45 * (-1.0 / 12.0),  p01 * e2 * p45 * (1.0 / 12.0),
                       p01 * p23 * e5 * (-1.0 / 24.0),  p01 * p23 * e4 * (1.0 / 120.0)};
  const double2* r = (const double2*)tb + (m - 2);
  double re = 0.0, im = 0.0;
#pragma unroll
  for (int a = 0; a < 6; a++) {
    const double2 v = __ldg(r + a);
    re = fma(w[a], v.x, re);
    im = fma(w[a], v.y, im);
  }
  const double ph = im - 2.0 * M_PI * rint(im * (0.5 / M_PI));
  float sn, cs;
  sincosf((float)ph, &sn, &cs);
  const float mag = expf((float)re);
  const float et = (float)eta;
  ct<float> poly;
  if (deriv == 0) poly = tmk<float>(1.0f, 0.0f);
  else if (deriv == 1) poly = tmk<float>(-nu1, -et);
  else poly = tmk<float>(nu1 * (nu1 - 1.0f) - et * et, et * (2.0f * nu1 - 1.0f));
  // poly / w, w = (l + 1 + nu1 - d + i eta) / 2
  const float wr = 0.5f * ((float)(l + 1 - deriv) + nu1), wi = 0.5f * et;
  const float rw = 1.0f / (wr * wr + wi * wi);
  const ct<float> fac = tmk<float>((poly.x * wr + poly.y * wi) * rw, (poly.y * wr - poly.x * wi) * rw);
  *g = tmul(tmk<float>(mag * cs, mag * sn), fac);
  return true;
}

// ---- 2. Gamma-ratio kernels at the multipoles where the recurrence
// (re)starts: l = 0, 1 in the mixed plan, from the plan's tables of their
// Gamma part (gl_table; entries beyond the tables directly); the first two
// multipoles of every 16-block in the FP64 plan, as the reference does,
// evaluated directly (Lanczos, FP64).  One CTA per (point, radial kernel,
// start multipole).
__global__ void __launch_bounds__(NL_NT) k_nl_gdirect(Params P, NLParams Q)
{
  const int pt = blockIdx.x, j = blockIdx.y, d = blockIdx.z;
  const int k = Q.direct_every ? (d / 2) * 16 + (d & 1) : d;
  if (k >= P.lmax_nolimber) return;
  if (j == 2) {
    // the magnification kernel is read only by bins with magnification bias
    if (!Q.any_mag[pt]) return;
  }
  const NLGeom geo = nl_geom_rec(Q, pt);
  const int N = Q.N[j];
  const int nq = N / 2 + 1;
  const double deta = 2.0 * M_PI / (geo.dlnx * N);
  double* out = Q.gdir + (((size_t)pt * 3 + j) * Q.ndirect + d) * Q.hstride * 2;
  const double* tb = (Q.gtab && k < 2) ? Q.gtab + (size_t)(j * 2 + k) * Q.gtab_m * 2 : nullptr;
  for (int i = threadIdx.x; i < nq; i += NL_NT) {
    ct<float> gf;
    if (tb && gl_table(Q, tb, Q.deriv[j], Q.nu1f[j], k, deta * i, &gf)) {
      out[2 * i] = f32_to_f64_int(gf.x);
      out[2 * i + 1] = f32_to_f64_int(gf.y);
      continue;
    }
    const cd g = gl_direct(Q.deriv[j], Q.nu[j], deta * i, k);
    out[2 * i] = g.x;
    out[2 * i + 1] = g.y;
  }
}

// g_k / g_{k-2} at eta = deta i (the two-step recurrence): fi = i as a
// float, (dh, dl) deta as an FP32 head/tail (FP32), deta (FP64)
template <typename T>
__device__ __forceinline__ ct<T> nl_ratio(const NLParams& Q, int j, int i, float fi, int k, double deta, float dh,
                                          float dl)
{
  T et;
  if constexpr (sizeof(T) == sizeof(float)) {
    et = fmaf(dh, fi, dl * fi);
  } else {
    et = deta * i;
  }
  const T kk = (T)k;
  T nuj;
  if constexpr (sizeof(T) == sizeof(float)) nuj = Q.nuf[j];  // no FP64 conversion per entry
  else nuj = Q.nu[j];
  ct<T> num, den;
  if (Q.deriv[j] == 0) { num = tmk<T>(kk - 2 + nuj, et); den = tmk<T>(kk + 1 - nuj, -et); }
  else if (Q.deriv[j] == 1) { num = tmk<T>(kk - 3 + nuj, et); den = tmk<T>(kk + 2 - nuj, -et); }
  else { num = tmk<T>(kk - 4 + nuj, et); den = tmk<T>(kk + 3 - nuj, -et); }
  if constexpr (sizeof(T) == sizeof(float)) {
    // num / den = num conj(den) / |den|^2: one reciprocal instead of
    // Smith's two divisions (|den| >= k + 1 - nu >= 2 at the recurrence's
    // multipoles k >= 2; |den|^2 stays far inside the FP32 range)
    const float r = __frcp_rn(fmaf(den.x, den.x, den.y * den.y));
    return tmk<T>((num.x * den.x + num.y * den.y) * r, (num.y * den.x - num.x * den.y) * r);
  } else {
    return tdiv(num, den);
  }
}

// exp(i a) for an FP64 angle, reduced to [-pi, pi] in FP64
template <typename T>
__device__ __forceinline__ ct<T> phasor(double a)
{
  a -= 2.0 * M_PI * rint(a * (0.5 / M_PI));
  T sp, cp;
  tsincos<T>((T)a, &sp, &cp);
  return tmk<T>(cp, sp);
}

// FP32 head/tail of an angle reduced to [-pi, pi] in FP64
__device__ __forceinline__ float2 red_angle(double a)
{
  a -= 2.0 * M_PI * rint(a * (0.5 / M_PI));
  const float h = (float)a;
  return make_float2(h, (float)(a - (double)h));
}

// x^nu (nu = 1 or 1.01) and, for magnification, x^2 more (l10x = log10(x)
// in units of Mpc/h, FP64 only)
template <typename T>
__device__ __forceinline__ T nl_power(const NLParams& Q, int j, T x, double l10x)
{
  T xp = x;
  if constexpr (sizeof(T) == sizeof(float)) {
    const float num1f = Q.nu1f[j];
    if (num1f != 0.0f) xp *= __expf(num1f * __logf(x));
  } else {
    const double num1 = Q.nu[j] - 1.0;
    if (num1 != 0.0) xp *= texp<T>((T)(num1 * l10x * 2.302585092994045684));
  }
  if (j == 2) xp *= x * x;
  return xp;
}

// Per point, what every lens-bin CTA of the loop would otherwise repeat:
// the z = 0 slice P_lin(k_i, z = 0) of the linear table (p_lin(k, 1),
// cosmo3D.c:306-358, linear in z between the table's two columns around
// z = 0) as a contiguous row (the table is k-major, so the column is a
// strided gather), and in the mixed plan the phase increments of every
// (radial kernel, multipole) (NLParams::phase) -- FP64 work that one
// thread of each loop CTA used to do while the others waited.
__global__ void __launch_bounds__(256) k_nl_slice(Params P, NLParams Q)
{
  const int pt = blockIdx.x;
  const int j0 = bsearch_d(P.pkl_z, P.pkl_nz, 0.0);
  const double dy = (0.0 - P.pkl_z[j0]) / (P.pkl_z[j0 + 1] - P.pkl_z[j0]);
  const double* tabL = P.lnPL + (size_t)pt * P.pkl_nk * P.pkl_nz;
  double* out = Q.pslice + (size_t)pt * P.pkl_nk;
  for (int i = threadIdx.x; i < P.pkl_nk; i += blockDim.x)
    out[i] = (1 - dy) * tabL[(size_t)i * P.pkl_nz + j0] + dy * tabL[(size_t)i * P.pkl_nz + j0 + 1];
  const NLGeom geo = nl_geom(P, pt);
  const int nchi = P.nl_nchi, nk = P.pkl_nk;
  if (threadIdx.x == 0) {
    double* r = Q.geom + (size_t)pt * NL_GEOM;
    r[0] = geo.rc;
    r[1] = geo.dlnchi;
    r[2] = geo.dlnx;
    r[3] = geo.x0;
    r[4] = geo.xlast;
    // no block of this point's bins has converged
    for (int q = 0; q < P.nl; q++) Q.conv_blk[(size_t)pt * P.nl + q] = NL_OPEN;
    int any = 0;
    for (int q = 0; q < P.nl; q++) any |= P.nu[pt].gb[4][q] != 0.0;
    Q.any_mag[pt] = any;
  }
  const double lnx0last = log(geo.x0 / geo.xlast);
  const int LNL = P.lmax_nolimber;
  // (rc / x)^3, log10(rc / (x coverH0)) and the kernels' powers of x at the
  // reversed index nchi-1-i (y = (l+1)/x[nchi-1-i])
  for (int i = threadIdx.x; i < nchi; i += blockDim.x) {
    const double x = geo.x0 * exp(geo.dlnchi * (nchi - 1 - i));
    const double lx = log10(geo.rc / (x * CL2PT_COVERH0));
    if (Q.phase) {
      float* xs = (float*)Q.xtab + (size_t)pt * NL_XROWS * nchi;
      const float rx = (float)geo.rc / (float)x;
      xs[i] = rx * rx * rx;
      xs[nchi + i] = (float)lx;
      for (int j = 0; j < 3; j++) xs[(2 + j) * nchi + i] = nl_power<float>(Q, j, (float)x, 0.0);
    } else {
      double* xs = (double*)Q.xtab + (size_t)pt * NL_XROWS * nchi;
      const double rx = geo.rc / x;
      xs[i] = rx * rx * rx;
      xs[nchi + i] = lx;
      for (int j = 0; j < 3; j++)
        xs[(2 + j) * nchi + i] = nl_power<double>(Q, j, x, log10(geo.rc / CL2PT_COVERH0) - lx);
    }
  }
  if (Q.phase) {
    for (int e = threadIdx.x; e < 3 * LNL; e += blockDim.x) {
      const int j = e / LNL, k = e - j * LNL;
      const double deta = 2.0 * M_PI / (geo.dlnx * Q.N[j]);
      const double lnbj = lnx0last - 2 * Q.pad[j] * geo.dlnx;
      Q.phase[((size_t)pt * 3 + j) * LNL + k] = red_angle(deta * (lnbj + Q.lnk1[k]));
    }
    // the slice's cells (head, tail, 1 / width of the FP32 axis, slope)
    __syncthreads();
    for (int i = threadIdx.x; i < nk; i += blockDim.x) {
      const double v = out[i];
      const float h = (float)v;
      float4 c = make_float4(h, (float)(v - (double)h), 0.0f, 0.0f);
      if (i + 1 < nk) {
        // the cell width of the FP32 axis, so dx = 1 at the upper edge
        c.z = 1.0f / ((float)P.pkl_lk[i + 1] - (float)P.pkl_lk[i]);
        c.w = (float)(out[i + 1] - v);
      }
      Q.pcell[(size_t)pt * nk + i] = c;
    }
  }
}

// exp(-i m theta) for theta = th.x + th.y in [-pi, pi] and integer m = fm
// in [0, 2^15),
// without FP64: m theta as an exact two-float product, reduced by 2 pi in
// three parts (Cody-Waite; m th.x / 2 pi < 2^14, so n C1 and p - n C1 are
// exact), then sincosf of the reduced angle (~2e-7 rad from the exact one)
__device__ __forceinline__ ct<float> phase_f(float fm, float2 th)
{
  constexpr float C1 = 6.28125f;
  constexpr float C2 = (float)(6.283185307179586476925 - 6.28125);
  constexpr float C3 = (float)(6.283185307179586476925 - 6.28125 - (double)C2);
  const float p = fm * th.x;
  const float e = fmaf(fm, th.x, -p);
  const float n = rintf(p * 0.159154943091895335769f);
  float r = fmaf(-n, C1, p);
  r = fmaf(-n, C2, r);
  r = fmaf(-n, C3, r);
  r += e + fm * th.y;
  float sn, cs;
  sincosf(r, &sn, &cs);
  return tmk<float>(cs, -sn);
}

// Cell of the z = 0 slice's FP32 log10 k axis (the bracketing search's
// answer: largest i <= nk - 2 with plk[i] <= v, else 0) from a table of
// the cells at NL_LUT(nk) equally spaced values, walked up or down to the
// exact cell -- a step or two on the usual log-spaced axes instead of the
// ~10 dependent steps of the search.  scale = (NL_LUT - 1) / (plk[nk-1] -
// plk[0]); the rounding to the nearest table entry is integer arithmetic
// (0 <= u < 2^22), not a conversion.
__device__ __forceinline__ int slice_cell(const float* __restrict__ plk, int nk, const unsigned short* lut,
                                          float scale, float umax, float v)
{
  const float u = fminf(fmaxf((v - plk[0]) * scale, 0.0f), umax);
  int lo = lut[__float_as_int(u + 12582912.0f) - 0x4B400000];
  while (lo < nk - 2 && plk[lo + 1] <= v) lo++;
  while (lo > 0 && plk[lo] > v) lo--;
  return lo;
}

// ---- 3a. phases and Gamma kernels of every multipole of a chunk: with the
// spectra of the radial kernels these are all that the transforms of the
// multipole blocks read, and they depend on the point's geometry alone, so
// they are formed once per point instead of once per (point, lens bin):
//   ctab [pt][l - l0][.]  exp(-i eta_i ln base) of every radial kernel
//   gtabl[pt][l - l0][.]  g_l(eta_i); the last two multipoles of a chunk are
//                         kept in gcar for the next chunk
// (the kernels' entries follow one another at Q.qoff).  FP32: the phase of
// entry i is a rotation of the phase of i mod nlt, nlt the threads of a block
// CTA.
//   ptab [pt][l - l0][i]  p_lin(k, 1) at the chi samples.
// grid (point, role): roles [0, 3 nc) the phases of (kernel, nc parts
// of the multipoles), then the Gamma kernels by (kernel, parity or block,
// part of the entries), then p_lin by nc parts of the multipoles.
constexpr int NLC_NT = 128, NLC_PART = 8;
// p_lin(k, 1) (cosmo3D.c:306-358) at the chi samples of multipoles l0 + part,
// + parts, ... of a chunk, from the z = 0 slice
template <typename T>
__device__ __forceinline__ void nl_ptab(const Params& P, const NLParams& Q, int pt, int l0, int l1, int part, int parts)
{
  const int nchi = P.nl_nchi, nk = P.pkl_nk;
  const T lc3 = (T)(1.0 / (CL2PT_COVERH0 * CL2PT_COVERH0 * CL2PT_COVERH0));
  T* out = (T*)Q.ptab + (size_t)pt * Q.lchunk * nchi;
  if constexpr (sizeof(T) == sizeof(float)) {
    const double* geom = Q.geom + (size_t)pt * NL_GEOM;
    // log10(rc / (x coverH0)) at the reversed index = lx0 + i lx1
    const double lx1d = geom[1] * 0.434294481903251827651;  // dlnchi log10(e)
    const float lx0f = (float)(log10(geom[0] / (geom[3] * CL2PT_COVERH0)) - (nchi - 1) * lx1d);
    const float lx1f = (float)lx1d;
    const float4* pcf = Q.pcell + (size_t)pt * nk;
    const float step = (float)NLC_NT;
    for (int l = l0 + part; l < l1; l += parts) {
      const float lk = Q.l10k1f[l];
      float fi = (float)threadIdx.x;  // i as a float, counted (no conversion per entry)
      for (int i = threadIdx.x; i < nchi; i += NLC_NT, fi += step) {
        const float lkt = lk + fmaf(fi, lx1f, lx0f);
        const int lo = slice_cell(Q.plkf, nk, Q.lut, Q.lscale, Q.lumax, lkt);
        // in-cell offset and exponent in FP32 from the per-cell split (head,
        // tail) of the slice, the slope from the cell's ends (lo <= nk - 2)
        const float4 c = pcf[lo], c1 = pcf[lo + 1];
        const float dx = (lkt - Q.plkf[lo]) * c.z;
        const float slope = (c1.x - c.x) + (c1.y - c.y);
        const float del = c.y + dx * slope;
        out[(size_t)(l - l0) * nchi + i] = __expf(c.x) * __expf(del) * lc3;
      }
    }
  } else {
    const double* lxk = (const double*)Q.xtab + ((size_t)pt * NL_XROWS + 1) * nchi;
    const double* psl = Q.pslice + (size_t)pt * nk;
    for (int l = l0 + part; l < l1; l += parts)
      for (int i = threadIdx.x; i < nchi; i += NLC_NT) {
        const double lkv = Q.l10k1[l] + lxk[i];
        const int lo = bsearch_d(P.pkl_lk, nk, lkv);
        const double dxd = (lkv - P.pkl_lk[lo]) * Q.pinv[lo];
        out[(size_t)(l - l0) * nchi + i] = exp(psl[lo] + dxd * (psl[lo + 1] - psl[lo])) * lc3;
      }
  }
}
template <typename T>
__global__ void __launch_bounds__(NLC_NT) k_nl_cg(Params P, NLParams Q, int l0, int l1, int nlt, int nc, int ng)
{
  const int pt = blockIdx.x, tid = threadIdx.x;
  constexpr bool F32 = sizeof(T) == sizeof(float);
  int role = blockIdx.y;
  if (role >= 3 * (nc + ng)) {
    nl_ptab<T>(P, Q, pt, l0, l1, role - 3 * (nc + ng), nc);
    return;
  }
  const bool phases = role < 3 * nc;
  if (!phases) role -= 3 * nc;
  const int per = phases ? nc : ng;
  const int j = role / per, part = role - j * per;
  if (j == 2 && !Q.any_mag[pt]) return;
  if (l0 > 0) {
    // a later chunk: nothing to do once every bin of the point converged
    bool open = false;
    for (int q = 0; q < P.nl; q++) open |= Q.conv_blk[(size_t)pt * P.nl + q] >= l0 / 16;
    if (!open) return;
  }
  const NLGeom geo = nl_geom_rec(Q, pt);
  const int N = Q.N[j], nq = N / 2 + 1, LNL = P.lmax_nolimber;
  const double deta = 2.0 * M_PI / (geo.dlnx * N);
  const size_t row = Q.qs;
  if (phases) {
    ct<T>* out = (ct<T>*)Q.ctab + (size_t)pt * Q.lchunk * row + Q.qoff[j];
    for (int l = l0 + part; l < l1; l += nc) {
      ct<T>* o = out + (size_t)(l - l0) * row;
      if constexpr (F32) {
        const float2 th = Q.phase[((size_t)pt * 3 + j) * LNL + l];
        const ct<float> s = phase_f((float)nlt, th);
        for (int t = tid; t < nlt; t += NLC_NT) {
          ct<float> e = phase_f((float)t, th);
          for (int i = t; i < nq; i += nlt) {
            o[i] = e;
            e = tmul(e, s);
          }
        }
      } else {
        const double lnb = log(geo.x0 / geo.xlast) - 2 * Q.pad[j] * geo.dlnx + Q.lnk1[l];
        for (int i = tid; i < nq; i += NLC_NT) o[i] = phasor<T>(-(deta * i) * lnb);
      }
    }
    return;
  }
  const float dh = (float)deta, dl = (float)(deta - (double)dh);
  ct<T>* out = (ct<T>*)Q.gtabl + (size_t)pt * Q.lchunk * row + Q.qoff[j];
  const double* gd = Q.gdir + ((size_t)pt * 3 + j) * Q.ndirect * Q.hstride * 2;
  if constexpr (F32) {
    // part = (entries' part) * 2 + parity: the recurrence from l = 0, 1
    const int par = part & 1;
    const int i = (part >> 1) * NLC_NT + tid;
    if (i >= nq) return;
    ct<float>* car = (ct<float>*)Q.gcar + (size_t)pt * 2 * row + Q.qoff[j];
    ct<float> g = tmk<float>(0.0f, 0.0f);
    if (l0 > 0) g = car[(size_t)par * row + i];
    for (int l = l0 + par; l < l1; l += 2) {
      if (l < 2) {
        const double* gk = gd + (size_t)l * Q.hstride * 2;
        g = tmk<float>((float)gk[2 * i], (float)gk[2 * i + 1]);
      } else {
        g = tmul(g, nl_ratio<float>(Q, j, i, (float)i, l, deta, dh, dl));
      }
      out[(size_t)(l - l0) * row + i] = g;
    }
    car[(size_t)par * row + i] = g;
  } else {
    // part = block of 16 multipoles: restarted from its first two
    const int ks = l0 + part * 16, ke = min(ks + 16, l1);
    for (int i = tid; i < nq; i += NLC_NT)
      for (int h = 0; h < 2; h++) {
        ct<double> g = tmk<double>(0.0, 0.0);
        for (int l = ks + h; l < ke; l += 2) {
          if (l < ks + 2) {
            const double* gk = gd + (size_t)((ks / 16) * 2 + h) * Q.hstride * 2;
            g = tmk<double>(gk[2 * i], gk[2 * i + 1]);
          } else {
            g = tmul(g, nl_ratio<double>(Q, j, i, 0.0f, l, deta, dh, dl));
          }
          out[(size_t)(l - l0) * row + i] = g;
        }
      }
  }
}

// The multiply-add forms of the spectra are fixed by intrinsics: the C_l
// below the hand-over are differences of FP32 sums of these, so a compiler's
// choice of the fused product would show at their rounding level.
__device__ __forceinline__ float r_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double r_add(double a, double b) { return a + b; }
__device__ __forceinline__ float r_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double r_sub(double a, double b) { return a - b; }
// FP64 to the loop precision, to nearest, without a conversion instruction
template <typename T> __device__ __forceinline__ T narrow(double v);
template <> __device__ __forceinline__ float narrow<float>(double v) { return split_f64_bits(v).x; }
template <> __device__ __forceinline__ double narrow<double>(double v) { return v; }
__device__ __forceinline__ double wide64(float a) { return f32_to_f64_int(a); }
__device__ __forceinline__ double wide64(double a) { return a; }
__device__ __forceinline__ float fma_t(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }
// (t c) g
__device__ __forceinline__ ct<float> nl_term(ct<float> t, ct<float> c, ct<float> g)
{
  const float ux = __fmaf_rn(t.x, c.x, -__fmul_rn(t.y, c.y)), uy = __fmaf_rn(t.x, c.y, __fmul_rn(t.y, c.x));
  return tmk<float>(__fmaf_rn(ux, g.x, -__fmul_rn(uy, g.y)), __fmaf_rn(uy, g.x, __fmul_rn(ux, g.y)));
}
__device__ __forceinline__ ct<double> nl_term(ct<double> t, ct<double> c, ct<double> g) { return tmul(tmul(t, c), g); }


// ---- 3b. multipole blocks (cfftlog_ells_p2 + C_cl_tomo sums and
// convergence, cosmo2D.c:4132-4769) in the loop precision T: one CTA per
// (point, bin) and block of 16 multipoles.  Two consecutive multipoles share
// one complex inverse transform: both outputs are real, so the spectrum
// X_k + i X_{k+1} (each Hermitian-completed) transforms to x_k + i x_{k+1}.
// The blocks of a (point, bin) are independent but for the stop at the first
// converged one, so they run on as many SMs as there are: the grid holds
// the blocks of all (point, bin) pairs lowest block first, and a CTA whose
// pair has already converged in a lower block returns at once.  A block that
// runs ahead of that only writes entries that k_nl_handover replaces.
// Bound by issue and barrier latency of small transforms (900-3072 points);
// the per-point tables keep the shared layout to the two FFT buffers and
// the radial sums, so more CTAs share an SM.
// the c2r scales of kernel j at multipoles k, k2
template <typename T>
__device__ __forceinline__ void nl_scales(const NLParams& Q, int j, int k, int k2, int LNL, T* sc0, T* sc1)
{
  if constexpr (sizeof(T) == sizeof(float)) {
    *sc0 = Q.sckf[j * LNL + k];
    *sc1 = Q.sckf[j * LNL + k2];
  } else {
    *sc0 = (T)Q.sck[j * LNL + k];
    *sc1 = (T)Q.sck[j * LNL + k2];
  }
}

// DFT_R of v with only the outputs wanted: emit(r, o_r) for every r with
// need(r).  The sums are dft_odd's, in its order.
template <typename T, int R, int SIGN, typename N, typename E>
__device__ __forceinline__ void dft_some(const ct<T>* vin, N need, E emit)
{
  ct<T> v[R];
#pragma unroll
  for (int r = 0; r < R; r++) v[r] = vin[r];
  if constexpr (R == 2 || R == 4 || sizeof(T) == sizeof(double)) {
    if constexpr (R == 2) dft2(v);
    else if constexpr (R == 4) dft4<T, SIGN>(v);
    else dft_odd<T, R, SIGN>(v);
#pragma unroll
    for (int r = 0; r < R; r++)
      if (need(r)) emit(r, v[r]);
  } else {
    if (need(0)) {
      ct<T> o = v[0];
#pragma unroll
      for (int r = 1; r < R; r++) o = tadd(o, v[r]);
      emit(0, o);
    }
#pragma unroll
    for (int t = 1; t <= R / 2; t++) {
      if (!need(t) && !need(R - t)) continue;
      ct<T> a = v[0], b = v[0];
#pragma unroll
      for (int r = 1; r < R; r++) {
        const float wr = (float)root_c<R>((r * t) % R), wi = SIGN * (float)root_s<R>((r * t) % R);
        const float m1 = __fmul_rn(v[r].y, wi), m2 = __fmul_rn(v[r].x, wi);
        a.x = __fadd_rn(a.x, __fmaf_rn(v[r].x, wr, -m1));
        a.y = __fadd_rn(a.y, __fmaf_rn(v[r].y, wr, m2));
        b.x = __fadd_rn(b.x, __fmaf_rn(v[r].x, wr, m1));
        b.y = __fadd_rn(b.y, __fmaf_rn(v[r].y, wr, -m2));
      }
      if (need(t)) emit(t, a);
      if (need(R - t)) emit(R - t, b);
    }
  }
}

// entry i <= N / 2 of X_k + i X_{k+1} (nl_term of both multipoles, conjugated)
// and its mirror N - i; lone: i = 0 or N / 2, where Hermitian spectra are real
template <typename T>
__device__ __forceinline__ void nl_pair(const NLParams& Q, int i, bool lone, const ct<T>* __restrict__ tj,
                                        const ct<T>* __restrict__ c, const ct<T>* __restrict__ g, bool two, ct<T>& d,
                                        ct<T>& m)
{
  const ct<T> tv = tj[i];
  const ct<T> v0 = nl_term(tv, c[i], g[i]);
  const ct<T> v1 = two ? nl_term(tv, c[Q.qs + i], g[Q.qs + i]) : tmk<T>((T)0, (T)0);
  d = lone ? tmk<T>(v0.x, v1.x) : tmk<T>(r_add(v0.x, v1.y), r_sub(v1.x, v0.y));
  m = tmk<T>(r_sub(v0.x, v1.y), r_add(v1.x, v0.y));
}

// The spectrum in natural order, for sizes whose first radix is odd (the size
// rule, next 7-smooth even number tried twice, leaves 735, 1225, 1715, 2205,
// 3125, 3675 for some radial grids): entries i and N - i by one thread.
template <typename T, int NT>
__device__ __forceinline__ void nl_spectrum(const NLParams& Q, int j, ct<T>* __restrict__ out,
                                            const ct<T>* __restrict__ tj, const ct<T>* __restrict__ c,
                                            const ct<T>* __restrict__ g, bool two)
{
  const int N = Q.N[j];
  for (int i = threadIdx.x; 2 * i <= N; i += NT) {
    const bool lone = i == 0 || 2 * i == N;
    ct<T> d, m;
    nl_pair<T>(Q, i, lone, tj, c, g, two, d, m);
    out[i] = d;
    if (!lone) out[N - i] = m;
  }
}

// First stage (radix R = 2 or 4, no twiddles) with the spectrum formed in
// registers: butterflies jb and NR - jb read each other's mirrored entries, so
// one thread takes both.
template <typename T, int R, int NT>
__device__ __forceinline__ void nl_first(const NLParams& Q, int j, ct<T>* __restrict__ out,
                                         const ct<T>* __restrict__ tj, const ct<T>* __restrict__ c,
                                         const ct<T>* __restrict__ g, bool two)
{
  const int N = Q.N[j], NR = N / R;
  for (int jb = threadIdx.x; 2 * jb <= NR; jb += NT) {
    ct<T> x[R], y[R];
    const bool self = jb == 0 || 2 * jb == NR;  // its own mirror
    if (!self) {
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int i = jb + r * NR;
        const bool up = 2 * i > N;
        ct<T> d, m;
        nl_pair<T>(Q, up ? N - i : i, false, tj, c, g, two, d, m);
        x[r] = up ? m : d;
        y[R - 1 - r] = up ? d : m;
      }
    } else {
      // entries r NR (mirror slot R - r), or (r + 1/2) NR (slot R - 1 - r)
      const bool zero = jb == 0;
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int mr = zero ? (R - r) % R : R - 1 - r;
        if (r > mr) continue;
        ct<T> d, m;
        nl_pair<T>(Q, jb + r * NR, r == mr, tj, c, g, two, d, m);
#pragma unroll
        for (int q = 0; q < R; q++) {
          if (q == mr && q != r) x[q] = m;
          if (q == r) x[q] = d;
        }
      }
#pragma unroll
      for (int r = 0; r < R; r++) y[r] = x[r];
    }
    if constexpr (R == 2) { dft2(x); dft2(y); }
    else { dft4<T, 1>(x); dft4<T, 1>(y); }
    ct<T>* o = out + jb * R;
#pragma unroll
    for (int r = 0; r < R; r++) o[r] = x[r];
    if (!self) {
      o = out + (NR - jb) * R;
#pragma unroll
      for (int r = 0; r < R; r++) o[r] = y[r];
    }
  }
}

// Last stage (Ns = NR, one block): emit(i, z) for the chi samples i of
// the result, which starts at pad
template <typename T, int R, int NT, typename E>
__device__ __forceinline__ void nl_last(const ct<T>* __restrict__ in, int NR, int pad, int nchi,
                                        const ct<T>* __restrict__ tw, E emit)
{
  for (int k = threadIdx.x; k < NR; k += NT) {
    ct<T> v[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
      ct<T> x = in[k + r * NR];
      if (r && k) x = tmul(x, tw[(r - 1) * NR + k]);
      v[r] = x;
    }
    auto need = [&](int r) { return (unsigned)(k + r * NR - pad) < (unsigned)nchi; };
    dft_some<T, R, 1>(v, need, [&](int r, ct<T> z) { emit(k + r * NR - pad, z); });
  }
}

// The transform of kernel j for the multipoles k, k + 1 of a pair: spectrum
// and first stage in registers, the middle stages over shared memory, and of
// the last stage only the chi samples, handed to emit(i, z) as they are
// formed.  A stage of its own for the spectrum and another for the samples
// cost two more passes over shared memory and two barriers of seven.  With
// the twiddles in reading order, p_lin and the powers of x from per-point
// tables, and the FP64 end of a block at once, k_nl_block took 3.42 -> 2.02 ms
// at 512 points of real_3x2pt and 24.6 -> 13.2 ms at 512 of fourier_serving
// (500 and 2048 chi samples); bound now by the latency of the table loads and
// barriers at 24 warps an SM.
// fa: the buffer to write first; on return the buffer that the last stage did
// not read (free at once: its last readers are a barrier behind).  Emitted
// values are other threads' to read only after a barrier.
// ODD: a kernel's first radix may be odd (nl_spectrum); a template parameter,
// because the branch cost the usual sizes 2 % of k_nl_block.
template <typename T, int NT, bool ODD, typename E>
__device__ __forceinline__ void nl_transform(const NLParams& Q, int j, int nchi, ct<T>*& fa, ct<T>*& fb,
                                             const ct<T>* __restrict__ tj, const ct<T>* __restrict__ c,
                                             const ct<T>* __restrict__ g, bool two, E emit)
{
  const NLStage* st = Q.st[j];
  const int nf = Q.nfac[j];
  const ct<T>* tw = (const ct<T>*)Q.twt[j];
  const int first = ODD ? (st[0].R == 4 || st[0].R == 2) : 1;
  if (ODD && !first) nl_spectrum<T, NT>(Q, j, fa, tj, c, g, two);
  else if (st[0].R == 4) nl_first<T, 4, NT>(Q, j, fa, tj, c, g, two);
  else nl_first<T, 2, NT>(Q, j, fa, tj, c, g, two);
  __syncthreads();
  const ct<T>* r = block_fft_t<T, 1>(fa, fb, st + first, nf - 1 - first, tw);
  if (r == fa) {
    fa = fb;
    fb = (ct<T>*)r;
  }
  const NLStage& S = st[nf - 1];
  switch (S.R) {
    case 2: nl_last<T, 2, NT>(r, S.NR, Q.pad[j], nchi, tw + S.off, emit); break;
    case 3: nl_last<T, 3, NT>(r, S.NR, Q.pad[j], nchi, tw + S.off, emit); break;
    case 4: nl_last<T, 4, NT>(r, S.NR, Q.pad[j], nchi, tw + S.off, emit); break;
    case 5: nl_last<T, 5, NT>(r, S.NR, Q.pad[j], nchi, tw + S.off, emit); break;
    default: nl_last<T, 7, NT>(r, S.NR, Q.pad[j], nchi, tw + S.off, emit); break;
  }
}

template <typename T, int NT, int MINB, bool ODD>
__global__ void __launch_bounds__(NT, MINB) k_nl_block(Params P, NLParams Q, int l0, int l1)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int item = blockIdx.x;
  const int blk = l0 / 16 + blockIdx.y;
  const int tid = threadIdx.x;
  constexpr int nlt = NT;
  __shared__ int skip;
  if (tid == 0) skip = *(volatile int*)&Q.conv_blk[item] < blk;
  __syncthreads();
  if (skip) return;
  const int pt = item / P.nl, q = item - (item / P.nl) * P.nl;
  const int nchi = P.nl_nchi, LNL = P.lmax_nolimber;
  const double bmag = P.nu[pt].gb[4][q];
  const int nj = (bmag != 0.0) ? 3 : 2;
  ct<T>* fa = (ct<T>*)smem_raw;
  ct<T>* fb = fa + Q.nmax;
  T* F0 = (T*)(fb + Q.nmax);
  T* F1 = F0 + nchi;
  __shared__ T red[16][NT / 32];
  const double dlnchi = Q.geom[(size_t)pt * NL_GEOM + 1];
  const T* xt = (const T*)Q.xtab + (size_t)pt * NL_XROWS * nchi;        // (rc / x)^3
  const T* xpt = xt + 2 * nchi;                                         // [3] the kernels' powers of x
  const T* ptab = (const T*)Q.ptab + (size_t)pt * Q.lchunk * nchi;
  const ct<T>* tout = (const ct<T>*)Q.tout + (size_t)item * Q.tout_stride;  // [3][hstride]
  const ct<T>* ctab = (const ct<T>*)Q.ctab + (size_t)pt * Q.lchunk * Q.qs;
  const ct<T>* gtab = (const ct<T>*)Q.gtabl + (size_t)pt * Q.lchunk * Q.qs;
  double* Cl = P.cnl + (size_t)item * LNL;
  const double* ggl = P.ggl + (size_t)item * LNL * 2;
  const T bmagt = (T)bmag;
  const int ks = blk * 16, ke = min(ks + 16, l1);
  T kf = (T)ks;  // k as a float, counted: conversions issue at the FP64 rate
  for (int k = ks; k < ke; k += 2, kf += (T)2) {
    const int k2 = k + 1;
    const bool two = k2 < ke;
    const T kp0 = kf + (T)1, kp1 = kf + (T)2;
    // bmag l(l+1)/(l+1)^2 = bmag l/(l+1)
    const T mag0 = bmagt * kf / kp0;
    const T mag1 = bmagt * kp0 / kp1;
    for (int j = 0; j < nj; j++) {
      T sc0, sc1;
      nl_scales<T>(Q, j, k, two ? k2 : k, LNL, &sc0, &sc1);
      const T* xp = xpt + (size_t)j * nchi;
      nl_transform<T, NT, ODD>(Q, j, nchi, fa, fb, tout + (size_t)j * Q.hstride,
                               ctab + (size_t)(k - l0) * Q.qs + Q.qoff[j],
                               gtab + (size_t)(k - l0) * Q.qs + Q.qoff[j], two,
                          [&](int i, ct<T> z) {
                            // summed in the order of the kernels (their
                            // barriers lie between)
                            const T p = xp[i], a0 = z.x * sc0, a1 = z.y * sc1;
                            if (j == 0) {
                              F0[i] = a0 * p;
                              F1[i] = a1 * p;
                            } else if (j == 1) {
                              F0[i] = fma_t(a0, p, F0[i]);
                              F1[i] = fma_t(a1, p, F1[i]);
                            } else {
                              F0[i] = fma_t(a0 * p, mag0, F0[i]);
                              F1[i] = fma_t(a1 * p, mag1, F1[i]);
                            }
                          });
    }
    __syncthreads();
    // chi sums of F^2 k^3 P_lin(k, a = 1), both multipoles
    const T cub0 = kp0 * kp0 * kp0, cub1 = kp1 * kp1 * kp1;  // exact for k < 255
    const T* p0 = ptab + (size_t)(k - l0) * nchi;
    const T* p1 = two ? p0 + nchi : p0;
    T part0 = 0, part1 = 0;
    for (int i = tid; i < nchi; i += nlt) {
      const T rx3 = xt[i], f0 = F0[i], f1 = F1[i];
      part0 = fma_t(f0 * f0 * (cub0 * rx3), p0[i], part0);
      part1 = fma_t(f1 * f1 * (cub1 * rx3), p1[i], part1);
    }
    // two block sums (mixed plan: FP32 within the warp, FP64 across)
    for (int o = 16; o > 0; o >>= 1) {
      part0 += __shfl_down_sync(0xffffffffu, part0, o);
      part1 += __shfl_down_sync(0xffffffffu, part1, o);
    }
    if ((tid & 31) == 0) {
      red[k - ks][tid >> 5] = part0;
      red[k - ks + 1][tid >> 5] = part1;
    }
  }
  __syncthreads();
  // the block's C_l at once, a lane each: done per pair by one thread, this
  // FP64 arithmetic (1/64 of the FP32 rate) held up the other warps at the
  // next barrier, 8 times a block
  const int m = tid;
  if (ks + m >= ke || m >= 16) return;
  double t = 0.0;
  for (int w2 = 0; w2 < nlt / 32; w2++) t += wide64(red[m][w2]);
  const double lim = ggl[(ks + m) * 2 + 0];
  t = t * dlnchi * 2. / M_PI + lim - ggl[(ks + m) * 2 + 1];
  Cl[ks + m] = t;
  // convergence at the block end (cosmo2D.c:4741-4750)
  if (ks + m == ke - 1 && fabs(lim) > 1e-300) {
    const double dev = t / lim - 1.0;
    if (isfinite(dev) && fabs(dev) < 0.01) atomicMin(&Q.conv_blk[item], blk);
  }
}

// ---- 3c. the hand-over (cosmo2D.c:4760-4765): the multipole after the first
// converged block, and the Limber C_l from there on.  One warp per
// (point, bin).
__global__ void __launch_bounds__(128) k_nl_handover(Params P, NLParams Q)
{
  const int item = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (item >= P.B * P.nl) return;
  const int LNL = P.lmax_nolimber;
  const int cb = Q.conv_blk[item];
  const int LM = cb == NL_OPEN ? LNL : min(cb * 16 + 16, LNL);
  if ((threadIdx.x & 31) == 0) P.conv_l[item] = LM;
  const double* tg = P.tab_gg + (size_t)item * P.nnode_g + P.nint;
  const double* ggl = P.ggl + (size_t)item * LNL * 2;
  double* Cl = P.cnl + (size_t)item * LNL;
  for (int k = LM + (threadIdx.x & 31); k < LNL; k += 32) {
    if (k > P.lmin_tab)
      Cl[k] = interpol1d_d(tg, P.n_ell, P.lim_g[0], P.lim_g[2], log((double)k));
    else
      Cl[k] = ggl[k * 2 + 0];
  }
}

// ---- 4. adjoint of the FFTLog part of C_cl_tomo.  For l < the hand-over
// multipole, C_l = (2/pi) dlnchi sum_i F_i^2 k_i^3 P_lin(k_i, 1) + ..., with
// F = b1 G0 + F_1 + bmag l(l+1) F_2 / y^2 linear in b1 (G0: the galaxy
// kernel's transform with b1 = 1, written to tout by k_nl_forward with
// unit_b1).  Given cbar[l] = dL/dC_l, one CTA per (point, bin) and block of
// 16 multipoles below the hand-over takes the forward's transforms again,
// keeps the b1-free galaxy term G0 and the bmag-free magnification term M0 of
// both multipoles of a pair, and accumulates
//   dL/db1     += cbar (2/pi) dlnchi sum_i 2 F_i G0_i k_i^3 P_i
//   dL/dbmag   += cbar (2/pi) dlnchi sum_i 2 F_i M0_i k_i^3 P_i  (bmag != 0;
//                 M0 = l(l+1) F_2 / y^2, the magnification term with bmag = 1)
//   dL/dpsl[m] += cbar (2/pi) dlnchi sum_i F_i^2 k_i^3 P_i (lerp weight)
// where psl is the z = 0 slice of the linear table.  FP64 plan: the slice
// adjoint of a block is summed in shared memory and spread onto the table's
// two z columns.  Mixed plan: the blocks store cbar (2/pi) dlnchi F_i^2 k_i^3
// P_i per multipole and sample (Q.gadj), and k_nl_adj_slice sums a bin's in
// the order of its multipoles in FP32, as one CTA walking them would: the
// blocks run in parallel and the FP32 sums keep their order.
// The chi-sum weight of a multipole with cotangent c in the loop precision:
// k_nl_adj skips (and does not store) the multipoles where it is 0, and
// k_nl_adj_slice must skip the same ones.  narrow flushes what is below the
// FP32 normal range; the conversion keeps it.
template <typename T>
__device__ __forceinline__ T nl_weight(double c, T wsum)
{
  T v = narrow<T>(c);
  if (v == (T)0) v = (T)c;
  return v * wsum;
}

// a slice adjoint onto the linear table's two z columns around z = 0
template <typename T, int NT>
__device__ __forceinline__ void nl_slice_flush(const Params& P, int pt, const T* pbar, double* __restrict__ lnpl_bar)
{
  const int nk = P.pkl_nk, j0 = bsearch_d(P.pkl_z, P.pkl_nz, 0.0);
  const double dyz = (0.0 - P.pkl_z[j0]) / (P.pkl_z[j0 + 1] - P.pkl_z[j0]);
  double* lb = lnpl_bar + (size_t)pt * nk * P.pkl_nz;
  for (int i = threadIdx.x; i < nk; i += NT) {
    const double v = (double)pbar[i];
    if (v != 0.0) {
      atomicAdd(&lb[(size_t)i * P.pkl_nz + j0], (1 - dyz) * v);
      atomicAdd(&lb[(size_t)i * P.pkl_nz + j0 + 1], dyz * v);
    }
  }
}

template <typename T, int NT, int MINB, bool ODD>
__global__ void __launch_bounds__(NT, MINB) k_nl_adj(Params P, NLParams Q, int lt, int l0, int l1,
                                                     const double* __restrict__ cbar, double* __restrict__ lnpl_bar,
                                                     cl2pt_nuisance* nu_bar)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr bool F32 = sizeof(T) == sizeof(float);
  const int item = blockIdx.x, tid = threadIdx.x;
  constexpr int nlt = NT;
  const int LNL = P.lmax_nolimber, nk = P.pkl_nk, nchi = P.nl_nchi;
  const int ks = l0 + blockIdx.y * 16, ke = min(min(ks + 16, l1), P.conv_l[item]);
  if (ks >= ke) return;
  const int pt = item / P.nl, q = item - (item / P.nl) * P.nl;
  const cl2pt_nuisance& nu = P.nu[pt];
  const double bmag = nu.gb[4][q];
  const int nj = (bmag != 0.0) ? 3 : 2;
  // shared: [fa, fb: nmax complex T][F0, F1, G00, G01: nchi T][pbar: nk T,
  // FP64 plan];
  // the magnification terms M00, M01 in the FFT buffer that the last (j = 2)
  // transform leaves free, until the pair's sums have read them
  ct<T>* fa = (ct<T>*)smem_raw;
  ct<T>* fb = fa + Q.nmax;
  T* F0 = (T*)(fb + Q.nmax);
  T* F1 = F0 + nchi;
  T* G00 = F1 + nchi;
  T* G01 = G00 + nchi;
  T* pbar = G01 + nchi;
  __shared__ T red[8][2][NT / 32];
  const double* geom = Q.geom + (size_t)pt * NL_GEOM;
  const double dlnchi = geom[1];
  const T* xt = (const T*)Q.xtab + (size_t)pt * NL_XROWS * nchi;        // (rc / x)^3
  const T* lxk = xt + nchi;                                             // log10(rc / (x coverH0))
  const T* xpt = xt + 2 * nchi;                                         // [3] the kernels' powers of x
  const float4* pcf = Q.pcell ? Q.pcell + (size_t)pt * nk : nullptr;
  const double* psl = Q.pslice + (size_t)pt * nk;
  const ct<T>* tout = (const ct<T>*)Q.tout + (size_t)item * Q.tout_stride;  // [3][hstride]
  const ct<T>* ctab = (const ct<T>*)Q.ctab + (size_t)pt * Q.lchunk * Q.qs;
  const ct<T>* gtab = (const ct<T>*)Q.gtabl + (size_t)pt * Q.lchunk * Q.qs;
  if constexpr (!F32)
    for (int i = tid; i < nk; i += nlt) pbar[i] = 0.0;
  float* gadj = F32 ? Q.gadj + ((size_t)item * Q.achunk + (ks - l0)) * nchi : nullptr;
  const T bmagt = (T)bmag;
  const T lc3 = (T)(1.0 / (CL2PT_COVERH0 * CL2PT_COVERH0 * CL2PT_COVERH0));
  const T wsum = (T)(dlnchi * 2. / M_PI);  // chi-sum weight of C_l
  const T b1t = (T)nu.gb[0][q];
  const double* cb = cbar + (size_t)item * LNL;
  T kf = (T)ks;  // k as a float, counted: conversions issue at the FP64 rate
  for (int k = ks; k < ke; k += 2, kf += (T)2) {
    const int k2 = k + 1;
    const bool two = k2 < ke;
    const T kp0 = kf + (T)1, kp1 = kf + (T)2;
    // bmag l(l+1)/(l+1)^2 = bmag l/(l+1), and with bmag = 1
    const T un0 = kf / kp0, un1 = kp0 / kp1;
    const T mag0 = bmagt * kf / kp0;
    const T mag1 = bmagt * kp0 / kp1;
    for (int j = 0; j < nj; j++) {
      T sc0, sc1;
      nl_scales<T>(Q, j, k, two ? k2 : k, LNL, &sc0, &sc1);
      const T* xp = xpt + (size_t)j * nchi;
      nl_transform<T, NT, ODD>(Q, j, nchi, fa, fb, tout + (size_t)j * Q.hstride,
                               ctab + (size_t)(k - lt) * Q.qs + Q.qoff[j],
                               gtab + (size_t)(k - lt) * Q.qs + Q.qoff[j], two,
                          [&](int i, ct<T> z) {
                            const T p = xp[i], a0 = z.x * sc0, a1 = z.y * sc1;
                            const T f0 = a0 * p, f1 = a1 * p;
                            if (j == 0) {
                              // the galaxy transform was taken with b1 = 1
                              G00[i] = f0;
                              G01[i] = f1;
                              F0[i] = f0 * b1t;
                              F1[i] = f1 * b1t;
                            } else if (j == 1) {
                              F0[i] = fma_t(a0, p, F0[i]);
                              F1[i] = fma_t(a1, p, F1[i]);
                            } else {
                              // 2 nmax T >= 2 nchi T of scratch (N >= nchi + 2 pad)
                              ((T*)fa)[i] = f0 * un0;
                              ((T*)fa)[nchi + i] = f1 * un1;
                              F0[i] = fma_t(f0, mag0, F0[i]);
                              F1[i] = fma_t(f1, mag1, F1[i]);
                            }
                          });
    }
    const T* M00 = (const T*)fa;
    const T* M01 = M00 + nchi;
    __syncthreads();
    // adjoint of C_l = (2/pi) dlnchi sum_i F_i^2 k_i^3 P_i for both
    // multipoles: P_lin slice adjoint (mixed plan: the terms, for
    // k_nl_adj_slice) and d/db1 through F = b1 G0 + ...
    const T wt0 = nl_weight<T>(cb[k], wsum), wt1 = two ? nl_weight<T>(cb[k2], wsum) : (T)0;
    const bool magk = nj == 3;
    T tb = 0, tm = 0;
    if (wt0 != (T)0 || wt1 != (T)0) {
      const double lk0 = F32 ? 0.0 : Q.l10k1[k], lk1 = F32 ? 0.0 : Q.l10k1[two ? k2 : k];
      const float lk0f = F32 ? Q.l10k1f[k] : 0.0f, lk1f = F32 ? Q.l10k1f[two ? k2 : k] : 0.0f;
      const T cub0 = kp0 * kp0 * kp0, cub1 = kp1 * kp1 * kp1;
      for (int i = tid; i < nchi; i += nlt) {
        const T rx3 = xt[i];
        for (int h = 0; h < (two ? 2 : 1); h++) {
          const T wt = h ? wt1 : wt0;
          if (wt == (T)0) continue;
          const T F = h ? F1[i] : F0[i];
          const T G = h ? G01[i] : G00[i];
          const T M = magk ? (h ? M01[i] : M00[i]) : (T)0;
          const T k3 = (h ? cub1 : cub0) * rx3;
          int lo;
          T dx, pl;
          if constexpr (F32) {
            const float lkt = (h ? lk1f : lk0f) + lxk[i];
            lo = slice_cell(Q.plkf, nk, Q.lut, Q.lscale, Q.lumax, lkt);
            const float4 c = pcf[lo];
            dx = (lkt - Q.plkf[lo]) * c.z;
            pl = __expf(c.x) * __expf(c.y + dx * c.w) * lc3;
          } else {
            const double lkv = (h ? lk1 : lk0) + lxk[i];
            lo = bsearch_d(P.pkl_lk, nk, lkv);
            dx = (lkv - P.pkl_lk[lo]) * Q.pinv[lo];
            pl = exp(psl[lo] + dx * (psl[lo + 1] - psl[lo])) * lc3;
          }
          const T g = wt * F * F * k3 * pl;
          if constexpr (F32) {
            gadj[(size_t)(k - ks + h) * nchi + i] = g;
          } else {
            atomicAdd(&pbar[lo], g * ((T)1 - dx));
            atomicAdd(&pbar[lo + 1], g * dx);
          }
          const T u = wt * (T)2 * F * k3 * pl;
          tb += u * G;
          tm += u * M;
        }
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      tb += __shfl_down_sync(0xffffffffu, tb, o);
      tm += __shfl_down_sync(0xffffffffu, tm, o);
    }
    if ((tid & 31) == 0) {
      red[(k - ks) >> 1][0][tid >> 5] = tb;
      red[(k - ks) >> 1][1][tid >> 5] = tm;
    }
    // also separates the reads of M0 from the next pair's spectrum
    __syncthreads();
  }
  if constexpr (!F32) {
    __syncthreads();
    nl_slice_flush<double, NT>(P, pt, pbar, lnpl_bar);
  }
  if (tid < (nj == 3 ? 2 : 1)) {
    double v = 0.0;
    for (int m = 0; m < (ke - ks + 1) >> 1; m++)
      for (int w2 = 0; w2 < nlt / 32; w2++) v += wide64(red[m][tid][w2]);
    atomicAdd(&nu_bar[pt].gb[tid ? 4 : 0][q], v);
  }
}

// The slice adjoint of a (point, bin) over the multipoles [l0, l1) of a
// chunk below its hand-over, from the blocks' stored terms; carried in
// Q.padj between chunks, onto the table with the last one.  The FP32 sum of a
// cell depends on the order of its terms (to ~1e-7 of the gradient), so one
// CTA adds them as a CTA walking the multipoles would: pair by pair, NT
// samples at a time, both multipoles.  Latency-bound: a chain of lookups and
// two shared-memory atomics per sample, so the tables lie in shared memory
// and a pair's terms are loaded ahead.
template <int NT>
__global__ void __launch_bounds__(NT) k_nl_adj_slice(Params P, NLParams Q, int l0, int l1,
                                                     const double* __restrict__ cbar, double* __restrict__ lnpl_bar)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int item = blockIdx.x, tid = threadIdx.x;
  const int pt = item / P.nl, nk = P.pkl_nk, nchi = P.nl_nchi, LNL = P.lmax_nolimber;
  const int LM = P.conv_l[item], ke = min(l1, LM);
  if (l0 > 0 && l0 >= LM) return;
  float* pbar = (float*)smem_raw;      // [nk]
  float* plk = pbar + nk;              // [nk]
  float* inv = plk + nk;               // [nk] 1 / width
  float* lxk = inv + nk;               // [nchi]
  unsigned short* lut = (unsigned short*)(lxk + nchi);
  float* carry = Q.padj + (size_t)item * nk;
  for (int i = tid; i < nk; i += NT) {
    pbar[i] = l0 > 0 ? carry[i] : 0.0f;
    plk[i] = Q.plkf[i];
    inv[i] = Q.pcell[(size_t)pt * nk + i].z;
  }
  for (int i = tid; i < nchi; i += NT) lxk[i] = ((const float*)Q.xtab)[((size_t)pt * NL_XROWS + 1) * nchi + i];
  for (int i = tid; i < nl_lut_size(nk); i += NT) lut[i] = Q.lut[i];
  __syncthreads();
  const double* cb = cbar + (size_t)item * LNL;
  const float wsum = (float)(Q.geom[(size_t)pt * NL_GEOM + 1] * 2. / M_PI);
  const float* gadj = Q.gadj + (size_t)item * Q.achunk * nchi;
  constexpr int U = 4;  // samples of a thread loaded ahead
  for (int k = l0; k < ke; k += 2) {
    const int k2 = k + 1 < ke ? k + 1 : k;
    const bool on[2] = {nl_weight<float>(cb[k], wsum) != 0.0f, k2 > k && nl_weight<float>(cb[k2], wsum) != 0.0f};
    const float lk[2] = {Q.l10k1f[k], Q.l10k1f[k2]};
    const float* gk = gadj + (size_t)(k - l0) * nchi;
    for (int i0 = tid; i0 < nchi; i0 += U * NT) {
      float g[U][2];
#pragma unroll
      for (int u = 0; u < U; u++)
#pragma unroll
        for (int h = 0; h < 2; h++) g[u][h] = (on[h] && i0 + u * NT < nchi) ? gk[(size_t)h * nchi + i0 + u * NT] : 0.0f;
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int i = i0 + u * NT;
        if (i >= nchi) break;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          if (!on[h]) continue;
          const float lkt = lk[h] + lxk[i];
          const int lo = slice_cell(plk, nk, lut, Q.lscale, Q.lumax, lkt);
          const float dx = (lkt - plk[lo]) * inv[lo];
          atomicAdd(&pbar[lo], __fmul_rn(g[u][h], __fsub_rn(1.0f, dx)));
          atomicAdd(&pbar[lo + 1], g[u][h] * dx);
        }
      }
    }
    __syncthreads();  // the pairs' terms add in order
  }
  if (l1 < LNL && l1 < LM) {
    for (int i = tid; i < nk; i += NT) carry[i] = pbar[i];
    return;
  }
  nl_slice_flush<float, NT>(P, pt, pbar, lnpl_bar);
}

// Threads of a block CTA.  128 give a 900-1500 point transform two or three
// butterflies a thread and stage between barriers, which several CTAs an SM
// overlap; 256 shorten the chain of the longer ones, and of few CTAs.
// real_3x2pt, us per evaluation (value and gradient in brackets):
//   chi samples       500            850            1000           1200           1500           2048
//   512 points, 128   11313 (28482)  12667 (32477)  13089 (34191)  14370 (37782)  15168 (41640)  18535 (53979)
//               256   11935 (30869)  13184 (34574)  13160 (34824)  14332 (38546)  14849 (40400)  16775 (46183)
//   37 points,  128    1386 (4063)    1550 (4827)    1540 (5030)    1711 (5611)    1860 (6152)    2040 (7612)
//               256    1410 (4114)    1535 (4562)    1508 (4611)    1594 (4976)    1702 (5312)    1861 (6014)
// The forms cross near 1100 samples at 512 points and near 600 at 37; the line
// below is at 910 samples with 600 k (1016 with 400).  It does not follow the
// number of points, because the count of threads fixes the order of the FP32
// partial sums and a point's result does not depend on its batch.
static int nl_threads(const Params& P, const NLParams& Q)
{
  if (P.prec == CL2PT_PREC_FP64) return 256;
  return 16 * (size_t)Q.nmax + 16 * (size_t)P.nl_nchi + 20 * (size_t)P.pkl_nk + 64 + 1024 <= 57 * 1024 ? 128 : 256;
}

template <typename T>
static size_t nl_block_smem(const Params& P, const NLParams& Q, bool adj)
{
  return sizeof(T) * (4 * (size_t)Q.nmax + (adj ? 4 : 2) * (size_t)P.nl_nchi +
                      (adj && sizeof(T) == sizeof(double) ? P.pkl_nk : 0));
}

// f(loop precision, odd sizes) of the plan
template <typename F>
static void by_form(const Params& P, const NLParams& Q, F f)
{
  const bool odd = (Q.N[0] | Q.N[1] | Q.N[2]) & 1;
  if (P.prec == CL2PT_PREC_FP64) odd ? f(0.0, std::true_type{}) : f(0.0, std::false_type{});
  else odd ? f(0.0f, std::true_type{}) : f(0.0f, std::false_type{});
}

template <typename T>
static void launch_nl_cg(const Params& P, const NLParams& Q, int l0, int l1, cudaStream_t s)
{
  // phases: the multipoles in parts of NLC_PART; Gamma kernels: entries in
  // parts of NLC_NT for both parities (FP32), blocks of 16 multipoles (FP64)
  const int nc = (l1 - l0 + NLC_PART - 1) / NLC_PART;
  const int ng = sizeof(T) == sizeof(float) ? 2 * ((Q.hstride + NLC_NT - 1) / NLC_NT) : (l1 - l0 + 15) / 16;
  k_nl_cg<T><<<dim3(P.B, 3 * (nc + ng) + nc), NLC_NT, 0, s>>>(P, Q, l0, l1, nl_threads(P, Q), nc, ng);
}

template <typename T, bool ODD>
static void launch_nl_vjp_t(const Params& P, const NLParams& Q, const double* cbar, double* lnpl_bar,
                            cl2pt_nuisance* nu_bar, cudaStream_t s, int* launches)
{
  const size_t sm1 = sizeof(double) * (2 * 2 * (size_t)Q.nmax + 3 * (size_t)P.nl_nchi) + 64;
  cudaFuncSetAttribute(k_nl_forward<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm1);
  k_nl_forward<T><<<dim3(P.B, P.nl), NL_NT, sm1, s>>>(P, Q, 1, 0, 1);
  (*launches)++;
  const size_t sm = nl_block_smem<T>(P, Q, true);
  const int nt = nl_threads(P, Q), LNL = P.lmax_nolimber;
  auto run = [&](auto kern, int lt, int l0, int l1) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    kern<<<dim3(P.B * P.nl, (l1 - l0 + 15) / 16), nt, sm, s>>>(P, Q, lt, l0, l1, cbar, lnpl_bar, nu_bar);
    (*launches)++;
  };
  for (int lt = 0; lt < LNL; lt += Q.lchunk) {
    const int le = lt + Q.lchunk < LNL ? lt + Q.lchunk : LNL;
    if (Q.lchunk < LNL) {  // else the forward's tables of this wave are still there
      launch_nl_cg<T>(P, Q, lt, le, s);
      (*launches)++;
    }
    if constexpr (sizeof(T) == sizeof(double)) {
      run(k_nl_adj<double, 256, 2, ODD>, lt, lt, le);
    } else {
      // as many multipoles at a time as the slice adjoint's terms have room for
      const size_t smk = sizeof(float) * (3 * (size_t)P.pkl_nk + P.nl_nchi) + sizeof(unsigned short) * nl_lut_size(P.pkl_nk);
      auto sum = [&](auto kern, int l0, int l1) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smk);
        kern<<<P.B * P.nl, nt, smk, s>>>(P, Q, l0, l1, cbar, lnpl_bar);
        (*launches)++;
      };
      for (int l0 = lt; l0 < le; l0 += Q.achunk) {
        const int l1 = l0 + Q.achunk < le ? l0 + Q.achunk : le;
        if (nt == 128) {
          run(k_nl_adj<float, 128, 6, ODD>, lt, l0, l1);
          sum(k_nl_adj_slice<128>, l0, l1);
        } else {
          run(k_nl_adj<float, 256, 2, ODD>, lt, l0, l1);
          sum(k_nl_adj_slice<256>, l0, l1);
        }
      }
    }
  }
}

void launch_nonlimber_vjp(const Params& P, const NLParams& Q, const double* cbar, double* lnpl_bar,
                          cl2pt_nuisance* nu_bar, cudaStream_t s, int* launches)
{
  by_form(P, Q, [&](auto t, auto odd) {
    launch_nl_vjp_t<decltype(t), decltype(odd)::value>(P, Q, cbar, lnpl_bar, nu_bar, s, launches);
  });
}

template <typename T>
static void launch_nl_prep_t(const Params& P, const NLParams& Q, cudaStream_t s)
{
  const size_t sm1 = sizeof(double) * (2 * 2 * (size_t)Q.nmax + 3 * (size_t)P.nl_nchi) + 64;
  cudaFuncSetAttribute(k_nl_forward<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm1);
  k_nl_slice<<<P.B, 256, 0, s>>>(P, Q);
  k_nl_gdirect<<<dim3(P.B, 3, Q.ndirect), NL_NT, 0, s>>>(P, Q);
  launch_nl_cg<T>(P, Q, 0, Q.lchunk < P.lmax_nolimber ? Q.lchunk : P.lmax_nolimber, s);
  k_nl_forward<T><<<dim3(P.B, P.nl), NL_NT, sm1, s>>>(P, Q, 0, 0, 3);
}

template <typename T, bool ODD>
static void launch_nl_loop_t(const Params& P, const NLParams& Q, cudaStream_t s, int* launches)
{
  const size_t sm = nl_block_smem<T>(P, Q, false);
  const int nt = nl_threads(P, Q), LNL = P.lmax_nolimber;
  auto run = [&](auto kern, int l0, int l1) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    kern<<<dim3(P.B * P.nl, (l1 - l0 + 15) / 16), nt, sm, s>>>(P, Q, l0, l1);
  };
  for (int l0 = 0; l0 < LNL; l0 += Q.lchunk) {
    const int l1 = l0 + Q.lchunk < LNL ? l0 + Q.lchunk : LNL;
    if (l0) {
      launch_nl_cg<T>(P, Q, l0, l1, s);
      (*launches)++;
    }
    if constexpr (sizeof(T) == sizeof(double)) run(k_nl_block<double, 256, 2, ODD>, l0, l1);
    else if (nt == 128) run(k_nl_block<float, 128, 6, ODD>, l0, l1);
    else run(k_nl_block<float, 256, 3, ODD>, l0, l1);
    (*launches)++;
  }
  k_nl_handover<<<(P.B * P.nl + 3) / 4, 128, 0, s>>>(P, Q);
  (*launches)++;
}

void launch_nonlimber_prep(const Params& P, const NLParams& Q, cudaStream_t s, int* launches, const Hook& hk)
{
  hk(CL2PT_K_NONLIMBER, 1);
  if (P.prec == CL2PT_PREC_FP64) launch_nl_prep_t<double>(P, Q, s);
  else launch_nl_prep_t<float>(P, Q, s);
  hk(CL2PT_K_NONLIMBER, 0);
  (*launches) += 4;
}

void launch_nonlimber_loop(const Params& P, const NLParams& Q, cudaStream_t s, int* launches, const Hook& hk)
{
  hk(CL2PT_K_NONLIMBER, 1);
  by_form(P, Q, [&](auto t, auto odd) { launch_nl_loop_t<decltype(t), decltype(odd)::value>(P, Q, s, launches); });
  hk(CL2PT_K_NONLIMBER, 0);
}

void launch_nonlimber(const Params& P, const NLParams& Q, cudaStream_t s, int* launches,
                      const Hook& hk)
{
  launch_nonlimber_prep(P, Q, s, launches, hk);
  launch_nonlimber_loop(P, Q, s, launches, hk);
}

}  // namespace cl2pt
