// fft_fx.cuh -- in-place mixed-radix FFTs of FP64 data in 64-bit block
// fixed point, one shared-memory buffer per CTA.
//
// GB300 issues FP64 at 1/64 of the FP32 rate (about 1.7 instructions per
// SM and cycle), so an FP64 transform of 12150 points takes one SM 210 us
// whatever else it does.  The integer units run 32 x 32 -> 64 bit multiply-
// adds and 64-bit sums some twenty times as fast, and 61 bits of a common
// scale hold more than the 53 of an FP64 number near the block's largest:
//   * the input is scaled by a power of two to 59 bits; each stage notes the
//     top bit of what it wrote, and the next shifts down (rounding) on the
//     way in, by as much as its radix could overflow and no more;
//   * a value times a twiddle is three of the four 31-bit limb products (the
//     low x low one is below half a unit);
//   * the result returns as FP64, rounded to nearest.
// 12150 points on one SM: about 210 -> 60 us, with an L2 error of 0.5 to 1.4
// units of 2^-53 at 5040 to 14406 points (noise, smooth, 26 decades) where
// fft64.cuh makes 3.4 to 5.2, both against extended precision; over the
// outputs below 1e-6 of the largest 0.5 to 0.9 against 2.7 to 3.3.  An entry
// is held to 2^-59 of its block's largest, finer than its first FP64 sum with
// that would leave it: one more than 2^-8 below has fewer than 53 bits of its
// own, one more than 2^-59 below is 0.  Bound by issue (about 100 integer
// instructions a point and stage).
// Any non-finite input gives NaN everywhere, as FP64 butterflies would.
//
// dif: natural order in, digit-reversed out (position p holds X[rev(p)]);
// dit: digit-reversed in, natural out; both sum_n x[n] exp(-+ 2 pi i n k / n),
// the + sign (inv) by exchanging real and imaginary parts on the way in and
// out.  Stage s (radix R, block length L, m = L / R): for each block b and
// j < m the R points b L + j + r m form one butterfly, with the twiddles
// exp(-2 pi i j k / L) after it (dif) or before it (dit).  Radices 6, 10, 12,
// 14, 15 are prime-factor products (no inner twiddles), so 12150 points take
// four stages (15, 15, 9, 6) with as many passes over shared memory.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <vector>

#include "common.cuh"

namespace cl2pt {
namespace fx {

#define FX_HD __host__ __device__ __forceinline__

constexpr int MAX_STAGES = 16;
constexpr int GENERIC_MAX_PER_THREAD = 16;
constexpr int BITS = 61;  // magnitudes stay below 2^BITS

struct Desc {
  int n, nst;
  int rad[MAX_STAGES], L[MAX_STAGES];  // L[0] = n
  FastDiv m[MAX_STAGES];               // L / rad as a divisor
  FastDiv r[MAX_STAGES];               // rad (generic stages)
};

// Bluestein form of a size with a large prime factor: X_k = w_k sum_n
// (x_n w_n) conj(w_{k-n}), w_n = exp(-i pi n^2 / n_fft), as a convolution of
// the size of another transform (at least 2 n_fft - 1 points)
struct Chirp {
  const int4* w;   // [n_fft] limbs
  const int4* b;   // transform of conj(w) at DIF positions, limbs of it / (its size 2^kb)
  int kb;
};

struct c64 { long long x, y; };

FX_HD c64 add(c64 a, c64 b) { return {a.x + b.x, a.y + b.y}; }
FX_HD c64 sub(c64 a, c64 b) { return {a.x - b.x, a.y - b.y}; }
FX_HD c64 sub_i(c64 a, c64 b) { return {a.x + b.y, a.y - b.x}; }  // a - i b
FX_HD c64 add_i(c64 a, c64 b) { return {a.x - b.y, a.y + b.x}; }  // a + i b

// limbs of a value: v = hi 2^31 + lo, lo in [0, 2^31); of a constant in
// units of 2^-61: lo in [-2^30, 2^30)
FX_HD int hi31(long long v) { return (int)(v >> 31); }
FX_HD int lo31(long long v) { return (int)((unsigned)v & 0x7fffffffu); }
FX_HD long long wide(int a, int b) { return (long long)a * b; }
// The low x low product is left out; its mean, half the constant's low limb a
// value's low limb being anywhere in [0, 2^31), joins the rounding: a bias
// would add up coherently in a few outputs.
FX_HD long long rnd(int l) { return (long long)((l >> 1) + (1 << 29)); }
FX_HD long long fin(long long hh, long long cr) { return hh + hh + (cr >> 30); }

// a (rh + i ih) with w = (rh, rl, ih, il)
FX_HD c64 mulw(c64 a, int4 w)
{
  const int xh = hi31(a.x), xl = lo31(a.x), yh = hi31(a.y), yl = lo31(a.y);
  const int nh = -w.z, nl = -w.w;
  return {fin(wide(xh, w.x) + wide(yh, nh), rnd(w.y + nl) + wide(xh, w.y) + wide(xl, w.x) + wide(yh, nl) + wide(yl, nh)),
          fin(wide(xh, w.z) + wide(yh, w.x), rnd(w.w + w.y) + wide(xh, w.w) + wide(xl, w.z) + wide(yh, w.y) + wide(yl, w.x))};
}
// v c for a real constant (h, l)
FX_HD long long mulc(long long v, int h, int l)
{
  const int vh = hi31(v), vl = lo31(v);
  return fin(wide(vh, h), rnd(l) + wide(vh, l) + wide(vl, h));
}
FX_HD c64 mulc(c64 v, int h, int l) { return {mulc(v.x, h, l), mulc(v.y, h, l)}; }
// a c + b d
FX_HD long long mulc2(long long a, int ch, int cl, long long b, int dh, int dl)
{
  const int ah = hi31(a), al = lo31(a), bh = hi31(b), bl = lo31(b);
  return fin(wide(ah, ch) + wide(bh, dh), rnd(cl + dl) + wide(ah, cl) + wide(al, ch) + wide(bh, dl) + wide(bl, dh));
}
FX_HD c64 mulc2(c64 a, int ch, int cl, c64 b, int dh, int dl)
{
  return {mulc2(a.x, ch, cl, b.x, dh, dl), mulc2(a.y, ch, cl, b.y, dh, dl)};
}
FX_HD c64 half(c64 a) { return {(a.x + 1) >> 1, (a.y + 1) >> 1}; }
FX_HD c64 quarter(c64 a) { return {(a.x + 2) >> 2, (a.y + 2) >> 2}; }
// shift down (s > 0), to nearest and half to even: the small shifts meet
// halves often
FX_HD long long rsh(long long v, int s) { return (v + ((1ll << (s - 1)) - 1) + ((v >> s) & 1)) >> s; }

// y_k = sum_r x_r exp(-2 pi i r k / R), in place; constants as limbs of 2^61
template <int R> struct Bfly;
template <> struct Bfly<2> {
  static FX_HD void run(c64* x)
  {
    const c64 a = x[0], b = x[1];
    x[0] = add(a, b);
    x[1] = sub(a, b);
  }
};
template <> struct Bfly<3> {
  static FX_HD void run(c64* x)
  {
    const c64 t = add(x[1], x[2]);
    const c64 d = mulc(sub(x[1], x[2]), 929887697, -666064268);  // sin(2 pi / 3)
    const c64 a = sub(x[0], half(t));
    x[0] = add(x[0], t);
    x[1] = sub_i(a, d);
    x[2] = add_i(a, d);
  }
};
template <> struct Bfly<4> {
  static FX_HD void run(c64* x)
  {
    const c64 a = add(x[0], x[2]), b = sub(x[0], x[2]), c = add(x[1], x[3]), d = sub(x[1], x[3]);
    x[0] = add(a, c);
    x[2] = sub(a, c);
    x[1] = sub_i(b, d);
    x[3] = add_i(b, d);
  }
};
template <> struct Bfly<5> {
  static FX_HD void run(c64* x)
  {
    // cos(2 pi/5) and cos(4 pi/5) = -1/4 +- sqrt(5)/4
    const c64 t1 = add(x[1], x[4]), t2 = add(x[2], x[3]), t3 = sub(x[1], x[4]), t4 = sub(x[2], x[3]);
    const c64 t = add(t1, t2);
    const c64 c = sub(x[0], quarter(t));
    const c64 e = mulc(sub(t1, t2), 600239927, 401909697);
    const c64 a1 = add(c, e), a2 = sub(c, e);
    const c64 b1 = mulc2(t3, 1021189159, -1001062562, t4, 631129609, -178627090);
    const c64 b2 = mulc2(t3, 631129609, -178627090, t4, -1021189159, 1001062562);
    x[0] = add(x[0], t);
    x[1] = sub_i(a1, b1);
    x[4] = add_i(a1, b1);
    x[2] = sub_i(a2, b2);
    x[3] = add_i(a2, b2);
  }
};
template <> struct Bfly<7> {
  static FX_HD void run(c64* x)
  {
    constexpr int c1h = 669467077, c1l = 200135021, c2h = -238930034, c2l = 1064214374, c3h = -967407956,
                  c3l = 883134254;
    constexpr int s1h = 839485162, s1l = 98454284, s2h = 1046820875, s2l = -655791900, s3h = 465879117,
                  s3l = 953540736;
    const c64 p1 = add(x[1], x[6]), p2 = add(x[2], x[5]), p3 = add(x[3], x[4]);
    const c64 m1 = sub(x[1], x[6]), m2 = sub(x[2], x[5]), m3 = sub(x[3], x[4]);
    const c64 x0 = x[0];
    const c64 a1 = add(x0, add(mulc2(p1, c1h, c1l, p2, c2h, c2l), mulc(p3, c3h, c3l)));
    const c64 a2 = add(x0, add(mulc2(p1, c2h, c2l, p2, c3h, c3l), mulc(p3, c1h, c1l)));
    const c64 a3 = add(x0, add(mulc2(p1, c3h, c3l, p2, c1h, c1l), mulc(p3, c2h, c2l)));
    const c64 b1 = add(mulc2(m1, s1h, s1l, m2, s2h, s2l), mulc(m3, s3h, s3l));
    const c64 b2 = add(mulc2(m1, s2h, s2l, m2, -s3h, -s3l), mulc(m3, -s1h, -s1l));
    const c64 b3 = add(mulc2(m1, s3h, s3l, m2, -s1h, -s1l), mulc(m3, s2h, s2l));
    x[0] = add(x0, add(p1, add(p2, p3)));
    x[1] = sub_i(a1, b1);
    x[6] = add_i(a1, b1);
    x[2] = sub_i(a2, b2);
    x[5] = add_i(a2, b2);
    x[3] = sub_i(a3, b3);
    x[4] = add_i(a3, b3);
  }
};
template <> struct Bfly<8> {
  static FX_HD void run(c64* x)
  {
    constexpr int h = 759250125, l = -12858223;  // sqrt(1/2)
    c64 a[4] = {x[0], x[2], x[4], x[6]}, b[4] = {x[1], x[3], x[5], x[7]};
    Bfly<4>::run(a);
    Bfly<4>::run(b);
    b[1] = mulc(sub_i(b[1], b[1]), h, l);                      // (1 - i) / sqrt 2
    b[2] = {b[2].y, -b[2].x};                                  // -i
    b[3] = mulc(c64{b[3].y - b[3].x, -b[3].x - b[3].y}, h, l);  // (-1 - i) / sqrt 2
#pragma unroll
    for (int k = 0; k < 4; k++) {
      x[k] = add(a[k], b[k]);
      x[k + 4] = sub(a[k], b[k]);
    }
  }
};
template <> struct Bfly<9> {
  static FX_HD void run(c64* x)
  {
    const int4 w1 = {822533958, -816826062, -690187940, -1008082092};
    const int4 w2 = {186453311, 48030313, -1057429273, -18618202};
    const int4 w4 = {-1008987269, 768795749, -367241333, 989463890};
    c64 y[3][3];
#pragma unroll
    for (int r = 0; r < 3; r++) {
      y[r][0] = x[r];
      y[r][1] = x[r + 3];
      y[r][2] = x[r + 6];
      Bfly<3>::run(y[r]);
    }
    y[1][1] = mulw(y[1][1], w1);
    y[1][2] = mulw(y[1][2], w2);
    y[2][1] = mulw(y[2][1], w2);
    y[2][2] = mulw(y[2][2], w4);
#pragma unroll
    for (int k = 0; k < 3; k++) {
      c64 t[3] = {y[0][k], y[1][k], y[2][k]};
      Bfly<3>::run(t);
      x[k] = t[0];
      x[k + 3] = t[1];
      x[k + 6] = t[2];
    }
  }
};
// R = A B, coprime: input (B n1 + A n2) mod R, output k = (k mod A, k mod B)
template <int A, int B> struct PFA {
  static FX_HD void run(c64* x)
  {
    constexpr int R = A * B;
    c64 y[B][A];
#pragma unroll
    for (int n2 = 0; n2 < B; n2++) {
#pragma unroll
      for (int n1 = 0; n1 < A; n1++) y[n2][n1] = x[(B * n1 + A * n2) % R];
      Bfly<A>::run(y[n2]);
    }
#pragma unroll
    for (int k1 = 0; k1 < A; k1++) {
      c64 t[B];
#pragma unroll
      for (int n2 = 0; n2 < B; n2++) t[n2] = y[n2][k1];
      Bfly<B>::run(t);
#pragma unroll
      for (int k = 0; k < R; k++)
        if (k % A == k1) x[k] = t[k % B];
    }
  }
};
template <> struct Bfly<6> : PFA<2, 3> {};
template <> struct Bfly<10> : PFA<2, 5> {};
template <> struct Bfly<12> : PFA<4, 3> {};
template <> struct Bfly<14> : PFA<2, 7> {};
template <> struct Bfly<15> : PFA<3, 5> {};

// the union of the magnitudes' high words
FX_HD void note(unsigned& top, c64 a)
{
  const int x = (int)(a.x >> 32), y = (int)(a.y >> 32);
  top |= (unsigned)(x ^ (x >> 31));
  top |= (unsigned)(y ^ (y >> 31));
}

FX_HD int quot(int n, const FastDiv& f)
{
#ifdef __CUDA_ARCH__
  return fdiv(n, f);
#else
  return (int)(((((unsigned long long)f.m * (unsigned)n) >> 32) + (unsigned)n) >> f.l);
#endif
}
#ifdef __CUDA_ARCH__
#define FX_TW(p) __ldg(p)
#else
#define FX_TW(p) (*(p))
#endif

// one butterfly of a stage
template <int R, bool DIF>
FX_HD void butterfly(c64* buf, int q, int L, int m, int tstep, const FastDiv& md, const int4* __restrict__ tw,
                     int sin, unsigned& top)
{
  const int b = quot(q, md), j = q - b * m;
  c64* p = buf + b * L + j;
  c64 x[R];
#pragma unroll
  for (int r = 0; r < R; r++) x[r] = p[r * m];
  if (sin) {
#pragma unroll
    for (int r = 0; r < R; r++) x[r] = {rsh(x[r].x, sin), rsh(x[r].y, sin)};
  }
  if (!DIF && j) {
#pragma unroll
    for (int k = 1; k < R; k++) x[k] = mulw(x[k], FX_TW(tw + j * k * tstep));
  }
  Bfly<R>::run(x);
  if (DIF && j) {
#pragma unroll
    for (int k = 1; k < R; k++) x[k] = mulw(x[k], FX_TW(tw + j * k * tstep));
  }
#pragma unroll
  for (int r = 0; r < R; r++) {
    note(top, x[r]);
    p[r * m] = x[r];
  }
}

// The two parts of a generic stage (any other prime R): the pre-shift and,
// for dit, the twiddle of entry i in place; then whole outputs
// y_k = sum_r x_r w_R^{rk}, output o of butterfly o / R
template <bool DIF>
FX_HD c64 generic_pre(c64 v, int i, int m, int R, int tstep, const FastDiv& md, const FastDiv& rd,
                      const int4* __restrict__ tw, int sin)
{
  if (sin) v = {rsh(v.x, sin), rsh(v.y, sin)};
  if (!DIF) {
    const int g = quot(i, md), j = i - g * m, r = g - quot(g, rd) * R;
    if (j && r) v = mulw(v, FX_TW(tw + j * r * tstep));
  }
  return v;
}
template <bool DIF>
FX_HD c64 generic_out(const c64* buf, int o, int& pos, int n, int L, int m, int R, const FastDiv& md,
                      const FastDiv& rd, const int4* __restrict__ tw)
{
  const int tstep = n / L, rstep = n / R;
  const int q = quot(o, rd), k = o - q * R;
  const int b = quot(q, md), j = q - b * m;
  const c64* p = buf + b * L + j;
  c64 acc = p[0];
  int e = 0;
  for (int r = 1; r < R; r++) {
    e += k;
    if (e >= R) e -= R;
    const c64 x = p[r * m];
    acc = e ? add(acc, mulw(x, FX_TW(tw + e * rstep))) : add(acc, x);
  }
  if (DIF && j && k) acc = mulw(acc, FX_TW(tw + j * k * tstep));
  pos = b * L + j + k * m;
  return acc;
}

// FP64 bits -> fixed point at scale 2^K (rounded to nearest; below half a
// unit 0; subnormals 0) and back (nearest; underflow 0)
FX_HD long long to_fx(unsigned long long u, int K)
{
  const int e = (int)(u >> 52) & 0x7ff;
  if (e == 0) return 0;
  unsigned long long v = (u & 0xfffffffffffffull) | 0x10000000000000ull;
  const int s = e - 1075 + K;
  if (s >= 0) v <<= s;
  else v = s > -62 ? (v + (1ull << (-s - 1))) >> -s : 0ull;
  return (long long)u < 0 ? -(long long)v : (long long)v;
}
FX_HD unsigned long long to_fp(long long v, int K)
{
  if (v == 0) return 0ull;
  const unsigned long long sgn = (unsigned long long)v & 0x8000000000000000ull;
  const unsigned long long u = (unsigned long long)(v < 0 ? -v : v);
#ifdef __CUDA_ARCH__
  const int e = 63 - __clzll((long long)u);
#else
  const int e = 63 - __builtin_clzll(u);
#endif
  const unsigned long long f = e <= 52 ? u << (52 - e) : (u + (1ull << (e - 53))) >> (e - 52);
  const int x = e + 1023 - K;
  if (x <= 0) return sgn;
  if (x >= 2046) return sgn | 0x7ff0000000000000ull;
  // the leading bit of f carries into the exponent field
  return sgn | (((unsigned long long)(x - 1) << 52) + f);
}

// Shift down before a stage of radix R: no part of a sum may pass 2^BITS.  Two
// bounds hold: R times the largest magnitude, whose high words' union is
// top, and the L1 norm, 2^l1 at the current scale (the fixed point of a
// smooth input's few large outputs; l1 follows the shifts).
FX_HD int room(unsigned top, int R, float& l1)
{
  // |re + i im| <= sqrt(2) 2^32 (top + 1)
  const float b = log2f(((float)top + 1.0f) * 1.4143f * (float)R) + 32.0f;
  const float need = fminf(b, l1) - ((float)BITS - 0.001f);
  const int s = need > 0.0f ? (int)ceilf(need) : 0;
  l1 -= (float)s;
  return s;
}

// a constant re + i im in units of 2^-61 as limbs
FX_HD int4 limbs(long long re, long long im)
{
  const int rh = (int)((re + (1ll << 30)) >> 31), ih = (int)((im + (1ll << 30)) >> 31);
  return make_int4(rh, (int)(re - ((long long)rh << 31)), ih, (int)(im - ((long long)ih << 31)));
}

// Host: the stages of an n-point transform. Few, wide stages (each is one pass
// over the buffer), no radix above 15 (60 registers of values, two rounds
// of 512 threads at 12150 points); false if n has a prime factor above 7 and
// !allow_generic, or too many stages.
inline bool make_desc(int n, Desc& d, bool allow_generic)
{
  d.n = n;
  d.nst = 0;
  int left = n;
  auto push = [&](int r) {
    if (d.nst >= MAX_STAGES) return false;
    const int L = left;
    left /= r;
    d.rad[d.nst] = r;
    d.L[d.nst] = L;
    d.m[d.nst] = make_fastdiv(left);
    d.r[d.nst] = make_fastdiv(r);
    d.nst++;
    return true;
  };
  const int order[] = {15, 14, 10, 12, 9, 8, 7, 6, 5, 4, 3, 2};
  for (int r : order)
    while (left % r == 0)
      if (!push(r)) return false;
  if (left > 1 && !allow_generic) return false;
  for (int f = 11; left > 1; f += 2)
    while (left % f == 0)
      if (!push(f)) return false;
  return true;
}

// DIF output position p holds frequency rev[p]
inline std::vector<int> digit_reverse(const Desc& d)
{
  std::vector<int> rev(d.n);
  for (int p = 0; p < d.n; p++) {
    int q = p, k = 0, mult = 1;
    for (int s = 0; s < d.nst; s++) {
      const int m = d.L[s] / d.rad[s], dg = q / m;
      q -= dg * m;
      k += dg * mult;
      mult *= d.rad[s];
    }
    rev[p] = k;
  }
  return rev;
}

// exp(-2 pi i j / n) in units of 2^-61, the angle folded to [0, pi / 4] in
// whole numbers
inline std::vector<c64> roots(int n)
{
  std::vector<c64> oct(n / 2 + 1, c64{-1, 0}), t(n);
  for (int j = 0; j < n; j++) {
    const int q = (int)(4ll * j / n);
    const int r = (int)(4ll * j - (long long)q * n);  // angle (pi / 2) (q + r / n)
    const bool up = 2ll * r > n;
    c64& o = oct[up ? n - r : r];
    if (o.x < 0) {
      const long double a = 1.57079632679489661923132169163975144L * (long double)(up ? n - r : r) / (long double)n;
      o = {llrintl(cosl(a) * 2305843009213693952.0L), llrintl(sinl(a) * 2305843009213693952.0L)};
    }
    c64 v = up ? c64{o.y, -o.x} : c64{o.x, -o.y};  // exp(-i angle)
    for (int k = 0; k < q; k++) v = {v.y, -v.x};
    t[j] = v;
  }
  return t;
}

inline std::vector<int4> twiddles(int n)
{
  const std::vector<c64> r = roots(n);
  std::vector<int4> t(n);
  for (int j = 0; j < n; j++) t[j] = limbs(r[j].x, r[j].y);
  return t;
}

// One dif stage on the host (sizes without other prime factors)
template <int R>
inline unsigned host_stage(c64* z, const Desc& d, int s, const int4* tw, int sin)
{
  unsigned top = 0;
  for (int q = 0; q < d.n / R; q++) butterfly<R, true>(z, q, d.L[s], d.L[s] / R, d.n / d.L[s], d.m[s], tw, sin, top);
  return top;
}

// Host: the tables of a Chirp of n points on transform d (d.n >= 2 n - 1);
// returns kb
inline int chirp_tables(int n, const Desc& d, const std::vector<int4>& tw, std::vector<int4>& w, std::vector<int4>& b)
{
  const int T = d.n;
  const std::vector<c64> r2 = roots(2 * n);
  std::vector<c64> z(T, c64{0, 0});
  w.resize(n);
  b.resize(T);
  int K = 59;
  for (int j = 0; j < n; j++) {
    const c64 v = r2[(int)((long long)j * j % (2ll * n))];
    w[j] = limbs(v.x, v.y);
    z[j] = {rsh(v.x, 2), -rsh(v.y, 2)};
    if (j) z[T - j] = z[j];
  }
  float l1 = 128.0f;
  unsigned top = (1u << 27);
  for (int s = 0; s < d.nst; s++) {
    const int sin = room(top, d.rad[s], l1);
    K -= sin;
    switch (d.rad[s]) {
      case 2: top = host_stage<2>(z.data(), d, s, tw.data(), sin); break;
      case 3: top = host_stage<3>(z.data(), d, s, tw.data(), sin); break;
      case 4: top = host_stage<4>(z.data(), d, s, tw.data(), sin); break;
      case 5: top = host_stage<5>(z.data(), d, s, tw.data(), sin); break;
      case 6: top = host_stage<6>(z.data(), d, s, tw.data(), sin); break;
      case 7: top = host_stage<7>(z.data(), d, s, tw.data(), sin); break;
      case 8: top = host_stage<8>(z.data(), d, s, tw.data(), sin); break;
      case 9: top = host_stage<9>(z.data(), d, s, tw.data(), sin); break;
      case 10: top = host_stage<10>(z.data(), d, s, tw.data(), sin); break;
      case 12: top = host_stage<12>(z.data(), d, s, tw.data(), sin); break;
      case 14: top = host_stage<14>(z.data(), d, s, tw.data(), sin); break;
      case 15: top = host_stage<15>(z.data(), d, s, tw.data(), sin); break;
    }
  }
  long double mx = 0;
  for (const c64& v : z) mx = std::max(mx, hypotl((long double)v.x, (long double)v.y));
  int kb;
  frexpl(ldexpl(mx, -K) / T, &kb);
  const long double sc = ldexpl(1.0L, BITS - K - kb) / T;
  for (int p = 0; p < T; p++) b[p] = limbs(llrintl((long double)z[p].x * sc), llrintl((long double)z[p].y * sc));
  return kb;
}

}  // namespace fx
}  // namespace cl2pt
