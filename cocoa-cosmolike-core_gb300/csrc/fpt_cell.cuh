// fpt_cell.cuh -- where a multipole and a node fall on the FAST-PT k grid.
//
// fpti_row / fptb_row (cosmo2D.c:1411-1445) read a table row at ln k =
// ln(l + 1/2) - ln chi, linear in ln k on the uniform grid and 0 off it.  The
// grid coordinate r = (ln k - lim0) / dlnk is a multipole's part minus a
// node's part, each formed once (FP64); the kernels form the difference for
// every (multipole, node).
//   FP64 plan: as the reference, in FP64.
//   mixed plan: the parts as FP32 head and tail, their difference as an exact
//   two-float sum, the in-cell weight good to FP32 rounding (6e-8 of a cell).
//   The FP64 form costs ~25 instructions of the FP64 pipe (1/64 of the FP32
//   rate on GB300), a division and conversions among them, which bound every
//   kernel that took it per (multipole, node).
#pragma once
#include "common.cuh"

namespace cl2pt {

__device__ __forceinline__ float2 split2(double v)
{
  const float h = (float)v;
  return make_float2(h, (float)(v - (double)h));
}

// an FP64 value in the loop precision (FP32: nearest, by integer arithmetic on
// the bits -- a conversion instruction issues at the FP64 rate)
template <typename T> __device__ __forceinline__ T round_to(double v);
template <> __device__ __forceinline__ double round_to<double>(double v) { return v; }
template <> __device__ __forceinline__ float round_to<float>(double v) { return split_f64_bits(v).x; }

// cell i and in-cell weight w; off the grid (in = false) the row counts as 0,
// in the last cell it is the last value (w = 0)
template <typename T>
struct FptCell {
  int i;
  T w;
  bool in;
};

template <typename T> struct FptPart;
template <> struct FptPart<double> {
  typedef double type;
  static __device__ __forceinline__ double of_l(const Params& P, double lnl) { return lnl; }
  static __device__ __forceinline__ double of_p(const Params& P, double lnchi) { return lnchi; }
};
template <> struct FptPart<float> {
  typedef float2 type;
  static __device__ __forceinline__ float2 of_l(const Params& P, double lnl)
  {
    return split2((lnl - P.fpt_lim0) / P.fpt_lim2);
  }
  static __device__ __forceinline__ float2 of_p(const Params& P, double lnchi) { return split2(lnchi / P.fpt_lim2); }
};

__device__ __forceinline__ FptCell<double> fpt_cell(const Params& P, double lnl, double lnchi)
{
  const double lnk = lnl - lnchi;
  FptCell<double> c;
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
__device__ __forceinline__ FptCell<float> fpt_cell(const Params& P, float2 a, float2 b)
{
  // r = a - b as an unevaluated sum rs + rt (TwoSum of the heads)
  const float rs = __fsub_rn(a.x, b.x);
  const float bb = __fsub_rn(rs, a.x);
  const float rt = __fadd_rn(__fsub_rn(a.x, __fsub_rn(rs, bb)), __fsub_rn(-b.x, bb)) + (a.y - b.y);
  const float r = rs + rt;
  FptCell<float> c;
  c.in = !(r < 0.0f);
  // floor(r) without a conversion (round r - 1/2), then the exact in-cell
  // offset from the two-float r
  int i = __float_as_int((r - 0.5f) + 12582912.0f) - 0x4B400000;
  float w = (rs - (float)i) + rt;
  if (w < 0.0f) { i -= 1; w += 1.0f; }
  if (w >= 1.0f) { i += 1; w -= 1.0f; }
  if (!c.in || i < 0) i = 0;
  if (i + 1 >= P.fpt_n) {
    // past the grid's upper end by the exact offset (r itself is rounded to
    // 6e-5 of a cell there)
    if (i > P.fpt_n || (i == P.fpt_n && w > 0.0f)) c.in = false;
    i = P.fpt_n - 1;
    w = 0.0f;
  }
  c.i = i;
  c.w = w;
  return c;
}

// a row at cell c (0 off the grid)
template <typename T>
__device__ __forceinline__ T fpt_val(const T* row, const FptCell<T>& c, int n)
{
  if (!c.in) return (T)0;
  const T v0 = row[c.i];
  if (c.i + 1 >= n) return v0;
  return c.w * (row[c.i + 1] - v0) + v0;
}

}  // namespace cl2pt
