// efe_fixed.cuh -- sums of products of doubles in 64-bit integers.
//
// This part issues FP64 at 1/64 of its FP32 rate (1.9 fused multiply-adds per clock and SM measured)
// but 32 x 32 + 64 bit integer multiply-adds at 55.  A double that shares a scale with the others of its sum is
// therefore carried as a 57-bit integer in two digits, v = (h 2^28 + l) 2^(em - 1079) with |h| <= 2^29 and
// |l| <= 2^27, and a product costs three multiply-adds into two accumulators (h h, and h l + l h together; l l, below
// 2^-60 of the largest product, is left out): 18 products per clock and SM, ten times the FP64 pipe.  The accumulation
// is exact; what is lost is the rounding of the operands to the common scale, 2^-58 of the largest operand (FP64
// rounds every product and sum at 2^-53).  The error is thus one of the largest operands' product, not of the sum's own
// terms: operands share a scale only where they are of one size by their nature, in an element the values of one component.
// The components of dN/dX of a thin element, and of the displacements of a plate, are not, and have scales of their own.
// At most 31 products to a sum (h h reaches 2^58).  em: biased exponent of the largest operand.  Scales are integers
// that may leave the exponent range; FX_NAN marks non-finite operands.
#pragma once
#include <cstdint>

namespace efe {

struct fx {
  int32_t h, l;
};
constexpr int FX_NAN = 1 << 20;

// biased exponent of |x| (0 for zero and subnormals; far above FX_NAN if not finite, so that sums of scales stay above it)
__device__ __forceinline__ int fx_exponent(double x) {
  const int e = (__double2hiint(x) >> 20) & 0x7ff;
  return e == 0x7ff ? 4 * FX_NAN : e;
}
// V = h 2^28 + l with |l| <= 2^27
__device__ __forceinline__ fx fx_split(int64_t V) {
  const int32_t h = (int32_t)((V + (1 << 27)) >> 28);
  return fx{h, (int32_t)((uint32_t)V - ((uint32_t)h << 28))};
}
// x (|x| < 2^(em - 1022)) at scale em, rounded to nearest; 0 where em is FX_NAN or x is subnormal
__device__ __forceinline__ fx fx_make(double x, int em) {
  const uint64_t X = (uint64_t)__double_as_longlong(x);
  const int e = (int)(X >> 52) & 0x7ff, s = e - em + 4;  // at most 4
  uint64_t m = e ? (X & 0xfffffffffffffull) | (1ull << 52) : 0ull;
  if (s < 0) m = s > -60 ? (m + (1ull << (-s - 1))) >> -s : 0ull;
  int64_t V = (int64_t)(s >= 0 ? m << s : m);
  if ((int64_t)X < 0) V = -V;
  return fx_split(V);
}
struct FxSum {
  int64_t hh, cr;
};
__device__ __forceinline__ void fx_fma(FxSum& s, fx a, fx b) {
  s.hh += (int64_t)a.h * b.h;
  s.cr += (int64_t)a.h * b.l;
  s.cr += (int64_t)a.l * b.h;
}
// V / 2^d rounded to nearest
__device__ __forceinline__ int64_t fx_shift(int64_t V, int d) { return d > 0 ? (V + (1ll << (d - 1))) >> d : V; }
// the sum in units of 2^(ema + emb - 2102 - B), B <= 27
__device__ __forceinline__ int64_t fx_int(const FxSum& s, int B = 0) {
  if (B < 0) return fx_shift(s.hh + (s.cr >> 28), -B);
  return (s.hh << B) + (B < 28 ? (s.cr + (1ll << 27 >> B)) >> (28 - B) : 0);
}
// V / 2^d rounded down, for sums that keep bits to spare: one unit is 2^-57 or less of what they can hold
__device__ __forceinline__ int64_t fx_down(int64_t V, int d) { return V >> min(d, 63); }
// A + B of scales sa, sb (fx_int of both with B = -1, so that the sum fits); sa becomes the sum's scale, less that shift
__device__ __forceinline__ int64_t fx_add(int64_t A, int& sa, int64_t B, int sb) {
  const int m = max(sa, sb);
  const int64_t v = fx_down(A, m - sa) + fx_down(B, m - sb);
  sa = m;
  return v;
}
// An operand of scale em as a float, from its upper digit: unit = fx_unit(em)
__device__ __forceinline__ float fx_unit(int em) {
  const int e = em - 1051 + 127;
  if (e > 0 && e < 255) return __int_as_float(e << 23);
  return em >= FX_NAN ? __int_as_float(0x7fc00000) : ldexpf(1.0f, max(-300, min(300, em - 1051)));
}
__device__ __forceinline__ float fx_float(fx v, float unit) { return (float)v.h * unit; }
// the upper 32 bits of |hh|, roughly: __clz of them (or of an OR of several) counts the places to spare
__device__ __forceinline__ int fx_bits(const FxSum& s) {
  const int h = (int)(s.hh >> 32);
  return h ^ (h >> 31);
}
// a b as an operand of scale ema + emb - 1022
__device__ __forceinline__ fx fx_mul(fx a, fx b) {
  FxSum s{0, 0};
  fx_fma(s, a, b);
  return fx_split(fx_int(s, -1));
}
// V 2^(em - 2102) with em the sum of the two operands' scales: one conversion, the exponent added in integers
__device__ __forceinline__ double fx_value(int64_t V, int em) {
  if (em >= FX_NAN) return __longlong_as_double(0x7ff8000000000000ll);
  if (V == 0) return 0.0;
  const double x = (double)V;
  const int hi = __double2hiint(x), e = ((hi >> 20) & 0x7ff) + em - 2102;
  if (e > 0 && e < 0x7ff) return __hiloint2double(hi + ((em - 2102) << 20), __double2loint(x));
  return scalbn(x, max(-2200, min(2200, em - 2102)));
}

}  // namespace efe
