// f64_slices.cuh -- FP64 operands of a tensor-core contraction as exact integer slices.
//
// A vector of FP64 numbers that share the biased exponent E of their largest magnitude is rounded to
// the integers X = round(x 2^(1075 - E)), |X| < 2^53: the largest binade keeps all its 53 bits, smaller
// values are rounded at the same absolute place.  X is cut into six balanced base-512 digits
// X = sum_l d_l 512^(5 - l), |d_l| <= 256, each an integer that BF16 holds exactly; slice l stores
// d_l 2^(-9 l).  Products of slices are integers of at most 2^16 (times 2^(-9 (i + j))), so that the
// tensor core's FP32 accumulators add the products of one level i + j <= 3 over 64 terms without
// rounding: (level + 1) 64 2^16 <= 2^24.  (The splitting is the error-free transformation of Ozaki,
// Ogita, Oishi and Rump, Numer. Algorithms 59, 95 (2012).)
//
// The digits are read from Y = X + bias, bias = sum_l 256 512^(5 - l): field l of Y (9 bits; the top one
// up to 512) is d_l + 256, so no carry has to be followed.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace cxc {
namespace f64s {

constexpr int kSlices = 6;
constexpr unsigned long long kBias = 256ull * (1ull + (1ull << 9) + (1ull << 18) + (1ull << 27) + (1ull << 36) +
                                               (1ull << 45));

// Y of x for the shared biased exponent E >= x's own; zeros and subnormal x give digits of zero.
__device__ __forceinline__ unsigned long long to_fixed(double x, int E) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const int ex = (int)((hi >> 20) & 0x7FFu);
  unsigned long long man = ((unsigned long long)((hi & 0xFFFFFu) | 0x100000u) << 32) | lo;
  const int sh = E - ex;
  man += sh > 0 ? (1ull << (sh < 55 ? sh - 1 : 0)) : 0ull;  // round half away from zero
  man = (ex == 0 || sh > 54) ? 0ull : man >> (sh < 64 ? sh : 63);
  return (hi >> 31) ? kBias - man : kBias + man;
}

// Slice l (d_l 2^(-9 l)) of Y as an FP32 number whose low 16 bits are zero (exact in BF16): the field is
// put into the low mantissa bits of 2^(23 - 9 l), whose unit in the last place is 2^(-9 l).
template <int l>
__device__ __forceinline__ uint32_t slice_bits(unsigned long long Y) {
  uint32_t f;
  if (l == 0)
    f = (uint32_t)(Y >> 45);
  else
    f = (uint32_t)(Y >> (45 - 9 * l)) & 511u;
  constexpr uint32_t kExp = (uint32_t)(127 + 23 - 9 * l) << 23;
  return __float_as_uint(__fsub_rn(__uint_as_float(kExp | f), __uint_as_float(kExp | 256u)));
}

// The slices of two neighbouring elements as packed BF16 pairs (a in the low half): w[l].
__device__ __forceinline__ void slice_pairs(unsigned long long a, unsigned long long b, uint32_t (&w)[kSlices]) {
  w[0] = __byte_perm(slice_bits<0>(a), slice_bits<0>(b), 0x7632);
  w[1] = __byte_perm(slice_bits<1>(a), slice_bits<1>(b), 0x7632);
  w[2] = __byte_perm(slice_bits<2>(a), slice_bits<2>(b), 0x7632);
  w[3] = __byte_perm(slice_bits<3>(a), slice_bits<3>(b), 0x7632);
  w[4] = __byte_perm(slice_bits<4>(a), slice_bits<4>(b), 0x7632);
  w[5] = __byte_perm(slice_bits<5>(a), slice_bits<5>(b), 0x7632);
}

// The level sums of one K group (level l: an integer times 2^(-9 l); the last one levels 4 and 5
// together) as one integer in units of 2^(-36), exact but for the last level's rounding.
__device__ __forceinline__ long long level_sum(float s0, float s1, float s2, float s3, float s4) {
  const int i0 = __float2int_rn(s0);
  const int i1 = __float2int_rn(s1 * 512.f);
  const int i2 = __float2int_rn(s2 * 262144.f);
  const int i3 = __float2int_rn(s3 * 134217728.f);
  const long long i4 = (long long)__float2int_rn(s4 * 68719476736.f);
  return ((long long)i0 << 36) + ((long long)i1 << 27) + ((long long)i2 << 18) + ((long long)i3 << 9) + i4;
}

// V 2^e as a double, by adding e to the FP64 pattern's exponent (V = 0 stays 0; kScaleMin <= e), or NaN from
// e = kScaleNan on (an operand vector of 2^957 and above, or with infinities or NaN).
constexpr int kScaleMin = -1000;
constexpr int kScaleNan = 957;
__device__ __forceinline__ double scaled_or_nan(long long V, int e) {
  const double d = __ll2double_rn(V);
  const int hi = V == 0 ? 0 : __double2hiint(d) + (e << 20);
  return __hiloint2double(e >= kScaleNan ? 0x7FF80000 : hi, __double2loint(d));
}

}  // namespace f64s
}  // namespace cxc
