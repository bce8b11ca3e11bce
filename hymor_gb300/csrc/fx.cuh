// Fixed-point products for FP64 sums on the integer pipe: the batched stencil matvec.
//
// On GB300 a warp's FP64 multiply-add occupies its sub-partition for ~70 cycles and its 32 x 32
// -> 64-bit integer multiply-add for ~5 (measured: 1.6 against 24 per SM and clock), so a sum of
// products is cheaper in integers: with every factor a 58-bit integer against a power of two
// that the factors of its sum share, split into a high and a low part of 29 bits each,
//   sum a x = 2^58 sum ah xh + 2^29 sum (ah xl + al xh) + sum al xl,
// three multiply-adds per product, the last sum dropped (below 2^-2 of the unit kept). The sums
// are exact in 64 bits for nine products: |ah|, |xh| <= 2^29, |al|, |xl| <= 2^28.
#pragma once

#include <cuda_runtime.h>

namespace hymor {

constexpr int kFxBits = 58, kFxLow = 29;

// A factor's shared exponent: E with |x| < 2^E for all of them, from the largest biased exponent
// field of their doubles; kFxZero when all are zero, kFxBad when one is not finite or E lies
// outside +-900 (the products' exponents then leave the double range's middle). A subnormal is not
// zero, and its product with a large factor is an ordinary number: it counts as the smallest
// normal exponent, so that factors of which it is the largest are kFxBad.
constexpr int kFxZero = -32768, kFxBad = 32767;
__device__ __forceinline__ int fx_field(double x) {
  const unsigned h = (unsigned)__double2hiint(x) << 1;
  return max((int)(h >> 21), (int)((h | (unsigned)__double2loint(x)) != 0u));
}
__device__ __forceinline__ int fx_exponent(int field) {
  if (field == 0) return kFxZero;
  const int e = field - 1022;
  return e > 900 || e < -900 ? kFxBad : e;
}

// x as a high and a low part of round(x 2^(58 - E)), |x| < 2^E
__device__ __forceinline__ int2 fx_split(double x, int E) {
  const long long b = __double_as_longlong(x);
  const int f = (int)((b >> 52) & 0x7ff);
  // x = +-m 2^(f - 1085), m with its leading bit at 62; the shift is at least 5
  const unsigned long long u = f ? ((unsigned long long)b << 10 & 0x3ffffffffffffc00ull) | 0x4000000000000000ull : 0;
  const int sh = 1085 - kFxBits + E - f;
  long long m = sh < 64 ? (long long)((u + (1ull << (sh - 1))) >> sh) : 0;
  if (b < 0) m = -m;
  const int h = (int)((m + (1ll << (kFxLow - 1))) >> kFxLow);
  return make_int2(h, (int)(m - ((long long)h << kFxLow)));
}

// T 2^k rounded to the nearest double (ties to even); ok is cleared when the result is not a
// normal double (T == 0 gives +0)
__device__ __forceinline__ double fx_to_double(long long T, int k, bool& ok) {
  if (T == 0) return 0.0;
  const unsigned long long n = T < 0 ? 0ull - (unsigned long long)T : (unsigned long long)T;
  const int lz = __clzll((long long)n);
  const unsigned long long m = n << lz;
  unsigned long long r = m >> 11;
  const unsigned rem = (unsigned)m & 0x7ffu;
  r += rem > 0x400u || (rem == 0x400u && (r & 1));
  const int be = 63 + k - lz + 1023;
  ok = ok && be > 0 && be < 2046;
  // r's leading bit adds one to the exponent field, as does a carry to 2^53
  const unsigned long long bits = ((unsigned long long)(be - 1) << 52) + r;
  return __longlong_as_double((long long)(bits | (T < 0 ? 0x8000000000000000ull : 0ull)));
}

}  // namespace hymor
