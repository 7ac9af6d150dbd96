// FP32 <-> FP64 conversions in integer arithmetic.
//
// GB300 converts between the two on its FP64 pipe: 2 lanes per clock per SM measured in both
// directions (594 G/s on 152 SMs), the rate of an FP64 fused multiply-add, against 64 and
// more per clock for integer operations.  In the mixed-precision kernels conversions were a
// third of the FP64-pipe work.  These give the hardware conversion's result bit for bit:
// f32 -> f64 is exact, f64 -> f32 rounds to nearest even, subnormals and infinities included
// (a NaN stays a NaN).  Normal numbers, nearly all, take the short path; the rest is integer
// arithmetic as well, because even a conversion whose lanes are all predicated off takes its
// slot on the FP64 pipe.
#pragma once
#include <stdint.h>

namespace nrt {

__device__ __forceinline__ double f2d(float f) {
  const uint32_t u = __float_as_uint(f), s = u & 0x80000000u, m = u & 0x7fffffffu;
  // normal: the exponent rebiased by 896, the mantissa shifted by 29
  uint32_t hi = (m >> 3) + 0x38000000u, lo = u << 29;
  if (m - 0x00800000u >= 0x7f000000u) {
    if (m >= 0x7f800000u) {  // infinity or NaN
      hi = 0x7ff00000u | (m >> 3);
    } else if (m == 0) {
      hi = lo = 0;
    } else {  // subnormal: m 2^-149, normalised
      const int k = __clz(m) - 8;
      const uint32_t q = (m << k) & 0x7fffffu;
      hi = ((uint32_t)(897 - k) << 20) | (q >> 3);
      lo = q << 29;
    }
  }
  return __hiloint2double((int)(s | hi), (int)lo);
}

__device__ __forceinline__ float d2f(double d) {
  const uint32_t hi = (uint32_t)__double2hiint(d), lo = (uint32_t)__double2loint(d);
  const uint32_t s = hi & 0x80000000u, e = hi & 0x7ff00000u;
  // normal in FP32: the exponent rebiased by 896, 23 mantissa bits, nearest with ties to even
  uint32_t v = __funnelshift_l(lo, hi, 3) - 0xc0000000u;
  v += ((lo & 0x1fffffffu) + 0x0fffffffu + (v & 1u)) >> 29;
  v &= 0x7fffffffu;
  if (e - 0x38100000u > 0x0fd00000u) {
    if (e > 0x47e00000u) {  // overflow, infinity, NaN
      const bool nan = e == 0x7ff00000u && ((hi & 0x000fffffu) | lo) != 0;
      v = nan ? 0x7fffffffu : 0x7f800000u;
    } else {  // subnormal in FP32 or zero: the 53-bit mantissa shifted right by 30 to 54
      const int k = 926 - (int)(e >> 20);
      const uint64_t m = ((uint64_t)((hi & 0x000fffffu) | 0x00100000u) << 32) | lo;
      v = 0;
      if (k <= 54) {
        const uint64_t q = m >> k, rest = m & (((uint64_t)1 << k) - 1), half = (uint64_t)1 << (k - 1);
        v = (uint32_t)q + (uint32_t)(rest > half || (rest == half && (q & 1)));
      }
    }
  }
  return __uint_as_float(v | s);
}

}  // namespace nrt
