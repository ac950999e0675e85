// bf16 activations as three block-scaled 8-bit terms for the block-scaled tensor-core path of the MXFP4 layers:
//   x = 2^(s - 127) * (hi + 2^-4 * mid + 2^-8 * lo),   all three e5m2, s = the e8m0 scale byte of x's 32-element block.
//
// A bf16 number has 8 significant bits.  hi takes three of them and leaves a remainder of at most 16 units of the
// number's last place; mid takes three bits of that and leaves at most one unit (two to eight where hi is subnormal
// or 0), which lo holds.  With the largest magnitude of the block in [2^14, 2^15) every element down to 2^-31 of it
// is exact, whatever the weights pick out of the block, and a smaller one is off by at most 2^-39 of the largest's
// power of two.  (The fp32 accumulators keep 2^-24 of it, so no sum that holds the largest element sees the
// difference.)  Two terms do not reach that far: of e5m2 + e4m3, which also carry 8 bits, the e4m3 one runs out 13
// powers of two below the largest, and a weight row that is 0 at the large elements of its blocks shows it.
// hi carries infinities and NaN (mid and lo are 0 there).
#pragma once
#include <stdint.h>

namespace xkb {
namespace mx {

// Scale byte (e8m0) of hi from the largest |x| of the block's finite elements, given as bf16 bits.  Blocks below
// 2^-105 keep the smallest byte that leaves room for the other terms': 2^-24 there is below bf16's smallest number.
constexpr uint32_t kMidShift = 4, kLoShift = 8;   // the scale bytes of mid and lo are hi's minus these
__device__ __forceinline__ uint32_t hi_scale(uint32_t max_abs_bits) {
  const uint32_t e = max_abs_bits >> 7;
  return e > 14u + kLoShift ? e - 14u : kLoShift;
}
__device__ __forceinline__ float hi_factor(uint32_t sh) { return __uint_as_float((254u - sh) << 23); }   // 2^(127 - sh)

__device__ __forceinline__ uint32_t finite_abs_bits(uint32_t bits16) {
  const uint32_t a = bits16 & 0x7FFFu;
  return a < 0x7F80u ? a : 0u;
}

__device__ __forceinline__ uint16_t to_e5m2x2(float x0, float x1, float& back0, float& back1) {
  uint16_t h;
  asm("cvt.rn.satfinite.e5m2x2.f32 %0, %1, %2;" : "=h"(h) : "f"(x1), "f"(x0));
  uint32_t f;
  asm("cvt.rn.f16x2.e5m2x2 %0, %1;" : "=r"(f) : "h"(h));
  const __half2 b = *reinterpret_cast<const __half2*>(&f);
  back0 = __low2float(b);
  back1 = __high2float(b);
  return h;
}

// Two elements (x0 in the low byte).  f0, f1 = hi_factor of their blocks' scales.
__device__ __forceinline__ void split_pair(float x0, float x1, float f0, float f1, uint32_t& hi2, uint32_t& mid2, uint32_t& lo2) {
  const float y0 = x0 * f0, y1 = x1 * f1;   // exact, as the differences are: powers of two
  float h0, h1, m0, m1, l0, l1;
  hi2 = to_e5m2x2(y0, y1, h0, h1);
  const float r0 = (y0 - h0) * 16.f, r1 = (y1 - h1) * 16.f;
  mid2 = to_e5m2x2(r0, r1, m0, m1);
  lo2 = to_e5m2x2((r0 - m0) * 16.f, (r1 - m1) * 16.f, l0, l1);
  const uint32_t a0 = __float_as_uint(x0) & 0x7FFFFFFFu, a1 = __float_as_uint(x1) & 0x7FFFFFFFu;
  if (a0 >= 0x7F800000u) {
    hi2 = (hi2 & 0xFF00u) | (a0 > 0x7F800000u ? 0x7Fu : (0x7Cu | (__float_as_uint(x0) >> 31 << 7)));
    mid2 &= 0xFF00u;
    lo2 &= 0xFF00u;
  }
  if (a1 >= 0x7F800000u) {
    hi2 = (hi2 & 0x00FFu) | ((a1 > 0x7F800000u ? 0x7Fu : (0x7Cu | (__float_as_uint(x1) >> 31 << 7))) << 8);
    mid2 &= 0x00FFu;
    lo2 &= 0x00FFu;
  }
}

}  // namespace mx
}  // namespace xkb
