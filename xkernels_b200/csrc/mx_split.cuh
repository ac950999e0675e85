// bf16 activations as two block-scaled 8-bit terms, x = 2^(sh - 127) * hi + 2^(sl - 127) * lo, for the
// block-scaled tensor-core path of the MXFP4 layers.
//
// A bf16 number has 8 significant bits.  Rounded to e5m2 (3 bits) it leaves a remainder of at most half a
// unit in that third place, which is an integer of at most 16 in units of the bf16 number's last place: e4m3
// (4 significant bits) holds every such integer.  So the two terms ARE the number, as long as the range lasts:
// with the largest magnitude of the 32-element block at 2^14 in e5m2 and its remainder at 2^8 in e4m3, every
// element down to 2^-13 of the block's largest is exact, and a smaller one is off by at most 2^-21 of the
// largest - below what the fp32 sum over the block keeps.  hi carries infinities and NaN (lo is 0 there).
#pragma once
#include <stdint.h>

namespace xkb {
namespace mx {

// Scale bytes (e8m0) of a block from the largest |x| of its finite elements, given as bf16 bits.
__device__ __forceinline__ uint32_t hi_scale(uint32_t max_abs_bits) {
  const uint32_t e = max_abs_bits >> 7;
  return e > 14u ? e - 14u : 0u;
}
constexpr uint32_t kLoShift = 3;   // lo's scale byte is hi's plus this: half of e5m2's last place at 2^14 is 2^11
__device__ __forceinline__ float hi_factor(uint32_t sh) { return __uint_as_float((254u - sh) << 23); }   // 2^(127 - sh)

__device__ __forceinline__ uint32_t finite_abs_bits(uint32_t bits16) {
  const uint32_t a = bits16 & 0x7FFFu;
  return a < 0x7F80u ? a : 0u;
}

// Two elements (x0 in the low byte).  f0, f1 = hi_factor of their blocks' scales.
__device__ __forceinline__ void split_pair(float x0, float x1, float f0, float f1, uint32_t& hi2, uint32_t& lo2) {
  const float y0 = x0 * f0, y1 = x1 * f1;   // exact: a power of two
  uint16_t h, l;
  asm("cvt.rn.satfinite.e5m2x2.f32 %0, %1, %2;" : "=h"(h) : "f"(y1), "f"(y0));
  uint32_t back;
  asm("cvt.rn.f16x2.e5m2x2 %0, %1;" : "=r"(back) : "h"(h));
  const __half2 hb = *reinterpret_cast<const __half2*>(&back);
  const float r0 = (y0 - __low2float(hb)) * 0.125f, r1 = (y1 - __high2float(hb)) * 0.125f;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(l) : "f"(r1), "f"(r0));
  hi2 = h;
  lo2 = l;
  const uint32_t a0 = __float_as_uint(x0) & 0x7FFFFFFFu, a1 = __float_as_uint(x1) & 0x7FFFFFFFu;
  if (a0 >= 0x7F800000u) {
    hi2 = (hi2 & 0xFF00u) | (a0 > 0x7F800000u ? 0x7Fu : (0x7Cu | (__float_as_uint(x0) >> 31 << 7)));
    lo2 &= 0xFF00u;
  }
  if (a1 >= 0x7F800000u) {
    hi2 = (hi2 & 0x00FFu) | ((a1 > 0x7F800000u ? 0x7Fu : (0x7Cu | (__float_as_uint(x1) >> 31 << 7))) << 8);
    lo2 &= 0x00FFu;
  }
}

}  // namespace mx
}  // namespace xkb
