// fp32 operands as pairs of half-precision numbers for tcgen05.mma kind::f16.
//
// v * s = hi + lo with s a power of two that brings the largest value of a row to 2 .. 4 (a row: what shares one index of the
// result, a pixel's or an output channel's values over the depth): hi is v * s rounded to 11 bits, lo the rest rounded to
// 11 bits, together 22 bits and a sign, or 2^-25 absolute where that is more, 2^-26 of the row's largest value.  Three MMAs, hi * hi +
// hi * lo + lo * hi, in fp32 accumulators make a product to 2^-24 of the row's norm; the result is multiplied by the two
// inverse powers of two, which is exact.
//
// Against tf32 pairs (11 + 11 bits cut off, as many MMAs): an operand takes half the bytes in shared and tensor memory and
// an MMA covers 16 of the depth in the time of 8.  Those kernels were bound by shared memory: 144 KB per step of 128 x 128 x 32
// at 128 bytes a cycle, 1150 cycles of which the MMAs were busy 768; 72 KB and 384 cycles now.
//
// A row's scale is that of the first step of 32 in which it has a value other than zero (zeros need none), so that nothing has
// to be read twice.  Later values may be 2^14 times larger; beyond that hi is infinite and the results of that row come out as
// NaN, like those of an infinite value or of a row below 2^-61, and are marked, and worked out again by fp32 FMAs.
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

// The scale of a row whose largest value is m > 0.  NaN below 2^-61: its products are then worked out again.
__device__ __forceinline__ float f32_row_scale(float m) {
  const uint32_t e = __float_as_uint(m) >> 23;  // biased; the scale's is 254 - e + 1
  if (e < 66u) return __uint_as_float(0x7fc00000u);
  return __uint_as_float((255u - min(e, 190u)) << 23);
}
// What a result is multiplied by: 1 / s, 0 for a row of zeros only (its scale is still 0).
__device__ __forceinline__ float f32_row_unscale(float s) {
  return s == 0.f ? 0.f : __uint_as_float(0x7f000000u - __float_as_uint(s));
}

__device__ __forceinline__ uint64_t f32_pair(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
// Two values v (packed) times s as hi and lo halves, the first value in the low half.
__device__ __forceinline__ void f32_split2(uint64_t v, uint64_t s, uint32_t &hi, uint32_t &lo) {
  uint64_t a, r;
  float a0, a1, r0, r1;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(a) : "l"(v), "l"(s));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a0), "=f"(a1) : "l"(a));
  const __half2 h = __floats2half2_rn(a0, a1);
  const float2 f = __half22float2(h);
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(f32_pair(f.x, f.y)));  // (exact)
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r0), "=f"(r1) : "l"(r));
  const __half2 l = __floats2half2_rn(r0, r1);
  hi = *reinterpret_cast<const uint32_t *>(&h);
  lo = *reinterpret_cast<const uint32_t *>(&l);
}
