// fp32 operands as pairs of half-precision numbers for tcgen05.mma kind::f16.
//
// v * s = hi + 2^-11 lo with s a power of two that brings the largest value of a row to 2^14 .. 2^15, where it is known (a row: what
// shares one index of the result, a pixel's or an output channel's values over the depth): hi is v * s rounded to 11 bits, lo the rest
// rounded to 11 bits, together 22 bits and a sign, or 2^-36 absolute where that is more, below 2^-28 of the row's largest value.  (At
// the scale of hi, lo would end at 2^-25; and with the largest at 2 .. 4 values below 2^-12 of it lost bits, which shows where small
// values meet large ones of the other operand: 6e-6 instead of 8e-8 with a column of X times 1000 and W's divided by it.)  Three MMAs, hi * hi in one fp32
// accumulator and hi * lo + lo * hi in another; the second one's 2^-11 and the two inverse powers of two are exact.
//
// Against tf32 pairs (11 + 11 bits cut off, as many MMAs): an operand takes half the bytes in shared and tensor memory and
// an MMA covers 16 of the depth in the time of 8.  Those kernels were bound by shared memory: 144 KB per step of 128 x 128 x 32
// at 128 bytes a cycle, 1150 cycles of which the MMAs were busy 768; 72 KB and 384 cycles now.
//
// Where a row's largest value is not known beforehand its scale is one that the values at hand allow, and follows them when they
// grow, or the tile is done once more.  Results of an infinite value come out as NaN, and are marked, and worked out again by fp32
// FMAs.
#pragma once

#include <cuda_fp16.h>

#include "common.cuh"

constexpr uint32_t F32_AGAIN = 0x7fc0a6a1u;  // stored for a result to be worked out again

// The scale that brings a row's largest value m > 0 to 2^TOP .. 2^(TOP + 1): at most 2^126, so that its inverse is a normal number
// too.  (Rows that it leaves smaller are below 2^-111 and have no bits that lo does not hold.)
template <int TOP = 14>
__device__ __forceinline__ float f32_row_scale(float m) {
  const uint32_t e = __float_as_uint(m) >> 23;  // biased; the scale's is 254 - e + TOP
  return __uint_as_float(min(254u + TOP - min(e, 254u), 253u) << 23);
}
constexpr float F32_HIGH = 65504.f;  // what no value times its scale may reach
// What a result is multiplied by: 1 / s, 0 for a row of zeros only (its scale is still 0).  X's and W's one after the other: their
// product may leave the range of fp32 where the result does not.
__device__ __forceinline__ float f32_row_unscale(float s) {
  return s == 0.f ? 0.f : __uint_as_float(0x7f000000u - __float_as_uint(s));
}

__device__ __forceinline__ uint64_t f32_pair(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 f32_parts(uint64_t v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ uint64_t f32_mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f32_fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

constexpr float F32_LO = 1.f / 2048.f;  // what the accumulator of the small products is multiplied by

// Two values v (packed) times s as hi and lo halves, the first value in the low half.
__device__ __forceinline__ void f32_split2(uint64_t v, uint64_t s, uint32_t &hi, uint32_t &lo) {
  const uint64_t a = f32_mul2(v, s);
  const float2 a2 = f32_parts(a);
  const __half2 h = __floats2half2_rn(a2.x, a2.y);
  const float2 f = __half22float2(h);
  uint64_t r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(f32_pair(f.x, f.y)));  // (exact)
  const float2 r2 = f32_parts(f32_mul2(r, f32_pair(1.f / F32_LO, 1.f / F32_LO)));
  const __half2 l = __floats2half2_rn(r2.x, r2.y);
  hi = *reinterpret_cast<const uint32_t *>(&h);
  lo = *reinterpret_cast<const uint32_t *>(&l);
}

__device__ __forceinline__ float f32_finite_abs(float v) {
  v = fabsf(v);
  return v < INFINITY ? v : 0.f;
}

// The scale of values that share one although they belong to several rows (the places of a convolution's patch or strip), from the
// largest finite ones that the warps which looked at them found (all zero: 0).  It brings the largest to 2^12 .. 2^13, and is fair
// for others whose largest comes to F32_LOW at least and stays below F32_HIGH.  A value of 2^-14 and more is then held to 22 bits,
// 2^-22 of the largest or less.  What does not fit (values that are not finite, and those beyond 2^20 times all that the other
// warps have, whose largest would be held to less than 2^-29 of it) is left out: its results come out as NaN and are worked out
// again, and the others keep their bits.
constexpr float F32_LOW = 256.f;
template <int WARPS>
__device__ __forceinline__ float f32_shared_scale(const volatile float *most) {
  float first = 0.f, second = 0.f;
#pragma unroll
  for (int i = 0; i < WARPS; ++i) {
    const float m = most[i];
    second = fmaxf(second, fminf(first, m));
    first = fmaxf(first, m);
  }
  if (second > 0.f && first * (1.f / 1048576.f) > second) first = second;
  return first > 0.f ? f32_row_scale<12>(first) : 0.f;
}

// What a result is worked out again by: fp32 FMAs, a warp per result, every lane the whole of it.  (Results to be worked out again
// come by the pixel, with all of its channels; 3x3, 128 -> 128 channels, one infinite value: 0.69 ms on top, 3.6 with a thread each.)
// Of a product's
// row and column ...
__device__ __forceinline__ float f32_warp_sum(float v) {
#pragma unroll
  for (int d = 16; d > 0; d /= 2) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}
__device__ __forceinline__ float f32_warp_dot(const float *x, int64_t x_ks, const float *w, int64_t K) {
  float sum = 0.f;
#pragma unroll 8  // (so many loads on their way)
  for (int64_t k = threadIdx.x & 31; k < K; k += 32) sum = fmaf(x[k * x_ks], w[k], sum);
  return f32_warp_sum(sum);
}
// ... and of a convolution's window with its corner at (top, left) of an image, padding left out.
__device__ __forceinline__ float f32_warp_window(const float *image, const float *filter, int channels, int H, int W, int KH, int KW,
                                                 int top, int left) {
  float sum = 0.f;
  const int taps = KH * KW;
#pragma unroll 4
  for (int e = threadIdx.x & 31; e < channels * taps; e += 32) {
    const int c = e / taps, tap = e - c * taps, i = tap / KW, h = top + i, v = left + tap - i * KW;
    if (h >= 0 && h < H && v >= 0 && v < W) sum = fmaf(image[(static_cast<int64_t>(c) * H + h) * W + v], filter[e], sum);
  }
  return f32_warp_sum(sum);
}
// The lanes of a warp whose result is to be worked out again, one after the other: again(lane) by all of them.
template <typename Again>
__device__ __forceinline__ void f32_each_again(bool mine, Again again) {
  for (uint32_t left = __ballot_sync(0xffffffffu, mine); left != 0; left &= left - 1) again(__ffs(left) - 1);
}
