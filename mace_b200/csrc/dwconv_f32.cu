// fp32 depthwise convolution in NCHW with bias and activation.
//
// Reference behaviour: ref::DepthwiseConv2d (mace/ops/ref/depthwise_conv_2d.cc:36-125), filter
// [multiplier][C][KH][KW], the sum of a value taken in (kh, kw) order.
#include <algorithm>

#include "common.cuh"

namespace {

struct DwF32Params {
  const float *in, *filter, *bias;
  float *out;
  uint32_t planes;          // N * C * multiplier
  int C, H, W, Ho, Wo, mult_ch, KH, KW, sh, sw, dh, dw, pad_t, pad_l;
  uint32_t strips;          // runs of RH output rows per plane
  uint32_t threads;         // planes * strips * Wo
  uint32_t wo_mul, wo_shift, strips_mul, strips_shift, oc_mul, oc_shift, mc_mul, mc_shift;
  int act;
  float max_limit, coef;
};

// A thread computes RH output rows of one output column; the lanes of a warp are neighbouring
// columns (and, for narrow maps, the columns of the next run or plane), so every load of a tap is
// one run of a row.  Bound by DRAM for large maps: the kernel must have enough bytes in flight
// and must not spend more issue slots than the bytes take.  A run of rows loads each input row
// once for up to K output rows, all loads of a run are independent of each other (the
// compiler issues them ahead of the arithmetic), and an index costs a few multiply-highs instead
// of 64-bit divisions: one output per thread with 64-bit index arithmetic and bounds tests per tap ran
// 64 channels of 112 x 112 -> 56 x 56, batch 32, in 105.7 us = 1.2 TB/s; this form takes 29.1 us = 4.4 TB/s (and the next one,
// which such rows now go to, 25.4).
template <int K, int S, int RH>
__global__ void __launch_bounds__(256) dwconv_f32_rows_kernel(const DwF32Params p) {
  mb_grid_dep_launch();
  const uint32_t tid = blockIdx.x * 256u + threadIdx.x;
  if (tid >= p.threads) return;
  const uint32_t q = fast_div(tid, p.wo_mul, p.wo_shift);
  const int w = static_cast<int>(tid - q * static_cast<uint32_t>(p.Wo));
  const uint32_t plane = fast_div(q, p.strips_mul, p.strips_shift);
  const int h0 = static_cast<int>(q - plane * p.strips) * RH;
  const uint32_t n = fast_div(plane, p.oc_mul, p.oc_shift);
  const uint32_t m = plane - n * static_cast<uint32_t>(p.C * p.mult_ch);
  const uint32_t c = fast_div(m, p.mc_mul, p.mc_shift);
  const uint32_t o = m - c * static_cast<uint32_t>(p.mult_ch);
  const float *in = p.in + (static_cast<int64_t>(n) * p.C + c) * (static_cast<int64_t>(p.H) * p.W);
  const float *fp = p.filter + (static_cast<int64_t>(o) * p.C + c) * (K * K);
  const int iw0 = w * S - p.pad_l, ih0 = h0 * S - p.pad_t;
  bool col_ok[K];
#pragma unroll
  for (int j = 0; j < K; ++j) col_ok[j] = iw0 + j >= 0 && iw0 + j < p.W;
  mb_grid_dep_wait();
  float f[K * K];
#pragma unroll
  for (int i = 0; i < K * K; ++i) f[i] = mb_load(fp + i);
  const float bias = p.bias != nullptr ? mb_load(p.bias + m) : 0.f;
  float acc[RH];
#pragma unroll
  for (int r = 0; r < RH; ++r) acc[r] = 0.f;
  const float *row = in + static_cast<int64_t>(ih0) * p.W + iw0;
#pragma unroll
  for (int i = 0; i < (RH - 1) * S + K; ++i) {
    const bool row_ok = ih0 + i >= 0 && ih0 + i < p.H;
    float x[K];
#pragma unroll
    for (int j = 0; j < K; ++j) x[j] = (row_ok && col_ok[j]) ? mb_load(row + j) : 0.f;
    row += p.W;
#pragma unroll
    for (int r = 0; r < RH; ++r) {
      const int kh = i - r * S;
      if (kh >= 0 && kh < K) {
#pragma unroll
        for (int j = 0; j < K; ++j) acc[r] = fmaf(x[j], f[kh * K + j], acc[r]);
      }
    }
  }
  float *out = p.out + (static_cast<int64_t>(plane) * p.Ho + h0) * p.Wo + w;
#pragma unroll
  for (int r = 0; r < RH; ++r) acc[r] += bias;
  mb_activate_n(acc, p.act, p.max_limit, p.coef);
#pragma unroll
  for (int r = 0; r < RH; ++r) {
    if (h0 + r < p.Ho) *out = acc[r];
    out += p.Wo;
  }
}

// The same for 3x3 filters on rows of whole 16-byte words: a thread computes V = 4 (stride 1) or 2 (stride 2) neighbouring
// columns, whose inputs are one 16-byte load and one or two single values per row instead of 3 V; the values of a
// row are in flight together.  64 channels of 112 x 112, batch 32: stride 2, 29.2 us one column per thread, 25.7 this way
// (5.0 TB/s); stride 1, 53.7 -> 38.0 us (5.4 TB/s).
template <int S, int RH>
__global__ void __launch_bounds__(256) dwconv_f32_wide_kernel(const DwF32Params p) {
  constexpr int V = S == 1 ? 4 : 2, COLS = (V - 1) * S + 3;
  mb_grid_dep_launch();
  const uint32_t tid = blockIdx.x * 256u + threadIdx.x;
  if (tid >= p.threads) return;
  const uint32_t q = fast_div(tid, p.wo_mul, p.wo_shift);  // (by the groups of V columns per row)
  const int w = static_cast<int>(tid - q * static_cast<uint32_t>(p.Wo / V)) * V;
  const uint32_t plane = fast_div(q, p.strips_mul, p.strips_shift);
  const int h0 = static_cast<int>(q - plane * p.strips) * RH;
  const uint32_t n = fast_div(plane, p.oc_mul, p.oc_shift);
  const uint32_t m = plane - n * static_cast<uint32_t>(p.C * p.mult_ch);
  const uint32_t c = fast_div(m, p.mc_mul, p.mc_shift);
  const uint32_t o = m - c * static_cast<uint32_t>(p.mult_ch);
  const float *in = p.in + (static_cast<int64_t>(n) * p.C + c) * (static_cast<int64_t>(p.H) * p.W);
  const float *fp = p.filter + (static_cast<int64_t>(o) * p.C + c) * 9;
  const int ih0 = h0 * S - p.pad_t;
  const bool left = w > 0, right = w * S + 4 < p.W;
  mb_grid_dep_wait();
  float f[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) f[i] = mb_load(fp + i);
  const float bias = p.bias != nullptr ? mb_load(p.bias + m) : 0.f;
  float acc[RH * V];
#pragma unroll
  for (int r = 0; r < RH * V; ++r) acc[r] = 0.f;
  const float *row = in + static_cast<int64_t>(ih0) * p.W + w * S;
#pragma unroll
  for (int i = 0; i < (RH - 1) * S + 3; ++i) {
    const bool row_ok = ih0 + i >= 0 && ih0 + i < p.H;
    const float4 mid = row_ok ? mb_load(reinterpret_cast<const float4 *>(row)) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float last = row_ok && right ? mb_load(row + 4) : 0.f;
    float x[COLS];
    if (S == 1) {
      x[0] = row_ok && left ? mb_load(row - 1) : 0.f;
      x[1] = mid.x; x[2] = mid.y; x[3] = mid.z; x[4] = mid.w;
    } else {
      x[0] = mid.x; x[1] = mid.y; x[2] = mid.z; x[3] = mid.w;
    }
    x[COLS - 1] = last;
    row += p.W;
#pragma unroll
    for (int r = 0; r < RH; ++r) {
      const int kh = i - r * S;
      if (kh >= 0 && kh < 3) {
#pragma unroll
        for (int v = 0; v < V; ++v)
#pragma unroll
          for (int j = 0; j < 3; ++j) acc[r * V + v] = fmaf(x[v * S + j], f[kh * 3 + j], acc[r * V + v]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < RH * V; ++r) acc[r] += bias;
  mb_activate_n(acc, p.act, p.max_limit, p.coef);
  float *out = p.out + (static_cast<int64_t>(plane) * p.Ho + h0) * p.Wo + w;
#pragma unroll
  for (int r = 0; r < RH; ++r) {
    if (h0 + r < p.Ho) {
      if (V == 4) *reinterpret_cast<float4 *>(out) = make_float4(acc[r * V], acc[r * V + 1], acc[r * V + 2], acc[r * V + 3]);
      else *reinterpret_cast<float2 *>(out) = make_float2(acc[r * V], acc[r * V + 1]);
    }
    out += p.Wo;
  }
}

// Any filter size, stride and dilation: one thread per output value.
__global__ void __launch_bounds__(256) dwconv_f32_kernel(const DwF32Params p) {
  const int64_t total = static_cast<int64_t>(p.planes) * p.Ho * p.Wo;
  const int64_t tid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (tid >= total) return;
  const int w = static_cast<int>(tid % p.Wo);
  int64_t r = tid / p.Wo;
  const int h = static_cast<int>(r % p.Ho);
  r /= p.Ho;
  const int OC = p.C * p.mult_ch;
  const int m = static_cast<int>(r % OC);
  const int n = static_cast<int>(r / OC);
  const int c = m / p.mult_ch, o = m % p.mult_ch;
  const float *ib = p.in + (static_cast<int64_t>(n) * p.C + c) * p.H * p.W;
  const float *fp = p.filter + (static_cast<int64_t>(o) * p.C + c) * p.KH * p.KW;
  float sum = 0.f;
  for (int kh = 0; kh < p.KH; ++kh) {
    const int ih = -p.pad_t + h * p.sh + kh * p.dh;
    if (ih < 0 || ih >= p.H) continue;
    for (int kw = 0; kw < p.KW; ++kw) {
      const int iw = -p.pad_l + w * p.sw + kw * p.dw;
      if (iw < 0 || iw >= p.W) continue;
      sum = fmaf(mb_load(ib + ih * p.W + iw), mb_load(fp + kh * p.KW + kw), sum);
    }
  }
  if (p.bias != nullptr) sum += p.bias[m];
  p.out[tid] = mb_activate(sum, p.act, p.max_limit, p.coef);
}

template <int K, int S, int RH>
int launch_rows(mb_context *ctx, DwF32Params &p) {
  p.strips = static_cast<uint32_t>(ceil_div64(p.Ho, RH));
  p.threads = p.planes * p.strips * static_cast<uint32_t>(p.Wo);
  fast_div_make(static_cast<uint32_t>(p.Wo), &p.wo_mul, &p.wo_shift);
  fast_div_make(p.strips, &p.strips_mul, &p.strips_shift);
  fast_div_make(static_cast<uint32_t>(p.C * p.mult_ch), &p.oc_mul, &p.oc_shift);
  fast_div_make(static_cast<uint32_t>(p.mult_ch), &p.mc_mul, &p.mc_shift);
  MB_CUDA(ctx, mb_launch_chained(ctx, dwconv_f32_rows_kernel<K, S, RH>, dim3((p.threads + 255u) / 256u), dim3(256), 0, p));
  ctx->launches++;
  return MB_SUCCESS;
}

template <int S, int RH>
int launch_wide(mb_context *ctx, DwF32Params &p) {
  const int groups = p.Wo / (S == 1 ? 4 : 2);
  p.strips = static_cast<uint32_t>(ceil_div64(p.Ho, RH));
  p.threads = p.planes * p.strips * static_cast<uint32_t>(groups);
  fast_div_make(static_cast<uint32_t>(groups), &p.wo_mul, &p.wo_shift);
  fast_div_make(p.strips, &p.strips_mul, &p.strips_shift);
  fast_div_make(static_cast<uint32_t>(p.C * p.mult_ch), &p.oc_mul, &p.oc_shift);
  fast_div_make(static_cast<uint32_t>(p.mult_ch), &p.mc_mul, &p.mc_shift);
  MB_CUDA(ctx, mb_launch_chained(ctx, dwconv_f32_wide_kernel<S, RH>, dim3((p.threads + 255u) / 256u), dim3(256), 0, p));
  ctx->launches++;
  return MB_SUCCESS;
}

// Rows per thread: long runs save loads (a row is read once for K output rows), short ones give a
// small problem more threads.  The line for the row kernel: a run is as long as it can be while 32 warps per SM remain
// (64 channels, 111 x 111, runs of 1, 2, 4, 8: stride 1, batch 4, 19.0, 11.7, 8.3, 7.1 us; stride 2, batch 8, 10.5, 7.2, 6.0, 7.3;
// 57 x 57, stride 1, batch 4, 6.1, 4.1, 3.9, 4.9).
template <int K, int S>
int launch_ks(mb_context *ctx, DwF32Params &p) {
  const int64_t outputs = static_cast<int64_t>(p.planes) * p.Ho * p.Wo;
  const int64_t want = static_cast<int64_t>(ctx->num_sms) * 1024;
  // Whole words per row, and the padding that puts a word under each group of columns.  Runs are longer while twice 32 warps
  // per SM remain at stride 1 (once for runs of two), four times at stride 2 (twice for two).  64 channels, 112 x 112, runs of 1, 2,
  // 4, 8: stride 1, batch 8, 13.1, 10.0, 9.1, 8.6 us, batch 32, 50.0, 40.0, 38.8, 37.8; stride 2, batch 8, 6.4, 5.4, 6.0, batch 32, 26.4, 26.4,
  // 25.4.
  if (K == 3 && p.W % 4 == 0 && p.Wo * S == p.W && p.pad_l == (S == 1 ? 1 : 0) &&
      ((reinterpret_cast<uintptr_t>(p.in) | reinterpret_cast<uintptr_t>(p.out)) & 15u) == 0) {
    if (S == 1 && outputs >= 64 * want) return launch_wide<S, S == 1 ? 8 : 4>(ctx, p);
    if (outputs >= 32 * want) return launch_wide<S, 4>(ctx, p);
    if (outputs >= 8 * want) return launch_wide<S, 2>(ctx, p);
    return launch_wide<S, 1>(ctx, p);
  }
  if (outputs >= 8 * want) return launch_rows<K, S, 8>(ctx, p);
  if (outputs >= 4 * want) return launch_rows<K, S, 4>(ctx, p);
  if (outputs >= 2 * want) return launch_rows<K, S, 2>(ctx, p);
  return launch_rows<K, S, 1>(ctx, p);
}

}  // namespace

int mb_dwconv_f32_launch(mb_context *ctx, const float *in, const float *filter, const float *bias, float *out,
                         int64_t N, int64_t C, int64_t H, int64_t W, int64_t mult_ch, int64_t KH, int64_t KW,
                         int stride_h, int stride_w, int dil_h, int dil_w, int pad_top, int pad_left, int64_t Ho,
                         int64_t Wo, int activation, float max_limit, float coefficient) {
  DwF32Params p = {};
  p.in = in; p.filter = filter; p.bias = bias; p.out = out;
  p.C = static_cast<int>(C); p.H = static_cast<int>(H); p.W = static_cast<int>(W);
  p.Ho = static_cast<int>(Ho); p.Wo = static_cast<int>(Wo); p.mult_ch = static_cast<int>(mult_ch);
  p.KH = static_cast<int>(KH); p.KW = static_cast<int>(KW);
  p.sh = stride_h; p.sw = stride_w; p.dh = dil_h; p.dw = dil_w; p.pad_t = pad_top; p.pad_l = pad_left;
  p.act = activation; p.max_limit = max_limit; p.coef = coefficient;
  const int64_t planes = N * C * mult_ch, outputs = planes * Ho * Wo;
  p.planes = static_cast<uint32_t>(planes);
  // the row kernel: square 3x3 / 5x5 filters without dilation, indices within 31 bits
  if (KH == KW && (KH == 3 || KH == 5) && stride_h == stride_w && stride_h <= 2 && dil_h == 1 && dil_w == 1 &&
      planes < (1ll << 31) && outputs < (1ll << 31) - 256 && H < (1 << 24) && W < (1 << 24)) {
    if (KH == 3) return stride_h == 1 ? launch_ks<3, 1>(ctx, p) : launch_ks<3, 2>(ctx, p);
    return stride_h == 1 ? launch_ks<5, 1>(ctx, p) : launch_ks<5, 2>(ctx, p);
  }
  if (planes >= (1ll << 32)) return mb_fail(ctx, MB_UNSUPPORTED, "mb_dwconv_f32_nchw: tensor too large");
  dwconv_f32_kernel<<<static_cast<unsigned>(ceil_div64(outputs, 256)), 256, 0, ctx->stream>>>(p);
  MB_CUDA(ctx, cudaGetLastError());
  ctx->launches++;
  return MB_SUCCESS;
}
