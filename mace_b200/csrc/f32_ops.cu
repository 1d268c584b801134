// fp32 kernels of the path: batched GEMM, GEMV and general Conv2D in NCHW, with bias and
// activation fused into the epilogue (depthwise: dwconv_f32.cu).
//
// Reference behaviour: ref::Gemm / ref::Gemv / ref::Conv2d (mace/ops/ref/gemm.cc:57-106,
// gemv.cc:45-81, conv_2d.cc:36-122), ref::BiasAdd (bias_add.cc:74-103) and
// ref::Activation (activation.cc:61-88).  The reference accumulates in fp32 in
// index order; these kernels accumulate in fp32 in a tiled order, so results
// agree to rounding (tests bound the difference at 1e-4 of the output range).
#include "common.cuh"
#include "conv_f32_direct.cuh"
#include "gemm_f32_gather.cuh"

bool mb_gemm_f32_tc_supported(const mb_context *ctx, const float *X, const float *W, int64_t Mdim,
                              int64_t Ndim, int64_t K, int64_t x_row_stride, int64_t x_batch_stride,
                              int64_t w_row_stride, int64_t w_batch_stride);
int mb_gemm_f32_tc_launch(mb_context *ctx, const float *X, const float *W, const float *bias, float *C,
                          int64_t batch, int64_t Mdim, int64_t Ndim, int64_t K, int64_t x_row_stride,
                          int64_t x_batch_stride, int64_t w_row_stride, int64_t w_batch_stride,
                          int64_t c_row_stride, int64_t c_batch_stride, int act, float max_limit,
                          float coef, const float *residual);

bool mb_gemm_f32_pairs_pays(const mb_context *ctx, int64_t batch, int64_t Mdim, int64_t Ndim, int64_t K, int w_batched);

int mb_dwconv_f32_launch(mb_context *ctx, const float *in, const float *filter, const float *bias, float *out,
                         int64_t N, int64_t C, int64_t H, int64_t W, int64_t mult_ch, int64_t KH, int64_t KW,
                         int stride_h, int stride_w, int dil_h, int dil_w, int pad_top, int pad_left, int64_t Ho,
                         int64_t Wo, int activation, float max_limit, float coefficient);

namespace {

// ---- GEMM: 64 x 64 tile per 128-thread block, 4 x 8 outputs per thread, one chain of FMAs in the order of k --------
// What the tensor cores cannot take with this accuracy: products of depth below 48 and from 65 to 71 in a layout that TMA does
// not take (mb_f32_gather_run).  Bound by latency: 12 warps per SM at best, of which 0.6 per scheduler are ready (FMA pipe 41 %
// busy); a panel of 32 k is on its way to registers while the one before is multiplied.  Measured, a panel of 16 k loaded,
// waited for and multiplied by 256 threads -> now: 16 x 16 x 16 4.2 -> 2.9 us, 64 x 64 x 64 9.3 -> 4.2, 384 x 384 x 64, batch 12,
// 21.7 -> 10.9, 1536 x 1536 x 16 10.2 -> 4.7.
constexpr int FT = 64;
constexpr int FK = 32;
constexpr int FP = FT + 4;  // row pitch of a panel

struct GemmF32Params {
  const float *A, *B;
  float *C;
  const float *bias;  // per row of C (output channel) or null
  int64_t M, N, K;
  int64_t a_rs, a_cs, b_rs, b_cs, c_rs, c_cs;  // element strides
  int64_t a_bs, b_bs, c_bs;                    // batch strides
  int act;
  float max_limit, coef;
};

// One thread's 16 values of a 64 x 32 panel.  Contiguous along k, a warp takes 4 rows x 8 k at a time: 32-byte sectors of
// the operand, all banks of the panel; else 32 rows of one k.
template <bool ALONG_K>
struct PanelThread {
  static constexpr int ROWS = ALONG_K ? 4 : 2;  // rows of this thread, 16 / ROWS values of each
  const float *src;                             // its first row at its first k
  int64_t rs, ks;
  int row0, k0;
  uint32_t in;
  __device__ __forceinline__ PanelThread(const float *base, int64_t rows, int64_t first, int64_t rs_, int64_t ks_)
      : rs(ALONG_K ? 4 * rs_ : 32), ks(ALONG_K ? 8 : ks_), in(0) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    row0 = ALONG_K ? warp * 16 + (lane >> 3) : lane;
    k0 = ALONG_K ? lane & 7 : warp * 8;
#pragma unroll
    for (int q = 0; q < ROWS; ++q) in |= (first + row0 + q * (ALONG_K ? 4 : 32) < rows ? 1u : 0u) << q;
    src = base + (first + row0) * rs_ + k0 * ks_;
  }
  __device__ __forceinline__ void load(float (&v)[16], int64_t kb, int64_t K) const {
    const float *at = src + kb * (ALONG_K ? 1 : ks);
    const int left = static_cast<int>(min(K - kb - k0, static_cast<int64_t>(FK)));
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int q = i % ROWS, j = i / ROWS;
      v[i] = (in >> q & 1u) != 0 && j * (ALONG_K ? 8 : 1) < left ? at[q * rs + j * ks] : 0.f;
    }
  }
  __device__ __forceinline__ void store(const float (&v)[16], float (*panel)[FP]) const {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int q = i % ROWS, j = i / ROWS;
      panel[k0 + j * (ALONG_K ? 8 : 1)][row0 + q * (ALONG_K ? 4 : 32)] = v[i];
    }
  }
};

// Two FMAs per instruction, each rounded as fmaf rounds.
__device__ __forceinline__ void fma2(uint64_t &acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t twice(float v) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
  return r;
}

__device__ __forceinline__ void panel_fma(uint64_t (&acc)[4][4], const float *a, const float *b) {
  const float4 a4 = *reinterpret_cast<const float4 *>(a);
  const ulonglong2 b0 = *reinterpret_cast<const ulonglong2 *>(b), b1 = *reinterpret_cast<const ulonglong2 *>(b + 32);
  const uint64_t av[4] = {twice(a4.x), twice(a4.y), twice(a4.z), twice(a4.w)}, bv[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) fma2(acc[i][j], av[i], bv[j]);
}

// AK, BK: the operand is contiguous along k (else along its rows, the columns of B)
template <bool AK, bool BK>
__global__ void __launch_bounds__(128) gemm_f32_kernel(const GemmF32Params p) {
  __shared__ __align__(16) float As[2][FK][FP];
  __shared__ __align__(16) float Bs[2][FK][FP];
  const int b = blockIdx.z;
  const int64_t m0 = static_cast<int64_t>(blockIdx.y) * FT, n0 = static_cast<int64_t>(blockIdx.x) * FT;
  const PanelThread<AK> pa(p.A + b * p.a_bs, p.M, m0, p.a_rs, p.a_cs);
  const PanelThread<BK> pb(p.B + b * p.b_bs, p.N, n0, p.b_cs, p.b_rs);
  float *C = p.C + b * p.c_bs;
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
  uint64_t acc2[4][4] = {};  // pairs of columns
  float va[16], vb[16];
  mb_grid_dep_launch();
  mb_grid_dep_wait();
  pa.load(va, 0, p.K);
  pb.load(vb, 0, p.K);
  int buf = 0;
  for (int64_t k0 = 0; k0 < p.K; k0 += FK, buf ^= 1) {
    pa.store(va, As[buf]);
    pb.store(vb, Bs[buf]);
    __syncthreads();  // (a thread is at most one panel ahead of the slowest, in the other buffer)
    if (k0 + FK < p.K) {
      pa.load(va, k0 + FK, p.K);
      pb.load(vb, k0 + FK, p.K);
    }
    const float *ap = &As[buf][0][ty * 4], *bp = &Bs[buf][0][tx * 4];
    if (k0 + FK <= p.K) {
#pragma unroll
      for (int kk = 0; kk < FK; ++kk) panel_fma(acc2, ap + kk * FP, bp + kk * FP);
    } else {
      for (int kk = 0; kk < static_cast<int>(p.K - k0); ++kk) panel_fma(acc2, ap + kk * FP, bp + kk * FP);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int64_t m = m0 + ty * 4 + i;
    if (m >= p.M) continue;
    float acc[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[2 * j]), "=f"(acc[2 * j + 1]) : "l"(acc2[i][j]));
    if (p.bias != nullptr) {
      const float bv = p.bias[m];
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += bv;
    }
    mb_activate_n(acc, p.act, p.max_limit, p.coef);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t n = n0 + h * 32 + tx * 4;
      float *dst = C + m * p.c_rs + n * p.c_cs;
      if (p.c_cs == 1 && n + 4 <= p.N && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
        *reinterpret_cast<float4 *>(dst) = make_float4(acc[h * 4], acc[h * 4 + 1], acc[h * 4 + 2], acc[h * 4 + 3]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (n + j < p.N) dst[j * p.c_cs] = acc[h * 4 + j];
      }
    }
  }
}

// ---- GEMV: one warp per matrix row and up to VECS vectors -----------------------------------
// Bound by the matrix's bytes: a row is read once for VECS vectors, 16 bytes per lane where the rows allow, with as
// many rows in flight as warps fit.
template <int VECS, bool VEC4>
__global__ void __launch_bounds__(256)
gemv_f32_kernel(const float *lhs, const float *rhs, const float *bias,
                float *__restrict__ out, int64_t batch, int64_t rows, int64_t K, int lhs_batched, int rhs_batched) {
  mb_grid_dep_launch();
  mb_grid_dep_wait();
  const int lane = threadIdx.x & 31;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  if (row >= rows) return;
  // (a grid has at most 65535 blocks along y; what the batch has beyond them is a further pass)
  for (int64_t b0 = static_cast<int64_t>(blockIdx.y) * VECS; b0 < batch; b0 += static_cast<int64_t>(gridDim.y) * VECS) {
    const float *lp = lhs + (lhs_batched ? b0 * rows * K : 0) + row * K;
    const float *rp = rhs + (rhs_batched ? b0 * K : 0);
    const int vecs = static_cast<int>(min(static_cast<int64_t>(VECS), batch - b0));
    float s[VECS];
#pragma unroll
    for (int v = 0; v < VECS; ++v) s[v] = 0.f;
    if (VEC4) {
#pragma unroll 4
      for (int64_t i = lane * 4; i < K; i += 128) {
        const float4 a = mb_load(reinterpret_cast<const float4 *>(lp + i));
#pragma unroll
        for (int v = 0; v < VECS; ++v) {
          if (v < vecs) {
            const float4 x = mb_load(reinterpret_cast<const float4 *>(rp + v * K + i));
            s[v] = fmaf(a.x, x.x, s[v]); s[v] = fmaf(a.y, x.y, s[v]);
            s[v] = fmaf(a.z, x.z, s[v]); s[v] = fmaf(a.w, x.w, s[v]);
          }
        }
      }
    } else {
#pragma unroll 4
      for (int64_t i = lane; i < K; i += 32) {
        const float a = mb_load(lp + i);
#pragma unroll
        for (int v = 0; v < VECS; ++v)
          if (v < vecs) s[v] = fmaf(a, mb_load(rp + v * K + i), s[v]);
      }
    }
#pragma unroll
    for (int v = 0; v < VECS; ++v) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s[v] += __shfl_xor_sync(0xffffffffu, s[v], o);
      if (lane == 0 && v < vecs) out[(b0 + v) * rows + row] = s[v] + (bias != nullptr ? mb_load(bias + row) : 0.f);
    }
  }
}

// ---- direct convolution ------------------------------------------------------------
struct ConvF32Params {
  const float *in, *filter, *bias;
  float *out;
  int N, C, H, W, O, KH, KW, sh, sw, dh, dw, pad_t, pad_l, Ho, Wo;
  int act;
  float max_limit, coef;
};

// One thread per output value; the loop order (c, kh, kw) is the reference's.
__global__ void __launch_bounds__(256) conv2d_f32_direct_kernel(const ConvF32Params p) {
  mb_grid_dep_launch();
  mb_grid_dep_wait();
  const int64_t total = static_cast<int64_t>(p.N) * p.O * p.Ho * p.Wo;
  const int64_t tid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (tid >= total) return;
  const int w = static_cast<int>(tid % p.Wo);
  int64_t r = tid / p.Wo;
  const int h = static_cast<int>(r % p.Ho);
  r /= p.Ho;
  const int m = static_cast<int>(r % p.O);
  const int n = static_cast<int>(r / p.O);
  float sum = 0.f;
  for (int c = 0; c < p.C; ++c) {
    const float *ib = p.in + (static_cast<int64_t>(n) * p.C + c) * p.H * p.W;
    const float *fp = p.filter + (static_cast<int64_t>(m) * p.C + c) * p.KH * p.KW;
    for (int kh = 0; kh < p.KH; ++kh) {
      const int ih = -p.pad_t + h * p.sh + kh * p.dh;
      if (ih < 0 || ih >= p.H) continue;
      for (int kw = 0; kw < p.KW; ++kw) {
        const int iw = -p.pad_l + w * p.sw + kw * p.dw;
        if (iw < 0 || iw >= p.W) continue;
        sum = fmaf(mb_load(ib + ih * p.W + iw), mb_load(fp + kh * p.KW + kw), sum);
      }
    }
  }
  if (p.bias != nullptr) sum += p.bias[m];
  p.out[tid] = mb_activate(sum, p.act, p.max_limit, p.coef);
}

// ---- im2col for the tensor-core route of the general convolution --------------------------
// col[k][...] with k = (c * KH + kh) * KW + kw, the order of an OIHW filter row.  Two layouts:
// per image (col_ns = K * col_rs: image n owns a [K x positions] matrix) and merged
// (col_ns = positions per image: the images of a chunk lie side by side in one
// [K x images * positions] matrix, which keeps 128-position tiles full when an image has few).
struct ColF32Params {
  const float *in;  // first image of the chunk
  float *col;
  int C, H, W, KH, KW, sh, sw, dh, dw, pad_t, pad_l, Ho, Wo, hw;
  int64_t col_rs, col_ns;
};

// One block per (group of output rows, channel and filter row, image): threadIdx.x walks along
// an output row and threadIdx.y picks the row, so no thread divides by anything, the KW taps
// of a pixel re-read the same input row from L1, and every store is a contiguous run.
__global__ void __launch_bounds__(128) im2col_f32_kernel(const ColF32Params p, int rows_per_block) {
  const int h = blockIdx.x * blockDim.y + threadIdx.y, n = blockIdx.z;
  if (h >= p.Ho) return;
  const float *in = p.in;
  float *__restrict__ col = p.col;
  const int y_end = min((static_cast<int>(blockIdx.y) + 1) * rows_per_block, p.C * p.KH);
  // Up to eight values are loaded before the first is stored: a store waits for the load that
  // feeds it, a warp issues in order, and the compiler may not move a load above a store to
  // memory it cannot tell apart.
  if (p.KW == 1) {
    for (int w = threadIdx.x; w < p.Wo; w += blockDim.x) {
      const int iw = w * p.sw - p.pad_l;
      const bool col_ok = iw >= 0 && iw < p.W;
      for (int y0 = blockIdx.y * rows_per_block; y0 < y_end; y0 += 8) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int y = y0 + j;
          const int c = y / p.KH, kh = y - c * p.KH;
          const int ih = h * p.sh - p.pad_t + kh * p.dh;
          const bool ok = y < y_end && col_ok && ih >= 0 && ih < p.H;
          v[j] = ok ? mb_load(in + ((static_cast<int64_t>(n) * p.C + c) * p.H + ih) * p.W + iw) : 0.f;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (y0 + j < y_end) col[static_cast<int64_t>(y0 + j) * p.col_rs + n * p.col_ns + h * p.Wo + w] = v[j];
      }
    }
    return;
  }
  for (int y = blockIdx.y * rows_per_block; y < y_end; ++y) {  // y = c * KH + kh
    const int c = y / p.KH, kh = y - c * p.KH;
    const int ih = h * p.sh - p.pad_t + kh * p.dh;
    const bool row_ok = ih >= 0 && ih < p.H;
    const float *src = in + ((static_cast<int64_t>(n) * p.C + c) * p.H + (row_ok ? ih : 0)) * p.W;
    float *dst = col + static_cast<int64_t>(y) * p.KW * p.col_rs + n * p.col_ns + h * p.Wo;
    for (int w = threadIdx.x; w < p.Wo; w += blockDim.x) {
      const int iw0 = w * p.sw - p.pad_l;
      for (int kw0 = 0; kw0 < p.KW; kw0 += 8) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int iw = iw0 + (kw0 + j) * p.dw;
          v[j] = (kw0 + j < p.KW && row_ok && iw >= 0 && iw < p.W) ? mb_load(src + iw) : 0.f;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (kw0 + j < p.KW) dst[(kw0 + j) * p.col_rs + w] = v[j];
      }
    }
  }
}

// rows of K floats -> rows of Kp floats (a 16-byte multiple, which a tensor map's strides need)
__global__ void __launch_bounds__(256)
repack_rows_f32_kernel(const float *src, float *__restrict__ dst, int64_t rows, int K, int Kp) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
  if (i >= rows * Kp) return;
  const int k = static_cast<int>(i % Kp);
  dst[i] = k < K ? mb_load(src + (i / Kp) * K + k) : 0.f;
}

// merged product [O][images * hw] (row stride src_rs) -> NCHW images
__global__ void __launch_bounds__(256)
unmerge_f32_kernel(const float *src, float *__restrict__ dst, int64_t total, int O, int hw,
                   int64_t src_rs) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
  if (i >= total) return;
  const int pos = static_cast<int>(i % hw);
  const int64_t r = i / hw;
  const int o = static_cast<int>(r % O);
  const int64_t n = r / O;
  dst[i] = mb_load(src + o * src_rs + n * hw + pos);
}

}  // namespace

// Whether the kernel that fetches its own operands takes a product (see gemm_f32_gather.cu); by_tma: the TMA-fed one of
// gemm_f32_tc.cu could; fp32_accuracy: the error may not be larger than that of fp32 FMAs, which is so for the products that
// no other tensor-core route can take.
static bool take_gather(mb_context *ctx, mb_f32_gemm &g, bool by_tma, bool fp32_accuracy) {
  if (fp32_accuracy) g.run = mb_f32_gather_run(g.K);
  if (ctx->f32_gather == 1 || !mb_gemm_f32_gather_supported(ctx, g)) return false;
  if (ctx->f32_gather == 2) return true;
  if (fp32_accuracy && g.run == 0) return false;
  if (!by_tma) return true;
  // The TMA-fed kernels: tiles of 128 columns of one image (or matrix), 1200 cycles per step, 2.6 us for the results of 128
  // channels (twice that with a residual), 4.4 us around them; from the size on where W is split in front (gemm_f32_pairs.cu) 750
  // (600 for 64 channels), 2 us for the results, 6 us around them.
  const int64_t images = g.conv ? g.M / (static_cast<int64_t>(g.Ho) * g.Wo) : g.batch;
  const int64_t columns = g.M / (g.conv ? images : 1), tiles_m = ceil_div64(columns, 128), steps = ceil_div64(g.K, 32);
  const bool pairs = mb_gemm_f32_pairs_pays(ctx, images, columns, g.N, g.K, g.w_bs != 0);
  int64_t tma = -1;
  for (int w : {128, 64}) {
    if (w == 128 && g.N <= 64) continue;
    const int64_t rounds = ceil_div64(images * tiles_m * ceil_div64(g.N, w), ctx->num_sms);
    const int64_t results = pairs ? (w == 128 ? 3800 : 2400) : (w == 128 ? 5000 : 3000) * (g.residual != nullptr ? 2 : 1);
    const int64_t step = !pairs ? 1200 : w == 128 ? 750 : 600;
    const int64_t cost = (pairs ? 11500 : 8300) + rounds * std::max<int64_t>(steps * step, results);
    if (tma < 0 || cost < tma) tma = cost;
  }
  return mb_gemm_f32_gather_cost(ctx, g) < tma;
}

// A 1x1 convolution whose input is the product's operand as it lies ...
static bool pointwise_in_place(int64_t KH, int64_t KW, int sh, int sw, int pad_t, int pad_l, int64_t H, int64_t W, int64_t Ho,
                               int64_t Wo) {
  return KH == 1 && KW == 1 && sh == 1 && sw == 1 && pad_t == 0 && pad_l == 0 && Ho == H && Wo == W;
}
// ... and with rows that fill the TMA-fed kernel's tiles.
static bool long_rows(int64_t hw) { return hw % 4 == 0 && hw >= 128; }

// Other convolutions of at least this much work go to the tensor cores by way of a column matrix (where the kernel that
// fetches its own operands cannot run); smaller ones stay on the one-thread-per-output kernel.
constexpr int64_t COLUMN_MIN_WORK = 1 << 18, COLUMN_MIN_POSITIONS = 32;

static bool column_route(int64_t N, int64_t C, int64_t O, int64_t KH, int64_t KW, int64_t Ho, int64_t Wo) {
  return N * O * Ho * Wo * C * KH * KW >= COLUMN_MIN_WORK && Ho * Wo * N >= COLUMN_MIN_POSITIONS && C * KH <= 65535 &&
         Ho * Wo < (1ll << 30);
}

// The convolution as that kernel sees it.
static mb_f32_gemm conv_gemm(const float *in, const float *filter, const float *bias, const float *residual, float *out,
                             int64_t N, int64_t C, int64_t H, int64_t W, int64_t O, int64_t KH, int64_t KW, int sh,
                             int sw, int dh, int dw, int pad_t, int pad_l, int64_t Ho, int64_t Wo, int act,
                             float max_limit, float coef) {
  mb_f32_gemm g;
  g.X = in; g.W = filter; g.bias = bias; g.residual = residual; g.C = out;
  g.M = N * Ho * Wo; g.N = O; g.K = C * KH * KW;
  g.act = act; g.max_limit = max_limit; g.coef = coef;
  g.conv = true;
  g.C_in = static_cast<int>(C); g.H = static_cast<int>(H); g.Wd = static_cast<int>(W);
  g.KH = static_cast<int>(KH); g.KW = static_cast<int>(KW);
  g.sh = sh; g.sw = sw; g.dh = dh; g.dw = dw; g.pad_t = pad_t; g.pad_l = pad_l;
  g.Ho = static_cast<int>(Ho); g.Wo = static_cast<int>(Wo);
  return g;
}

// Strided batched fp32 GEMM with optional per-row bias and activation; the
// building block of the 1x1 convolution and of the Winograd batched product.
int mb_gemm_f32_strided(mb_context *ctx, const float *A, const float *B, float *C,
                        const float *bias_per_row, int64_t batch, int64_t M, int64_t N, int64_t K,
                        int64_t a_rs, int64_t a_cs, int64_t a_bs, int64_t b_rs, int64_t b_cs,
                        int64_t b_bs, int64_t c_rs, int64_t c_cs, int64_t c_bs, int act,
                        float max_limit, float coef) {
  mb_f32_gemm g;
  if (c_cs == 1 || bias_per_row != nullptr) {  // the columns of C are the tensor core's M
    g.X = B; g.x_ks = b_rs; g.x_ms = b_cs; g.x_bs = b_bs;
    g.W = A; g.w_ns = a_rs; g.w_ks = a_cs; g.w_bs = a_bs;
    g.M = N; g.N = M; g.c_ns = c_rs; g.c_ms = c_cs;
  } else {
    g.X = A; g.x_ks = a_cs; g.x_ms = a_rs; g.x_bs = a_bs;
    g.W = B; g.w_ns = b_cs; g.w_ks = b_rs; g.w_bs = b_bs;
    g.M = M; g.N = N; g.c_ns = c_cs; g.c_ms = c_rs;
  }
  g.batch = batch; g.K = K; g.C = C; g.c_bs = c_bs; g.bias = bias_per_row;
  g.act = act; g.max_limit = max_limit; g.coef = coef;
  const bool by_tma = a_cs == 1 && b_cs == 1 && c_cs == 1 &&
                      mb_gemm_f32_tc_supported(ctx, B, A, N, M, K, b_rs, b_bs, a_rs, a_bs);
  const bool gather = take_gather(ctx, g, by_tma, !by_tma);
  // Both depths contiguous, where its estimate is the smaller: a batch of 8, 992 x 352 x 768: 73.1 us fetching its own operands,
  // 56.8 this way; 4 of 240 x 64 x 80: 6.4 and 7.3.  Up to 64 deep the former's three accumulators are the more accurate.
  if (!by_tma && ctx->f32_rows != 1 && mb_gemm_f32_rows_supported(ctx, g) &&
      (ctx->f32_rows == 2 ||
       (gather && ctx->f32_gather == 0 && g.run != 0 && K > 64 && mb_gemm_f32_rows_cost(ctx, g) < mb_gemm_f32_gather_cost(ctx, g))))
    return mb_gemm_f32_rows_launch(ctx, g);
  if (gather) return mb_gemm_f32_gather_launch(ctx, g);
  // C = A * B with A [M x K] k-contiguous, B [K x N] n-contiguous and C n-contiguous is the
  // tensor-core kernel's layout with the roles X = B (pixels x channels side), W = A.
  if (by_tma) {
    return mb_gemm_f32_tc_launch(ctx, B, A, bias_per_row, C, batch, N, M, K, b_rs, b_bs, a_rs, a_bs,
                                 c_rs, c_bs, act, max_limit, coef, nullptr);
  }
  if (batch > 65535 || ceil_div64(M, FT) > 65535) {
    if (ctx->f32_gather != 1 && mb_gemm_f32_gather_supported(ctx, g)) return mb_gemm_f32_gather_launch(ctx, g);
    return mb_fail(ctx, MB_UNSUPPORTED, "fp32 GEMM: batch or M too large for this kernel");
  }
  GemmF32Params p;
  p.A = A; p.B = B; p.C = C; p.bias = bias_per_row;
  p.M = M; p.N = N; p.K = K;
  p.a_rs = a_rs; p.a_cs = a_cs; p.b_rs = b_rs; p.b_cs = b_cs; p.c_rs = c_rs; p.c_cs = c_cs;
  p.a_bs = a_bs; p.b_bs = b_bs; p.c_bs = c_bs;
  p.act = act; p.max_limit = max_limit; p.coef = coef;
  dim3 grid(static_cast<unsigned>(ceil_div64(N, FT)), static_cast<unsigned>(ceil_div64(M, FT)),
            static_cast<unsigned>(batch));
  auto kern = a_cs == 1 ? (b_rs == 1 ? gemm_f32_kernel<true, true> : gemm_f32_kernel<true, false>)
                        : (b_rs == 1 ? gemm_f32_kernel<false, true> : gemm_f32_kernel<false, false>);
  MB_CUDA(ctx, mb_launch_chained(ctx, kern, grid, dim3(128), 0, p));
  MB_CUDA(ctx, cudaGetLastError());
  ctx->launches++;
  return MB_SUCCESS;
}

// General convolution as im2col + GEMM (the tensor-core kernel when the shapes allow it).
// Images are processed in chunks so that the column matrix stays below the context's budget
// (1 GiB unless the option col_budget_mb changes it).
static int conv2d_f32_im2col(mb_context *ctx, const float *in, const float *filter, const float *bias,
                             float *out, int64_t N, int64_t C, int64_t H, int64_t W, int64_t O,
                             int64_t KH, int64_t KW, int sh, int sw, int dh, int dw, int pad_t,
                             int pad_l, int64_t Ho, int64_t Wo, int act, float max_limit, float coef) {
  const int64_t K = C * KH * KW, hw = Ho * Wo;
  const int64_t Kp = (K + 3) / 4 * 4;
  const bool merged = (hw % 4 != 0) || hw < 128;
  const int64_t hwp = (hw + 3) / 4 * 4;
  const int64_t per_image = K * (merged ? hw : hwp) * 4;
  int64_t chunk = std::max<int64_t>(1, std::min<int64_t>(N, ctx->col_budget_bytes / std::max<int64_t>(per_image, 1)));
  chunk = std::min<int64_t>(chunk, 65535);
  const bool repack = (K % 4 != 0) || (reinterpret_cast<uintptr_t>(filter) & 15u);
  const int64_t merged_rs = (chunk * hw + 3) / 4 * 4;
  size_t off = 0;
  const size_t off_f = off; off += repack ? align_up(sizeof(float) * O * Kp, 256) : 0;
  const size_t off_col = off; off += align_up(sizeof(float) * K * (merged ? merged_rs : chunk * hwp), 256);
  const size_t off_c2 = off; off += merged ? align_up(sizeof(float) * O * merged_rs, 256) : 0;
  uint8_t *scratch = nullptr;
  MB_RETURN_IF_ERROR(mb_scratch(ctx, off, reinterpret_cast<void **>(&scratch)));
  const float *wmat = filter;
  int64_t w_rs = K;
  if (repack) {
    float *wf = reinterpret_cast<float *>(scratch + off_f);
    repack_rows_f32_kernel<<<static_cast<unsigned>(ceil_div64(O * Kp, 256)), 256, 0, ctx->stream>>>(
        filter, wf, O, static_cast<int>(K), static_cast<int>(Kp));
    MB_CUDA(ctx, cudaGetLastError());
    ctx->launches++;
    wmat = wf;
    w_rs = Kp;
  }
  float *col = reinterpret_cast<float *>(scratch + off_col);
  float *c2 = reinterpret_cast<float *>(scratch + off_c2);
  ColF32Params p;
  p.col = col;
  p.C = static_cast<int>(C); p.H = static_cast<int>(H); p.W = static_cast<int>(W);
  p.KH = static_cast<int>(KH); p.KW = static_cast<int>(KW);
  p.sh = sh; p.sw = sw; p.dh = dh; p.dw = dw; p.pad_t = pad_t; p.pad_l = pad_l;
  p.Ho = static_cast<int>(Ho); p.Wo = static_cast<int>(Wo); p.hw = static_cast<int>(hw);
  for (int64_t n0 = 0; n0 < N; n0 += chunk) {
    const int64_t nc = std::min(chunk, N - n0);
    p.in = in + n0 * C * H * W;
    p.col_rs = merged ? merged_rs : hwp;
    p.col_ns = merged ? hw : K * hwp;
    int bw = 8;  // threads along a row: the power of two that covers Wo, at most 128
    while (bw < Wo && bw < 128) bw *= 2;
    dim3 block(bw, 128 / bw);
    // a block of few useful threads (narrow or single-tap rows) takes several (channel,
    // filter row) pairs, so that its launch cost is spread over more than a handful of values
    const int rows_per_block = (C * KH >= 64 && Wo * KW < 512) ? 8 : 1;
    dim3 grid(static_cast<unsigned>(ceil_div64(Ho, block.y)),
              static_cast<unsigned>(ceil_div64(C * KH, rows_per_block)), static_cast<unsigned>(nc));
    im2col_f32_kernel<<<grid, block, 0, ctx->stream>>>(p, rows_per_block);
    MB_CUDA(ctx, cudaGetLastError());
    ctx->launches++;
    float *dst = out + n0 * O * hw;
    if (!merged) {
      // out_n [O x hw] = filter [O x K] * col_n [K x hw]
      MB_RETURN_IF_ERROR(mb_gemm_f32_strided(ctx, wmat, col, dst, bias, nc, O, hw, K, w_rs, 1, 0, hwp, 1,
                                             K * hwp, hw, 1, O * hw, act, max_limit, coef));
    } else {
      MB_RETURN_IF_ERROR(mb_gemm_f32_strided(ctx, wmat, col, c2, bias, 1, O, nc * hw, K, w_rs, 1, 0,
                                             merged_rs, 1, 0, merged_rs, 1, 0, act, max_limit, coef));
      const int64_t total = nc * O * hw;
      unmerge_f32_kernel<<<static_cast<unsigned>(ceil_div64(total, 256)), 256, 0, ctx->stream>>>(
          c2, dst, total, static_cast<int>(O), static_cast<int>(hw), merged_rs);
      MB_CUDA(ctx, cudaGetLastError());
      ctx->launches++;
    }
  }
  return MB_SUCCESS;
}

extern "C" {

int mb_gemm_f32(mb_context *ctx, const float *A, const float *B, float *C, int64_t batch,
                int64_t M, int64_t N, int64_t K, int a_col_major, int b_col_major,
                int c_col_major, int a_batched, int b_batched) {
  if (ctx == nullptr) return MB_INVALID_ARGS;
  if (batch < 0 || M < 0 || N < 0 || K < 0)
    return mb_fail(ctx, MB_INVALID_ARGS, "mb_gemm_f32: negative dimension");
  if (batch == 0 || M == 0 || N == 0) return MB_SUCCESS;
  if (A == nullptr || B == nullptr || C == nullptr)
    return mb_fail(ctx, MB_INVALID_ARGS, "mb_gemm_f32: null operand");
  MB_CUDA(ctx, cudaSetDevice(ctx->device));
  return mb_gemm_f32_strided(ctx, A, B, C, nullptr, batch, M, N, K, a_col_major ? 1 : K,
                             a_col_major ? M : 1, a_batched ? M * K : 0, b_col_major ? 1 : N,
                             b_col_major ? K : 1, b_batched ? K * N : 0, c_col_major ? 1 : N,
                             c_col_major ? M : 1, M * N, 0, 0.f, 0.f);
}

int mb_gemv_f32(mb_context *ctx, const float *lhs, const float *rhs, const float *bias,
                float *out, int64_t batch, int64_t rows, int64_t K, int lhs_batched,
                int rhs_batched) {
  if (ctx == nullptr) return MB_INVALID_ARGS;
  if (batch < 0 || rows < 0 || K < 0)
    return mb_fail(ctx, MB_INVALID_ARGS, "mb_gemv_f32: negative dimension");
  if (batch == 0 || rows == 0) return MB_SUCCESS;
  if (lhs == nullptr || rhs == nullptr || out == nullptr)
    return mb_fail(ctx, MB_INVALID_ARGS, "mb_gemv_f32: null operand");
  MB_CUDA(ctx, cudaSetDevice(ctx->device));
  // Whole groups of 32 and more vectors against one matrix: the vectors are the tensor core's M, the matrix its N.  Fewer,
  // and ragged ones, keep the accuracy of the CUDA-core kernel (a sum per lane, then over the lanes: 4e-8 to 2e-7 where the
  // tensor cores' shortest runs give 1.3e-7 to 2e-7), in which up to eight vectors share a pass over the matrix.
  const bool whole = batch >= 32 && batch % 4 == 0 && K % 4 == 0 && rows >= 16 && (reinterpret_cast<uintptr_t>(lhs) & 15u) == 0;
  if (!lhs_batched && rhs_batched && (whole || ctx->f32_gather == 2)) {
    mb_f32_gemm g;
    g.X = rhs; g.x_ks = 1; g.x_ms = K;
    g.W = lhs; g.w_ns = K; g.w_ks = 1;
    g.bias = bias; g.C = out; g.c_ns = 1; g.c_ms = rows;
    g.M = batch; g.N = rows; g.K = K;
    if (take_gather(ctx, g, false, false)) return mb_gemm_f32_gather_launch(ctx, g);
  }
  const bool shared = !lhs_batched && rhs_batched;  // (one matrix, several vectors: up to eight per pass)
  const int vecs = !shared || batch == 1 ? 1 : batch == 2 ? 2 : batch <= 4 ? 4 : 8;
  const dim3 grid(static_cast<unsigned>(ceil_div64(rows, 8)),
                  static_cast<unsigned>(std::min<int64_t>(ceil_div64(batch, vecs), 65535)));
  const bool vec4 = K % 4 == 0 && ((reinterpret_cast<uintptr_t>(lhs) | reinterpret_cast<uintptr_t>(rhs)) & 15u) == 0;
#define MB_GEMV(V_)                                                                                                   \
  MB_CUDA(ctx, vec4 ? mb_launch_chained(ctx, gemv_f32_kernel<V_, true>, grid, dim3(256), 0, lhs, rhs, bias, out, batch, \
                                        rows, K, lhs_batched, rhs_batched)                                            \
                    : mb_launch_chained(ctx, gemv_f32_kernel<V_, false>, grid, dim3(256), 0, lhs, rhs, bias, out, batch, \
                                        rows, K, lhs_batched, rhs_batched));
  if (vecs == 8) { MB_GEMV(8) } else if (vecs == 4) { MB_GEMV(4) } else if (vecs == 2) { MB_GEMV(2) } else { MB_GEMV(1) }
#undef MB_GEMV
  ctx->launches++;
  return MB_SUCCESS;
}

static int check_conv_f32(mb_context *ctx, const char *who, const float *in, const float *filter,
                          float *out, int64_t N, int64_t C, int64_t H, int64_t W, int64_t O,
                          int64_t KH, int64_t KW, int sh, int sw, int dh, int dw, int pt, int pl,
                          int64_t Ho, int64_t Wo, int act, bool *empty) {
  *empty = false;
  if (N < 0 || C < 1 || H < 1 || W < 1 || O < 1 || KH < 1 || KW < 1 || sh < 1 || sw < 1 ||
      dh < 1 || dw < 1 || pt < 0 || pl < 0 || Ho < 0 || Wo < 0)
    return mb_fail(ctx, MB_INVALID_ARGS, "%s: bad shape argument", who);
  if (!(act == 0 || act == 1 || act == 2 || act == 6))
    return mb_fail(ctx, MB_UNSUPPORTED, "%s: activation %d is not fused here", who, act);
  if (N == 0 || Ho == 0 || Wo == 0) {
    *empty = true;
    return MB_SUCCESS;
  }
  if (in == nullptr || filter == nullptr || out == nullptr)
    return mb_fail(ctx, MB_INVALID_ARGS, "%s: null operand", who);
  if (N * O * Ho * Wo >= (1ll << 38) || N * C * H * W >= (1ll << 38))
    return mb_fail(ctx, MB_UNSUPPORTED, "%s: tensor too large", who);
  return MB_SUCCESS;
}

int mb_conv2d_f32_nchw(mb_context *ctx, const float *in, const float *filter, const float *bias,
                       float *out, int64_t N, int64_t C, int64_t H, int64_t W, int64_t O,
                       int64_t KH, int64_t KW, int stride_h, int stride_w, int dil_h, int dil_w,
                       int pad_top, int pad_left, int64_t Ho, int64_t Wo, int activation,
                       float max_limit, float coefficient) {
  if (ctx == nullptr) return MB_INVALID_ARGS;
  bool empty;
  MB_RETURN_IF_ERROR(check_conv_f32(ctx, "mb_conv2d_f32_nchw", in, filter, out, N, C, H, W, O, KH,
                                    KW, stride_h, stride_w, dil_h, dil_w, pad_top, pad_left, Ho,
                                    Wo, activation, &empty));
  if (empty) return MB_SUCCESS;
  MB_CUDA(ctx, cudaSetDevice(ctx->device));
  const bool pointwise = pointwise_in_place(KH, KW, stride_h, stride_w, pad_top, pad_left, H, W, Ho, Wo);
  {
    const bool by_tma = pointwise && long_rows(H * W) && mb_gemm_f32_tc_supported(ctx, in, filter, H * W, O, C, H * W, C * H * W, C, 0);
    const bool on_cores = pointwise && long_rows(H * W) ? !by_tma : !column_route(N, C, O, KH, KW, Ho, Wo);
    mb_f32_gemm g = conv_gemm(in, filter, bias, nullptr, out, N, C, H, W, O, KH, KW, stride_h, stride_w, dil_h, dil_w, pad_top,
                              pad_left, Ho, Wo, activation, max_limit, coefficient);
    // Stride 1, the output as large as the input: every input value split once instead of once per tap.  Nine taps and more:
    // with fewer the input's way through registers is what a block waits for (512 -> 128 channels, 1x1, 28 x 28, batch 16:
    // 35 us against 17; 64 -> 64, 5x5, 56 x 56, batch 24: 69 against 130).
    mb_f32_conv d;
    d.X = in; d.filter = filter; d.bias = bias; d.out = out;
    d.N = N; d.C = C; d.H = H; d.W = W; d.O = O; d.KH = static_cast<int>(std::min<int64_t>(KH, 99)); d.KW = static_cast<int>(std::min<int64_t>(KW, 99));
    d.act = activation; d.max_limit = max_limit; d.coef = coefficient;
    d.run = static_cast<int>(std::max<int64_t>(1, 10 / KW));  // an error of 3.5e-7 to 4e-7, the self-fetching kernel's at depth 60
    if (stride_h == 1 && stride_w == 1 && dil_h == 1 && dil_w == 1 && pad_top == KH / 2 && pad_left == KW / 2 && Ho == H && Wo == W &&
        ctx->f32_direct != 1 && mb_conv_f32_direct_supported(ctx, d) &&
        (ctx->f32_direct == 2 || (ctx->f32_gather == 0 && !on_cores && KH * KW >= 9 && C * KH * KW >= 128 &&
                                  mb_gemm_f32_gather_supported(ctx, g) &&
                                  mb_conv_f32_direct_cost(ctx, d) < mb_gemm_f32_gather_cost(ctx, g)))) {
      bool done = false;
      MB_RETURN_IF_ERROR(mb_conv_f32_direct_launch(ctx, d, &done));
      if (done) return MB_SUCCESS;
    }
    // Few input channels, a stride of two columns: input values split once, not once per tap, where the estimate is the smaller
    // (3 -> 64 channels, 7x7, 224 x 224, batch 8: 30 us fetching its own operands, 22 this way; 2: 12.9 and 13.6).  Up to 64 deep
    // the self-fetching kernel's form with three accumulators is the more accurate.
    if (dil_h == 1 && dil_w == 1 && ctx->f32_stem != 1 && mb_conv_f32_stem_supported(ctx, d, stride_h, stride_w, pad_left, Ho, Wo) &&
        (ctx->f32_stem == 2 || (ctx->f32_gather == 0 && !on_cores && C * KH * KW > 64 && mb_gemm_f32_gather_supported(ctx, g) &&
                                mb_conv_f32_stem_cost(ctx, d, stride_h, Ho, Wo) < mb_gemm_f32_gather_cost(ctx, g))))
      return mb_conv_f32_stem_launch(ctx, d, stride_h, pad_top, pad_left, Ho, Wo);
    // However small: the one-thread-per-output kernel is a serial chain over the depth (depth 64, 4 x 4 pixels, 22.8 us against
    // 6.5; 144, 3 x 3, 18.8 against 6.6; near the line, 48 to 54, 4.5 to 14 against 5.0 to 6.7).
    if (take_gather(ctx, g, by_tma, on_cores)) return mb_gemm_f32_gather_launch(ctx, g);
  }
  if (pointwise && (long_rows(H * W) || !ctx->use_tensor_cores)) {
    // out_n[O x HW] = filter[O x C] * in_n[C x HW] for every image n
    // (arm::Conv2dK1x1, mace/ops/arm/base/conv_2d_1x1.cc:61-68)
    const int64_t hw = H * W;
    return mb_gemm_f32_strided(ctx, filter, in, out, bias, N, O, hw, C, C, 1, 0, hw, 1, C * hw, hw,
                               1, O * hw, activation, max_limit, coefficient);
  }
  // (beyond the limits of the kernel that fetches its own operands:) enough work to fill tensor-core tiles: gather columns
  // and multiply.  Else the one-thread-per-output kernel.
  if (column_route(N, C, O, KH, KW, Ho, Wo)) {
    return conv2d_f32_im2col(ctx, in, filter, bias, out, N, C, H, W, O, KH, KW, stride_h, stride_w, dil_h,
                             dil_w, pad_top, pad_left, Ho, Wo, activation, max_limit, coefficient);
  }
  ConvF32Params p;
  p.in = in; p.filter = filter; p.bias = bias; p.out = out;
  p.N = static_cast<int>(N); p.C = static_cast<int>(C); p.H = static_cast<int>(H); p.W = static_cast<int>(W);
  p.O = static_cast<int>(O); p.KH = static_cast<int>(KH); p.KW = static_cast<int>(KW);
  p.sh = stride_h; p.sw = stride_w; p.dh = dil_h; p.dw = dil_w; p.pad_t = pad_top; p.pad_l = pad_left;
  p.Ho = static_cast<int>(Ho); p.Wo = static_cast<int>(Wo);
  p.act = activation; p.max_limit = max_limit; p.coef = coefficient;
  const int64_t total = N * O * Ho * Wo;
  MB_CUDA(ctx, mb_launch_chained(ctx, conv2d_f32_direct_kernel, dim3(static_cast<unsigned>(ceil_div64(total, 256))),
                                 dim3(256), 0, p));
  ctx->launches++;
  return MB_SUCCESS;
}

int mb_conv2d_f32_nchw_residual(mb_context *ctx, const float *in, const float *filter, const float *bias,
                                const float *residual, float *out, int64_t N, int64_t C, int64_t H,
                                int64_t W, int64_t O, int64_t KH, int64_t KW, int stride_h, int stride_w,
                                int dil_h, int dil_w, int pad_top, int pad_left, int64_t Ho, int64_t Wo,
                                int activation, float max_limit, float coefficient) {
  if (ctx == nullptr) return MB_INVALID_ARGS;
  if (residual == nullptr)
    return mb_conv2d_f32_nchw(ctx, in, filter, bias, out, N, C, H, W, O, KH, KW, stride_h, stride_w, dil_h,
                              dil_w, pad_top, pad_left, Ho, Wo, activation, max_limit, coefficient);
  bool empty;
  MB_RETURN_IF_ERROR(check_conv_f32(ctx, "mb_conv2d_f32_nchw_residual", in, filter, out, N, C, H, W, O, KH,
                                    KW, stride_h, stride_w, dil_h, dil_w, pad_top, pad_left, Ho, Wo,
                                    activation, &empty));
  if (empty) return MB_SUCCESS;
  MB_CUDA(ctx, cudaSetDevice(ctx->device));
  const int64_t hw = H * W;
  const bool pointwise_rows = pointwise_in_place(KH, KW, stride_h, stride_w, pad_top, pad_left, H, W, Ho, Wo) && long_rows(hw);
  const bool by_tma = pointwise_rows && mb_gemm_f32_tc_supported(ctx, in, filter, hw, O, C, hw, C * hw, C, 0);
  const bool on_cores = pointwise_rows ? !by_tma : !column_route(N, C, O, KH, KW, Ho, Wo);
  mb_f32_gemm g = conv_gemm(in, filter, bias, residual, out, N, C, H, W, O, KH, KW, stride_h, stride_w, dil_h, dil_w, pad_top,
                            pad_left, Ho, Wo, activation, max_limit, coefficient);
  if (take_gather(ctx, g, by_tma, on_cores)) return mb_gemm_f32_gather_launch(ctx, g);
  // 1x1 stride 1 on the tensor cores: the sum and the activation ride in the GEMM's epilogue
  if (by_tma && (reinterpret_cast<uintptr_t>(residual) & 3u) == 0) {
    return mb_gemm_f32_tc_launch(ctx, in, filter, bias, out, N, hw, O, C, hw, C * hw, C, 0, hw, O * hw,
                                 activation, max_limit, coefficient, residual);
  }
  // every other shape: the convolution without activation, then sum + activation in place
  // (of a copy of the residual where it lies in the output)
  const int64_t count = N * O * Ho * Wo;
  float *copy = nullptr;
  if (mb_ranges_meet(residual, out, count * 4)) {
    MB_CUDA(ctx, cudaMallocAsync(reinterpret_cast<void **>(&copy), count * 4, ctx->stream));
    MB_CUDA(ctx, cudaMemcpyAsync(copy, residual, count * 4, cudaMemcpyDeviceToDevice, ctx->stream));
    residual = copy;
  }
  int status = mb_conv2d_f32_nchw(ctx, in, filter, bias, out, N, C, H, W, O, KH, KW, stride_h, stride_w, dil_h, dil_w, pad_top,
                                  pad_left, Ho, Wo, 0, 0.f, 0.f);
  if (status == MB_SUCCESS)
    status = mb_eltwise_act_f32(ctx, out, residual, out, count, 0, 0.f, 0, 0.f, 0.f, 0, activation, max_limit, coefficient);
  if (copy != nullptr) MB_CUDA(ctx, cudaFreeAsync(copy, ctx->stream));
  return status;
}

int mb_dwconv_f32_nchw(mb_context *ctx, const float *in, const float *filter, const float *bias,
                       float *out, int64_t N, int64_t C, int64_t H, int64_t W, int64_t mult_ch,
                       int64_t KH, int64_t KW, int stride_h, int stride_w, int dil_h, int dil_w,
                       int pad_top, int pad_left, int64_t Ho, int64_t Wo, int activation,
                       float max_limit, float coefficient) {
  if (ctx == nullptr) return MB_INVALID_ARGS;
  bool empty;
  MB_RETURN_IF_ERROR(check_conv_f32(ctx, "mb_dwconv_f32_nchw", in, filter, out, N, C, H, W,
                                    mult_ch, KH, KW, stride_h, stride_w, dil_h, dil_w, pad_top,
                                    pad_left, Ho, Wo, activation, &empty));
  if (empty) return MB_SUCCESS;
  MB_CUDA(ctx, cudaSetDevice(ctx->device));
  return mb_dwconv_f32_launch(ctx, in, filter, bias, out, N, C, H, W, mult_ch, KH, KW, stride_h, stride_w, dil_h,
                              dil_w, pad_top, pad_left, Ho, Wo, activation, max_limit, coefficient);
}

}  // extern "C"
