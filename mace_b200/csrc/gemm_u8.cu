// mb_gemm_u8: argument checks, operand preparation (row/column byte sums for
// the zero-point correction, copies of rows that TMA cannot address) and the
// choice between the kernels: the persistent one (gemm_u8_tc.cu), one tile per
// CTA with the depth cut over a cluster (gemm_u8_cut.cu: operands by TMA;
// gemm_u8_gather.cu: rows of any alignment), a few rows on CUDA cores
// (gemm_u8_skinny.cu), and a CUDA-core kernel that takes any depth and size and
// runs for ragged products of up to 2^18 multiplications, depths beyond 33000
// and with the tensor cores switched off.
//
// Reference behaviour: MatMulFixpointImpl (mace/ops/matmul.cc:228-394) and the
// GEMM of the quantized Conv2D (mace/ops/conv_2d.cc:301-315).
#include <algorithm>

#include "common.cuh"
#include "gemm_u8_cut.cuh"

bool mb_gemm_u8_tc_supported(const mb_context *ctx, const void *A, const void *B, int64_t M, int64_t N, int64_t K,
                             int64_t lda, int64_t ldb);

namespace {

// ---- CUDA-core GEMM: any major order, any size --------------------------------
// 64 x 64 output tile per 256-thread block, 4 x 4 outputs per thread.  Operands
// are read element-wise with their own strides, the zero points are subtracted
// on load, so no correction terms and no overflow for any depth whose true
// result fits int32.
constexpr int GT = 64;   // tile edge
constexpr int GK = 32;   // depth per step

struct GenericParams {
  const uint8_t *A, *B;
  const int32_t *bias;
  void *C;
  int64_t M, N, K;
  int64_t a_rs, a_cs;  // strides of A(m,k): m * a_rs + k * a_cs
  int64_t b_rs, b_cs;  // strides of B(k,n): k * b_rs + n * b_cs
  int64_t a_bs, b_bs;  // batch strides (0 when not batched)
  int32_t zp_a, zp_b;
  mb_requant_params rq;
  int out_is_int32, bias_per_row;
};

__global__ void __launch_bounds__(256) gemm_u8_generic_kernel(const GenericParams p) {
  __shared__ int16_t As[GK][GT + 2];
  __shared__ int16_t Bs[GK][GT + 2];
  mb_grid_dep_launch();
  mb_grid_dep_wait();
  const int b = blockIdx.z;
  const int64_t m0 = static_cast<int64_t>(blockIdx.y) * GT;
  const int64_t n0 = static_cast<int64_t>(blockIdx.x) * GT;
  const uint8_t *A = p.A + b * p.a_bs;
  const uint8_t *B = p.B + b * p.b_bs;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  int32_t acc[4][4] = {};
  for (int64_t k0 = 0; k0 < p.K; k0 += GK) {
    for (int i = threadIdx.x; i < GK * GT; i += 256) {
      // pick the fastest-varying index so that loads coalesce for either major
      int kk, mm;
      if (p.a_cs == 1) { kk = i % GK; mm = i / GK; } else { mm = i % GT; kk = i / GT; }
      const int64_t m = m0 + mm, k = k0 + kk;
      As[kk][mm] = (m < p.M && k < p.K)
                       ? static_cast<int16_t>(static_cast<int32_t>(A[m * p.a_rs + k * p.a_cs]) - p.zp_a)
                       : 0;
      int nn;
      if (p.b_cs == 1) { nn = i % GT; kk = i / GT; } else { kk = i % GK; nn = i / GK; }
      const int64_t n = n0 + nn;
      const int64_t kb = k0 + kk;
      Bs[kk][nn] = (n < p.N && kb < p.K)
                       ? static_cast<int16_t>(static_cast<int32_t>(B[kb * p.b_rs + n * p.b_cs]) - p.zp_b)
                       : 0;
    }
    __syncthreads();
#pragma unroll 8
    for (int kk = 0; kk < GK; ++kk) {
      int32_t a[4], bv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) bv[j] = Bs[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += a[i] * bv[j];
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int64_t m = m0 + ty * 4 + i;
    if (m >= p.M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t n = n0 + tx * 4 + j;
      if (n >= p.N) continue;
      int32_t v = acc[i][j];
      if (p.bias != nullptr) v += p.bias_per_row ? p.bias[m] : p.bias[n];
      const int64_t idx = (static_cast<int64_t>(b) * p.M + m) * p.N + n;
      if (p.out_is_int32) {
        static_cast<int32_t *>(p.C)[idx] = v;
      } else {
        static_cast<uint8_t *>(p.C)[idx] =
            static_cast<uint8_t>(mb_requant_fast(v, p.rq));
      }
    }
  }
}

// ---- rows of any length -> rows of a 16-byte pitch ---------------------------------------
// TMA addresses rows that start 16-byte aligned.  An operand whose rows do not (an odd depth, an odd
// sequence length, a base inside another tensor) is copied once into scratch with its rows apart by
// the next multiple of 16, the gap filled with one value; its major order stays.  Both operands in one
// launch.  A thread writes one word per step: it reads the two aligned words that hold its four bytes
// (neighbouring lanes read neighbouring words, whatever the alignment) and shifts.  Only words
// that hold at least one byte of the row are read.  Bound by its launch for operands of a few
// megabytes (they stay in L2): 333 x 1001 x 777, batch 4, both operands copied: 14 us in all, 195 us on the
// CUDA-core kernel.
struct RepackJob {
  const uint8_t *src;
  uint8_t *dst;
  int64_t len, ld;          // bytes of a row; bytes from row to row in dst
  uint32_t words;           // of dst
  uint32_t fill;            // four times the byte of the gaps
  uint32_t row_mul, row_shift;
  int blocks;
};

constexpr int REPACK_STEPS = 4;

__global__ void __launch_bounds__(256) repack_rows_u8_kernel(const RepackJob a, const RepackJob b) {
  mb_grid_dep_launch();
  const bool first = static_cast<int>(blockIdx.x) < a.blocks;
  const RepackJob &j = first ? a : b;
  const uint32_t block = first ? blockIdx.x : blockIdx.x - a.blocks;
  const uint32_t row_words = static_cast<uint32_t>(j.ld >> 2);
  mb_grid_dep_wait();
  uint32_t lo[REPACK_STEPS], hi[REPACK_STEPS];
  int sh[REPACK_STEPS], left[REPACK_STEPS];
#pragma unroll
  for (int s = 0; s < REPACK_STEPS; ++s) {
    const uint32_t w = (block * REPACK_STEPS + s) * 256u + threadIdx.x;
    const uint32_t row = fast_div(w, j.row_mul, j.row_shift);
    const int64_t at = static_cast<int64_t>(w - row * row_words) * 4;
    left[s] = w < j.words ? static_cast<int>(max(min(j.len - at, static_cast<int64_t>(4)), static_cast<int64_t>(0))) : 0;
    const uint8_t *q = j.src + static_cast<int64_t>(row) * j.len + at;
    const int off = static_cast<int>(reinterpret_cast<uintptr_t>(q) & 3u);
    const uint32_t *aligned = reinterpret_cast<const uint32_t *>(q - off);
    sh[s] = off * 8;
    lo[s] = left[s] > 0 ? mb_load(aligned) : 0u;
    hi[s] = left[s] + off > 4 ? mb_load(aligned + 1) : 0u;
  }
#pragma unroll
  for (int s = 0; s < REPACK_STEPS; ++s) {
    const uint32_t w = (block * REPACK_STEPS + s) * 256u + threadIdx.x;
    uint32_t v = __funnelshift_r(lo[s], hi[s], sh[s]);
    if (left[s] < 4) {
      const uint32_t mask = (1u << (8 * left[s])) - 1u;
      v = (v & mask) | (j.fill & ~mask);
    }
    if (w < j.words) reinterpret_cast<uint32_t *>(j.dst)[w] = v;
  }
}

int launch_generic(mb_context *ctx, const uint8_t *A, const uint8_t *B, const int32_t *bias,
                   void *C, int out_is_int32, int64_t batch, int64_t M, int64_t N, int64_t K,
                   bool a_mn, bool b_mn, int a_batched, int b_batched, int32_t zp_a,
                   int32_t zp_b, int32_t mult, int32_t shift, int32_t zp_c, int bias_per_row) {
  GenericParams p;
  p.A = A; p.B = B; p.bias = bias; p.C = C;
  p.M = M; p.N = N; p.K = K;
  // A K-major: (m,k) at m*K + k.  A MN-major: (m,k) at k*M + m.
  p.a_rs = a_mn ? 1 : K; p.a_cs = a_mn ? M : 1;
  // B MN-major (row-major K x N): (k,n) at k*N + n.  B K-major: n*K + k.
  p.b_rs = b_mn ? N : 1; p.b_cs = b_mn ? 1 : K;
  p.a_bs = a_batched ? M * K : 0; p.b_bs = b_batched ? K * N : 0;
  p.zp_a = zp_a; p.zp_b = zp_b;
  p.rq = mb_make_requant(mult, shift, zp_c);
  p.out_is_int32 = out_is_int32; p.bias_per_row = bias_per_row;
  const int64_t gx = ceil_div64(N, GT), gy = ceil_div64(M, GT);
  if (gy > 65535 || batch > 65535)
    return mb_fail(ctx, MB_UNSUPPORTED, "generic GEMM: M or batch too large for this path");
  dim3 grid(static_cast<unsigned>(gx), static_cast<unsigned>(gy), static_cast<unsigned>(batch));
  MB_CUDA(ctx, mb_launch_chained(ctx, gemm_u8_generic_kernel, grid, dim3(256), 0, p));
  ctx->launches++;
  return MB_SUCCESS;
}

}  // namespace

// Rows of a_len bytes at A -> rows lda bytes apart at a_dst (lda a multiple of 16, fewer than 2^33 bytes in
// all), the gap filled with fill_a; the same for B.  Either source may be null.
int mb_repack_rows_u8(mb_context *ctx, const uint8_t *A, uint8_t *a_dst, int64_t a_rows, int64_t a_len, int64_t lda,
                      int fill_a, const uint8_t *B, uint8_t *b_dst, int64_t b_rows, int64_t b_len, int64_t ldb,
                      int fill_b) {
  auto make = [](const uint8_t *src, uint8_t *dst, int64_t rows, int64_t len, int64_t ld, int fill) {
    RepackJob j = {};
    if (src == nullptr) return j;
    j.src = src; j.dst = dst; j.len = len; j.ld = ld;
    j.fill = static_cast<uint32_t>(fill & 255) * 0x01010101u;
    j.words = static_cast<uint32_t>(rows * ld / 4);
    fast_div_make(static_cast<uint32_t>(ld / 4), &j.row_mul, &j.row_shift);
    j.blocks = static_cast<int>(ceil_div64(j.words, 256 * REPACK_STEPS));
    return j;
  };
  const RepackJob ja = make(A, a_dst, a_rows, a_len, lda, fill_a), jb = make(B, b_dst, b_rows, b_len, ldb, fill_b);
  MB_CUDA(ctx, mb_launch_chained(ctx, repack_rows_u8_kernel, dim3(static_cast<unsigned>(ja.blocks + jb.blocks)),
                                 dim3(256), 0, ja, jb));
  ctx->launches++;
  return MB_SUCCESS;
}

bool mb_gemm_u8_skinny_supported(int64_t batch, int64_t M, int64_t N, int64_t K, bool a_mn, bool b_mn,
                                 const void *A, const void *B);
int mb_gemm_u8_skinny_launch(mb_context *ctx, const uint8_t *A, const uint8_t *B, const int32_t *bias,
                             void *C, int out_is_int32, int64_t M, int64_t N, int64_t K, int32_t zp_a,
                             int32_t zp_b, int32_t mult, int32_t shift, int32_t zp_c, int bias_per_row);

int mb_operand_sums_slices(const mb_context *ctx, bool mn, int64_t nb, int64_t K, int64_t cols);
int mb_gemm_u8_tc_launch_sliced(mb_context *ctx, const uint8_t *A, const uint8_t *B,
                                const uint32_t *sum_a, const uint32_t *sum_b, int sum_a_slices, int sum_b_slices,
                                const int32_t *bias, void *C, int out_is_int32, int64_t batch, int64_t M, int64_t N,
                                int64_t K, int64_t lda, int64_t ldb, bool a_mn, bool b_mn, int a_batched, int b_batched,
                                int32_t zp_a, int32_t zp_b, int32_t mult, int32_t shift, int32_t zp_c,
                                int bias_per_row);
int mb_operand_sums_launch(mb_context *ctx, const uint8_t *A, bool a_mn, int64_t nb_a, int64_t M, uint32_t *sum_a,
                           const uint8_t *B, bool b_mn, int64_t nb_b, int64_t N, uint32_t *sum_b, int64_t K,
                           int k_split, int64_t lda, int64_t ldb);
int mb_gemm_u8_tc_launch_splitk(mb_context *ctx, const uint8_t *A, const uint8_t *B,
                                const uint32_t *sum_a, const uint32_t *sum_b, int sum_a_slices, int sum_b_slices,
                                int32_t *parts, int k_split, int bn, int64_t M, int64_t N, int64_t K, bool a_mn,
                                bool b_mn, int32_t zp_a, int32_t zp_b);

namespace {

// ---- few output tiles, long depth: the depth cut into runs ----------------------------
// A product of 128 rows against a 4096 x 4096 matrix has 32 output tiles for 148 SMs, and each
// of the 32 pulls a megabyte through one SM.  Cutting the depth into S runs gives S times the
// CTAs, each streaming 1/S of the bytes; the S exact int32 partial results (zero-point terms
// included: they are linear in the depth) are added here, then bias and the fixed-point
// output stage as in the GEMM's own epilogue (mace/ops/common/gemmlowp_util.h:37-74).
struct SplitReduceParams {
  const int32_t *parts;   // [splits][M][N]
  const int32_t *bias;
  void *C;
  int64_t M, N;
  int splits, bias_per_row, out_is_int32;
  mb_requant_params rq;
};

template <int VEC>
__global__ void __launch_bounds__(256) gemm_u8_split_reduce_kernel(const SplitReduceParams p) {
  mb_grid_dep_launch();
  mb_grid_dep_wait();
  const int64_t total = p.M * p.N / VEC;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * 256) {
    const int64_t e = i * VEC;
    const int64_t m = e / p.N, n = e % p.N;
    int32_t acc[VEC];
#pragma unroll
    for (int j = 0; j < VEC; ++j) acc[j] = 0;
    for (int s = 0; s < p.splits; ++s) {
      const int32_t *src = p.parts + s * p.M * p.N + e;
      if (VEC == 4) {
        const int4 v = *reinterpret_cast<const int4 *>(src);
        acc[0] += v.x; acc[1 % VEC] += v.y; acc[2 % VEC] += v.z; acc[3 % VEC] += v.w;
      } else {
        acc[0] += src[0];
      }
    }
    if (p.bias != nullptr) {
#pragma unroll
      for (int j = 0; j < VEC; ++j) acc[j] += p.bias[p.bias_per_row ? m : n + j];
    }
    if (p.out_is_int32) {
#pragma unroll
      for (int j = 0; j < VEC; ++j) static_cast<int32_t *>(p.C)[e + j] = acc[j];
    } else if (VEC == 4) {
      uint32_t w = 0;
#pragma unroll
      for (int j = 0; j < VEC; ++j) w |= mb_requant_fast(acc[j], p.rq) << (8 * j);
      *reinterpret_cast<uint32_t *>(static_cast<uint8_t *>(p.C) + e) = w;
    } else {
      static_cast<uint8_t *>(p.C)[e] = static_cast<uint8_t>(mb_requant_fast(acc[0], p.rq));
    }
  }
}

// The number of runs for this shape (1: do not cut), and the tile width to run them with.
int split_k_choice(const mb_context *ctx, int64_t batch, int64_t M, int64_t N, int64_t K, int *bn) {
  if (!ctx->split_k || batch != 1 || K < 2048) return 1;
  *bn = N >= 128 ? 128 : 64;
  const int64_t tiles = ceil_div64(M, 128) * ceil_div64(N, *bn);
  int best = 1;
  for (int s : {2, 4, 8}) {
    if (tiles * s > ctx->num_sms) break;
    if (K % (static_cast<int64_t>(s) * 128) != 0 || K / s < 512) break;
    best = s;
  }
  // two runs do not pay for the extra kernel and the int32 round trip (measured at
  // M = 256, K = N = 4096: 15.2 us against 13.9 us undivided)
  return best >= 4 ? best : 1;
}

}  // namespace

// ---- the choice between the tensor-core kernels ----------------------------------------
// Estimated SM cycles of the persistent kernel (gemm_u8_tc.cu), from its times at 1024^3 (7.4 us), 512^3 (5.9 us),
// 16 x 1024 x 1024 (7.3 us), 256 x 4096 x 4096 (17 us) and 4096^3 (58 us): about 4.4 us around the steps, a row-major
// B whose column sums come from the tiles paces them; beyond a depth of 1024 (or with a column-major A) the sums
// are a kernel of their own.
int64_t mb_gemm_u8_persistent_cost(const mb_context *ctx, const mb_cut_gemm &g) {
  const int64_t tiles_m = ceil_div64(g.M, 128), steps = ceil_div64(g.K, 128);
  const bool fused = !g.a_mn && g.K <= 1024;
  int64_t best = -1;
  for (int w : {256, 128, 64}) {
    if (w > 64 && g.N <= w / 2) continue;
    const int64_t rounds = ceil_div64(g.batch * tiles_m * ceil_div64(g.N, w), ctx->num_sms);
    const int64_t step = fused ? (g.b_mn ? (w == 256 ? 1400 : w == 128 ? 930 : 720) : (w == 256 ? 900 : 700)) : (w == 256 ? 900 : w == 128 ? 600 : 520);
    const int64_t cost = rounds * std::max<int64_t>(steps * step, w == 256 ? 2600 : w == 128 ? 1500 : 900);
    if (best < 0 || cost < best) best = cost;
  }
  return best + (fused ? 8300 : 13300);
}

namespace {

// The same of the few-row kernel (gemm_u8_skinny.cu), which takes panels of 256 rows of B, from 1, 4, 8 and 16 rows against
// 256 .. 1024 x 20004 .. 200004 (1 row: 6.2 us at 256 x 20004, 18.5 at 200004; 16 rows: 14.4, 191 at 1024 x 200004).
int64_t skinny_cost(int64_t M, int64_t N, int64_t K) {
  const int64_t bytes = ceil_div64(K, 256) * 256 * N;
  return M <= 1 ? 9200 + bytes / 1950 : M <= 4 ? 13400 + bytes / 1950 : M <= 8 ? 16000 + bytes / 1200 : 22000 + bytes / 600;
}

// Runs the product on a cluster-cut kernel where that is estimated to be the fastest way: as it lies, or, with rows that
// TMA cannot address, on copies that it can (2.4 us for the extra launch and the bytes at about 4 TB/s); or, few ragged
// rows, on the kernel made for them.  Else the caller takes the persistent kernel, on copies.
bool try_cut(mb_context *ctx, const mb_cut_gemm &g, bool a_copy, bool b_copy, int *status) {
  const mb_cut_plan direct = mb_gemm_u8_cut_plan(ctx, g);
  int64_t other = mb_gemm_u8_persistent_cost(ctx, g);
  if (!a_copy && !b_copy) {
    if (direct.cost < 0 || (ctx->cut_aligned == 0 ? direct.cost >= other : ctx->cut_aligned == 1)) return false;
    *status = mb_gemm_u8_cut_launch(ctx, g, direct);
    return true;
  }
  const int64_t a_rows = (g.a_batched ? g.batch : 1) * (g.a_mn ? g.K : g.M), b_rows = (g.b_batched ? g.batch : 1) * (g.b_mn ? g.K : g.N);
  const int64_t a_len = g.a_mn ? g.M : g.K, b_len = g.b_mn ? g.N : g.K;
  const int64_t lda = static_cast<int64_t>(align_up(static_cast<size_t>(a_len), 16)), ldb = static_cast<int64_t>(align_up(static_cast<size_t>(b_len), 16));
  const int64_t copy_cost = 4500 + ((a_copy ? 2 * a_rows * a_len : 0) + (b_copy ? 2 * b_rows * b_len : 0)) / 2000;
  mb_cut_gemm c = g;
  if (a_copy) { c.A = nullptr; c.lda = lda; }
  if (b_copy) { c.B = nullptr; c.ldb = ldb; }
  const mb_cut_plan copied = mb_gemm_u8_cut_plan(ctx, c);
  other += copy_cost;
  if (g.M <= ctx->skinny_max_m && mb_gemm_u8_skinny_supported(g.batch, g.M, g.N, g.K, g.a_mn, g.b_mn, g.A, g.B)) {
    const int64_t skinny = skinny_cost(g.M, g.N, g.K);
    if (skinny < other && (direct.cost < 0 || skinny < direct.cost) && (copied.cost < 0 || skinny < copied.cost + copy_cost)) {
      *status = mb_gemm_u8_skinny_launch(ctx, g.A, g.B, g.bias, g.C, g.out_is_int32, g.M, g.N, g.K, g.zp_a, g.zp_b, g.rq.mult,
                                         g.rq.sh - 31, g.rq.zp, g.bias_per_row);
      return true;
    }
  }
  if (direct.cost >= 0 && direct.cost <= other && (copied.cost < 0 || direct.cost <= copied.cost + copy_cost)) {
    *status = mb_gemm_u8_cut_launch(ctx, g, direct);
    return true;
  }
  if (copied.cost < 0 || copied.cost + copy_cost >= other || (a_copy && a_rows * lda >= (1ll << 33)) || (b_copy && b_rows * ldb >= (1ll << 33)))
    return false;
  const size_t a_bytes = a_copy ? align_up(static_cast<size_t>(a_rows * lda), 256) : 0;
  uint8_t *scratch = nullptr;
  *status = mb_scratch(ctx, a_bytes + (b_copy ? static_cast<size_t>(b_rows * ldb) : 0), reinterpret_cast<void **>(&scratch));
  if (*status != MB_SUCCESS) return true;
  *status = mb_repack_rows_u8(ctx, a_copy ? g.A : nullptr, scratch, a_rows, a_len, lda, 0, b_copy ? g.B : nullptr,
                              scratch + a_bytes, b_rows, b_len, ldb, 0);
  if (*status != MB_SUCCESS) return true;
  if (a_copy) c.A = scratch;
  if (b_copy) c.B = scratch + a_bytes;
  *status = mb_gemm_u8_cut_launch(ctx, c, copied);
  return true;
}

}  // namespace

// Row-major-C GEMM on device operands; a_mn / b_mn as in mb_gemm_u8_tc_launch.
int mb_gemm_u8_rowmajor(mb_context *ctx, const uint8_t *A, const uint8_t *B, const int32_t *bias,
                        void *C, int out_is_int32, int64_t batch, int64_t M, int64_t N,
                        int64_t K, bool a_mn, bool b_mn, int a_batched, int b_batched,
                        int32_t zp_a, int32_t zp_b, int32_t mult, int32_t shift, int32_t zp_c,
                        int bias_per_row) {
  bool use_tc = ctx->use_tensor_cores && ctx->encode_tiled != nullptr && K <= 33000 && M < (1ll << 31) && N < (1ll << 31);
  // Each operand reaches the tensor core in its own major order, in place when its rows are 16-byte
  // aligned, else through a copy with a 16-byte pitch.
  const int64_t a_len = a_mn ? M : K, b_len = b_mn ? N : K;
  const bool a_copy = a_len % 16 != 0 || (reinterpret_cast<uintptr_t>(A) & 15u) != 0;
  const bool b_copy = b_len % 16 != 0 || (reinterpret_cast<uintptr_t>(B) & 15u) != 0;
  // A ragged product of a few thousand multiplications per SM is not worth the copy: one launch of the
  // CUDA-core kernel is over before the copy's successor could start.
  if ((a_copy || b_copy) && batch * M * N * K <= (1 << 18)) use_tc = false;
  const bool cut_rule = use_tc && ctx->split_k && ctx->skinny_max_m > 0 && !ctx->pair_gemm && (ctx->force_bn == 0 || a_copy || b_copy);
  if (cut_rule) {
    mb_cut_gemm g;
    g.A = A; g.B = B; g.bias = bias; g.C = C; g.out_is_int32 = out_is_int32; g.bias_per_row = bias_per_row;
    g.batch = batch; g.M = M; g.N = N; g.K = K; g.a_mn = a_mn; g.b_mn = b_mn;
    g.a_batched = a_batched; g.b_batched = b_batched; g.zp_a = zp_a; g.zp_b = zp_b;
    g.rq = mb_make_requant(mult, shift, zp_c);
    g.rq_variant = mb_requant_variant(shift, zp_c);
    int st = MB_SUCCESS;
    // Up to 16 rows of a row-major B always: what else there is for them (a streaming kernel on CUDA cores) takes 4.6 to 10.5
    // us where the cut takes 3.9 (3 .. 16 rows, 256 x 864 .. 4096).
    if (!a_copy && !b_copy && M <= ctx->skinny_max_m && ctx->cut_aligned == 0 &&
        mb_gemm_u8_skinny_supported(batch, M, N, K, a_mn, b_mn, A, B)) {
      const mb_cut_plan plan = mb_gemm_u8_cut_plan(ctx, g);
      if (plan.cost >= 0) return mb_gemm_u8_cut_launch(ctx, g, plan);
    }
    if (try_cut(ctx, g, a_copy, b_copy, &st)) return st;
  }
  // With the cluster-cut kernels off (split_k or skinny_max_m = 0), or beyond their depth: a few rows against a large
  // row-major B on CUDA cores, or on the tensor cores with the depth cut into runs through global memory.
  if (ctx->use_tensor_cores && !(cut_rule && (a_copy || b_copy)) && M <= ctx->skinny_max_m && mb_gemm_u8_skinny_supported(batch, M, N, K, a_mn, b_mn, A, B)) {
    int bn_unused = 0;
    const bool runs_apply = M >= ctx->runs_min_m && use_tc && !a_copy && !b_copy &&
                            split_k_choice(ctx, batch, M, N, K, &bn_unused) > 1;
    if (!runs_apply)
      return mb_gemm_u8_skinny_launch(ctx, A, B, bias, C, out_is_int32, M, N, K, zp_a, zp_b, mult, shift,
                                      zp_c, bias_per_row);
  }
  if (!use_tc) {
    return launch_generic(ctx, A, B, bias, C, out_is_int32, batch, M, N, K, a_mn, b_mn,
                          a_batched, b_batched, zp_a, zp_b, mult, shift, zp_c, bias_per_row);
  }
  const int64_t nb_a = a_batched ? batch : 1, nb_b = b_batched ? batch : 1;
  int split_bn = 0;
  const int splits = (a_copy || b_copy) ? 1 : split_k_choice(ctx, batch, M, N, K, &split_bn);
  if (splits > 1 && mb_gemm_u8_tc_supported(ctx, A, B, M, N, K / splits, a_len, b_len)) {
    const int64_t Ks = K / splits;
    // runs no longer than 1024 with a K-major A: the kernel sums the bytes of its own tiles
    const bool fused = !a_mn && Ks <= 1024;
    const bool want_a = zp_b != 0 && !fused, want_b = zp_a != 0 && !fused;
    const int sl_a = want_a ? mb_operand_sums_slices(ctx, a_mn, splits, Ks, M) : 1;
    const int sl_b = want_b ? mb_operand_sums_slices(ctx, b_mn, splits, Ks, N) : 1;
    size_t off = 0;
    const size_t off_parts = off; off += align_up(sizeof(int32_t) * splits * M * N, 256);
    const size_t off_sa = off; off += want_a ? align_up(sizeof(uint32_t) * splits * M * sl_a, 256) : 0;
    const size_t off_sb = off; off += want_b ? align_up(sizeof(uint32_t) * splits * N * sl_b, 256) : 0;
    uint8_t *scratch = nullptr;
    MB_RETURN_IF_ERROR(mb_scratch(ctx, off, reinterpret_cast<void **>(&scratch)));
    int32_t *parts = reinterpret_cast<int32_t *>(scratch + off_parts);
    uint32_t *sum_a = want_a ? reinterpret_cast<uint32_t *>(scratch + off_sa) : nullptr;
    uint32_t *sum_b = want_b ? reinterpret_cast<uint32_t *>(scratch + off_sb) : nullptr;
    if (want_a || want_b)
      MB_RETURN_IF_ERROR(mb_operand_sums_launch(ctx, A, a_mn, 1, M, sum_a, B, b_mn, 1, N, sum_b, K, splits, a_len, b_len));
    ctx->pdl_next_gemm = (want_a || want_b) ? 1 : 0;
    MB_RETURN_IF_ERROR(mb_gemm_u8_tc_launch_splitk(ctx, A, B, sum_a, sum_b, sl_a, sl_b, parts, splits, split_bn, M, N,
                                                   K, a_mn, b_mn, zp_a, zp_b));
    SplitReduceParams rp;
    rp.parts = parts; rp.bias = bias; rp.C = C; rp.M = M; rp.N = N;
    rp.splits = splits; rp.bias_per_row = bias_per_row; rp.out_is_int32 = out_is_int32;
    rp.rq = mb_make_requant(mult, shift, zp_c);
    const bool vec4 = N % 4 == 0 && (reinterpret_cast<uintptr_t>(C) & 3u) == 0;
    const int64_t work = M * N / (vec4 ? 4 : 1);
    const unsigned grid = static_cast<unsigned>(std::min<int64_t>(ceil_div64(work, 256), 8ll * ctx->num_sms));
    if (vec4) {
      MB_CUDA(ctx, mb_launch_chained(ctx, gemm_u8_split_reduce_kernel<4>, dim3(grid), dim3(256), 0, rp));
    } else {
      MB_CUDA(ctx, mb_launch_chained(ctx, gemm_u8_split_reduce_kernel<1>, dim3(grid), dim3(256), 0, rp));
    }
    MB_CUDA(ctx, cudaGetLastError());
    ctx->launches++;
    return MB_SUCCESS;
  }
  // A K-major A with K <= 1024 (B in either order): the tensor-core kernel sums the operand
  // bytes itself from the tiles it has in shared memory.
  // (option pair = 2, the CTA-pair kernel wherever it can run, takes its sums from the sums kernel)
  const bool fused_sums = !a_mn && K <= 1024 && ctx->pair_gemm != 2;
  const bool need_sum_a = zp_b != 0 && !fused_sums, need_sum_b = zp_a != 0 && !fused_sums;
  const int64_t lda = a_copy ? static_cast<int64_t>(align_up(a_len, 16)) : a_len;
  const int64_t ldb = b_copy ? static_cast<int64_t>(align_up(b_len, 16)) : b_len;
  const int64_t a_rows = nb_a * (a_mn ? K : M), b_rows = nb_b * (b_mn ? K : N);
  if (!mb_gemm_u8_tc_supported(ctx, nullptr, nullptr, M, N, K, lda, ldb) ||
      (a_copy && a_rows * lda >= (1ll << 33)) || (b_copy && b_rows * ldb >= (1ll << 33))) {
    return launch_generic(ctx, A, B, bias, C, out_is_int32, batch, M, N, K, a_mn, b_mn,
                          a_batched, b_batched, zp_a, zp_b, mult, shift, zp_c, bias_per_row);
  }
  size_t off = 0;
  // (an operand that reaches the tensor core MN-major gets its column sums as a few partial rows)
  const int sl_a = need_sum_a ? mb_operand_sums_slices(ctx, a_mn, nb_a, K, M) : 1;
  const int sl_b = need_sum_b ? mb_operand_sums_slices(ctx, b_mn, nb_b, K, N) : 1;
  const size_t off_sum_a = off; off += need_sum_a ? align_up(sizeof(uint32_t) * nb_a * M * sl_a, 256) : 0;
  const size_t off_sum_b = off; off += need_sum_b ? align_up(sizeof(uint32_t) * nb_b * N * sl_b, 256) : 0;
  const size_t off_at = off; off += a_copy ? align_up(a_rows * lda, 256) : 0;
  const size_t off_bt = off; off += b_copy ? align_up(b_rows * ldb, 256) : 0;

  uint8_t *scratch = nullptr;
  if (off > 0) MB_RETURN_IF_ERROR(mb_scratch(ctx, off, reinterpret_cast<void **>(&scratch)));
  uint32_t *sum_a = need_sum_a ? reinterpret_cast<uint32_t *>(scratch + off_sum_a) : nullptr;
  uint32_t *sum_b = need_sum_b ? reinterpret_cast<uint32_t *>(scratch + off_sum_b) : nullptr;
  const uint8_t *a_use = a_copy ? scratch + off_at : A, *b_use = b_copy ? scratch + off_bt : B;
  if (a_copy || b_copy)
    MB_RETURN_IF_ERROR(mb_repack_rows_u8(ctx, a_copy ? A : nullptr, scratch + off_at, a_rows, a_len, lda, 0,
                                         b_copy ? B : nullptr, scratch + off_bt, b_rows, b_len, ldb, 0));
  // both operands' sums in one launch (see operand_sums.cu)
  if (need_sum_a || need_sum_b)
    MB_RETURN_IF_ERROR(mb_operand_sums_launch(ctx, a_use, a_mn, nb_a, M, sum_a, b_use, b_mn, nb_b, N, sum_b, K, 1,
                                              lda, ldb));
  // The operand-sum kernel was the last launch: the GEMM may overlap it (programmatic
  // dependent launch); its operands were complete before that kernel started.
  ctx->pdl_next_gemm = (need_sum_a || need_sum_b) ? 1 : 0;
  return mb_gemm_u8_tc_launch_sliced(ctx, a_use, b_use, sum_a, sum_b, sl_a, sl_b, bias, C, out_is_int32, batch, M,
                                     N, K, lda, ldb, a_mn, b_mn, a_batched, b_batched, zp_a, zp_b, mult, shift,
                                     zp_c, bias_per_row);
}

extern "C" int mb_gemm_u8(mb_context *ctx, const uint8_t *A, const uint8_t *B,
                          const int32_t *bias, void *C, int out_is_int32, int64_t batch,
                          int64_t M, int64_t N, int64_t K, int a_col_major, int b_col_major,
                          int c_col_major, int a_batched, int b_batched, int32_t zp_a,
                          int32_t zp_b, int32_t multiplier, int32_t right_shift, int32_t zp_c,
                          int bias_per_row) {
  if (ctx == nullptr) return MB_INVALID_ARGS;
  if (batch < 0 || M < 0 || N < 0 || K < 0)
    return mb_fail(ctx, MB_INVALID_ARGS, "mb_gemm_u8: negative dimension");
  if (batch == 0 || M == 0 || N == 0) return MB_SUCCESS;  // empty output
  if (A == nullptr || B == nullptr || C == nullptr)
    return mb_fail(ctx, MB_INVALID_ARGS, "mb_gemm_u8: null operand");
  if (!out_is_int32) {
    // GetOutputMultiplierAndShift (mace/core/quantize.h:116-126) yields a
    // multiplier in [2^30, 2^31) and a right shift >= 0; RoundingDivideByPOT
    // is defined for shifts up to 31.
    if (multiplier <= 0 || right_shift < 0 || right_shift > 31)
      return mb_fail(ctx, MB_INVALID_ARGS, "mb_gemm_u8: bad multiplier %d / shift %d",
                     multiplier, right_shift);
    if (zp_c < 0 || zp_c > 255)
      return mb_fail(ctx, MB_INVALID_ARGS, "mb_gemm_u8: output zero point %d outside uint8", zp_c);
  }
  if (K == 0) {
    // Empty depth: the accumulator is zero, the pipeline still applies.
    return mb_fail(ctx, MB_UNSUPPORTED, "mb_gemm_u8: K == 0");
  }
  MB_CUDA(ctx, cudaSetDevice(ctx->device));
  // A(m,k) is K-major unless a_col_major; B(k,n) is K-major iff b_col_major.
  if (!c_col_major) {
    return mb_gemm_u8_rowmajor(ctx, A, B, bias, C, out_is_int32, batch, M, N, K,
                               a_col_major != 0, b_col_major == 0, a_batched, b_batched, zp_a,
                               zp_b, multiplier, right_shift, zp_c, bias_per_row);
  }
  // Column-major C (M x N) is row-major C^T (N x M) = B^T * A^T: swap the
  // roles of the operands.  A'(n,k) = B(k,n) is MN-major iff B is; likewise B'.
  return mb_gemm_u8_rowmajor(ctx, B, A, bias, C, out_is_int32, batch, N, M, K,
                             /*a_mn=*/b_col_major == 0, /*b_mn=*/a_col_major != 0, b_batched,
                             a_batched, zp_b, zp_a, multiplier, right_shift, zp_c,
                             bias != nullptr ? !bias_per_row : 0);
}
