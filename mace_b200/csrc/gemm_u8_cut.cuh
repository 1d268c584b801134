// uint8 GEMMs whose depth may be cut over a cluster of CTAs, in one launch: the description their callers --
// MatMul of few or ragged rows, k x k convolution, FullyConnected on a batch -- give, and the rule that
// picks the kernel (gemm_u8_cut.cu: operands by TMA; gemm_u8_gather.cu: operands at any alignment).
#pragma once

#include "common.cuh"

struct mb_cut_gemm {
  const uint8_t *A = nullptr, *B = nullptr;
  const int32_t *bias = nullptr;
  void *C = nullptr;  // row-major [batch][M][N], uint8 or int32
  int out_is_int32 = 0, bias_per_row = 0;
  int64_t batch = 1, M = 0, N = 0, K = 0;
  // A is [M x K] (K contiguous) or, a_mn, [K x M]; B is [N x K] or, b_mn, [K x N]; lda, ldb: bytes
  // from row to row (0: no gaps)
  int64_t lda = 0, ldb = 0;
  bool a_mn = false, b_mn = false;
  int a_batched = 0, b_batched = 0;
  int32_t zp_a = 0, zp_b = 0;
  mb_requant_params rq = {};
  int rq_variant = 0;  // mb_requant_variant(), or 8 for the Gemv delegators' float rule
  float mult_f = 0.f, zp_f = 0.f;
  // conv: A is the NHWC input of a convolution, M its output pixels and K = KH * KW * C its windows
  // in filter-row order (C = C_in, a multiple of 16), taps outside the image holding zp_a
  bool conv = false;
  int H = 0, W = 0, C_in = 0, KH = 1, KW = 1, sh = 1, sw = 1, pad_t = 0, pad_l = 0, Ho = 0, Wo = 0;
};

struct mb_cut_plan {
  int bn = 0, splits = 1;
  bool by_tma = true, two_per_sm = false;
  bool persistent = false;  // convolution on the persistent kernel of gemm_u8_tc.cu
  int64_t cost = -1;  // estimated SM cycles; negative: not possible
};

// The cheapest way for the product as it lies (by_tma only where every row is 16-byte aligned).
mb_cut_plan mb_gemm_u8_cut_plan(mb_context *ctx, const mb_cut_gemm &g);
// The same of the persistent kernel (gemm_u8_tc.cu; gemm_u8.cu has the estimate).
int64_t mb_gemm_u8_persistent_cost(const mb_context *ctx, const mb_cut_gemm &g);
int mb_gemm_u8_cut_launch(mb_context *ctx, const mb_cut_gemm &g, const mb_cut_plan &plan);
int mb_gemm_u8_gather_launch(mb_context *ctx, const mb_cut_gemm &g, int bn, int splits);

// CTAs of clusters of `s` that the device holds at once with one CTA per SM.
int64_t mb_resident_cluster_ctas(mb_context *ctx, int s);

// Rows of any length copied to a 16-byte pitch (gemm_u8.cu).
int mb_repack_rows_u8(mb_context *ctx, const uint8_t *A, uint8_t *a_dst, int64_t a_rows, int64_t a_len, int64_t lda,
                      int fill_a, const uint8_t *B, uint8_t *b_dst, int64_t b_rows, int64_t b_len, int64_t ldb,
                      int fill_b);

// A launch in clusters of `cluster` CTAs along x (1: none), chained like mb_launch_chained.
template <typename... KArgs, typename... Args>
static inline cudaError_t mb_launch_clusters(mb_context *ctx, void (*kern)(KArgs...), unsigned grid, unsigned threads,
                                             size_t smem, int cluster, Args &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[2];
  unsigned n = 0;
  if (cluster > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = static_cast<unsigned>(cluster);
    attr[n].val.clusterDim.y = 1;
    attr[n++].val.clusterDim.z = 1;
  }
  if (ctx->pdl_chain) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}
