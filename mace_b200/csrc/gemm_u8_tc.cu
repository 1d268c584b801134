// uint8 x uint8 -> int32 GEMM on the Blackwell tensor cores (tcgen05.mma
// kind::i8) with the whole gemmlowp output pipeline fused into the epilogue.
//
// What it replaces: gemmlowp::GemmWithOutputPipeline as called by MACE's
// quantized MatMul and Conv2D (mace/ops/matmul.cc:283-301, :369-385;
// mace/ops/conv_2d.cc:301-315) with the output stages of
// mace/ops/common/gemmlowp_util.h:37-74.
//
// Formulation.  The tensor core multiplies the raw bytes:
//   raw[m,n] = sum_k A[m,k] * B[k,n]                      (exact in int32)
// and the epilogue applies the zero-point correction
//   acc = raw - zp_b * rowsum_A[m] - zp_a * colsum_B[n] + K * zp_a * zp_b
// then + bias, fixed-point requantization, + zp_c, clamp, store.
//
// Structure (one persistent CTA per SM, 704 threads):
//   warp 0       TMA producer: 128-byte-swizzled tiles of A and B into a
//                multi-stage shared-memory ring (mbarrier full/empty pairs)
//   warp 1       MMA issuer: one thread issues tcgen05.mma 128 x BN x 32 steps
//                into one of two TMEM accumulator buffers
//   warps 2..5   preparation: per tile, the row and column terms of the
//                epilogue (zero-point corrections, bias) into shared memory.
//                With FUSE_SUMS they also add up the operand bytes of every
//                stage straight from the tiles in shared memory, so the
//                correction needs no extra pass over the operands; that mode
//                serves K-major operands with K <= 1024 (pointwise
//                convolutions), where the tensor pipe has time to spare.
//                Large-K GEMMs take their sums from separate kernels, because
//                the extra shared-memory reads would slow their main loop.
//   warps 6..21  epilogue: sets of four warps (one per TMEM lane quarter), each set on
//                a 64-column slice of a tile; BN / 64 sets share a tile and the other
//                sets drain the following tiles from their own accumulator buffers.
//                Per 16-column chunk: tcgen05.ld (the next chunk is in flight while
//                the current one is processed), add the terms, requantize (one 64-bit
//                multiply-add per value), pack; two chunks are staged in shared memory
//                (32 rows x 32 bytes, 32-byte swizzle) and written by one TMA store,
//                which also clips the ragged edges of M and N.  Outputs TMA cannot
//                address (int32, unaligned rows) take plain stores.
//   K <= 64      K-major operands use 64- or 32-byte rows (64B / 32B swizzle) so that
//                the TMA boxes of the first pointwise convolutions carry no padding.
// Every wait is bounded; on a timeout the kernel records a status word, lets
// outstanding copies land, frees its TMEM and returns.
#include "gemm_u8_tc.cuh"

using namespace mb_tc;

int mb_tc_dispatch_plain(mb_context *ctx, const TcChoice &c, const CUtensorMap &ta, const CUtensorMap &tb,
                         const CUtensorMap &tc, TcParams &p);
int mb_tc_dispatch_conv_plain(mb_context *ctx, int bn, int kb, const CUtensorMap &ta, const CUtensorMap &tb,
                              const CUtensorMap &tc, ConvTcParams &p);

// 3-D uint8 tensor map: dims {inner, rows, batch}; 128-byte swizzle for the operand
// tiles, 32-byte swizzle for the output staging boxes; row_pitch 0: no gaps.
int mb_make_map_u8(mb_context *ctx, CUtensorMap *map, const void *base, uint64_t inner,
                uint64_t rows, uint64_t batch, uint64_t batch_stride_bytes, uint32_t box_inner,
                uint32_t box_rows, CUtensorMapSwizzle swizzle,
                uint64_t row_pitch) {
  const cuuint64_t dims[3] = {inner, rows, batch};
  const cuuint64_t strides[2] = {row_pitch != 0 ? row_pitch : inner, batch_stride_bytes};
  const cuuint32_t box[3] = {box_inner, box_rows, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = reinterpret_cast<EncodeTiledFn>(ctx->encode_tiled)(
      map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void *>(base), dims, strides, box, estr,
      CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return mb_fail(ctx, MB_RUNTIME_ERROR, "cuTensorMapEncodeTiled failed (%d)", static_cast<int>(r));
  return MB_SUCCESS;
}

namespace {

// The CTA-pair kernel: clusters of two, as many as there are SM pairs (or tiles).
template <bool A_MN, bool B_MN>
int launch_pair(mb_context *ctx, const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &tc, TcParams &p) {
  using Cfg = TileCfg<256, B_MN, BK, false, true>;
  auto kern = gemm_u8_tc_kernel<256, A_MN, B_MN, false, BK, false, true, false, false>;
  constexpr int cfg_id = 56 + (A_MN ? 2 : 0) + (B_MN ? 1 : 0);
  if (!(ctx->func_attr_mask & (1ull << cfg_id))) {
    MB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
    ctx->func_attr_mask |= (1ull << cfg_id);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(NUM_THREADS);
  // The tiles are dealt out to the clusters once, so every cluster of the launch has to be
  // resident at the same time: ask how many fit (the SMs of a pair share a TPC, and not every
  // TPC of every GPC need be available), once per context.
  if (ctx->max_pair_clusters == 0) {
    cudaLaunchConfig_t probe = {};
    probe.gridDim = dim3(2 * (ctx->num_sms / 2));
    probe.blockDim = dim3(NUM_THREADS);
    probe.dynamicSmemBytes = Cfg::SMEM_BYTES;
    cudaLaunchAttribute pa[1];
    pa[0].id = cudaLaunchAttributeClusterDimension;
    pa[0].val.clusterDim.x = 2;
    pa[0].val.clusterDim.y = 1;
    pa[0].val.clusterDim.z = 1;
    probe.attrs = pa;
    probe.numAttrs = 1;
    int n = 0;
    MB_CUDA(ctx, cudaOccupancyMaxActiveClusters(&n, kern, &probe));
    if (n < 1) return mb_fail(ctx, MB_RUNTIME_ERROR, "no CTA pair of the GEMM kernel fits the device");
    ctx->max_pair_clusters = n;
  }
  const int64_t pairs = std::min<int64_t>(ctx->num_sms / 2, ctx->max_pair_clusters);
  const int clusters = static_cast<int>(p.total_tiles < pairs ? p.total_tiles : pairs);
  p.step_m = clusters % p.tiles_m;
  p.step_n = (clusters / p.tiles_m) % p.tiles_n;
  p.step_b = (clusters / p.tiles_m) / p.tiles_n;
  ctx->pdl_next_gemm = 0;
  cfg.gridDim = dim3(2 * clusters);
  cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctx->pdl_chain ? 2 : 1;
  MB_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, ta, tb, tc, p));
  MB_CUDA(ctx, cudaGetLastError());
  ctx->launches++;
  ctx->launches_tc++;
  ctx->launches_pair++;
  return MB_SUCCESS;
}

}  // namespace

// Whether the tensor-core path can take this problem: TMA needs 16-byte
// aligned bases and row pitches (lda, ldb), and raw byte products must not wrap int32.
bool mb_gemm_u8_tc_supported(const mb_context *ctx, const void *A, const void *B, int64_t M, int64_t N, int64_t K,
                             int64_t lda, int64_t ldb) {
  if (ctx->encode_tiled == nullptr) return false;
  if (M < 1 || N < 1 || K < 1) return false;
  if (K > 33000) return false;  // 255*255*K must stay below 2^31
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15u) return false;
  if ((lda % 16) || (ldb % 16)) return false;  // (matrices of a batch are whole rows apart)
  if (M > (1ll << 31) || N > (1ll << 31)) return false;
  return true;
}

// Launch the tensor-core GEMM.  A is [M x K] K-major (a_mn = false) or
// [K x M] MN-major; B^T is [N x K] K-major (b_mn = false) or B is [K x N]
// MN-major.  C is row-major M x N.  sum_a / sum_b are the per-row byte sums of
// the operands (may be null when the other zero point is 0).
static int tc_launch_impl(mb_context *ctx, const uint8_t *A, const uint8_t *B,
                          const uint32_t *sum_a, const uint32_t *sum_b, int sum_a_slices, int sum_b_slices,
                          const int32_t *bias,
                          void *C, int out_is_int32, int64_t batch, int64_t M, int64_t N,
                          int64_t K, bool a_mn, bool b_mn, int a_batched, int b_batched,
                          int32_t zp_a, int32_t zp_b, int32_t mult, int32_t shift, int32_t zp_c,
                          int bias_per_row, int float_rule, float mult_f, int add_zp, int k_split = 1,
                          int bn_forced = 0, int64_t lda = 0, int64_t ldb = 0) {
  // lda, ldb: bytes from row to row of the stored operands (0: no gap between rows).
  // k_split > 1: one product whose depth is cut into k_split equal runs, computed as a batch of
  // k_split products (int32 results [k_split][M][N], each with its own zero-point terms, which
  // are linear in the depth); the caller adds them up.
  if (lda == 0) lda = a_mn ? M : K;
  if (ldb == 0) ldb = b_mn ? N : K;
  if (k_split > 1) {
    K /= k_split;
    batch = k_split;
    a_batched = b_batched = 1;
  }
  // Operand sums computed inside the kernel: K-major operands, short K, and the
  // caller passed no precomputed sums although a zero point needs them.
  // Rows of 64 or 32 bytes for K-major operands with K <= 64 (the first pointwise
  // convolutions of a network): the TMA boxes then hold no out-of-range bytes.  These
  // shapes always take the fused kernel (it also serves zero points of 0).
  const bool kmajor_free = !a_mn && !b_mn && sum_a == nullptr && sum_b == nullptr;
  const int KBsel = (kmajor_free && K <= 32) ? 32 : (kmajor_free && K <= 64) ? 64 : BK;
  const bool fuse = kmajor_free && K <= 8 * BK && (zp_a != 0 || zp_b != 0 || KBsel != BK);
  // a K-major A against a row-major B with a depth (or depth run) of at most 1024: B's column
  // sums are taken from the tiles too, word by word (depth runs are bound by the bytes each SM
  // can pull and short-depth products by their epilogue: the tile readers have the time)
  const bool fuse_bmn = !a_mn && b_mn && sum_a == nullptr && sum_b == nullptr && K <= 8 * BK &&
                        (zp_a != 0 || zp_b != 0);
  // Tile width.  Long main loops (K > 1024) want the widest tile for operand
  // reuse -- unless that leaves most SMs without a tile (a few rows against a
  // large B): then the width with the fewest columns per SM wins, wider on a
  // tie, so that B streams through as many SMs as possible.  Short main loops
  // are bound by the epilogue, whose cost grows with the width, plus a fixed
  // cost per tile: pick the width with the fewest rounds of (width + overhead)
  // over the SMs.
  int BN = 64;
  {
    const int64_t tm = ceil_div64(M, BM);
    const int widths[3] = {256, 128, 64};
    int64_t best = -1;
    bool widest_seen = false, spread = false;
    for (int w : widths) {
      if (w > 64 && N <= w / 2) continue;  // more than half of the tile would be padding
      const int64_t tiles = batch * tm * ceil_div64(N, w);
      const int64_t rounds = ceil_div64(tiles, ctx->num_sms);
      if (K > 1024) {
        if (!widest_seen) {
          widest_seen = true;
          BN = w;
          if (tiles >= ctx->num_sms) break;  // every SM has work at the widest width
          spread = true;
          best = rounds * w;
          continue;
        }
        if (spread && rounds * w < best) {
          best = rounds * w;
          BN = w;
        }
        continue;
      }
      const int64_t cost = rounds * (w + 96);
      if (best < 0 || cost < best) {
        best = cost;
        BN = w;
      }
    }
    if (ctx->force_bn != 0 && !(ctx->force_bn > 64 && N <= ctx->force_bn / 2)) BN = ctx->force_bn;
    if (bn_forced != 0) BN = bn_forced;
  }
  TcParams p;
  p.M = M; p.N = N; p.K = K; p.batch = batch;
  p.tiles_m = static_cast<int>(ceil_div64(M, BM));
  p.tiles_n = static_cast<int>(ceil_div64(N, BN));
  p.k_blocks = static_cast<int>(ceil_div64(K, KBsel));
  p.total_tiles = batch * p.tiles_m * p.tiles_n;
  p.sum_a = sum_a; p.sum_b = sum_b;
  p.sum_a_slices = sum_a_slices; p.sum_b_slices = sum_b_slices;
  p.sum_a_bstride = M * sum_a_slices; p.sum_b_bstride = N * sum_b_slices;
  p.a_batched = a_batched; p.b_batched = b_batched;
  p.bias = bias; p.bias_per_row = bias_per_row;
  p.zp_a = zp_a; p.zp_b = zp_b;
  p.rq = mb_make_requant(mult, shift, zp_c);
  p.rq_variant = float_rule ? 8 : mb_requant_variant(shift, zp_c);
  p.mult_f = mult_f;
  p.zp_f = add_zp ? static_cast<float>(zp_c) : 0.f;
  p.kzz = static_cast<int32_t>(static_cast<uint32_t>(K) * static_cast<uint32_t>(zp_a) *
                               static_cast<uint32_t>(zp_b));
  p.C = C; p.out_is_int32 = out_is_int32;
  const uintptr_t cbase = reinterpret_cast<uintptr_t>(C);
  p.c_tma = (!out_is_int32 && cbase % 16 == 0 && N % 16 == 0 && N >= 64 && M >= 32) ? 1 : 0;
  p.status = ctx->dev_status;
  p.timeline = ctx->tc_timeline;
  p.b_const = (ctx->gemm_b_const && ctx->b_prefetch) ? 1 : 0;
  p.sums_pending = (ctx->pdl_next_gemm && ctx->pdl_chain && (sum_a != nullptr || sum_b != nullptr)) ? 1 : 0;
  // At least one round of 256 x 256 tiles over the SM pairs: two CTAs per tile, each loading
  // half of it (the lone-CTA kernel is bound by the bytes its 128 x 256 tiles pull from L2).
  // (option value 2 takes the pair kernel wherever it can run, for tests on small shapes)
  const bool pair = ctx->pair_gemm && !fuse && !fuse_bmn && k_split == 1 && p.c_tma && ctx->num_sms >= 2 &&
                    (ctx->pair_gemm == 2 ||
                     (BN == 256 && K >= 512 && batch * ceil_div64(M, 256) * ceil_div64(N, 256) >= ctx->num_sms / 2));
  if (pair) {
    BN = 256;
    p.tiles_n = static_cast<int>(ceil_div64(N, 256));
    p.tiles_m = static_cast<int>(ceil_div64(M, 256));
    p.total_tiles = batch * p.tiles_m * p.tiles_n;
  }

  CUtensorMap ta, tb, tc;
  if (p.c_tma) {
    // the staged box is 32 bytes wide for 256-wide tiles, else 64 (TileCfg::STG_CHUNKS)
    if (BN == 256) {
      MB_RETURN_IF_ERROR(mb_make_map_u8(ctx, &tc, C, N, M, batch, M * N, 32, 32, CU_TENSOR_MAP_SWIZZLE_32B, 0));
    } else {
      MB_RETURN_IF_ERROR(mb_make_map_u8(ctx, &tc, C, N, M, batch, M * N, 64, 32, CU_TENSOR_MAP_SWIZZLE_64B, 0));
    }
  } else {
    memset(&tc, 0, sizeof(tc));
  }
  const uint64_t nb_a = a_batched ? batch : 1, nb_b = b_batched ? batch : 1;
  const CUtensorMapSwizzle kswz = KBsel == 32   ? CU_TENSOR_MAP_SWIZZLE_32B
                                  : KBsel == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                                                : CU_TENSOR_MAP_SWIZZLE_128B;
  // (a run of the depth: K-major rows keep the pitch of the whole matrix and the runs lie side by
  // side; MN-major runs are whole row blocks, one behind the other)
  if (a_mn) {
    MB_RETURN_IF_ERROR(mb_make_map_u8(ctx, &ta, A, M, K, nb_a, K * lda, 128, BK, CU_TENSOR_MAP_SWIZZLE_128B, lda));
  } else {
    MB_RETURN_IF_ERROR(mb_make_map_u8(ctx, &ta, A, K, M, nb_a, k_split > 1 ? K : M * lda, KBsel, BM, kswz, lda));
  }
  if (b_mn) {
    MB_RETURN_IF_ERROR(mb_make_map_u8(ctx, &tb, B, N, K, nb_b, K * ldb, BN < 128 ? 64 : 128, BK,
                                      BN < 128 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, ldb));
  } else {
    MB_RETURN_IF_ERROR(mb_make_map_u8(ctx, &tb, B, K, N, nb_b, k_split > 1 ? K : N * ldb, KBsel, pair ? 128 : BN, kswz, ldb));
  }
  if (pair) {
    if (a_mn) {
      if (b_mn) return launch_pair<true, true>(ctx, ta, tb, tc, p);
      return launch_pair<true, false>(ctx, ta, tb, tc, p);
    }
    if (b_mn) return launch_pair<false, true>(ctx, ta, tb, tc, p);
    return launch_pair<false, false>(ctx, ta, tb, tc, p);
  }

  const TcChoice choice{BN, KBsel, a_mn, b_mn, fuse, fuse_bmn};
  return p.c_tma ? dispatch<false>(ctx, choice, ta, tb, tc, p) : mb_tc_dispatch_plain(ctx, choice, ta, tb, tc, p);
}

int mb_gemm_u8_tc_launch(mb_context *ctx, const uint8_t *A, const uint8_t *B,
                         const uint32_t *sum_a, const uint32_t *sum_b, const int32_t *bias,
                         void *C, int out_is_int32, int64_t batch, int64_t M, int64_t N,
                         int64_t K, bool a_mn, bool b_mn, int a_batched, int b_batched,
                         int32_t zp_a, int32_t zp_b, int32_t mult, int32_t shift, int32_t zp_c,
                         int bias_per_row) {
  return tc_launch_impl(ctx, A, B, sum_a, sum_b, 1, 1, bias, C, out_is_int32, batch, M, N, K, a_mn, b_mn,
                        a_batched, b_batched, zp_a, zp_b, mult, shift, zp_c, bias_per_row, 0, 0.f, 0);
}

// The same with each operand's sums given as `slices` partial rows ([batch or 1][slices][extent]),
// as mb_operand_sums_launch writes the column sums of an MN-major operand.
int mb_gemm_u8_tc_launch_sliced(mb_context *ctx, const uint8_t *A, const uint8_t *B,
                                const uint32_t *sum_a, const uint32_t *sum_b, int sum_a_slices, int sum_b_slices,
                                const int32_t *bias, void *C, int out_is_int32, int64_t batch, int64_t M, int64_t N,
                                int64_t K, int64_t lda, int64_t ldb, bool a_mn, bool b_mn, int a_batched, int b_batched,
                                int32_t zp_a, int32_t zp_b, int32_t mult, int32_t shift, int32_t zp_c,
                                int bias_per_row) {
  return tc_launch_impl(ctx, A, B, sum_a, sum_b, sum_a_slices, sum_b_slices, bias, C, out_is_int32, batch, M, N, K,
                        a_mn, b_mn, a_batched, b_batched, zp_a, zp_b, mult, shift, zp_c, bias_per_row, 0, 0.f, 0, 1, 0,
                        lda, ldb);
}

// One product with its depth cut into k_split equal runs (K % (k_split * 128) == 0): `parts`
// receives the k_split int32 results [k_split][M][N], each the exact sum over its run of
// (A - zp_a)(B - zp_b); the sums are per run ([k_split][...], see mb_operand_sums_launch).
int mb_gemm_u8_tc_launch_splitk(mb_context *ctx, const uint8_t *A, const uint8_t *B,
                                const uint32_t *sum_a, const uint32_t *sum_b, int sum_a_slices, int sum_b_slices,
                                int32_t *parts, int k_split, int bn, int64_t M, int64_t N, int64_t K, bool a_mn,
                                bool b_mn, int32_t zp_a, int32_t zp_b) {
  return tc_launch_impl(ctx, A, B, sum_a, sum_b, sum_a_slices, sum_b_slices, nullptr, parts, 1, 1, M, N, K, a_mn,
                        b_mn, 0, 0, zp_a, zp_b, 1 << 30, 0, 0, 0, 0, 0.f, 0, k_split, bn);
}

// The same product with the Gemv delegators' float requantization rule (see
// requant_float_rule): K-major operands, operand sums taken inside the kernel.
int mb_gemm_u8_tc_launch_float_rule(mb_context *ctx, const uint8_t *A, const uint8_t *B,
                                    const int32_t *bias, void *C, int out_is_int32, int64_t M,
                                    int64_t N, int64_t K, int32_t zp_a, int32_t zp_b, float mult_f,
                                    int32_t zp_c, int add_zp) {
  return tc_launch_impl(ctx, A, B, nullptr, nullptr, 1, 1, bias, C, out_is_int32, 1, M, N, K, false, false, 0,
                        0, zp_a, zp_b, 1 << 30, 0, zp_c, 0, 1, mult_f, add_zp);
}

// A convolution (g.conv) with tiles of 128 pixels x bn channels, depth rows of kbt bytes; map_a in im2col mode, map_b
// the filter as [taps][O][C].
int mb_gemm_u8_tc_launch_conv(mb_context *ctx, const mb_cut_gemm &g, const CUtensorMap &map_a, const CUtensorMap &map_b,
                              int bn, int kbt, int c_blocks, int patch) {
  ConvTcParams p = {};
  p.M = g.M; p.N = g.N; p.K = g.K; p.batch = 1;
  p.tiles_m = static_cast<int>(ceil_div64(g.M, BM));
  p.tiles_n = static_cast<int>(ceil_div64(g.N, bn));
  p.k_blocks = g.KH * g.KW * c_blocks;
  p.total_tiles = static_cast<int64_t>(p.tiles_m) * p.tiles_n;
  p.bias = g.bias;
  p.zp_a = g.zp_a; p.zp_b = g.zp_b;
  p.rq = g.rq; p.rq_variant = g.rq_variant;
  p.kzz = static_cast<int32_t>(static_cast<uint32_t>(g.K) * static_cast<uint32_t>(g.zp_a) * static_cast<uint32_t>(g.zp_b));
  p.C = g.C;
  p.c_tma = (reinterpret_cast<uintptr_t>(g.C) % 16 == 0 && g.N % 16 == 0 && g.N >= 64 && g.M >= 32) ? 1 : 0;
  p.patch = patch;
  p.H = g.H; p.W = g.W; p.Cin = g.C_in; p.KW = g.KW; p.sh = g.sh; p.sw = g.sw; p.pad_t = g.pad_t; p.pad_l = g.pad_l;
  p.Ho = g.Ho; p.Wo = g.Wo; p.c_blocks = c_blocks;
  fast_div_make(static_cast<uint32_t>(g.Wo), &p.wo_mul, &p.wo_shift);
  fast_div_make(static_cast<uint32_t>(g.Ho), &p.ho_mul, &p.ho_shift);
  p.status = ctx->dev_status;
  CUtensorMap tc;
  memset(&tc, 0, sizeof(tc));
  if (p.c_tma) MB_RETURN_IF_ERROR(mb_make_map_u8(ctx, &tc, g.C, g.N, g.M, 1, g.M * g.N, 64, 32, CU_TENSOR_MAP_SWIZZLE_64B, 0));
  return p.c_tma ? dispatch_conv<false>(ctx, bn, kbt, map_a, map_b, tc, p)
                 : mb_tc_dispatch_conv_plain(ctx, bn, kbt, map_a, map_b, tc, p);
}
