// The persistent tensor-core uint8 GEMM kernel and the choice of its instances, compiled twice: gemm_u8_tc.cu (results
// through TMA stores) and gemm_u8_tc_plain.cu (plain stores), which halves the build's longest file.
#pragma once

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "gemm_u8_cut.cuh"
#include "sm100_ptx.cuh"

namespace mb_tc {

using namespace sm100;

constexpr int BM = 128;        // rows of A per tile == TMEM lanes
constexpr int BK = 128;        // bytes of K per pipeline stage (one swizzle row); K-major
                               // operands with K <= 64 use rows of 64 or 32 bytes (template KB)
constexpr int UMMA_K = 32;     // K per tcgen05.mma for 8-bit operands
constexpr int PREP_WARPS = 4;
constexpr int EPI_WARPS = 16;
constexpr int FIRST_EPI_WARP = 2 + PREP_WARPS;
constexpr int NUM_THREADS = (2 + PREP_WARPS + EPI_WARPS) * 32;
constexpr int CHUNK = 16;      // accumulator columns per tcgen05.ld
constexpr long long WAIT_BUDGET = 1ll << 31;  // ~1 s of SM clocks per wait
constexpr uint32_t SWIZZLE_128B = 2;

struct TcParams {
  int64_t M, N, K, batch;
  int tiles_m, tiles_n, k_blocks;
  int64_t total_tiles;

  // gridDim.x as (step_b, step_n, step_m) in tile coordinates: advancing a CTA to its next
  // tile is three additions and two carries instead of 64-bit divisions
  int step_m, step_n, step_b;
  // Operand byte sums, each as `slices` partial rows that are added up here:
  const uint32_t *sum_a;  // [batch or 1][sum_a_slices][M]; null when fused or zp_b == 0
  const uint32_t *sum_b;  // [batch or 1][sum_b_slices][N]; null when fused or zp_a == 0
  int64_t sum_a_bstride, sum_b_bstride;
  int sum_a_slices, sum_b_slices;
  int a_batched, b_batched;
  const int32_t *bias;
  int bias_per_row;
  int32_t zp_a, zp_b, kzz;
  mb_requant_params rq;
  int rq_variant;  // mb_requant_variant() (0..5), or 8 = the Gemv delegators' float rule
                   // (mult_f, zp_f)
  float mult_f, zp_f;
  void *C;
  int out_is_int32;
  int c_tma;  // uint8 C written by TMA stores (base and rows 16-byte aligned)
  // The kernel in front of this one in the stream only computes sum_a / sum_b (the operands
  // themselves were complete before it started): the main loop starts without waiting for it,
  // only the preparation warps wait, where they read the sums.
  int sums_pending;
  int b_const;  // B is a weight: its first tiles may be asked into L2 before the wait for the kernel in front
  int *status;
  // null, or clock stamps written by CTA 0 (profiling aid): 32 milestone slots, then 5
  // slots for each of its first 16 tiles (TMA issued, tile landed, MMAs committed,
  // epilogue begins, epilogue ends); the buffer holds 128 values
  long long *timeline;
};

// CONV: A is the NHWC input of a convolution, fetched by TMA in im2col mode (a step is one channel run of
// one filter tap); `patch`: windows reach outside the image and its zero point is not 0.
struct ConvTcParams : TcParams {
  int patch, H, W, Cin, KW, sh, sw, pad_t, pad_l, Ho, Wo, c_blocks;
  uint32_t wo_mul, wo_shift, ho_mul, ho_shift;
};

// Clock stamp of a pipeline milestone, CTA 0 only, when a buffer was given.  Compiled in
// only with -DMB_TC_TIMELINE: the checks sit on the single-thread roles' critical path.
#ifdef MB_TC_TIMELINE
#define MB_STAMP(slot)                                                    \
  do {                                                                    \
    if (p.timeline != nullptr && blockIdx.x == 0) p.timeline[slot] = clock64(); \
  } while (0)
#else
#define MB_STAMP(slot) do { } while (0)
#endif

// Per-tile stamp k (0..4) of CTA 0's n-th tile, first 16 tiles only.
#ifndef MB_TC_TIMELINE
#define MB_STAMP_TILE(tile, k) do { (void)(tile); } while (0)
#else
#define MB_STAMP_TILE(tile, k)                                                       \
  do {                                                                              \
    if (p.timeline != nullptr && blockIdx.x == 0 && (tile) < 16)                    \
      p.timeline[32 + (tile) * 5 + (k)] = clock64();                                \
  } while (0)
#endif

// TCR ("row sums on the tensor core"): the B tile of every stage is followed by 16 constant rows
// of ones, and the MMA runs with N = BN + 16: accumulator columns BN .. BN + 15 of row m then
// hold the byte sum of A's row m, which the zero-point correction needs, at the price of an
// eighth (BN = 128) or a quarter (BN = 64) more work for a tensor pipe that short-K tiles leave
// idle anyway -- instead of a pass of the preparation warps over every A tile in shared memory,
// which cost these issue-bound kernels a fifth of their instructions.
// PAIR: two CTAs of a cluster work on one 256 x 256 tile: each holds 128 rows of A and 128 of
// the 256 columns of B in its shared memory (two thirds of the operand bytes per row of C that
// a lone CTA pulls for 128 x 256), and its own 128 rows of the accumulator in its tensor memory.
template <int BN, bool B_MN, int KB = BK, bool TCR = false, bool PAIR = false>
struct TileCfg {
  static_assert(!PAIR || (BN == 256 && KB == 128 && !TCR), "pairs: 256 columns, 128-byte rows");
  static_assert(KB == 128 || !B_MN, "short rows are for K-major operands");
  static_assert(!TCR || (!B_MN && BN <= 128), "ones rows follow a K-major B tile of at most 128 rows");
  // a row-major B comes in panels of 128 columns (64 for tiles of 64, whose other half nobody would read)
  static constexpr int PANEL = BN < 128 ? 64 : 128;
  static constexpr int BNX = TCR ? BN + 16 : BN;  // MMA N and TMEM columns per accumulator
  static constexpr int A_BYTES = BM * KB;
  static constexpr int B_TMA_BYTES = PAIR ? 128 * KB : BN * KB;  // what TMA brings
  static constexpr int B_BYTES = B_TMA_BYTES + (TCR ? 16 * KB : 0);
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGE_TX = A_BYTES + B_TMA_BYTES;
  // epilogue staging for the TMA stores: 1 KB (32 rows x 32 bytes) per epilogue warp
  // ... 2 KB (32 rows x 64 bytes: one store per warp and tile) where the ring leaves room
  static constexpr int STG_CHUNKS = BN == 256 ? 2 : 4;   // 16-byte chunks per staged row
  static constexpr int STAGING_BYTES = EPI_WARPS * 32 * STG_CHUNKS * 16;
  static constexpr int RING_BUDGET = 208 * 1024 - STAGING_BYTES;
  static constexpr int STAGES = RING_BUDGET / STAGE_BYTES > 8 ? 8 : RING_BUDGET / STAGE_BYTES;
  // all 512 TMEM columns as accumulator buffers: 2 for BN = 256, 4 for 128, 8 for 64, so
  // that narrow tiles (short main loops) keep several tiles in flight
  static constexpr int NUM_ACC = 512 / BNX;
  static constexpr int TMEM_COLS = 512;
  static constexpr int BAR_BYTES = 512;
  // + for a row-major B: the preparation warps' partial column sums, [tile parity][k quarter][columns]
  static constexpr int PART_INTS = B_MN ? 4 * ((BN + 127) / 128) * 128 : 0;
  static constexpr int TERM_BYTES = NUM_ACC * (128 + BN) * 4 + 2 * PART_INTS * 4;
  static constexpr int SMEM_BYTES =
      STAGES * STAGE_BYTES + STAGING_BYTES + 1024 /*align*/ + BAR_BYTES + TERM_BYTES;
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
};

// Adds up the `slices` partial rows of an operand sum for one row / column: eight loads in
// flight at a time (one after the other they would cost an L2 round trip each, and the terms
// of a tile have to be ready within the tile's main loop).
__device__ __forceinline__ uint32_t sum_partials(const uint32_t *p, int slices, int64_t stride) {
  uint32_t a0 = 0, a1 = 0, a2 = 0, a3 = 0, a4 = 0, a5 = 0, a6 = 0, a7 = 0;
  int sl = 0;
  for (; sl + 8 <= slices; sl += 8) {
    const uint32_t *q = p + sl * stride;
    const uint32_t v0 = mb_load(q), v1 = mb_load(q + stride), v2 = mb_load(q + 2 * stride), v3 = mb_load(q + 3 * stride);
    const uint32_t v4 = mb_load(q + 4 * stride), v5 = mb_load(q + 5 * stride), v6 = mb_load(q + 6 * stride),
                   v7 = mb_load(q + 7 * stride);
    a0 += v0; a1 += v1; a2 += v2; a3 += v3; a4 += v4; a5 += v5; a6 += v6; a7 += v7;
  }
  for (; sl < slices; ++sl) a0 += mb_load(p + sl * stride);
  return ((a0 + a1) + (a2 + a3)) + ((a4 + a5) + (a6 + a7));
}

// Tile coordinates of a persistent CTA: tile index = (b * tiles_n + tn) * tiles_m + tm,
// advanced by gridDim.x per step.
struct TileIter {
  int tm, tn, b;
  __device__ __forceinline__ TileIter(const TcParams &p, bool pair = false) {
    const unsigned t = pair ? blockIdx.x >> 1 : blockIdx.x;  // < tiles of the first wave, one division pair per kernel
    tm = t % p.tiles_m;
    const unsigned q = t / p.tiles_m;
    tn = q % p.tiles_n;
    b = q / p.tiles_n;
  }
  __device__ __forceinline__ bool valid(const TcParams &p) const { return b < p.batch; }
  __device__ __forceinline__ void next(const TcParams &p) {
    tm += p.step_m;
    tn += p.step_n;
    b += p.step_b;
    if (tm >= p.tiles_m) { tm -= p.tiles_m; ++tn; }
    if (tn >= p.tiles_n) { tn -= p.tiles_n; ++b; }
  }
};

// Requantizes one 16-column chunk of an accumulator row and packs it into four words.
// MODE: 0..3 = mb_requant_t<ZP0 = bit 0, SGE1 = bit 1>; 4 / 5 = packed saturating form
// (zero point != 0 / == 0); 8 = the Gemv delegators' float rule.
template <int MODE>
__device__ __forceinline__ void requant_chunk(const uint32_t (&raw)[CHUNK], int32_t row_term,
                                              const int4 *ct, const TcParams &p,
                                              uint32_t (&packed)[CHUNK / 4]);

// The float rule of the Gemv delegators (mace/ops/arm/q8/gemv.cc:151-164):
// Saturate<uint8_t>(roundf(acc * multiplier [+ zp_out])), product and sum rounded separately
// (zp_f is 0 for the REF delegator's formula, which omits the zero point).
__device__ __forceinline__ uint32_t requant_float_rule(int32_t acc, float mult_f, float zp_f) {
  const float v = __fadd_rn(__fmul_rn(static_cast<float>(acc), mult_f), zp_f);
  return mb_saturate_round_u8(v);
}

template <int MODE>
__device__ __forceinline__ void requant_chunk(const uint32_t (&raw)[CHUNK], int32_t row_term,
                                              const int4 *ct, const TcParams &p,
                                              uint32_t (&packed)[CHUNK / 4]) {
#pragma unroll
  for (int q = 0; q < CHUNK / 4; ++q) {
    const int4 t = ct[q];  // broadcast read: all lanes, same address
    const int32_t a0 = static_cast<int32_t>(raw[4 * q + 0]) + row_term + t.x;
    const int32_t a1 = static_cast<int32_t>(raw[4 * q + 1]) + row_term + t.y;
    const int32_t a2 = static_cast<int32_t>(raw[4 * q + 2]) + row_term + t.z;
    const int32_t a3 = static_cast<int32_t>(raw[4 * q + 3]) + row_term + t.w;
    if (MODE == 4 || MODE == 5) {
      packed[q] = mb_requant_pack4<MODE == 5>(a0, a1, a2, a3, p.rq);
    } else {
      uint32_t b0, b1, b2, b3;
      if (MODE == 8) {
        b0 = requant_float_rule(a0, p.mult_f, p.zp_f); b1 = requant_float_rule(a1, p.mult_f, p.zp_f);
        b2 = requant_float_rule(a2, p.mult_f, p.zp_f); b3 = requant_float_rule(a3, p.mult_f, p.zp_f);
      } else {
        b0 = mb_requant_t<(MODE & 1) != 0, (MODE & 2) != 0>(a0, p.rq);
        b1 = mb_requant_t<(MODE & 1) != 0, (MODE & 2) != 0>(a1, p.rq);
        b2 = mb_requant_t<(MODE & 1) != 0, (MODE & 2) != 0>(a2, p.rq);
        b3 = mb_requant_t<(MODE & 1) != 0, (MODE & 2) != 0>(a3, p.rq);
      }
      packed[q] = __byte_perm(__byte_perm(b0, b1, 0x0040), __byte_perm(b2, b3, 0x0040), 0x5410);
    }
  }
}

// What an epilogue warp needs for one tile on the TMA-store path.
struct EpiTile {
  uint32_t tbase;          // TMEM address of the warp's 32 lanes x 64 columns
  int32_t row_term;
  const int32_t *ct_base;  // column terms of the 64 columns (shared memory)
  uint32_t tempty;         // barrier that returns the accumulator buffer
  uint32_t tempty_leader;  // pairs, odd CTA: the even CTA's barrier too (shared::cluster address)
  uint4 *stage_row;        // this lane's row of the staging buffer (STG chunks of 16 bytes)
  int swz;
  uint32_t stage_addr;
  int64_t n_first;
  int m0, b, lane;
};

// 32 rows x 64 columns of one tile: four 16-column chunks from TMEM (the next one in flight
// while the current one is requantized), staged STG chunks at a time for a TMA store of
// 32 rows x 16*STG bytes.
template <int STG, int MODE, bool PAIR = false>
__device__ __forceinline__ void epi_tma_tile(const EpiTile &e, const CUtensorMap &tmap_c,
                                             const TcParams &p) {
  uint32_t r[2][CHUNK];
  tmem_ld_32x32b_x16(e.tbase, r[0]);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    tmem_ld_wait_x16(r[i & 1]);
    if (i + 1 < 4) tmem_ld_32x32b_x16(e.tbase + (i + 1) * CHUNK, r[(i + 1) & 1]);
    uint32_t packed[CHUNK / 4];
    requant_chunk<MODE>(r[i & 1], e.row_term, reinterpret_cast<const int4 *>(e.ct_base + i * CHUNK), p, packed);
    if (i == 3) {
      // The accumulator is in registers and the tile's terms have been read: hand the buffer
      // (TMEM columns and term slots; the preparation warps refill the latter on the same
      // barrier) back before the staging and the store.
      tc_fence_before_sync();
      __syncwarp();
      if (e.lane == 0) {
        mbar_arrive(e.tempty);
        if (PAIR && e.tempty_leader != 0) mbar_arrive_cluster(e.tempty_leader);
      }
    }
    if ((i & (STG - 1)) == 0) {
      // the previous store must have read the staging buffer before it is refilled
      if (e.lane == 0) bulk_wait_group_read<0>();
      __syncwarp();
    }
    e.stage_row[(i & (STG - 1)) ^ e.swz] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    if ((i & (STG - 1)) == STG - 1) {
      fence_proxy_async();
      __syncwarp();
      const int64_t n0 = e.n_first + (i - (STG - 1)) * CHUNK;
      if (e.lane == 0 && n0 < p.N && e.m0 < p.M) {
        tma_store_3d(&tmap_c, e.stage_addr, static_cast<int>(n0), e.m0, e.b);
        bulk_commit_group();
      }
    }
  }
}

// A uint8 output whose rows TMA cannot address (their pitch is no multiple of 16 bytes, e.g. the 1001
// columns of a product of odd size, or few rows): the same 32 x 64 values staged in shared memory, then
// written along the rows, so that a store instruction fills adjacent bytes of one or two rows and not
// one byte in each of 32.
struct PlainTile {
  uint32_t tbase;
  int32_t row_term;
  const int32_t *ct_base;
  uint8_t *stage;  // 32 rows x 16 * STG bytes
  uint8_t *out;    // first value of the warp's 32 x 64
  int64_t pitch;
  int rows, cols;  // of them inside the matrix (may be <= 0)
  int swz;
};

template <int STG, int MODE>
__device__ __forceinline__ void epi_plain_tile(const PlainTile &e, const TcParams &p) {
  const int lane = threadIdx.x & 31;
  uint4 *stage_row = reinterpret_cast<uint4 *>(e.stage + lane * (STG * 16));
  const bool words_ok = ((e.pitch | static_cast<int64_t>(reinterpret_cast<uintptr_t>(e.out))) & 3) == 0;
#pragma unroll 1
  for (int i = 0; i < 4; i += STG) {
    uint32_t r[2][CHUNK];
    tmem_ld_32x32b_x16(e.tbase + i * CHUNK, r[0]);
    __syncwarp();  // the staging buffer has been read
#pragma unroll
    for (int q = 0; q < STG; ++q) {
      tmem_ld_wait_x16(r[q & 1]);
      if (q + 1 < STG) tmem_ld_32x32b_x16(e.tbase + (i + q + 1) * CHUNK, r[(q + 1) & 1]);
      uint32_t packed[CHUNK / 4];
      requant_chunk<MODE>(r[q & 1], e.row_term, reinterpret_cast<const int4 *>(e.ct_base + (i + q) * CHUNK), p, packed);
      stage_row[q ^ e.swz] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    }
    __syncwarp();
    const int cols = e.cols - i * CHUNK;  // of the 16 * STG columns staged
    uint8_t *out = e.out + i * CHUNK;
    // column c of row r lies in the row's 16-byte chunk (c / 16) ^ (the row's swizzle, see stage_row)
    if (words_ok) {
      // whole words (the row pitch and hence the edge of the matrix are multiples of four)
      constexpr int WPR = STG * 4;
      const int w = lane % WPR;
#pragma unroll 4
      for (int row = lane / WPR; row < 32; row += 32 / WPR) {
        const int swz = STG == 2 ? ((row >> 2) & 1) : ((row >> 1) & 3);
        const uint32_t v = *reinterpret_cast<const uint32_t *>(e.stage + row * (STG * 16) + (((w >> 2) ^ swz) << 4) + (w & 3) * 4);
        if (row < e.rows && w * 4 < cols) *reinterpret_cast<uint32_t *>(out + row * e.pitch + w * 4) = v;
      }
    } else {
#pragma unroll 4
      for (int row = 0; row < 32; ++row) {
        if (row >= e.rows) break;
        const int swz = STG == 2 ? ((row >> 2) & 1) : ((row >> 1) & 3);
#pragma unroll
        for (int h = 0; h < STG / 2; ++h) {
          const int c = h * 32 + lane;
          const uint8_t v = e.stage[row * (STG * 16) + (((c >> 4) ^ swz) << 4) + (c & 15)];
          if (c < cols) out[row * e.pitch + c] = v;
        }
      }
    }
  }
}

// Top-left corner of output pixel `pix`'s window.
__device__ __forceinline__ void conv_corner(const ConvTcParams &p, int pix, int &n, int &h, int &w) {
  const uint32_t r = fast_div(static_cast<uint32_t>(pix), p.wo_mul, p.wo_shift);
  const uint32_t img = fast_div(r, p.ho_mul, p.ho_shift);
  n = static_cast<int>(img);
  h = static_cast<int>(r - img * static_cast<uint32_t>(p.Ho)) * p.sh - p.pad_t;
  w = (pix - static_cast<int>(r) * p.Wo) * p.sw - p.pad_l;
}

// PLAIN: the output does not go through TMA stores (int32, or rows whose pitch is no multiple of 16 bytes).  A template
// parameter, so that neither kind of epilogue costs the other's instances registers or instructions.
template <int BN, bool A_MN, bool B_MN, bool FUSE_SUMS, int KB, bool TCR_ON, bool PAIR, bool CONV, bool PLAIN>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_u8_tc_kernel(const __grid_constant__ CUtensorMap tmap_a,
                  const __grid_constant__ CUtensorMap tmap_b,
                  const __grid_constant__ CUtensorMap tmap_c, const std::conditional_t<CONV, ConvTcParams, TcParams> p) {
  constexpr bool TCR = TCR_ON && FUSE_SUMS && BN <= 128;
  static_assert(!PAIR || !FUSE_SUMS, "pairs take their operand sums from the sums kernel");
  static_assert(!CONV || (TCR && !A_MN && !B_MN), "convolutions take A's sums from the tensor core");
  bool patch = false;
  if constexpr (CONV) patch = p.patch != 0;
  using Cfg = TileCfg<BN, B_MN, KB, TCR, PAIR>;
  constexpr int STAGES = Cfg::STAGES;
  constexpr int TILE_M = PAIR ? 2 * BM : BM;  // rows of C per tile (of the pair)
  // pairs: the even CTA issues the MMAs for both; rank is this CTA's half of the rows and columns
  const uint32_t rank = PAIR ? cluster_ctarank() : 0u;
  constexpr int BNX = Cfg::BNX;
  // the preparation warps read the operand tiles in shared memory only for the sums the tensor
  // core does not deliver: B's (needed when zp_a != 0), and A's without the ones rows
  const bool prep_reads_tiles = patch || (FUSE_SUMS && ((!TCR && p.zp_b != 0) || p.zp_a != 0));
  // shared-memory descriptor fields for rows of KB bytes: swizzle mode and the distance
  // between 8-row groups
  constexpr uint32_t SWZ = KB == 128 ? 2u : KB == 64 ? 4u : 6u;
  constexpr uint32_t SBO = 8 * KB;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t *smem_aligned = smem_raw + (smem_base - smem_u32(smem_raw));
  // barrier block after the tile ring
  uint64_t *bars =
      reinterpret_cast<uint64_t *>(smem_aligned + STAGES * Cfg::STAGE_BYTES + Cfg::STAGING_BYTES);
  const uint32_t full_bar = smem_u32(bars);                  // [STAGES] tile landed
  const uint32_t empty_bar = full_bar + 8 * STAGES;          // [STAGES] tile consumed
  constexpr int NUM_ACC = Cfg::NUM_ACC;
  const uint32_t tfull_bar = empty_bar + 8 * STAGES;         // [NUM_ACC] accumulator complete
  const uint32_t tempty_bar = tfull_bar + 8 * NUM_ACC;       // [NUM_ACC] accumulator drained
  const uint32_t terms_bar = tempty_bar + 8 * NUM_ACC;       // [NUM_ACC] epilogue terms ready
  const uint32_t part_bar = terms_bar + 8 * NUM_ACC;          // the four quarters of a tile's column sums are written
  const uint32_t ready_bar = part_bar + 8;                    // CONV: [STAGES] outside pixels overwritten
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + (CONV ? 3 : 2) * STAGES + 3 * NUM_ACC + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  // per accumulator buffer: row terms [128] and column terms [BN]
  int32_t *row_term_sm =
      reinterpret_cast<int32_t *>(smem_aligned + STAGES * Cfg::STAGE_BYTES + Cfg::STAGING_BYTES +
                                  Cfg::BAR_BYTES);
  int32_t *col_term_sm = row_term_sm + NUM_ACC * 128;
  uint32_t *part_sm = reinterpret_cast<uint32_t *>(col_term_sm + NUM_ACC * BN);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  mb_grid_dep_launch();  // the kernel behind this one may start its own prologue

  if (threadIdx.x == 0) {
    MB_STAMP(0);
    prefetch_tensormap(&tmap_a);
    prefetch_tensormap(&tmap_b);
    if (!PLAIN) prefetch_tensormap(&tmap_c);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar + 8 * s, 1);
      mbar_init(empty_bar + 8 * s, prep_reads_tiles ? 1 + PREP_WARPS : 1);
      if (CONV) mbar_init(ready_bar + 8 * s, PREP_WARPS);
    }
    mbar_init(part_bar, PREP_WARPS);
    for (int b = 0; b < NUM_ACC; ++b) {
      mbar_init(tfull_bar + 8 * b, 1);
      // (pairs: the even CTA's barrier also counts the odd CTA's epilogue warps)
      mbar_init(tempty_bar + 8 * b, (PAIR && rank == 0 ? 2 : 1) * 4 * (BN / 64));
      mbar_init(terms_bar + 8 * b, PREP_WARPS);
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    if (PAIR) {
      tmem_alloc_pair(smem_u32(tmem_slot), Cfg::TMEM_COLS);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(smem_u32(tmem_slot), Cfg::TMEM_COLS);
      tmem_relinquish();
    }
  }
  if (TCR) {
    // the 16 rows of ones behind every stage's B tile (TMA never writes there)
    constexpr int ONES_VECS = 16 * KB / 16;
    for (int i = threadIdx.x; i < STAGES * ONES_VECS; i += NUM_THREADS) {
      const int st = i / ONES_VECS, v = i - st * ONES_VECS;
      *reinterpret_cast<uint4 *>(smem_aligned + st * Cfg::STAGE_BYTES + Cfg::A_BYTES + Cfg::B_TMA_BYTES + v * 16) =
          make_uint4(0x01010101u, 0x01010101u, 0x01010101u, 0x01010101u);
    }
    fence_proxy_async();  // generic-proxy writes, read by the tensor core through the async proxy
  }
  tc_fence_before_sync();
  __syncthreads();
  if (PAIR) cluster_sync_all();  // both CTAs' barriers exist before either arrives on the other's
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  if (threadIdx.x == 0) MB_STAMP(1);
  // Everything above touched only this CTA's shared and tensor memory (and the kernel's
  // parameters); from here on the roles read and write global memory, which the kernel in
  // front of this one in the stream may still be producing.
  // (with sums_pending only the preparation warps, which read the sums, wait; the operands were
  // complete before the sums kernel started, and C is not touched by it)
  if (!PAIR && !CONV && p.b_const && warp == 0 && lane == 0) {
    // a weight matrix is usually not in L2 any more (the activations of a whole network pass have
    // gone through it since): ask for this CTA's first B tiles now, so that they travel from HBM
    // while the kernel in front finishes
    TileIter it(p, PAIR);
    if (it.valid(p)) {
      const int bb = p.b_batched ? it.b : 0;
      const int ahead = p.k_blocks < STAGES ? p.k_blocks : STAGES;
      for (int kb = 0; kb < ahead; ++kb) {
        if (B_MN) {
#pragma unroll
          for (int j = 0; j < (BN + 127) / 128; ++j) tma_prefetch_3d(&tmap_b, it.tn * BN + j * 128, kb * KB, bb);
        } else {
          tma_prefetch_3d(&tmap_b, kb * KB, it.tn * BN, bb);
        }
      }
    }
  }
  if (!p.sums_pending || (warp >= 2 && warp < 2 + PREP_WARPS)) mb_grid_dep_wait();

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    // One thread runs the role (see the MMA issuer); the other lanes wait at the warp barrier.
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      int local = 0;  // this CTA's tile counter (profiling stamps)
      // When every tile of the launch reads the same B tile (one column of tiles, one K step,
      // B shared by the batch: a pointwise convolution with few channels), each stage's copy
      // of B is loaded once, on the first pass through the ring, and then left in place: TMA
      // handles short rows one by one, and the B rows would be a third to a half of them.
      const bool b_once = !CONV && p.tiles_n == 1 && p.k_blocks == 1 && !p.b_batched;
      for (TileIter it(p, PAIR); ok && it.valid(p); it.next(p), ++local) {
        const int b = it.b, tm = it.tm, tn = it.tn;
        const int ab = p.a_batched ? b : 0, bb = p.b_batched ? b : 0;
        int img = 0, h0 = 0, w0 = 0, tap_h = 0, tap_w = 0, tap = 0, cb = 0;
        if constexpr (CONV) conv_corner(p, tm * BM, img, h0, w0);
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (!mbar_wait(empty_bar + 8 * stage, phase ^ 1, abort_flag, WAIT_BUDGET)) {
            *abort_flag = 1;
            atomicCAS(p.status, 0, MB_DEV_TIMEOUT_PRODUCER);
            ok = false;
            break;
          }
          const uint32_t fb = full_bar + 8 * stage;
          const uint32_t sa = smem_base + stage * Cfg::STAGE_BYTES;
          const uint32_t sb = sa + Cfg::A_BYTES;
          const bool skip_b = b_once && local >= STAGES;
          if (PAIR) {
            // Both CTAs' bytes are counted on the even CTA's barrier, which its MMA thread
            // waits on: this CTA's 128 rows of A and 128 of the tile's 256 columns of B.
            if (rank == 0) mbar_arrive_expect_tx(fb, 2 * Cfg::STAGE_TX);
            const uint32_t fbc = mapa_shared(fb, 0);
            if (A_MN) tma_load_3d_pair(sa, &tmap_a, fbc, tm * TILE_M + rank * BM, kb * KB, ab);
            else tma_load_3d_pair(sa, &tmap_a, fbc, kb * KB, tm * TILE_M + rank * BM, ab);
            if (B_MN) tma_load_3d_pair(sb, &tmap_b, fbc, tn * BN + rank * 128, kb * KB, bb);
            else tma_load_3d_pair(sb, &tmap_b, fbc, kb * KB, tn * BN + rank * 128, bb);
          } else {
          mbar_arrive_expect_tx(fb, skip_b ? Cfg::A_BYTES : Cfg::STAGE_TX);
          if constexpr (CONV) {
            tma_load_im2col_4d(sa, &tmap_a, fb, cb * KB, w0, h0, img, static_cast<uint16_t>(tap_w), static_cast<uint16_t>(tap_h));
          } else if (A_MN) {
            tma_load_3d(sa, &tmap_a, fb, tm * BM, kb * KB, ab);
          } else {
            tma_load_3d(sa, &tmap_a, fb, kb * KB, tm * BM, ab);
          }
          if constexpr (CONV) {
            tma_load_3d(sb, &tmap_b, fb, cb * KB, tn * BN, tap);
            if (++cb == p.c_blocks) {
              cb = 0;
              ++tap;
              if (++tap_w == p.KW) {
                tap_w = 0;
                ++tap_h;
              }
            }
          } else if (skip_b) {
            // B of this stage is already in place
          } else if (B_MN) {
#pragma unroll
            for (int j = 0; j < (BN + 127) / 128; ++j)
              tma_load_3d(sb + j * 128 * KB, &tmap_b, fb, tn * BN + j * 128, kb * KB, bb);
          } else {
            tma_load_3d(sb, &tmap_b, fb, kb * KB, tn * BN, bb);
          }
          }
          if (local == 0) MB_STAMP(2 + (kb < 3 ? kb : 3));  // TMA of k-block kb issued
          if (kb == 0) MB_STAMP_TILE(local, 0);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    // One thread runs the whole role; the other lanes go straight to the warp barrier below.
    // What the thread does between two MMAs has to fit into the time the tensor pipe's short
    // queue keeps it busy, and for tiles of one K step it is on the critical path outright:
    // the descriptors are one add per step and nothing in the loop is warp-collective.
    if (PAIR && rank != 0) {
      // the odd CTA issues no MMAs: the even CTA's thread drives both tensor cores
    } else if (lane == 0) {
      constexpr uint32_t idesc = make_idesc(/*c s32*/ 2, /*a u8*/ 0, /*b u8*/ 0, A_MN, B_MN, TILE_M, BNX);
      // K-major tile: rows of KB bytes, 8-row groups SBO bytes apart; a K step moves 32 bytes
      // inside the swizzled row.  MN-major tile: k-rows of 128 bytes (128 elements of M or N),
      // 8-k-row groups 1024 bytes apart, 128-element atoms 128 * KB bytes apart; a K step moves
      // 32 k-rows = 4096 bytes.  The address field counts 16-byte units.
      const uint64_t a_base = A_MN ? make_smem_desc(0, 128 * KB, 1024, SWIZZLE_128B) : make_smem_desc(0, 16, SBO, SWZ);
      const uint64_t b_base = B_MN ? make_smem_desc(0, Cfg::PANEL * KB, 8 * Cfg::PANEL, Cfg::PANEL == 128 ? 2 : 4)
                                   : make_smem_desc(0, 16, SBO, SWZ);
      constexpr uint32_t a_step = (A_MN ? UMMA_K * 128 : UMMA_K) >> 4;
      constexpr uint32_t b_step = (B_MN ? UMMA_K * Cfg::PANEL : UMMA_K) >> 4;
      const int last_ksteps = CONV ? KB / UMMA_K :
          static_cast<int>((p.K - static_cast<int64_t>(p.k_blocks - 1) * KB + UMMA_K - 1) / UMMA_K);
      int stage = 0;
      uint32_t phase = 0;
      int acc_buf = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      int local = 0;
      for (TileIter it(p, PAIR); ok && it.valid(p); it.next(p), ++local) {
        if (!mbar_wait(tempty_bar + 8 * acc_buf, acc_phase ^ 1, abort_flag, WAIT_BUDGET)) {
          *abort_flag = 1;
          atomicCAS(p.status, 0, MB_DEV_TIMEOUT_MMA);
          break;
        }
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + acc_buf * BNX;
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (!mbar_wait((patch ? ready_bar : full_bar) + 8 * stage, phase, abort_flag, WAIT_BUDGET)) {
            *abort_flag = 1;
            atomicCAS(p.status, 0, MB_DEV_TIMEOUT_MMA);
            ok = false;
            break;
          }
          tc_fence_after_sync();
          if (local == 0) MB_STAMP(6 + (kb < 3 ? kb : 3));  // k-block kb landed
          if (kb == p.k_blocks - 1) MB_STAMP_TILE(local, 1);
          const uint32_t sa = smem_base + stage * Cfg::STAGE_BYTES;
          const uint64_t a_desc = a_base | static_cast<uint64_t>((sa >> 4) & 0x3FFFu);
          const uint64_t b_desc = b_base | static_cast<uint64_t>(((sa + Cfg::A_BYTES) >> 4) & 0x3FFFu);
          if (PAIR) {
            const int ksteps = (kb + 1 < p.k_blocks) ? KB / UMMA_K : last_ksteps;
            for (int j = 0; j < ksteps; ++j)
              mma_i8_ss_pair(d_tmem, a_desc + j * a_step, b_desc + j * b_step, idesc, (kb > 0 || j > 0) ? 1u : 0u);
            mma_commit_pair(empty_bar + 8 * stage, 3);  // frees the stage in both CTAs
          } else {
          if (kb + 1 < p.k_blocks || last_ksteps == KB / UMMA_K) {
#pragma unroll
            for (int j = 0; j < KB / UMMA_K; ++j)
              mma_i8_ss(d_tmem, a_desc + j * a_step, b_desc + j * b_step, idesc, (kb > 0 || j > 0) ? 1u : 0u);
          } else {
            for (int j = 0; j < last_ksteps; ++j)
              mma_i8_ss(d_tmem, a_desc + j * a_step, b_desc + j * b_step, idesc, (kb > 0 || j > 0) ? 1u : 0u);
          }
          mma_commit(empty_bar + 8 * stage);  // frees the stage when the MMAs have read it
          }
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        if (PAIR) mma_commit_pair(tfull_bar + 8 * acc_buf, 3);  // accumulator complete, in both CTAs
        else mma_commit(tfull_bar + 8 * acc_buf);               // accumulator complete
        if (local == 0) MB_STAMP(10);
        MB_STAMP_TILE(local, 2);
        if (++acc_buf == NUM_ACC) {
          acc_buf = 0;
          acc_phase ^= 1;
        }
      }
    }
    __syncwarp();
  } else if (warp < FIRST_EPI_WARP) {
    // ---------------- preparation: operand sums (fused) and epilogue terms ----------------
    const int r = (warp - 2) * 32 + lane;  // 0..127: row of the A tile / column slot
    int stage = 0;
    uint32_t phase = 0;
    int acc_buf = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    int local = 0;
    int last_tn = -1;
    uint32_t last_sum = 0;
    for (TileIter it(p, PAIR); ok && it.valid(p); it.next(p), ++local) {
      const int b = it.b, tm = it.tm, tn = it.tn;
      uint32_t sa_sum = 0, sb_sum[(BN + 127) / 128];
      uint32_t cs[(BN + 127) / 128][8];  // row-major B: 16 columns of each panel over this lane's k rows, 16-bit counts
#pragma unroll
      for (int j = 0; j < (BN + 127) / 128; ++j) {
        sb_sum[j] = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) cs[j][i] = 0;
      }
      // global inputs of the terms, requested before the main loop is followed
      const int64_t m = static_cast<int64_t>(tm) * TILE_M + rank * BM + r;
      int32_t row_bias = 0, col_bias[(BN + 127) / 128];
      if (p.bias != nullptr && p.bias_per_row && m < p.M) row_bias = mb_load(p.bias + m);
      if (!FUSE_SUMS && p.sum_a != nullptr && m < p.M) {
        sa_sum = sum_partials(p.sum_a + (p.a_batched ? b : 0) * p.sum_a_bstride + m, p.sum_a_slices, p.M);
      }
#pragma unroll
      for (int j = 0; j < (BN + 127) / 128; ++j) {
        const int64_t n = static_cast<int64_t>(tn) * BN + j * 128 + r;
        col_bias[j] = (p.bias != nullptr && !p.bias_per_row && n < p.N) ? mb_load(p.bias + n) : 0;
        if (!FUSE_SUMS && p.sum_b != nullptr && n < p.N) {
          sb_sum[j] = sum_partials(p.sum_b + (p.b_batched ? b : 0) * p.sum_b_bstride + n, p.sum_b_slices, p.N);
        }
      }
      if (prep_reads_tiles) {
        // (a convolution's filter: the sums of a column of tiles serve every tile of it in turn)
        const bool want_a = !TCR && p.zp_b != 0, want_b = p.zp_a != 0 && !(CONV && tn == last_tn);
        int img, h0 = 0, w0 = 0, tap_h = 0, tap_w = 0, cb = 0;
        if constexpr (CONV) conv_corner(p, static_cast<int>(m), img, h0, w0);
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (!mbar_wait_warp(full_bar + 8 * stage, phase, abort_flag, WAIT_BUDGET)) {
            *abort_flag = 1;
            atomicCAS(p.status, 0, MB_DEV_TIMEOUT_EPILOGUE);
            ok = false;
            break;
          }
          const uint8_t *ta = smem_aligned + stage * Cfg::STAGE_BYTES;
          const uint8_t *tb = ta + Cfg::A_BYTES;
          if constexpr (CONV) if (patch) {
            const int h = h0 + tap_h, w = w0 + tap_w;
            const bool outside = h < 0 || h >= p.H || w < 0 || w >= p.W;
            if (outside) {
              // this pixel's channel run lies outside the image, TMA left zeros: the zero point, in the real channels
              const uint32_t z = static_cast<uint32_t>(p.zp_a) * 0x01010101u;
              const int chunks = min(KB, p.Cin - cb * KB) / 16;
              const int rs = KB == 128 ? (r & 7) : KB == 64 ? ((r >> 1) & 3) : ((r >> 2) & 1);
              uint8_t *row = smem_aligned + stage * Cfg::STAGE_BYTES + r * KB;
              for (int c = 0; c < chunks; ++c) *reinterpret_cast<uint4 *>(row + ((c ^ rs) << 4)) = make_uint4(z, z, z, z);
            }
            if (++cb == p.c_blocks) {
              cb = 0;
              if (++tap_w == p.KW) {
                tap_w = 0;
                ++tap_h;
              }
            }
            if (__any_sync(0xffffffffu, outside)) {
              fence_proxy_async();
              __syncwarp();
            }
            if (lane == 0) mbar_arrive(ready_bar + 8 * stage);
          }
          // a row is KB bytes = KB / 16 chunks of 16; start at chunk (r mod chunks) so that
          // the threads of a quarter warp spread over the bank groups.  The swizzle only
          // permutes chunks inside a row, which a sum does not see.
          if (want_a) {
            uint32_t s1 = 0, s2 = 0, s3 = 0;  // (four chains: one would be 32 dependent instructions per step)
#pragma unroll
            for (int i = 0; i < KB / 16; ++i) {
              const uint4 v = *reinterpret_cast<const uint4 *>(ta + r * KB + ((i + r) & (KB / 16 - 1)) * 16);
              sa_sum = __dp4a(v.x, 0x01010101u, sa_sum);
              s1 = __dp4a(v.y, 0x01010101u, s1);
              s2 = __dp4a(v.z, 0x01010101u, s2);
              s3 = __dp4a(v.w, 0x01010101u, s3);
            }
            sa_sum += s1 + (s2 + s3);
          }
#pragma unroll
          for (int j = 0; j < (BN + 127) / 128; ++j) {
            const int row = j * 128 + r;
            if (B_MN) {
              // The tile is [panel][KB depth rows][128 or 64 bytes], the 16-byte chunks of a row permuted by
              // the row's low bits.  Warp q takes depth rows 32 q .. 32 q + 31, four (eight) at a time, a lane
              // one chunk (16 columns).  The bytes are added as pairs of 16-bit counts, which hold the
              // rows a lane sees in all of the at most eight steps (64 x 255); lanes and warps meet below.
              if (want_b) {
                constexpr int CH = Cfg::PANEL / 16, RPP = 32 / CH, PASSES = 32 / RPP;  // chunks of a row, rows per pass
                const int c = lane % CH, k0 = (warp - 2) * 32 + lane / CH;
                const uint8_t *pan = tb + j * 128 * KB + k0 * Cfg::PANEL;
                uint4 v[PASSES];
#pragma unroll
                for (int i = 0; i < PASSES; ++i) {
                  const int k = k0 + RPP * i;
                  v[i] = *reinterpret_cast<const uint4 *>(pan + i * RPP * Cfg::PANEL + ((c ^ (Cfg::PANEL == 128 ? k & 7 : (k >> 1) & 3)) << 4));
                }
#pragma unroll
                for (int i = 0; i < PASSES; i += 2) {
                  const uint32_t w0[4] = {v[i].x, v[i].y, v[i].z, v[i].w}, w1[4] = {v[i + 1].x, v[i + 1].y, v[i + 1].z, v[i + 1].w};
#pragma unroll
                  for (int w = 0; w < 4; ++w) {
                    cs[j][w] += (w0[w] & 0x00ff00ffu) + (w1[w] & 0x00ff00ffu);
                    cs[j][4 + w] += __byte_perm(w0[w], 0, 0x4341) + __byte_perm(w1[w], 0, 0x4341);
                  }
                }
              }
            } else if (want_b && row < BN) {
              uint32_t s1 = 0, s2 = 0, s3 = 0;
#pragma unroll
              for (int i = 0; i < KB / 16; ++i) {
                const uint4 v = *reinterpret_cast<const uint4 *>(tb + row * KB + ((i + r) & (KB / 16 - 1)) * 16);
                sb_sum[j] = __dp4a(v.x, 0x01010101u, sb_sum[j]);
                s1 = __dp4a(v.y, 0x01010101u, s1);
                s2 = __dp4a(v.z, 0x01010101u, s2);
                s3 = __dp4a(v.w, 0x01010101u, s3);
              }
              sb_sum[j] += s1 + (s2 + s3);
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(empty_bar + 8 * stage);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        if (B_MN && want_b) {
          // the four k quarters of every column: through shared memory (two buffers, by tile parity)
          constexpr int COLS = ((BN + 127) / 128) * 128;
          uint32_t *part = part_sm + (local & 1) * Cfg::PART_INTS;
#pragma unroll
          for (int j = 0; j < (BN + 127) / 128; ++j) {
#pragma unroll
            for (int w = 0; w < 4; ++w) {
              uint32_t t[4] = {cs[j][w] & 0xffffu, cs[j][4 + w] & 0xffffu, cs[j][w] >> 16, cs[j][4 + w] >> 16};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
#pragma unroll
                for (int o = Cfg::PANEL / 16; o < 32; o <<= 1) t[i] += __shfl_xor_sync(0xffffffffu, t[i], o);
              }
              if (lane < Cfg::PANEL / 16)
                *reinterpret_cast<uint4 *>(part + (warp - 2) * COLS + j * 128 + lane * 16 + w * 4) = make_uint4(t[0], t[1], t[2], t[3]);
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(part_bar);
          if (!mbar_wait_warp(part_bar, static_cast<uint32_t>(local & 1), abort_flag, WAIT_BUDGET)) {
            *abort_flag = 1;
            atomicCAS(p.status, 0, MB_DEV_TIMEOUT_EPILOGUE);
            break;
          }
#pragma unroll
          for (int j = 0; j < (BN + 127) / 128; ++j)
            sb_sum[j] = part[j * 128 + r] + part[COLS + j * 128 + r] + part[2 * COLS + j * 128 + r] +
                        part[3 * COLS + j * 128 + r];
        }
      }
      if (CONV) {
        if (tn == last_tn) sb_sum[0] = last_sum;
        last_tn = tn;
        last_sum = sb_sum[0];
      }
      // terms of this tile (operand sums are zero where no correction is needed)
      const int32_t row_term = row_bias - p.zp_b * static_cast<int32_t>(sa_sum);
      int32_t col_term[(BN + 127) / 128];
#pragma unroll
      for (int j = 0; j < (BN + 127) / 128; ++j)
        col_term[j] = p.kzz + col_bias[j] - p.zp_a * static_cast<int32_t>(sb_sum[j]);
      // the terms of this buffer's previous tile must have been consumed
      if (!mbar_wait_warp(tempty_bar + 8 * acc_buf, acc_phase ^ 1, abort_flag, WAIT_BUDGET)) {
        *abort_flag = 1;
        atomicCAS(p.status, 0, MB_DEV_TIMEOUT_EPILOGUE);
        break;
      }
      row_term_sm[acc_buf * 128 + r] = row_term;
#pragma unroll
      for (int j = 0; j < (BN + 127) / 128; ++j)
        if (j * 128 + r < BN) col_term_sm[acc_buf * BN + j * 128 + r] = col_term[j];
      __syncwarp();
      if (lane == 0) mbar_arrive(terms_bar + 8 * acc_buf);
      if (local == 0 && warp == 2 && lane == 0) MB_STAMP(11);
      if (++acc_buf == NUM_ACC) {
        acc_buf = 0;
        acc_phase ^= 1;
      }
    }
  } else {
    // ---------------- epilogue ----------------
    // Four consecutive warps cover the four TMEM lane quarters of a 64-column slice of a
    // tile; BN / 64 such sets work on one tile, and the remaining sets on the tiles after
    // it (GROUPS tiles are drained at the same time, each from its own accumulator
    // buffer).  Per tile a warp handles 32 rows x 64 columns in four 16-column chunks.
    constexpr int SETS_PER_TILE = BN / 64;             // 1, 2, 4
    constexpr int GROUPS = 4 / SETS_PER_TILE;          // 4, 2, 1 tiles in flight
    constexpr int CHUNKS_PER_WARP = 4;
    const int quarter = warp & 3;                      // TMEM lanes [32*quarter, +32) are this warp's
    const int set = (warp - FIRST_EPI_WARP) >> 2;      // 0..3
    const int slice = set % SETS_PER_TILE;             // which 64 columns of the tile
    const int group = set / SETS_PER_TILE;             // which tiles: local % GROUPS == group
    // staging for the TMA store: 32 rows x 32 bytes (two chunks), 32-byte swizzle:
    // 16-byte half h of row r sits at r*32 + ((h ^ (r >> 2)) & 1)*16, which keeps the
    // quarter-warps' 16-byte writes free of bank conflicts
    constexpr int STG = Cfg::STG_CHUNKS;
    uint8_t *stage_ptr = smem_aligned + STAGES * Cfg::STAGE_BYTES + (warp - FIRST_EPI_WARP) * (32 * STG * 16);
    const uint32_t stage_addr = smem_u32(stage_ptr);
    uint4 *stage_row = reinterpret_cast<uint4 *>(stage_ptr + lane * (STG * 16));
    // 32-byte rows, 32-byte swizzle: half h of row r at ((h ^ (r >> 2)) & 1); 64-byte rows,
    // 64-byte swizzle: chunk c of row r at (c ^ (r >> 1)) & 3
    const int swz = STG == 2 ? ((lane >> 2) & 1) : ((lane >> 1) & 3);
    int local = 0;
    for (TileIter it(p, PAIR); it.valid(p); it.next(p), ++local) {
      if (local % GROUPS != group) continue;
      const int b = it.b, tm = it.tm, tn = it.tn;
      const int acc_buf = local % NUM_ACC;
      const uint32_t acc_phase = (local / NUM_ACC) & 1;
      if (!mbar_wait_warp(tfull_bar + 8 * acc_buf, acc_phase, abort_flag, WAIT_BUDGET) ||
          !mbar_wait_warp(terms_bar + 8 * acc_buf, acc_phase, abort_flag, WAIT_BUDGET)) {
        *abort_flag = 1;
        atomicCAS(p.status, 0, MB_DEV_TIMEOUT_EPILOGUE);
        break;
      }
      tc_fence_after_sync();
      if (local == 0 && warp == FIRST_EPI_WARP && lane == 0) MB_STAMP(12);
      if (warp == FIRST_EPI_WARP && lane == 0) MB_STAMP_TILE(local, 3);
      const int m0 = tm * TILE_M + rank * BM + quarter * 32;  // first row of this warp
      const int64_t m = static_cast<int64_t>(m0) + lane;
      const bool row_ok = m < p.M;
      int32_t row_term = row_term_sm[acc_buf * 128 + quarter * 32 + lane];
      const uint32_t tbase = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc_buf * BNX +
                             slice * 64;
      if (TCR) {
        // columns BN .. BN + 15 of this lane's row: the byte sum of A's row (all 16 alike)
        uint32_t ones_cols[CHUNK];
        tmem_ld_32x32b_x16(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc_buf * BNX + BN, ones_cols);
        tmem_ld_wait_x16(ones_cols);
        row_term -= p.zp_b * static_cast<int32_t>(ones_cols[0]);
      }
      const int32_t *ct_base = col_term_sm + acc_buf * BN + slice * 64;
      const int64_t n_first = static_cast<int64_t>(tn) * BN + slice * 64;
      if constexpr (!PLAIN) {
        // one decision per tile (not per chunk or value: with so few warps per scheduler
        // a branch's latency is not hidden)
        const EpiTile e{tbase, row_term, ct_base, tempty_bar + 8 * acc_buf,
                        (PAIR && rank != 0) ? mapa_shared(tempty_bar + 8 * acc_buf, 0) : 0u, stage_row, swz,
                        stage_addr, n_first, m0, b, lane};
        switch (p.rq_variant) {
          case 8: epi_tma_tile<STG, 8, PAIR>(e, tmap_c, p); break;
          case 5: epi_tma_tile<STG, 5, PAIR>(e, tmap_c, p); break;
          case 4: epi_tma_tile<STG, 4, PAIR>(e, tmap_c, p); break;
          case 3: epi_tma_tile<STG, 3, PAIR>(e, tmap_c, p); break;
          case 2: epi_tma_tile<STG, 2, PAIR>(e, tmap_c, p); break;
          case 1: epi_tma_tile<STG, 1, PAIR>(e, tmap_c, p); break;
          default: epi_tma_tile<STG, 0, PAIR>(e, tmap_c, p); break;
        }
      } else {
        // plain stores: int32 output, or a uint8 output whose rows TMA cannot address
        if (!p.out_is_int32) {
          const PlainTile e{tbase, row_term, ct_base, stage_ptr,
                            static_cast<uint8_t *>(p.C) + (static_cast<int64_t>(b) * p.M + m0) * p.N + n_first, p.N, static_cast<int>(min(static_cast<int64_t>(32), p.M - m0)),
                            static_cast<int>(min(static_cast<int64_t>(64), p.N - n_first)), swz};
          switch (p.rq_variant) {
            case 8: epi_plain_tile<STG, 8>(e, p); break;
            case 5: epi_plain_tile<STG, 5>(e, p); break;
            case 4: epi_plain_tile<STG, 4>(e, p); break;
            case 3: epi_plain_tile<STG, 3>(e, p); break;
            case 2: epi_plain_tile<STG, 2>(e, p); break;
            case 1: epi_plain_tile<STG, 1>(e, p); break;
            default: epi_plain_tile<STG, 0>(e, p); break;
          }
        } else {
        int32_t *c32 = static_cast<int32_t *>(p.C) + (static_cast<int64_t>(b) * p.M + m) * p.N;
        const bool quads_ok = (p.N & 3) == 0 && (reinterpret_cast<uintptr_t>(p.C) & 15u) == 0;
        uint32_t r[1][CHUNK];
        tmem_ld_32x32b_x16(tbase, r[0]);
#pragma unroll 1
        for (int i = 0; i < CHUNKS_PER_WARP; ++i) {
          uint32_t v[CHUNK];
          tmem_ld_wait_x16(r[0]);
#pragma unroll
          for (int j = 0; j < CHUNK; ++j) v[j] = r[0][j];
          if (i + 1 < CHUNKS_PER_WARP) tmem_ld_32x32b_x16(tbase + (i + 1) * CHUNK, r[0]);
          const int64_t n0 = n_first + i * CHUNK;
          const int32_t *ct = ct_base + i * CHUNK;
          if (quads_ok && n0 + CHUNK <= p.N) {
            // a whole chunk of an int32 row: four 16-byte stores instead of sixteen words
            if (row_ok) {
              int4 *cq = reinterpret_cast<int4 *>(c32 + n0);
#pragma unroll
              for (int q = 0; q < CHUNK / 4; ++q)
                cq[q] = make_int4(static_cast<int32_t>(v[4 * q + 0]) + row_term + ct[4 * q + 0],
                                  static_cast<int32_t>(v[4 * q + 1]) + row_term + ct[4 * q + 1],
                                  static_cast<int32_t>(v[4 * q + 2]) + row_term + ct[4 * q + 2],
                                  static_cast<int32_t>(v[4 * q + 3]) + row_term + ct[4 * q + 3]);
            }
          } else if (row_ok && n0 < p.N) {
#pragma unroll
            for (int j = 0; j < CHUNK; ++j)
              if (n0 + j < p.N) c32[n0 + j] = static_cast<int32_t>(v[j]) + row_term + ct[j];
          }
        }
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(tempty_bar + 8 * acc_buf);
          if (PAIR && rank != 0) mbar_arrive_cluster(mapa_shared(tempty_bar + 8 * acc_buf, 0));
        }
      }
      if (warp == FIRST_EPI_WARP && lane == 0) MB_STAMP(local == 0 ? 13 : 14);
      if (warp == FIRST_EPI_WARP && lane == 0) MB_STAMP_TILE(local, 4);
    }
    // the staging buffer must outlive the last store's read, and the kernel its writes
    if (lane == 0) bulk_wait_group<0>();
    __syncwarp();
  }

  __syncthreads();
  if (threadIdx.x == 0) MB_STAMP(15);
  if (*abort_flag != 0) {
    // Give copies and MMAs that are still in flight time to land before the
    // shared memory and TMEM they target go away (bounded: about 2 ms).
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    __syncthreads();
  }
  // pairs: neither CTA's shared or tensor memory may go away while the other can still reach
  // it (the even CTA's MMAs read the odd CTA's tiles; the odd CTA arrives on the even one's
  // barriers)
  if (PAIR) cluster_sync_all();
  if (warp == 1) {
    tc_fence_after_sync();
    if (PAIR) tmem_dealloc_pair(tmem_base, Cfg::TMEM_COLS);
    else tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}



template <bool PLAIN, int BN, bool A_MN, bool B_MN, bool FUSE_SUMS = false, int KB = BK, bool TCR_ON = false>
int launch_cfg(mb_context *ctx, const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &tc,
               TcParams &p) {
  using Cfg = TileCfg<BN, B_MN, KB, TCR_ON && FUSE_SUMS && BN <= 128>;
  auto kern = gemm_u8_tc_kernel<BN, A_MN, B_MN, FUSE_SUMS, KB, TCR_ON, false, false, PLAIN>;
  // The opt-in shared-memory limit is a per-device function attribute; set it
  // once per context.
  constexpr int cfg_id = (BN == 256 ? 0 : BN == 128 ? 1 : 2) * 4 + (A_MN ? 2 : 0) + (B_MN ? 1 : 0) +
                         (FUSE_SUMS ? 12 : 0) + (KB == 64 ? 3 : KB == 32 ? 6 : 0) + (TCR_ON ? 24 : 0);
  uint64_t &mask = PLAIN ? ctx->func_attr_mask_plain : ctx->func_attr_mask;
  if (!(mask & (1ull << cfg_id))) {
    MB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      Cfg::SMEM_BYTES));
    mask |= (1ull << cfg_id);
  }
  const int grid = static_cast<int>(p.total_tiles < ctx->num_sms ? p.total_tiles : ctx->num_sms);
  p.step_m = grid % p.tiles_m;
  p.step_n = (grid / p.tiles_m) % p.tiles_n;
  p.step_b = (grid / p.tiles_m) / p.tiles_n;
  ctx->pdl_next_gemm = 0;
  MB_CUDA(ctx, mb_launch_chained(ctx, kern, dim3(grid), dim3(NUM_THREADS), Cfg::SMEM_BYTES, ta, tb, tc, p));
  MB_CUDA(ctx, cudaGetLastError());
  ctx->launches++;
  ctx->launches_tc++;
  return MB_SUCCESS;
}

// A convolution: one K-major instance per tile width and depth row.
template <bool PLAIN, int BN, int KB>
int launch_conv(mb_context *ctx, const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &tc, ConvTcParams &p) {
  using Cfg = TileCfg<BN, false, KB, true>;
  auto kern = gemm_u8_tc_kernel<BN, false, false, true, KB, true, false, true, PLAIN>;
  constexpr int bit = 32 + (PLAIN ? 6 : 0) + (BN == 128 ? 3 : 0) + (KB == 128 ? 0 : KB == 64 ? 1 : 2);
  if (!(ctx->func_attr_mask2 & (1ull << bit))) {
    MB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
    ctx->func_attr_mask2 |= (1ull << bit);
  }
  const int grid = static_cast<int>(p.total_tiles < ctx->num_sms ? p.total_tiles : ctx->num_sms);
  p.step_m = grid % p.tiles_m;
  p.step_n = (grid / p.tiles_m) % p.tiles_n;
  p.step_b = (grid / p.tiles_m) / p.tiles_n;
  MB_CUDA(ctx, mb_launch_chained(ctx, kern, dim3(grid), dim3(NUM_THREADS), Cfg::SMEM_BYTES, ta, tb, tc, p));
  ctx->launches++;
  ctx->launches_tc++;
  return MB_SUCCESS;
}

// Which instance: tile width, bytes of a depth row, operand orders, where the operand sums come from.
struct TcChoice {
  int bn, kb;
  bool a_mn, b_mn, fuse, fuse_bmn;
};

template <bool PLAIN>
int dispatch(mb_context *ctx, const TcChoice &c, const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &tc,
             TcParams &p) {
#define MB_TC_DISPATCH(BN_)                                                         \
  if (c.a_mn) {                                                                       \
    if (c.b_mn) return launch_cfg<PLAIN, BN_, true, true>(ctx, ta, tb, tc, p);                   \
    return launch_cfg<PLAIN, BN_, true, false>(ctx, ta, tb, tc, p);                            \
  } else {                                                                          \
    if (c.b_mn) return launch_cfg<PLAIN, BN_, false, true>(ctx, ta, tb, tc, p);                  \
    return launch_cfg<PLAIN, BN_, false, false>(ctx, ta, tb, tc, p);                           \
  }
  if (c.fuse_bmn) {
    if (c.bn == 256) return launch_cfg<PLAIN, 256, false, true, true>(ctx, ta, tb, tc, p);
    if (c.bn == 128) return launch_cfg<PLAIN, 128, false, true, true>(ctx, ta, tb, tc, p);
    return launch_cfg<PLAIN, 64, false, true, true>(ctx, ta, tb, tc, p);
  }
  if (c.fuse) {
#define MB_TC_FUSED(KB_)                                                                  \
  if (c.bn == 256) return launch_cfg<PLAIN, 256, false, false, true, KB_>(ctx, ta, tb, tc, p);     \
  if (ctx->tc_rowsum) {                                                                            \
    if (c.bn == 128) return launch_cfg<PLAIN, 128, false, false, true, KB_, true>(ctx, ta, tb, tc, p); \
    return launch_cfg<PLAIN, 64, false, false, true, KB_, true>(ctx, ta, tb, tc, p);             \
  }                                                                                                \
  if (c.bn == 128) return launch_cfg<PLAIN, 128, false, false, true, KB_>(ctx, ta, tb, tc, p);     \
  return launch_cfg<PLAIN, 64, false, false, true, KB_>(ctx, ta, tb, tc, p);
    if (c.kb == 32) { MB_TC_FUSED(32) }
    if (c.kb == 64) { MB_TC_FUSED(64) }
    MB_TC_FUSED(128)
#undef MB_TC_FUSED
  }
  if (c.bn == 256) { MB_TC_DISPATCH(256) }
  if (c.bn == 128) { MB_TC_DISPATCH(128) }
  MB_TC_DISPATCH(64)
#undef MB_TC_DISPATCH
}

template <bool PLAIN>
int dispatch_conv(mb_context *ctx, int bn, int kb, const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &tc,
                  ConvTcParams &p) {
  if (bn == 128) {
    if (kb == 128) return launch_conv<PLAIN, 128, 128>(ctx, ta, tb, tc, p);
    if (kb == 64) return launch_conv<PLAIN, 128, 64>(ctx, ta, tb, tc, p);
    return launch_conv<PLAIN, 128, 32>(ctx, ta, tb, tc, p);
  }
  if (kb == 128) return launch_conv<PLAIN, 64, 128>(ctx, ta, tb, tc, p);
  if (kb == 64) return launch_conv<PLAIN, 64, 64>(ctx, ta, tb, tc, p);
  return launch_conv<PLAIN, 64, 32>(ctx, ta, tb, tc, p);
}

}  // namespace mb_tc
