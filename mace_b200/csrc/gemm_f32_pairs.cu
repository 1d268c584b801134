// Large fp32 GEMMs on tcgen05 (kind::f16 on pairs of halves, see f32_split.cuh), bias, residual and activation fused:
//     C[b][n][m] = act(bias[n] + sum_k X[b][k][m] * W[b][n][k] [+ R[b][n][m]])
// What it serves: what gemm_f32_tc.cu does, in the same layout (X [K x Mdim] with m contiguous, W [Ndim x K] with k contiguous, C
// [Ndim x Mdim] with m contiguous; TMA's alignments), from the size on where its smaller steps pay for a launch of their own
// that splits W: the 1x1 convolution on a batch (arm::Conv2dK1x1, mace/ops/arm/base/conv_2d_1x1.cc:61-68), the
// products of a Winograd convolution (conv_2d_3x3_winograd.cc:147-170), MatMul / Gemm (mace/ops/arm/base/gemm.cc:520-683).
//
// Where the operands live.  X (the MMA's A, 128 pixels = 128 TMEM lanes) lands as fp32 in shared memory; a warp reads its 32
// pixels' values (one word per lane and k: conflict-free), splits them and writes hi and lo to tensor memory, from where the
// MMA takes A.  W has been split by f32_presplit_kernel.  A residual tile comes by TMA into the buffer that the result leaves
// from.
//
// What bounds it: shared memory at 128 bytes a cycle and the clocks that the power limit leaves.  A step of 128 x 128 x 32 moves
// 16 KB of X in and out, 16 KB of W in and 24 KB into the MMAs: 576 cycles, of which the MMAs are busy 384 (tf32 pairs split
// in the kernel: 144 KB, 1150 cycles, 768 busy; 750 measured now).  A tile of few steps is bound by HBM.
// Measured, tf32 pairs -> this kernel (1x1 convolutions, batch 256, us; in brackets with a residual): 64 -> 256 channels at 56 x 56
// 220 -> 226 (394 -> 346), 256 -> 64 214 -> 180, 512 -> 128 at 28 x 28 148 -> 128, 128 -> 512 170 -> 148 (258 -> 206), 256 -> 1024 at
// 14 x 14 156 -> 139 (194 -> 154), 1024 -> 256 147 -> 123, 1024 -> 512 282 -> 227.
//
// A row of X has the scale of its first step that has a value.  Where a later one is beyond 2^11 (with wide ranges 2^3) times that the
// row's results are no finite numbers; the tiles that have some are marked, and a second pass over them has scales from all of a row.  512 -> 128 at
// 28 x 28 with channels 2^14 times larger from the 32nd on: in all pixels 497 us (7170 by FMAs), in one of 1000 233 (1863).
//
// Structure (one persistent CTA per SM):
//   warp 0        TMA producer: X as one [32 k x 128 m] box (no swizzle) and a step of W, mbarrier ring
//   warp 1        MMA issuer: A from TMEM, B from shared memory
//   warps 2..9    X split, two warps per TMEM lane quarter, 16 k each
//   warps 10..17  epilogue: two sets of four warps (one per TMEM lane quarter), each on half of the tile's columns
//   warps 18, 19  a set's result and residual copies (one thread each)
// TMEM columns: with 64 channels two accumulators of 64 columns of large products and 64 of small ones; with 128 two of large
// products and one of small ones, which the epilogue adds to the large ones first, in tensor memory, so that it is free some
// 500 cycles into the next tile, whose large products run ahead meanwhile.  Then STAGES x 32 columns of A (hi 16, lo 16).
// Every wait is bounded; on a timeout the kernel records a status word, lets outstanding
// copies land, frees its TMEM and returns.
#include "common.cuh"
#include "f32_split.cuh"
#include "sm100_ptx.cuh"

namespace {

using namespace sm100;

constexpr int FBM = 128;       // pixels (m) per tile == TMEM lanes
constexpr int FKB = 32;        // k per pipeline stage
constexpr int F_X_WARPS = 8, F_EPI_WARPS = 8, F_FIRST_X = 2, FIRST_EPI = F_FIRST_X + F_X_WARPS, FIRST_STORE = FIRST_EPI + F_EPI_WARPS;
constexpr int F_THREADS = (FIRST_STORE + 2) * 32;
constexpr long long F_WAIT_BUDGET = 1ll << 31;
// Scales of so many tiles: X is at most F32Cfg::STAGES tiles of one step ahead of the MMAs, these are two ahead of the epilogue.
constexpr int F_SCALE_SLOTS = 16;
constexpr int MARKS = 512;     // tiles of a CTA with a mark of their own (of results that are no finite numbers)
constexpr int F_BUFS = 4;      // result buffers per set, 16 channels x 128 pixels each

struct F32TcParams {
  const float *X, *W;
  int64_t Mdim, Ndim, K, batch;
  int64_t x_rs, x_bs, w_rs, w_bs;
  int tiles_m, tiles_n, k_blocks;
  int step_m, step_n, step_b;
  int x_batched, w_batched;
  const float *w_unscale;     // 1 / scale per row of W, all batches' rows one behind the other
  const float *bias;  // per n, or null
  const float *residual;  // null, or a tensor laid out like C that is added before the activation
  int act;
  float max_limit, coef;
  float *C;
  int64_t c_row_stride, c_batch_stride;  // elements between consecutive n / batch entries
  int c_tma;  // rows of C (and of the residual) are 16-byte aligned: results and residual by TMA through shared memory
  int *status;
};

template <int BN>
struct F32Cfg {
  static constexpr int X_BYTES = FBM * FKB * 4;   // [32 k][128 m]
  // 32 halves of hi and 32 of lo per channel
  static constexpr int W_BYTES = BN * FKB * 4;
  static constexpr int STAGE_BYTES = X_BYTES + W_BYTES;
  static constexpr int BUF_BYTES = 16 * FBM * 4;
  static constexpr int STAGING_BYTES = 2 * F_BUFS * BUF_BYTES;
  static constexpr int XSCALE_BYTES = F_SCALE_SLOTS * FBM * 4;
  static constexpr int UB_BYTES = F_EPI_WARPS * (BN / 2) * 8;  // (1 / scale, bias) of the channels of an epilogue warp
  static constexpr int BAR_BYTES = 512 + 2 * MARKS;
  static constexpr int FIXED = STAGING_BYTES + XSCALE_BYTES + UB_BYTES + BAR_BYTES + 1024;
  static constexpr int NUM_ACC = 2;
  static constexpr int TMEM_COLS = 512;
  // 64 channels: the hi rows of W with the lo rows behind them, hi of X times both is one MMA of 128 columns
  static constexpr bool WIDE = BN == 64;
  static constexpr int ACC_COLS = 128;
  static constexpr int SMALL_COL0 = WIDE ? 64 : NUM_ACC * ACC_COLS;  // small products (WIDE: of the accumulator)
  static constexpr int A_COL0 = (NUM_ACC + (WIDE ? 0 : 1)) * ACC_COLS;  // first TMEM column of the A ring
  static constexpr int MAX_TMEM_STAGES = (TMEM_COLS - A_COL0) / FKB;
  static constexpr int SMEM_STAGES = (227 * 1024 - FIXED) / STAGE_BYTES;
  static constexpr int STAGES = SMEM_STAGES < MAX_TMEM_STAGES ? SMEM_STAGES : MAX_TMEM_STAGES;
  static_assert(STAGES >= 2, "pipeline needs two stages");
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + FIXED;
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
  static constexpr int BARRIERS = 3 * STAGES + 2 * NUM_ACC + 4 * F_BUFS + 1;
  static_assert(8 * BARRIERS + 2 * MARKS + 16 <= BAR_BYTES, "barriers, marks, flags");
};

// Column tiles first: the CTAs that read one tile of X run side by side and fetch it from HBM once.  With `only` the CTA's nth tiles
// that are marked there (the nth + i * MARKS ones with them).
struct FTileIter {
  int tm, tn, b, nth = 0;
  const volatile uint8_t *only;
  __device__ __forceinline__ FTileIter(const F32TcParams &p, const volatile uint8_t *marked = nullptr) : only(marked) {
    const unsigned t = blockIdx.x;
    tn = t % p.tiles_n;
    const unsigned q = t / p.tiles_n;
    tm = q % p.tiles_m;
    b = q / p.tiles_m;
    skip(p);
  }
  __device__ __forceinline__ bool valid(const F32TcParams &p) const { return b < p.batch; }
  __device__ __forceinline__ void next(const F32TcParams &p) {
    step(p);
    skip(p);
  }

 private:
  __device__ __forceinline__ void step(const F32TcParams &p) {
    ++nth;
    tm += p.step_m;
    tn += p.step_n;
    b += p.step_b;
    if (tn >= p.tiles_n) { tn -= p.tiles_n; ++tm; }
    if (tm >= p.tiles_m) { tm -= p.tiles_m; ++b; }
  }
  __device__ __forceinline__ void skip(const F32TcParams &p) {
    if (only == nullptr) return;
    while (valid(p) && only[nth % MARKS] == 0) step(p);
  }
};

// A result that the second pass has as no finite number either is stored as F32_AGAIN; when its tiles are done a CTA that stored
// one works those out again, by fp32 FMAs.
__device__ __noinline__ void tile_again(const F32TcParams &p, int m0, int n0, int bn, int b) {
  for (int i = threadIdx.x; i < FBM * bn; i += blockDim.x) {
    // (a warp: one channel, 32 pixels)
    const int64_t m_first = m0 + (i & (FBM - 32)), n = n0 + i / FBM, m = m_first + (i & 31);
    const int64_t at_first = b * p.c_batch_stride + n * p.c_row_stride + m_first;
    const bool mine = m < p.Mdim && n < p.Ndim &&
                      __float_as_uint(*reinterpret_cast<volatile float *>(p.C + at_first + (i & 31))) == F32_AGAIN;
    f32_each_again(mine, [&](int lane) {
      float sum = f32_warp_dot(p.X + b * p.x_bs + m_first + lane, p.x_rs, p.W + b * p.w_bs + n * p.w_rs, p.K);
      if ((i & 31) != lane) return;
      const int64_t at = at_first + lane;
      if (p.bias != nullptr) sum += p.bias[n];
      if (p.residual != nullptr) sum += p.residual[at];
      p.C[at] = mb_activate(sum, p.act, p.max_limit, p.coef);
    });
  }
}

// W [rows][K] -> [rows][K / 32 rounded up][32 halves of hi, 32 of lo] and 1 / scale per row, `group` threads per row.
__global__ void __launch_bounds__(256)
f32_presplit_kernel(const float *W, uint8_t *dst, float *unscale, int64_t rows, int64_t K, int64_t rows_per_batch, int64_t w_rs,
                    int64_t w_bs, int k_blocks, int group) {
  __shared__ float warp_most[8];
  mb_grid_dep_launch();
  mb_grid_dep_wait();
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (256 / group) + threadIdx.x / group;
  const int g = threadIdx.x & (group - 1);
  const bool in = row < rows;
  const int64_t b = in ? row / rows_per_batch : 0;
  const float *src = W + b * w_bs + (in ? row - b * rows_per_batch : 0) * w_rs;
  const int chunks = k_blocks * 8;  // of four values; the row is 16-byte aligned
  auto load = [&](int c) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    const int64_t k = static_cast<int64_t>(c) * 4;
    if (in && k + 4 <= K) return mb_load(reinterpret_cast<const float4 *>(src + k));
    if (in && k < K) v.x = mb_load(src + k);
    if (in && k + 1 < K) v.y = mb_load(src + k + 1);
    if (in && k + 2 < K) v.z = mb_load(src + k + 2);
    return v;
  };
  float most = 0.f;
#pragma unroll 4
  for (int c = g; c < chunks; c += group) {
    const float4 v = load(c);
    most = fmaxf(most, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
  }
  for (int d = 1; d < group && d < 32; d *= 2) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, d));
  if (group > 32) {
    if ((threadIdx.x & 31) == 0) warp_most[threadIdx.x >> 5] = most;
    __syncthreads();
    const int first = threadIdx.x / group * (group / 32);
    for (int w = 0; w < group / 32; ++w) most = fmaxf(most, warp_most[first + w]);
  }
  if (!in) return;
  const float s = most > 0.f ? f32_row_scale(most) : 0.f;
  if (g == 0) unscale[row] = f32_row_unscale(s);
  const uint64_t scales = f32_pair(s, s);
  uint8_t *out = dst + row * k_blocks * 128;
#pragma unroll 4
  for (int c = g; c < chunks; c += group) {
    const float4 v = load(c);
    uint2 hi, lo;
    f32_split2(f32_pair(v.x, v.y), scales, hi.x, lo.x);
    f32_split2(f32_pair(v.z, v.w), scales, hi.y, lo.y);
    uint8_t *to = out + (c >> 3) * 128 + (c & 7) * 8;
    *reinterpret_cast<uint2 *>(to) = hi;
    *reinterpret_cast<uint2 *>(to + 64) = lo;
  }
}

// Where what lies in shared memory behind the stages.
template <int BN>
struct FShared {
  using Cfg = F32Cfg<BN>;
  static constexpr int STAGING_AT = Cfg::STAGES * Cfg::STAGE_BYTES, XSCALE_AT = STAGING_AT + Cfg::STAGING_BYTES;
  static constexpr int UB_AT = XSCALE_AT + Cfg::XSCALE_BYTES, BAR_AT = UB_AT + Cfg::UB_BYTES;
  uint8_t *base;             // 1024-byte aligned
  uint32_t base_u32;
  uint32_t full_bar, split_bar, empty_bar;  // [STAGES] raw tiles landed, hi/lo ready, stage consumed
  uint32_t tfull_bar, tempty_bar;           // [NUM_ACC] accumulator complete, drained
  uint32_t free_bar, ready_bar;             // [2][F_BUFS] result buffer free (its residual landed), written
  uint32_t sempty_bar;                      // accumulator of the small products drained (128 channels)
  volatile uint8_t *marks;   // [2][MARKS] tiles with a result that is no finite number, of the first pass and the second
  uint32_t *tmem_slot;
  volatile int *abort_flag, *again;         // again: [2] any such tile
  __device__ __forceinline__ explicit FShared(uint8_t *raw) {
    base_u32 = (smem_u32(raw) + 1023u) & ~1023u;
    base = raw + (base_u32 - smem_u32(raw));
    full_bar = base_u32 + BAR_AT;
    split_bar = full_bar + 8 * Cfg::STAGES;
    empty_bar = split_bar + 8 * Cfg::STAGES;
    tfull_bar = empty_bar + 8 * Cfg::STAGES;
    tempty_bar = tfull_bar + 8 * Cfg::NUM_ACC;
    free_bar = tempty_bar + 8 * Cfg::NUM_ACC;
    ready_bar = free_bar + 8 * 2 * F_BUFS;
    sempty_bar = ready_bar + 8 * 2 * F_BUFS;
    marks = base + BAR_AT + 8 * Cfg::BARRIERS;
    tmem_slot = reinterpret_cast<uint32_t *>(base + BAR_AT + 8 * Cfg::BARRIERS + 2 * MARKS);
    abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    again = abort_flag + 1;
  }
  __device__ __forceinline__ void init_barriers() const {
    for (int s = 0; s < Cfg::STAGES; ++s) {
      mbar_init(full_bar + 8 * s, 1);
      mbar_init(split_bar + 8 * s, F_X_WARPS);
      mbar_init(empty_bar + 8 * s, 1);
    }
    for (int b = 0; b < Cfg::NUM_ACC; ++b) {
      mbar_init(tfull_bar + 8 * b, 1);
      mbar_init(tempty_bar + 8 * b, F_EPI_WARPS);
    }
    mbar_init(sempty_bar, F_EPI_WARPS);
    for (int b = 0; b < 2 * F_BUFS; ++b) {
      mbar_init(free_bar + 8 * b, 1);
      mbar_init(ready_bar + 8 * b, F_EPI_WARPS / 2);
    }
    fence_barrier_init();
  }
};

// The warps' roles over the CTA's tiles.  EPI selects the epilogue's arithmetic: 0 = the accumulator is the result (the Winograd
// products); 1 = bias and a clamp (NOOP / RELU / RELUX), 2 = with a residual too; 3 and 4 = the same with the leaky term.
// SECOND: once more over the tiles that the first pass marked; the split warps look at all of a row first.
template <int BN, int EPI, bool SECOND>
__device__ __forceinline__ void run_tiles(const CUtensorMap &tmap_x, const CUtensorMap &tmap_w, const CUtensorMap &tmap_c,
                                          const CUtensorMap &tmap_r, const F32TcParams &p, const FShared<BN> &sh,
                                          const uint32_t tmem_base, const int warp, const int lane) {
  using Cfg = F32Cfg<BN>;
  constexpr int STAGES = Cfg::STAGES;
  constexpr int NUM_ACC = Cfg::NUM_ACC;
  constexpr bool RES = EPI == 2 || EPI == 4, LEAKY = EPI >= 3;
  constexpr int STAGING_AT = FShared<BN>::STAGING_AT, UB_AT = FShared<BN>::UB_AT;
  const uint32_t smem_base = sh.base_u32;
  uint8_t *smem_aligned = sh.base;
  float *x_unscale = reinterpret_cast<float *>(smem_aligned + FShared<BN>::XSCALE_AT);  // [F_SCALE_SLOTS][FBM]
  const uint32_t full_bar = sh.full_bar, split_bar = sh.split_bar, empty_bar = sh.empty_bar, tfull_bar = sh.tfull_bar;
  const uint32_t tempty_bar = sh.tempty_bar, free_bar = sh.free_bar, ready_bar = sh.ready_bar, sempty_bar = sh.sempty_bar;
  volatile int *abort_flag = sh.abort_flag;
  const volatile uint8_t *only = SECOND ? sh.marks : nullptr;
  auto fail = [&](int code) {
    *abort_flag = 1;
    atomicCAS(p.status, 0, code);
  };

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    // One thread runs the role (see the MMA issuer); the other lanes wait at the warp barrier.
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (FTileIter it(p, only); ok && it.valid(p); it.next(p)) {
        const int xb = p.x_batched ? it.b : 0, wb = p.w_batched ? it.b : 0;
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (!mbar_wait(empty_bar + 8 * stage, phase ^ 1, abort_flag, F_WAIT_BUDGET)) {
            fail(MB_DEV_TIMEOUT_PRODUCER);
            ok = false;
            break;
          }
          const uint32_t fb = full_bar + 8 * stage;
          const uint32_t sx = smem_base + stage * Cfg::STAGE_BYTES;
          const uint32_t sw = sx + Cfg::X_BYTES;
          mbar_arrive_expect_tx(fb, Cfg::X_BYTES + Cfg::W_BYTES);
          tma_load_3d(sx, &tmap_x, fb, it.tm * FBM, kb * FKB, xb);  // [32 k][128 m], 512-byte rows
          const int w_row = wb * static_cast<int>(p.Ndim) + it.tn * BN;
          tma_load_3d(sw, &tmap_w, fb, 0, Cfg::WIDE ? 2 * kb : kb, w_row);
          if (Cfg::WIDE) tma_load_3d(sw + Cfg::W_BYTES / 2, &tmap_w, fb, 0, 2 * kb + 1, w_row);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      // (the MMAs have released every stage when the pass ends)
      for (int s = 0; ok && s < STAGES; ++s) {
        if (!mbar_wait(empty_bar + 8 * stage, phase ^ 1, abort_flag, F_WAIT_BUDGET)) {
          fail(MB_DEV_TIMEOUT_PRODUCER);
          ok = false;
        }
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    // The warp runs the role and one of its threads issues.  The tensor pipe queues only a few MMAs, so everything between the
    // last MMA of one K step and the first of the next (commit, barrier poll, descriptor arithmetic) has to fit into the
    // time those queued MMAs take to execute, or the pipe idles: the descriptors are one add per K step and in uniform
    // registers, the common case is unrolled, the next step's barrier is asked ahead.
    {
      constexpr uint32_t idesc = make_idesc(/*c f32*/ 1, /*a f16*/ 0, /*b f16*/ 0, /*a mn*/ false, /*b mn*/ false, FBM, 128);
      constexpr uint32_t idesc_64 = make_idesc(1, 0, 0, false, false, FBM, 64);
      // W (K-major), 16 of k are 32 bytes inside the swizzled row (+2 in the descriptor's address field): rows of 128 bytes, hi
      // then lo; or of 64 bytes, the hi rows before the lo rows.
      const uint64_t w0 = Cfg::WIDE ? make_smem_desc(smem_base + Cfg::X_BYTES, 16, 512, 4)
                                    : make_smem_desc(smem_base + Cfg::X_BYTES, 16, 1024, 2);
      const int k_blocks = p.k_blocks;
      const bool odd_end = (p.K + 15) / 16 % 2 != 0;  // the last step has only 16 of k
      uint32_t stage = 0, phase = 0;
      uint32_t acc_buf = 0, acc_phase = 0;
      uint32_t small_phase = 1;  // (of sempty_bar, which the first tile need not wait for)
      bool ok = true, ready = false;
      int tiles = static_cast<int>((p.batch * p.tiles_m * p.tiles_n - blockIdx.x + gridDim.x - 1) / gridDim.x);
      if (SECOND) {
        tiles = 0;
        for (FTileIter it(p, only); it.valid(p); it.next(p)) ++tiles;
      }
      for (; ok && tiles > 0; --tiles, small_phase ^= 1) {
        if (!mbar_wait_warp(tempty_bar + 8 * acc_buf, acc_phase ^ 1, abort_flag, F_WAIT_BUDGET)) {
          fail(MB_DEV_TIMEOUT_MMA);
          break;
        }
        const uint32_t d_tmem = tmem_base + acc_buf * Cfg::ACC_COLS, s_tmem = (Cfg::WIDE ? d_tmem : tmem_base) + Cfg::SMALL_COL0;
        bool small_free = Cfg::WIDE;
        int owed = 0;              // steps whose small products are still to be issued: the last ones, up to this one
        uint32_t owed_stage = stage;
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!ready && !mbar_wait_warp(split_bar + 8 * stage, phase, abort_flag, F_WAIT_BUDGET)) {
            fail(MB_DEV_TIMEOUT_MMA);
            ok = false;
            break;
          }
          tc_fence_after_sync();
          // whether the next step is there is asked before this one's MMAs are issued and looked at after them
          const uint32_t next = stage + 1 == STAGES ? 0 : stage + 1, next_phase = next == 0 ? phase ^ 1 : phase;
          ready = __all_sync(0xffffffffu, mbar_test_wait(split_bar + 8 * next, next_phase));
          // A (TMEM): lane = pixel, two k per column; hi in the first 16 columns of the stage's slot, lo in the next 16
          const uint32_t a_hi = tmem_base + Cfg::A_COL0 + stage * FKB, a_lo = a_hi + 16;
          const uint64_t w_hi = w0 + stage * (Cfg::STAGE_BYTES >> 4);
          const bool both = !odd_end || kb + 1 < k_blocks;
          if (Cfg::WIDE) {
            mma_f16_ts_elect(d_tmem, a_hi, w_hi, idesc, kb > 0 ? 1u : 0u);
            mma_f16_ts_elect(s_tmem, a_lo, w_hi, idesc_64, 1u);
            if (both) {
              mma_f16_ts_elect(d_tmem, a_hi + 8, w_hi + 2, idesc, 1u);
              mma_f16_ts_elect(s_tmem, a_lo + 8, w_hi + 2, idesc_64, 1u);
            }
            mma_commit_elect(empty_bar + 8 * stage);
          } else if (small_free) {
            mma_f16_ts_elect(d_tmem, a_hi, w_hi, idesc, 1u);
            mma_f16_ts_elect(s_tmem, a_hi, w_hi + 4, idesc, 1u);
            mma_f16_ts_elect(s_tmem, a_lo, w_hi, idesc, 1u);
            if (both) {
              mma_f16_ts_elect(d_tmem, a_hi + 8, w_hi + 2, idesc, 1u);
              mma_f16_ts_elect(s_tmem, a_hi + 8, w_hi + 6, idesc, 1u);
              mma_f16_ts_elect(s_tmem, a_lo + 8, w_hi + 2, idesc, 1u);
            }
            mma_commit_elect(empty_bar + 8 * stage);
          } else {
            mma_f16_ts_elect(d_tmem, a_hi, w_hi, idesc, kb > 0 ? 1u : 0u);
            if (both) mma_f16_ts_elect(d_tmem, a_hi + 8, w_hi + 2, idesc, 1u);
            ++owed;
            small_free = __all_sync(0xffffffffu, mbar_test_wait(sempty_bar, small_phase));
            if (!small_free && (owed == STAGES || kb + 1 == k_blocks)) {
              if (!mbar_wait_warp(sempty_bar, small_phase, abort_flag, F_WAIT_BUDGET)) {
                fail(MB_DEV_TIMEOUT_MMA);
                ok = false;
                break;
              }
              small_free = true;
            }
            if (small_free) {
              tc_fence_after_sync();
#pragma unroll 1
              for (; owed > 0; --owed) {
                const int step = kb + 1 - owed;
                const uint32_t x_hi = tmem_base + Cfg::A_COL0 + owed_stage * FKB, x_lo = x_hi + 16;
                const uint64_t w = w0 + owed_stage * (Cfg::STAGE_BYTES >> 4);
                mma_f16_ts_elect(s_tmem, x_hi, w + 4, idesc, step > 0 ? 1u : 0u);
                mma_f16_ts_elect(s_tmem, x_lo, w, idesc, 1u);
                if (both || owed > 1) {
                  mma_f16_ts_elect(s_tmem, x_hi + 8, w + 6, idesc, 1u);
                  mma_f16_ts_elect(s_tmem, x_lo + 8, w + 2, idesc, 1u);
                }
                mma_commit_elect(empty_bar + 8 * owed_stage);
                if (++owed_stage == STAGES) owed_stage = 0;
              }
            }
          }
          stage = next;
          phase = next_phase;
        }
        if (!ok) break;
        mma_commit_elect(tfull_bar + 8 * acc_buf);
        if (++acc_buf == NUM_ACC) {
          acc_buf = 0;
          acc_phase ^= 1;
        }
      }
    }
    __syncwarp();
  } else if (warp < FIRST_EPI) {
    // ---------------- X split: shared memory -> hi / lo in tensor memory ----------------
    const int quarter = warp & 3;  // the TMEM lanes this warp may touch: 32 * (warp % 4) ...
    const int half = (warp - F_FIRST_X) >> 2;
    const uint32_t a_lane = static_cast<uint32_t>(quarter * 32) << 16;
    int stage = 0, tile = 0;
    uint32_t phase = 0;
    bool ok = true;
    float v[16];
    auto landed = [&](int at) { return reinterpret_cast<const float *>(smem_aligned + at * Cfg::STAGE_BYTES) + quarter * 32 + lane; };
    auto load = [&](int at) {
      const float *xs = landed(at) + half * 16 * FBM;
#pragma unroll
      for (int k = 0; k < 16; ++k) v[k] = xs[k * FBM];
    };
    bool loaded = false;  // v holds this step's values
    for (FTileIter it(p, only); ok && it.valid(p); it.next(p), ++tile) {
      const int64_t m = static_cast<int64_t>(it.tm) * FBM + quarter * 32 + lane;
      const bool inside = m < p.Mdim;
      float scale = 0.f;
      bool known = false;  // every pixel of the warp has its scale
      if (SECOND) {
        const float *x = p.X + it.b * p.x_bs + min(m, p.Mdim - 1);
        float most = 0.f;
#pragma unroll 16
        for (int64_t k = 0; k < p.K; ++k) most = fmaxf(most, f32_finite_abs(mb_load(x + k * p.x_rs)));
        if (most > 0.f) scale = f32_row_scale(most);
        if (half == 0) x_unscale[(tile % F_SCALE_SLOTS) * FBM + quarter * 32 + lane] = f32_row_unscale(scale);
        known = true;
      }
      for (int kb = 0; kb < p.k_blocks; ++kb) {
        if (!loaded) {
          if (!mbar_wait_warp(full_bar + 8 * stage, phase, abort_flag, F_WAIT_BUDGET)) {
            fail(MB_DEV_TIMEOUT_EPILOGUE);
            ok = false;
            break;
          }
          load(stage);
        }
        // The slot's previous contents are dead: the producer refilled this stage only after
        // the MMAs that read the slot had completed.
        tc_fence_after_sync();
        if (!known) {
          // (both warps of a pixel look at all 32 values, and so come to the same scale)
          const float *other = landed(stage) + (half ^ 1) * 16 * FBM;
          // The largest value goes to 2^4 .. 2^5, room for larger ones and smaller ones to come.  Where it stands out, the largest of
          // another eight does, if it can: small values beside a large one keep their bits.
          float most = 0.f, group[4] = {};
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            group[k >> 3] = fmaxf(group[k >> 3], fabsf(v[k]));
            group[2 + (k >> 3)] = fmaxf(group[2 + (k >> 3)], fabsf(other[k * FBM]));
          }
#pragma unroll
          for (int g = 0; g < 4; ++g) most = fmaxf(most, group[g]);
          if (scale == 0.f && most > 0.f) {
            scale = f32_row_scale<4>(most);
#pragma unroll
            for (int g = 0; g < 4; ++g)
              if (group[g] > 0.f) scale = fmaxf(scale, fminf(f32_row_scale<4>(group[g]), f32_row_scale<12>(most)));
          }
          if (half == 0) x_unscale[(tile % F_SCALE_SLOTS) * FBM + quarter * 32 + lane] = f32_row_unscale(scale);
          known = __all_sync(0xffffffffu, scale != 0.f || !inside);
        }
        const uint32_t a_col = tmem_base + a_lane + Cfg::A_COL0 + stage * FKB + half * 8;
        const uint64_t scales = f32_pair(scale, scale);
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) f32_split2(f32_pair(v[2 * j], v[2 * j + 1]), scales, hi[j], lo[j]);
        tmem_st_32x32b_x8(a_col, hi);
        tmem_st_32x32b_x8(a_col + 16, lo);
        // the next step's values, if they have landed, are on their way while this step's reach tensor memory
        const int done = stage;
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
        loaded = __all_sync(0xffffffffu, mbar_test_wait(full_bar + 8 * stage, phase));
        if (loaded) load(stage);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(split_bar + 8 * done);
      }
    }
  } else if (warp < FIRST_STORE) {
    // ---------------- epilogue ----------------
    const int quarter = warp & 3;
    const int set = (warp - FIRST_EPI) >> 2;  // 0, 1: which half of the columns
    constexpr int CHUNKS = BN / 16 / 2;              // 16-column chunks per warp
    // The activation as clamp + negative-slope term, with the choice made once: a branch
    // per value costs more than the arithmetic (few warps are there to hide its latency).
    //   NOOP: [-inf, inf], 0   RELU: [0, inf], 0   RELUX: [0, max_limit], 0   LEAKYRELU: [0, inf], coef
    const float act_lo = p.act == 0 ? -INFINITY : 0.f;
    const float act_hi = p.act == 2 ? p.max_limit : INFINITY;
    const float act_slope = p.act == 6 ? p.coef : 0.f;
    const int64_t Ndim = p.Ndim;
    const int c_tma = p.c_tma;
    // Result buffers of a set: [buffer][channel j][128 pixels]; a lane's 16 accesses of a chunk go to 16 different rows, a
    // warp's access to one row covers all 32 banks.
    float *stage_f = reinterpret_cast<float *>(smem_aligned + STAGING_AT) + set * (F_BUFS * 16 * FBM);
    // of two channels each: 1 / scale, bias
    float4 *table = reinterpret_cast<float4 *>(smem_aligned + UB_AT) + (warp - FIRST_EPI) * (BN / 4);
    const uint32_t my_free_bar = free_bar + 8 * (set * F_BUFS), my_ready_bar = ready_bar + 8 * (set * F_BUFS);
    int acc_buf = 0;
    uint32_t acc_phase = 0;
    int tile = 0;
    int q = 0;        // chunks of this set so far
    bool ok = true;
    for (FTileIter it(p, only); ok && it.valid(p); it.next(p), ++tile) {
      const int64_t m = static_cast<int64_t>(it.tm) * FBM + quarter * 32 + lane;
      const bool m_ok = m < p.Mdim;
      const int64_t n_first = static_cast<int64_t>(it.tn) * BN + set * (BN / 2);
      // the warp's table of (1 / scale, bias)
      constexpr int PER = BN / 64;  // channels per lane
      float u[PER], b[PER];
#pragma unroll
      for (int j = 0; j < PER; ++j) {
        const int64_t n = n_first + j * 32 + lane;
        u[j] = n < Ndim ? mb_load(p.w_unscale + (p.w_batched ? it.b * Ndim : 0) + n) : 0.f;
        b[j] = EPI != 0 && p.bias != nullptr && n < Ndim ? mb_load(p.bias + n) : 0.f;
      }
      if (!mbar_wait_warp(tfull_bar + 8 * acc_buf, acc_phase, abort_flag, F_WAIT_BUDGET)) {
        fail(MB_DEV_TIMEOUT_EPILOGUE);
        break;
      }
      tc_fence_after_sync();
      const uint32_t lanes = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
      const uint32_t tbase = lanes + acc_buf * Cfg::ACC_COLS + set * (BN / 2);
      const uint32_t sbase = (Cfg::WIDE ? tbase : lanes + set * (BN / 2)) + Cfg::SMALL_COL0;
      uint32_t r[16], r2[16];
      if (!Cfg::WIDE) {
        // the small products join the large ones (the first chunk's in registers), and leave their accumulator to the next tile
#pragma unroll
        for (int i = CHUNKS - 1; i >= 0; --i) {
          tmem_ld_32x32b_x16(tbase + i * 16, r);
          tmem_ld_32x32b_x16(sbase + i * 16, r2);
          tmem_ld_wait_x16(r);
          tmem_ld_wait_x16(r2);
#pragma unroll
          for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(fmaf(__uint_as_float(r2[j]), F32_LO, __uint_as_float(r[j])));
          if (i > 0) tmem_st_32x32b_x16(tbase + i * 16, r);
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(sempty_bar);
        tmem_st_wait();
      }
      auto load = [&](int i) {
        tmem_ld_32x32b_x16(tbase + i * 16, r);
        if (Cfg::WIDE) tmem_ld_32x32b_x16(sbase + i * 16, r2);
      };
      if (Cfg::WIDE) load(0);
#pragma unroll
      for (int j = 0; j < PER; ++j) {
        float *entry = reinterpret_cast<float *>(table + j * 16 + (lane >> 1)) + (lane & 1);
        entry[0] = u[j];
        entry[2] = b[j];
      }
      const float unscale = x_unscale[(tile % F_SCALE_SLOTS) * FBM + quarter * 32 + lane];
      const uint64_t unscales = f32_pair(unscale, unscale);
      __syncwarp();
      float *c = p.C + it.b * p.c_batch_stride + m;
#pragma unroll
      for (int i = 0; i < CHUNKS; ++i, ++q) {
        if (Cfg::WIDE || i > 0) tmem_ld_wait_x16(r);
        if (Cfg::WIDE) tmem_ld_wait_x16(r2);
        float a[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          a[j] = Cfg::WIDE ? fmaf(__uint_as_float(r2[j]), F32_LO, __uint_as_float(r[j])) : __uint_as_float(r[j]);
        }
        if (i + 1 < CHUNKS) load(i + 1);
        if (i == CHUNKS - 1) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(tempty_bar + 8 * acc_buf);
        }
        const int64_t n0 = n_first + i * 16;
        float *buf = stage_f + (q & 3) * (16 * FBM) + quarter * 32 + lane;
        if (c_tma && !mbar_wait_warp(my_free_bar + 8 * (q & 3), (q >> 2) & 1, abort_flag, F_WAIT_BUDGET)) {
          fail(MB_DEV_TIMEOUT_EPILOGUE);
          ok = false;
          break;
        }
        if (RES && !c_tma) {
          // (from clamped addresses instead of guarded by branches; each thread reads back what it writes here)
          const float *res = p.residual + it.b * p.c_batch_stride + min(m, p.Mdim - 1);
#pragma unroll
          for (int j = 0; j < 16; ++j) buf[j * FBM] = mb_load(res + min(n0 + j, Ndim - 1) * p.c_row_stride);
        }
        uint64_t z2 = 0;
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          const float4 t = table[i * 8 + j / 2];
          // (the products with powers of two are exact, so the sum with the bias rounds once)
          uint64_t x2 = f32_mul2(f32_pair(a[j], a[j + 1]), unscales);
          x2 = EPI == 0 ? f32_mul2(x2, f32_pair(t.x, t.y)) : f32_fma2(x2, f32_pair(t.x, t.y), f32_pair(t.z, t.w));
          z2 = f32_fma2(x2, 0, z2);
          const float2 both = f32_parts(x2);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float x = h == 0 ? both.x : both.y;
            if (EPI != 0) {
              // (acc + bias) + residual: the rounding order of a convolution followed by a sum
              if (RES) x += buf[(j + h) * FBM];
              const float neg = LEAKY ? fminf(x, 0.f) * act_slope : 0.f;
              x = fminf(fmaxf(x, act_lo), act_hi);
              if (LEAKY) x += neg;
            }
            a[j + h] = x;
          }
        }
        const float2 z = f32_parts(z2);
        if (z.x + z.y != 0.f) {
          sh.again[SECOND] = 1;
          sh.marks[SECOND * MARKS + (SECOND ? it.nth : tile) % MARKS] = 1;
#pragma unroll
          for (int j = 0; SECOND && j < 16; ++j) a[j] = __uint_as_float(F32_AGAIN);
        }
        if (c_tma) {
#pragma unroll
          for (int j = 0; j < 16; ++j) buf[j * FBM] = a[j];
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) mbar_arrive(my_ready_bar + 8 * (q & 3));
        } else if (m_ok) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (n0 + j < Ndim) c[(n0 + j) * p.c_row_stride] = a[j];
        }
      }
      __syncwarp();  // (the table is written again)
      if (++acc_buf == NUM_ACC) {
        acc_buf = 0;
        acc_phase ^= 1;
      }
    }
  } else if (p.c_tma && lane == 0) {
    // ---------------- result copies of a set: one thread ----------------
    // A buffer leaves by a single TMA store of 512-byte rows (stores of 128-byte rows, one per warp, ran at half the rate), and
    // the residual of the chunk four further on comes into it as soon as that store has read it.  (Issuing a copy takes its
    // thread some 200 cycles: with the epilogue's own warps taking turns at it, each chunk waited for the one before.)
    constexpr int CHUNKS = BN / 16 / 2;
    const int set = warp - FIRST_STORE;
    const uint32_t bufs = smem_base + STAGING_AT + set * (F_BUFS * Cfg::BUF_BYTES);
    const uint32_t my_free_bar = free_bar + 8 * (set * F_BUFS), my_ready_bar = ready_bar + 8 * (set * F_BUFS);
    FTileIter rt(p, only);  // where the next chunk to be given out lies
    int rc = 0, rq = 0;
    auto give = [&]() {
      if (RES) {
        if (!rt.valid(p)) return;
        mbar_arrive_expect_tx(my_free_bar + 8 * (rq & 3), Cfg::BUF_BYTES);
        tma_load_3d(bufs + (rq & 3) * Cfg::BUF_BYTES, &tmap_r, my_free_bar + 8 * (rq & 3), rt.tm * FBM, rt.tn * BN + set * (BN / 2) + rc * 16,
                    rt.b);
        if (++rc == CHUNKS) {
          rc = 0;
          rt.next(p);
        }
      } else {
        mbar_arrive(my_free_bar + 8 * (rq & 3));
      }
      ++rq;
    };
    for (int i = 0; i < F_BUFS; ++i) give();
    int q = 0;
    bool ok = true;
    for (FTileIter it(p, only); ok && it.valid(p); it.next(p)) {
      const int n_first = it.tn * BN + set * (BN / 2);
      for (int i = 0; i < CHUNKS; ++i, ++q) {
        if (!mbar_wait(my_ready_bar + 8 * (q & 3), (q >> 2) & 1, abort_flag, F_WAIT_BUDGET)) {
          fail(MB_DEV_TIMEOUT_EPILOGUE);
          ok = false;
          break;
        }
        if (n_first + i * 16 < p.Ndim) tma_store_3d(&tmap_c, bufs + (q & 3) * Cfg::BUF_BYTES, it.tm * FBM, n_first + i * 16, it.b);
        bulk_commit_group();
        if (q > 0) {
          bulk_wait_group_read<1>();  // the store before has read its buffer
          give();
        }
      }
    }
    bulk_wait_group<0>();  // staging must outlive the stores' reads
  }
}

template <int BN, int EPI>
__global__ void __launch_bounds__(F_THREADS, 1)
gemm_f32_pairs_kernel(const __grid_constant__ CUtensorMap tmap_x,
                   const __grid_constant__ CUtensorMap tmap_w,
                   const __grid_constant__ CUtensorMap tmap_c, const __grid_constant__ CUtensorMap tmap_r,
                   const __grid_constant__ F32TcParams p) {
  using Cfg = F32Cfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  const FShared<BN> sh(smem_raw);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  mb_grid_dep_launch();  // the kernel behind this one may start its own prologue

  if (threadIdx.x == 0) {
    prefetch_tensormap(&tmap_x);
    prefetch_tensormap(&tmap_w);
    if (p.c_tma) prefetch_tensormap(&tmap_c);
    if ((EPI == 2 || EPI == 4) && p.c_tma) prefetch_tensormap(&tmap_r);
    sh.init_barriers();
    *sh.abort_flag = 0;
    sh.again[0] = sh.again[1] = 0;
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(sh.tmem_slot), Cfg::TMEM_COLS);
    tmem_relinquish();
    for (int i = lane; i < 2 * MARKS; i += 32) sh.marks[i] = 0;
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *sh.tmem_slot;
  // everything above touched only this CTA's shared and tensor memory; from here on the roles read
  // and write global memory, which the kernel in front of this one may still be producing
  mb_grid_dep_wait();

  run_tiles<BN, EPI, false>(tmap_x, tmap_w, tmap_c, tmap_r, p, sh, tmem_base, warp, lane);
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (sh.again[0] != 0 && *sh.abort_flag == 0) {
    // (no copy, MMA or arrival of the first pass is on its way any more)
    if (threadIdx.x == 0) {
      for (int i = 0; i < Cfg::BARRIERS; ++i) mbar_inval(sh.full_bar + 8 * i);
      sh.init_barriers();
    }
    __syncthreads();
    run_tiles<BN, EPI, true>(tmap_x, tmap_w, tmap_c, tmap_r, p, sh, tmem_base, warp, lane);
    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
  }
  if (*sh.abort_flag != 0) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  if (sh.again[1] != 0 && *sh.abort_flag == 0) {
    asm volatile("fence.proxy.async;" ::: "memory");  // (the results were written by TMA stores, which have completed)
    for (FTileIter it(p, sh.marks + MARKS); it.valid(p); it.next(p)) tile_again(p, it.tm * FBM, it.tn * BN, BN, it.b);
  }
}

// 3-D fp32 tensor map: dims {inner, rows, batch} in elements, no swizzle, zero fill.
// Every stride must be a multiple of 16 bytes, that of a batch dimension of extent 1 too:
// callers pass row stride x rows there.
int make_map_f32(mb_context *ctx, CUtensorMap *map, const void *base, uint64_t inner, uint64_t rows,
                 uint64_t batch, uint64_t row_stride_elems, uint64_t batch_stride_elems,
                 uint32_t box_inner, uint32_t box_rows) {
  const cuuint64_t dims[3] = {inner, rows, batch};
  const cuuint64_t strides[2] = {row_stride_elems * 4, batch_stride_elems * 4};
  const cuuint32_t box[3] = {box_inner, box_rows, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = reinterpret_cast<EncodeTiledFn>(ctx->encode_tiled)(
      map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void *>(base), dims, strides, box, estr,
      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return mb_fail(ctx, MB_RUNTIME_ERROR, "cuTensorMapEncodeTiled (fp32) failed (%d)", static_cast<int>(r));
  return MB_SUCCESS;
}

// The split W as f32_presplit_kernel lays it out: boxes of bn rows' 128 bytes of one step (64 rows: of their 64 bytes of hi or lo).
int make_map_split(mb_context *ctx, CUtensorMap *map, const void *base, uint64_t k_blocks, uint64_t rows, int bn) {
  const uint32_t per = bn == 64 ? 2 : 1, halves = 64 / per;
  const cuuint64_t dims[3] = {halves, k_blocks * per, rows};
  const cuuint64_t strides[2] = {halves * 2, k_blocks * 128};
  const cuuint32_t box[3] = {halves, 1, static_cast<cuuint32_t>(bn)};
  const cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = reinterpret_cast<EncodeTiledFn>(ctx->encode_tiled)(
      map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void *>(base), dims, strides, box, estr,
      CU_TENSOR_MAP_INTERLEAVE_NONE, bn == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return mb_fail(ctx, MB_RUNTIME_ERROR, "cuTensorMapEncodeTiled (split fp32) failed (%d)", static_cast<int>(r));
  return MB_SUCCESS;
}

template <int BN, int EPI>
int launch_f32(mb_context *ctx, const CUtensorMap &tx, const CUtensorMap &tw, const CUtensorMap &tc, const CUtensorMap &tr,
               F32TcParams &p) {
  using Cfg = F32Cfg<BN>;
  auto kern = gemm_f32_pairs_kernel<BN, EPI>;
  constexpr uint32_t bit = 1u << (EPI * 2 + (BN == 128 ? 1 : 0));
  if (!(ctx->f32_pairs_attr_mask & bit)) {
    MB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
    ctx->f32_pairs_attr_mask |= bit;
  }
  const int64_t total = p.batch * p.tiles_m * p.tiles_n;
  const int grid = static_cast<int>(total < ctx->num_sms ? total : ctx->num_sms);
  p.step_n = grid % p.tiles_n;
  p.step_m = (grid / p.tiles_n) % p.tiles_m;
  p.step_b = (grid / p.tiles_n) / p.tiles_m;
  MB_CUDA(ctx, mb_launch_chained(ctx, kern, dim3(grid), dim3(F_THREADS), Cfg::SMEM_BYTES, tx, tw, tc, tr, p));
  MB_CUDA(ctx, cudaGetLastError());
  ctx->launches++;
  ctx->launches_tc++;
  return MB_SUCCESS;
}

}  // namespace

// Whether the kernel pays: from about 60 steps per CTA on, less what the split of W costs beyond its launch, two passes over W
// (32 images of 512 -> 256 channels at 28 x 28, 64 steps: 44.6 us as tf32 pairs, 40.4 here; 256 -> 1024 at 14 x 14, 32 steps: 26.2
// and 28.4; 24 of 736 x 176 x 384, 12 steps and 27 MB of W: 19.6 and 27.9).
bool mb_gemm_f32_pairs_pays(const mb_context *ctx, int64_t batch, int64_t Mdim, int64_t Ndim, int64_t K, int w_batched) {
  if (ctx->f32_pairs != 0) return ctx->f32_pairs == 2;
  const int64_t tiles = batch * ceil_div64(Mdim, FBM) * ceil_div64(Ndim, Ndim > 64 ? 128 : 64);
  const int64_t steps = ceil_div64(tiles, ctx->num_sms) * ceil_div64(K, FKB);
  return (steps - 60) * 400 > (w_batched ? batch : 1) * Ndim * K * 8 / 1700;
}

// *done is false where nothing was launched: the residual lies in C, or there is no room for the split W (see mb_weight_scratch).
int mb_gemm_f32_pairs_launch(mb_context *ctx, const float *X, const float *W, const float *bias, float *C,
                          int64_t batch, int64_t Mdim, int64_t Ndim, int64_t K, int64_t x_row_stride,
                          int64_t x_batch_stride, int64_t w_row_stride, int64_t w_batch_stride,
                          int64_t c_row_stride, int64_t c_batch_stride, int act, float max_limit,
                          float coef, const float *residual, bool *done) {
  *done = false;
  // A result that is worked out again needs its residual once more, which must not lie where the first one was stored.
  if (mb_ranges_meet(residual, C, ((batch - 1) * c_batch_stride + (Ndim - 1) * c_row_stride + Mdim) * 4)) return MB_SUCCESS;
  const int BN = Ndim > 64 ? 128 : 64;
  F32TcParams p = {};
  p.X = X; p.W = W;
  p.Mdim = Mdim; p.Ndim = Ndim; p.K = K; p.batch = batch;
  p.x_rs = x_row_stride; p.x_bs = x_batch_stride; p.w_rs = w_row_stride; p.w_bs = w_batch_stride;
  p.tiles_m = static_cast<int>(ceil_div64(Mdim, FBM));
  p.tiles_n = static_cast<int>(ceil_div64(Ndim, BN));
  p.k_blocks = static_cast<int>(ceil_div64(K, FKB));
  p.x_batched = x_batch_stride != 0; p.w_batched = w_batch_stride != 0;
  p.bias = bias; p.residual = residual; p.act = act; p.max_limit = max_limit; p.coef = coef;
  p.C = C; p.c_row_stride = c_row_stride; p.c_batch_stride = c_batch_stride;
  p.status = ctx->dev_status;
  CUtensorMap tx, tw, tc, tr;
  memset(&tc, 0, sizeof(tc));
  memset(&tr, 0, sizeof(tr));
  MB_RETURN_IF_ERROR(make_map_f32(ctx, &tx, X, Mdim, K, p.x_batched ? batch : 1, x_row_stride,
                                  p.x_batched ? x_batch_stride : x_row_stride * K, FBM, FKB));
  p.c_tma = ((reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(residual)) & 15u) == 0 && c_row_stride % 4 == 0 &&
            c_batch_stride % 4 == 0 && Ndim >= 16;
  if (p.c_tma) {
    MB_RETURN_IF_ERROR(make_map_f32(ctx, &tc, C, Mdim, Ndim, batch, c_row_stride,
                                    batch > 1 ? c_batch_stride : c_row_stride * Ndim, FBM, 16));
    if (residual != nullptr)
      MB_RETURN_IF_ERROR(make_map_f32(ctx, &tr, residual, Mdim, Ndim, batch, c_row_stride,
                                      batch > 1 ? c_batch_stride : c_row_stride * Ndim, FBM, 16));
  }
  const int64_t w_rows = Ndim * (p.w_batched ? batch : 1);
  const size_t split_bytes = static_cast<size_t>(w_rows) * p.k_blocks * 128;
  if (w_rows >= (1ll << 31) || split_bytes > WEIGHT_SCRATCH_BYTES) return MB_SUCCESS;
  uint8_t *split = nullptr;
  MB_RETURN_IF_ERROR(mb_weight_scratch(ctx, align_up(split_bytes, 256) + w_rows * 4, reinterpret_cast<void **>(&split)));
  if (split == nullptr) return MB_SUCCESS;
  float *unscale = reinterpret_cast<float *>(split + align_up(split_bytes, 256));
  int group = 8;
  while (group < 256 && group * 4 < p.k_blocks * 8) group *= 2;
  MB_RETURN_IF_ERROR(make_map_split(ctx, &tw, split, p.k_blocks, w_rows, BN));
  MB_CUDA(ctx, mb_launch_chained(ctx, f32_presplit_kernel, dim3(static_cast<unsigned>(ceil_div64(w_rows, 256 / group))), dim3(256), 0,
                                 W, split, unscale, w_rows, K, Ndim, w_row_stride, w_batch_stride, p.k_blocks, group));
  ctx->launches++;
  p.w_unscale = unscale;
  *done = true;
#define MB_F32_PAIRS(EPI_) \
  return BN == 128 ? launch_f32<128, EPI_>(ctx, tx, tw, tc, tr, p) : launch_f32<64, EPI_>(ctx, tx, tw, tc, tr, p);
  if (bias == nullptr && residual == nullptr && act == 0) MB_F32_PAIRS(0)
  if (act != 6 && residual == nullptr) MB_F32_PAIRS(1)
  if (act != 6) MB_F32_PAIRS(2)
  if (residual == nullptr) MB_F32_PAIRS(3)
  MB_F32_PAIRS(4)
#undef MB_F32_PAIRS
}
