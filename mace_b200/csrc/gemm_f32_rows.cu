// fp32 GEMM on tcgen05 (kind::f16 on pairs of halves, see f32_split.cuh) for operands that both have their depth contiguous:
//     C[b][n][m] = act(bias[n] + sum_k X[b][m][k] * W[b][n][k])
// What it serves: MatMul / Gemm with a transposed right-hand side (mace/ops/arm/base/gemm.cc:520-683): attention scores,
// products with a weight matrix stored by output.
//
// A step is 32 of the depth of 128 rows of X and BN of W: rows of 128 bytes, by TMA in the 128-byte swizzle, which eight warps
// rewrite in place as 32 halves of hi and 32 of lo.  Both operands of the MMA then lie in shared memory, so that all of
// tensor memory is there for accumulators: the large products hi * hi in one, cut off once per 16 of k, hi * lo + lo * hi
// in another, both twice.  Every `run` steps the result warps take them and carry the sums on in registers: with one step the
// error is 1.16e-7, with three 1.76e-7 (2-norm against float64; the self-fetching kernel on tf32: 1.37e-7, 2.06e-7).  A run's rows
// have scales of their own, for which the warps that split look at all of its steps first.  (With a scale per tile, from its first
// step, rows that grew beyond 2^14 times that were worked out again by FMAs.)
//
// What bounds it: launch, first copies and results for few steps; else the split, whose warps wait for a run, look at it, split
// it step by step and hand each on (1860 cycles per step of 128 x 128 in runs of three, 2150 in runs of one).
// Against the kernel whose warps fetch X from where it lies (a lane a row: 32 lines per instruction): see cost_of.
//
// Roles: warp 0 copies, warp 1 MMAs, 8 warps split, 8 or 16 results (32 columns of n per thread).  Persistent over the tiles.
#include <algorithm>

#include "f32_split.cuh"
#include "gemm_f32_gather.cuh"
#include "sm100_ptx.cuh"

int mb_make_map_w_f32(mb_context *ctx, CUtensorMap *map, const float *W, int64_t K, int64_t N, int64_t batch, int64_t w_ns,
                      int64_t w_bs, int bn);

namespace {

using namespace sm100;

constexpr int BM = 128, KB = 32;
constexpr int FIRST_SPLIT = 2, SPLIT_WARPS = 8, FIRST_OUT = FIRST_SPLIT + SPLIT_WARPS;
constexpr int MAX_RUN = 3;
constexpr int SCALE_SLOTS = 16;  // runs: the split is at most STAGES ahead of the MMAs, these two of the results
constexpr long long WAIT_BUDGET = 1ll << 31;  // ~1 s of SM clocks per wait

// Where four k (chunk 0 .. 7 of a step) of a row's hi half lie: in the first 64 of its 128 bytes, in the tensor core's 128-byte
// swizzle.  Its lo half lies at 64 ^ that.
__device__ __forceinline__ uint32_t hi_at(int row, int chunk) {
  return static_cast<uint32_t>(row * 128 + (((chunk >> 1) ^ (row & 7)) << 4) + (chunk & 1) * 8);
}

struct Params {
  const float *X, *W, *bias;
  float *C;
  int M, N, K, batch;
  int64_t x_ms, x_bs, w_ns, w_bs, c_ns, c_bs;
  int tiles_m, tiles_n, k_blocks, run;
  int act;
  float max_limit, coef;
  int *status;
};

template <int BN>
struct Cfg {
  static constexpr int ROWS = BM + BN, STAGE_BYTES = ROWS * 128;
  static constexpr int STAGES = BN == 128 ? 6 : 8;  // (two runs and more)
  static_assert(STAGES >= MAX_RUN && STAGES + 3 <= SCALE_SLOTS, "a run is split when all of it has landed");
  static constexpr int OUT_WARPS = BN / 8, THREADS = (FIRST_OUT + OUT_WARPS) * 32;
  static constexpr int ACC_COLS = 2 * BN, ACCS = 2, TMEM_COLS = ACCS * ACC_COLS;
  static constexpr int SCALE_AT = STAGES * STAGE_BYTES, BAR_AT = SCALE_AT + SCALE_SLOTS * ROWS * 4;
  static constexpr int SMEM_BYTES = BAR_AT + 256 + 1024 /*align*/;
  static_assert(8 * (3 * STAGES + 2 * ACCS) + 16 <= 256 && SMEM_BYTES <= 227 * 1024, "shared memory");
};

// Results of a tile that are not finite, by fp32 FMAs.
__device__ __noinline__ void tile_again(const Params &p, int m0, int n0, int bn, int b) {
  for (int i = threadIdx.x; i < BM * bn; i += blockDim.x) {
    // (a warp: one n, 32 of m)
    const int m_first = m0 + (i & (BM - 32)), n = n0 + i / BM, m = m_first + (i & 31);
    float *c = p.C + b * p.c_bs + n * p.c_ns + m;
    f32_each_again(m < p.M && n < p.N && __float_as_uint(*c) == F32_AGAIN, [&](int lane) {
      float sum = f32_warp_dot(p.X + b * p.x_bs + (m_first + lane) * p.x_ms, 1, p.W + b * p.w_bs + n * p.w_ns, p.K);
      if ((i & 31) != lane) return;
      if (p.bias != nullptr) sum += p.bias[n];
      *c = mb_activate(sum, p.act, p.max_limit, p.coef);
    });
  }
}

template <int BN>
__global__ void __launch_bounds__(Cfg<BN>::THREADS, 1)
gemm_f32_rows_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                     const __grid_constant__ Params p) {
  using C = Cfg<BN>;
  constexpr int STAGES = C::STAGES;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t *smem = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t landed_bar = smem_base + C::BAR_AT, full_bar = landed_bar + 8 * STAGES, empty_bar = full_bar + 8 * STAGES;
  const uint32_t tfull_bar = empty_bar + 8 * STAGES, tempty_bar = tfull_bar + 8 * C::ACCS;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + C::BAR_AT + 8 * (3 * STAGES + 2 * C::ACCS));
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  volatile int *again = abort_flag + 1;
  float *unscales = reinterpret_cast<float *>(smem + C::SCALE_AT);  // [SCALE_SLOTS][ROWS]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  mb_grid_dep_launch();
  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_x);
    prefetch_tensormap(&map_w);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(landed_bar + 8 * s, 1);
      mbar_init(full_bar + 8 * s, SPLIT_WARPS);
      mbar_init(empty_bar + 8 * s, 1);
    }
    for (int s = 0; s < C::ACCS; ++s) {
      mbar_init(tfull_bar + 8 * s, 1);
      mbar_init(tempty_bar + 8 * s, C::OUT_WARPS);
    }
    *abort_flag = 0;
    *again = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), C::TMEM_COLS);
    tmem_relinquish();
  }
  auto fail = [&](int code) {
    *abort_flag = 1;
    atomicCAS(p.status, 0, code);
  };
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  mb_grid_dep_wait();
  const int tiles = p.tiles_m * p.tiles_n * p.batch, k_blocks = p.k_blocks;

  if (warp == 0) {
    // ---- copies ----
    if (lane == 0) {
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
        const int tn = t % p.tiles_n, q = t / p.tiles_n, tm = q % p.tiles_m, b = q / p.tiles_m;
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!mbar_wait(empty_bar + 8 * stage, phase ^ 1, abort_flag, WAIT_BUDGET)) {
            fail(MB_DEV_TIMEOUT_PRODUCER);
            ok = false;
            break;
          }
          const uint32_t at = smem_base + stage * C::STAGE_BYTES, bar = landed_bar + 8 * stage;
          mbar_arrive_expect_tx(bar, C::STAGE_BYTES);
          tma_load_3d(at, &map_x, bar, kb * KB, tm * BM, p.x_bs != 0 ? b : 0);
          tma_load_3d(at + BM * 128, &map_w, bar, kb * KB, tn * BN, p.w_bs != 0 ? b : 0);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---- MMAs ----
    constexpr uint32_t idesc = make_idesc(/*c f32*/ 1, /*a f16*/ 0, /*b f16*/ 0, false, false, BM, BN);
    const uint64_t first = make_smem_desc(smem_base, 16, 1024, 2);
    uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0;
    bool ok = true, ready = false;
    for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
      uint32_t d = 0;
      int left = 0;  // steps of this run still to come
      for (int kb = 0; kb < k_blocks; ++kb) {
        uint32_t add = 1u;
        if (left == 0) {
          if (!mbar_wait_warp(tempty_bar + 8 * acc, acc_phase ^ 1, abort_flag, WAIT_BUDGET)) {
            fail(MB_DEV_TIMEOUT_MMA);
            ok = false;
            break;
          }
          d = tmem + acc * C::ACC_COLS;
          left = min(p.run, k_blocks - kb);
          add = 0u;
        }
        if (!ready && !mbar_wait_warp(full_bar + 8 * stage, phase, abort_flag, WAIT_BUDGET)) {
          fail(MB_DEV_TIMEOUT_MMA);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const uint32_t next = stage + 1 == STAGES ? 0 : stage + 1, next_phase = next == 0 ? phase ^ 1 : phase;
        ready = __all_sync(0xffffffffu, mbar_test_wait(full_bar + 8 * next, next_phase));
        const uint64_t x = first + stage * (C::STAGE_BYTES >> 4), w = x + (BM * 128 >> 4);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          mma_f16_ss_elect(d, x + 2 * j, w + 2 * j, idesc, j > 0 ? 1u : add);
          mma_f16_ss_elect(d + BN, x + 2 * j, w + 4 + 2 * j, idesc, j > 0 ? 1u : add);
          mma_f16_ss_elect(d + BN, x + 4 + 2 * j, w + 2 * j, idesc, 1u);
        }
        mma_commit_elect(empty_bar + 8 * stage);
        stage = next;
        phase = next_phase;
        if (--left == 0) {
          mma_commit_elect(tfull_bar + 8 * acc);
          if ((acc ^= 1) == 0) acc_phase ^= 1;
        }
      }
    }
    __syncwarp();
  } else if (warp < FIRST_OUT) {
    // ---- split: a row of 32 fp32 values becomes one of 32 hi and 32 lo halves, in place; eight lanes per row ----
    constexpr int CH = C::ROWS / 32;  // rows per thread, a chunk of four k of each
    const int r0 = (warp - FIRST_SPLIT) * 4 + (lane >> 3);  // row of chunk i: i * 32 + r0
    const int chunk = (lane & 7) ^ (r0 & 7);                // (TMA lays the rows out in the 128-byte swizzle)
    const bool swap = ((lane >> 3) & 1) != 0;               // of two rows that share their banks, one writes lo first
    uint32_t stage = 0, phase = 0, run = 0;
    bool ok = true;
    float4 v[CH];
    auto load = [&](uint32_t at) {
      const uint8_t *rows = smem + at * C::STAGE_BYTES + r0 * 128 + (lane & 7) * 16;
#pragma unroll
      for (int i = 0; i < CH; ++i) v[i] = *reinterpret_cast<const float4 *>(rows + i * 4096);
    };
    for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
      for (int kb = 0; ok && kb < k_blocks; kb += p.run, ++run) {
        // the largest values of the run's rows, its first step last, whose values stay: the eight lanes of a row halve their rows
        // between them and end with one each
        const int steps = min(p.run, k_blocks - kb);
        float most[8] = {};
        for (int i = steps - 1; i >= 0; --i) {
          const uint32_t at = stage + i, wrapped = at >= static_cast<uint32_t>(STAGES) ? 1u : 0u;
          if (!mbar_wait_warp(landed_bar + 8 * (at - wrapped * STAGES), phase ^ wrapped, abort_flag, WAIT_BUDGET)) {
            fail(MB_DEV_TIMEOUT_EPILOGUE);
            ok = false;
            break;
          }
          load(at - wrapped * STAGES);
#pragma unroll
          for (int j = 0; j < CH; ++j) most[j] = fmaxf(fmaxf(most[j], fmaxf(fabsf(v[j].x), fabsf(v[j].y))), fmaxf(fabsf(v[j].z), fabsf(v[j].w)));
        }
        if (!ok) break;
#pragma unroll
        for (int d = 4; d > 0; d /= 2)
#pragma unroll
          for (int i = 0; i < d; ++i) {
            const bool up = (lane & d) != 0;
            most[i] = fmaxf(up ? most[i + d] : most[i], __shfl_xor_sync(0xffffffffu, up ? most[i] : most[i + d], d));
          }
        const float mine = most[0] > 0.f ? f32_row_scale(most[0]) : 0.f;
        if ((lane & 7) < CH) unscales[(run % SCALE_SLOTS) * C::ROWS + (lane & 7) * 32 + r0] = f32_row_unscale(mine);
        for (int i = 0; i < steps; ++i) {
          if (i > 0) load(stage);
          __syncwarp();  // (a row is rewritten by the warp that read it)
          uint8_t *rows = smem + stage * C::STAGE_BYTES;
#pragma unroll
          for (int j = 0; j < CH; ++j) {
            const float scale = __shfl_sync(0xffffffffu, mine, (lane & 24) + j);
            const uint64_t scales = f32_pair(scale, scale);
            uint2 hi, lo;
            f32_split2(f32_pair(v[j].x, v[j].y), scales, hi.x, lo.x);
            f32_split2(f32_pair(v[j].z, v[j].w), scales, hi.y, lo.y);
            const uint32_t at = hi_at(j * 32 + r0, chunk);
            *reinterpret_cast<uint2 *>(rows + (swap ? at ^ 64 : at)) = swap ? lo : hi;
            *reinterpret_cast<uint2 *>(rows + (swap ? at : at ^ 64)) = swap ? hi : lo;
          }
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) mbar_arrive(full_bar + 8 * stage);
          if (++stage == static_cast<uint32_t>(STAGES)) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else {
    // ---- results: a lane per m, 32 of n per thread ----
    const int quarter = warp & 3, c0 = (warp - FIRST_OUT) / 4 * 32;
    const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
    uint32_t acc = 0, acc_phase = 0, run = 0;
    bool ok = true;
    for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
      const int tn = t % p.tiles_n, q = t / p.tiles_n, tm = q % p.tiles_m, b = q / p.tiles_m;
      const int m = tm * BM + quarter * 32 + lane, n0 = tn * BN + c0;
      const float b_mine = p.bias != nullptr && n0 + lane < p.N ? mb_load(p.bias + n0 + lane) : 0.f;
      uint64_t sums[16];  // of two channels each
#pragma unroll
      for (int j = 0; j < 16; ++j) sums[j] = 0;
#pragma unroll 1
      for (int kb = 0; kb < k_blocks; kb += p.run, ++run) {
        if (!mbar_wait_warp(tfull_bar + 8 * acc, acc_phase, abort_flag, WAIT_BUDGET)) {
          fail(MB_DEV_TIMEOUT_EPILOGUE);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const uint32_t src = tmem + lanes + acc * C::ACC_COLS + c0;
        const float *slot = unscales + (run % SCALE_SLOTS) * C::ROWS;
        const uint64_t unscale = f32_pair(slot[quarter * 32 + lane], slot[quarter * 32 + lane]);
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
          uint32_t r[8], s[8];
          tmem_ld_32x32b_x8(src + j, r);
          tmem_ld_32x32b_x8(src + BN + j, s);
          tmem_ld_wait_x8(r);
          tmem_ld_wait_x8(s);
#pragma unroll
          for (int k = 0; k < 8; k += 4) {
            const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(slot + BM + c0 + j + k);  // (one address: a broadcast)
#pragma unroll
            for (int h = 0; h < 4; h += 2) {
              const uint64_t x = f32_fma2(f32_pair(__uint_as_float(s[k + h]), __uint_as_float(s[k + h + 1])), f32_pair(F32_LO, F32_LO),
                                          f32_pair(__uint_as_float(r[k + h]), __uint_as_float(r[k + h + 1])));
              sums[(j + k + h) / 2] = f32_fma2(f32_mul2(x, unscale), h == 0 ? w.x : w.y, sums[(j + k + h) / 2]);
            }
          }
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty_bar + 8 * acc);
        if ((acc ^= 1) == 0) acc_phase ^= 1;
      }
      if (!ok) break;
      float z = 0.f, sum[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const float2 both = f32_parts(sums[j / 2]);
        const float x = j % 2 == 0 ? both.x : both.y;
        z = fmaf(x, 0.f, z);
        sum[j] = p.bias != nullptr ? x + __shfl_sync(0xffffffffu, b_mine, j) : x;
      }
      mb_activate_n(sum, p.act, p.max_limit, p.coef);
      if (z != 0.f) {
        *again = 1;
#pragma unroll
        for (int j = 0; j < 32; ++j) sum[j] = __uint_as_float(F32_AGAIN);
      }
      if (m < p.M) {
        float *dst = p.C + b * p.c_bs + n0 * p.c_ns + m;
        if (n0 + 32 <= p.N) {
#pragma unroll
          for (int j = 0; j < 32; ++j) dst[j * p.c_ns] = sum[j];
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (n0 + j < p.N) dst[j * p.c_ns] = sum[j];
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (*abort_flag != 0) {
    // MMAs and copies in flight must not outlive the memory they use (bounded: about 2 ms)
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) tmem_dealloc(tmem, C::TMEM_COLS);
  if (*again == 0 || *abort_flag != 0) return;
  for (int t = blockIdx.x; t < tiles; t += gridDim.x)
    tile_again(p, t / p.tiles_n % p.tiles_m * BM, t % p.tiles_n * BN, BN, t / p.tiles_n / p.tiles_m);
}

template <int BN>
int launch(mb_context *ctx, Params &p) {
  using Cf = Cfg<BN>;
  CUtensorMap mx, mw;
  MB_RETURN_IF_ERROR(mb_make_map_w_f32(ctx, &mx, p.X, p.K, p.M, p.x_bs != 0 ? p.batch : 1, p.x_ms, p.x_bs, BM));
  MB_RETURN_IF_ERROR(mb_make_map_w_f32(ctx, &mw, p.W, p.K, p.N, p.w_bs != 0 ? p.batch : 1, p.w_ns, p.w_bs, BN));
  auto kern = gemm_f32_rows_kernel<BN>;
  if (!ctx->f32_rows_smem[BN == 128]) {
    MB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cf::SMEM_BYTES));
    ctx->f32_rows_smem[BN == 128] = true;
  }
  const int64_t tiles = static_cast<int64_t>(p.batch) * p.tiles_m * p.tiles_n;
  MB_CUDA(ctx, mb_launch_chained(ctx, kern, dim3(static_cast<unsigned>(std::min<int64_t>(tiles, ctx->num_sms))), dim3(Cf::THREADS),
                                 Cf::SMEM_BYTES, mx, mw, p));
  ctx->launches++;
  ctx->launches_tc++;
  return MB_SUCCESS;
}

// Estimated SM cycles, from 1536 x 1536 x 1024 (128 columns 37.8 us, 64 49.3), 1024^3 (37.5, 26.9), 257 x 200 x 260, batch 5 (17.4,
// 12.8), 1024 x 1024 x 64, batch 8 (19.7, 20.0) and single tiles (6.5, 4.9).  The self-fetching kernel: 49.6, 36.4, -, 21.0, 6.2 us.
int64_t cost_of(const mb_context *ctx, const mb_f32_gemm &g, int bn) {
  const int64_t rounds = ceil_div64(g.batch * ceil_div64(g.M, BM) * ceil_div64(g.N, bn), ctx->num_sms);
  const int64_t step = g.run > 1 ? (bn == 128 ? 1860 : 1300) : (bn == 128 ? 2150 : 1560);  // (runs of three steps, of one)
  return (bn == 128 ? 12000 : 10000) + rounds * std::max<int64_t>(ceil_div64(g.K, KB) * step, bn == 128 ? 6200 : 4400);
}
int pick_bn(const mb_context *ctx, const mb_f32_gemm &g) {
  if (ctx->f32_bn != 0) return ctx->f32_bn;
  return g.N <= 64 || cost_of(ctx, g, 64) < cost_of(ctx, g, 128) ? 64 : 128;
}

}  // namespace

bool mb_gemm_f32_rows_supported(const mb_context *ctx, const mb_f32_gemm &g) {
  if (!ctx->use_tensor_cores || ctx->encode_tiled == nullptr || g.conv || g.residual != nullptr || g.x_ks != 1 || g.w_ks != 1 || g.c_ms != 1)
    return false;
  if ((reinterpret_cast<uintptr_t>(g.X) | reinterpret_cast<uintptr_t>(g.W)) & 15u) return false;
  if (g.x_ms % 4 != 0 || g.x_bs % 4 != 0 || g.w_ns % 4 != 0 || g.w_bs % 4 != 0) return false;
  if (g.M < 1 || g.N < 1 || g.K < 1 || g.batch < 1 || g.M >= (1ll << 30) || g.N >= (1ll << 30) || g.K >= (1ll << 30)) return false;
  return g.batch * ceil_div64(g.M, BM) * ceil_div64(g.N, 64) < (1ll << 30);
}

int64_t mb_gemm_f32_rows_cost(const mb_context *ctx, const mb_f32_gemm &g) { return cost_of(ctx, g, pick_bn(ctx, g)); }

int mb_gemm_f32_rows_launch(mb_context *ctx, const mb_f32_gemm &g) {
  const int bn = pick_bn(ctx, g);
  Params p = {};
  p.X = g.X; p.W = g.W; p.bias = g.bias; p.C = g.C;
  p.M = static_cast<int>(g.M); p.N = static_cast<int>(g.N); p.K = static_cast<int>(g.K); p.batch = static_cast<int>(g.batch);
  p.x_ms = g.x_ms; p.x_bs = g.x_bs; p.w_ns = g.w_ns; p.w_bs = g.w_bs; p.c_ns = g.c_ns; p.c_bs = g.c_bs;
  p.tiles_m = static_cast<int>(ceil_div64(g.M, BM));
  p.tiles_n = static_cast<int>(ceil_div64(g.N, bn));
  p.k_blocks = static_cast<int>(ceil_div64(g.K, KB));
  p.run = g.run > 1 ? MAX_RUN : 1;
  p.act = g.act; p.max_limit = g.max_limit; p.coef = g.coef;
  p.status = ctx->dev_status;
  return bn == 128 ? launch<128>(ctx, p) : launch<64>(ctx, p);
}
