// fp32 stride-1 convolution with SAME padding, NCHW, as a direct product on tcgen05 (kind::f16 on pairs of halves, see
// f32_split.cuh): no column matrix, no Winograd intermediates, every input value split once per tile and not once per tap.
//
// What it serves: arm::Conv2dK3x3Winograd's layers (mace/ops/arm/base/conv_2d_3x3_winograd.cc:31-787) where the batch fills the
// GPU, and the general Conv2D of those shapes (conv_2d_general.cc:26-197).
//
// The input as the kernel sees it is one line of pixels over all images: rows of W + p_w values (the p_w zeros behind a row are
// the padding of that row's end and of the next one's beginning), images of H + p_h rows.  A tile is 128 consecutive places
// of that line (the few that fall on padding are computed and dropped), and a filter tap is a shift of it: the tile and its
// surroundings lie in shared memory once, split, 16 bytes (8 channels) per pixel in planes without swizzle, so that the MMA's
// A operand of a tap is the same memory at another start address.  32 channels at a time, two such patches.
//
//     place t, tap (i, j):  row  t + i * (W + p_w) + j  of the patch, whose row 0 is place  t0 - p_h * (W + p_w) - p_w.
//
// W (the filter) comes split by f32_conv_presplit_kernel, a step being 32 channels of one tap: a tile of hi rows with a tile
// of lo rows behind it, so that hi x [w_hi | w_lo] is one MMA of twice the columns, lo x w_hi goes to the second half, and the
// large products have an accumulator of their own, which is cut off once per 16 of k (2e-8 each time).  Every `run` filter rows of
// 32 channels the result warps take both and carry the sums on in registers, where they round: errors (2-norm against float64, 3x3) of
// 1.3e-7 with a row at a time, 3.5e-7 with three, whatever the depth; Winograd's are 3.1e-8 times the root of the channels with
// F(2,3) and 2e-6 and more with F(6,3).  So every patch may have a scale of its own: it takes that of the one before where its largest
// value allows it, which is known when the patch has been written, and else its own, and is written again.
//
// What bounds it: shared memory, 470 cycles per tap of 128 channels (40 KB into the MMAs, 16 KB of W in), of which the MMAs are
// busy 384, at the clocks that the power limit leaves; with 64 channels the issue of small MMAs, 350 against 235.
// Measured, Winograd's three kernels -> this one (3x3, us, errors in the 2-norm against float64): 64 -> 64 channels, 56 x 56, batch 32
// 55.3 -> 40.2 with inputs that are not in L2, 37.7 with the same ones (4.9e-6 -> 3.8e-7), batch 256 397 -> 220; 128 -> 128, 28 x 28,
// batch 256 287 -> 172; 256 -> 256, 14 x 14 290 -> 178; 512 -> 512, 7 x 7 225 -> 195; self-fetching kernel -> this one, 5x5: 64 -> 64,
// 56 x 56, batch 24 130 -> 69.  Blocks of channels of different size are split twice: 64 -> 64 with the second block 2^12 times larger
// or smaller 40 -> 56, 128 -> 128 at 28 x 28, batch 64, 51 -> 54.
//
// Roles: warp 0 W by TMA, warp 1 MMAs, 8 or 16 warps input, 8 or 16 warps results.  Persistent over the tiles.
#include <algorithm>

#include "common.cuh"
#include "conv_f32_direct.cuh"
#include "f32_split.cuh"
#include "sm100_ptx.cuh"

namespace {

using namespace sm100;

constexpr int BM = 128, KC = 32;                   // places per tile, channels per block
constexpr int FIRST_IN = 2, IN_WARPS = 8;         // input warps per group
constexpr long long WAIT_BUDGET = 1ll << 31;       // ~1 s of SM clocks per wait
constexpr int SCALE_SLOTS = 8;                     // patches: input is at most two ahead of the MMAs, these two runs of the results
constexpr int MAX_W_STAGES = 12;

struct Params {
  const float *X, *filter, *bias, *w_unscale;
  float *C;
  int N, C_in, H, W, O, KH, KW, ph, pw;
  int pitch, image;          // places per row and per image
  int64_t places;            // all of them
  int tiles_m, tiles_n, blocks, taps, run;  // run: filter rows, of one block
  int patch_rows;            // a multiple of 32
  int w_stages;              // filter rows in shared memory
  int w_stays;               // ... which are all there are
  int act;
  float max_limit, coef;
  uint32_t image_mul, image_shift, pitch_mul, pitch_shift;
  int *status;
};

template <int BN>
struct Cfg {
  // Input in two groups that take the tiles in turn where a tile's MMAs are over sooner than the first loads of the next one
  // (64 channels, 56 x 56, batch 32: 45.3 -> 42.3 us).
  static constexpr int IN_GROUPS = BN == 64 ? 2 : 1;
  static constexpr int FIRST_OUT = FIRST_IN + IN_GROUPS * IN_WARPS;
  static constexpr int OUT_WARPS = BN / 8;         // 32 channels per thread
  static constexpr int THREADS = (FIRST_OUT + OUT_WARPS) * 32;
  static constexpr int W_BYTES = BN * 128;         // a tap of 32 channels: hi rows of 64 bytes, then lo rows
  static constexpr int ACC_COLS = 2 * BN;          // large products, small ones
  static constexpr int ACCS = 2, TMEM_COLS = ACCS * ACC_COLS;
};

// Place f of the line (possibly outside of it): where its value of channel 0 lies in the tensor, or -1.
__device__ __forceinline__ int64_t value_at(const Params &p, int64_t f) {
  if (f < 0 || f >= p.places) return -1;
  const uint32_t img = fast_div(static_cast<uint32_t>(f), p.image_mul, p.image_shift);
  const uint32_t in = static_cast<uint32_t>(f) - img * p.image;
  const uint32_t y = fast_div(in, p.pitch_mul, p.pitch_shift), x = in - y * p.pitch;
  if (static_cast<int>(y) >= p.H || static_cast<int>(x) >= p.W) return -1;
  return static_cast<int64_t>(img) * p.C_in * p.H * p.W + y * p.W + x;
}

// A result by fp32 FMAs, by a warp.
__device__ __noinline__ void store_exact(const Params &p, int64_t f, int o) {
  const uint32_t img = fast_div(static_cast<uint32_t>(f), p.image_mul, p.image_shift);
  const uint32_t in = static_cast<uint32_t>(f) - img * p.image;
  const int y = static_cast<int>(fast_div(in, p.pitch_mul, p.pitch_shift)), x = static_cast<int>(in) - y * p.pitch;
  const int64_t hw = static_cast<int64_t>(p.H) * p.W;
  float sum = f32_warp_window(p.X + static_cast<int64_t>(img) * p.C_in * hw, p.filter + static_cast<int64_t>(o) * p.C_in * p.taps,
                               p.C_in, p.H, p.W, p.KH, p.KW, y - p.ph, x - p.pw);
  if ((threadIdx.x & 31) != 0) return;
  if (p.bias != nullptr) sum += p.bias[o];
  p.C[(static_cast<int64_t>(img) * p.O + o) * hw + static_cast<int64_t>(y) * p.W + x] = mb_activate(sum, p.act, p.max_limit, p.coef);
}

// OIHW filter -> [block][tap][hi, lo][O][32 channels] halves and 1 / scale per output channel, a block of threads per channel,
// whose values wait in shared memory while their largest is found (staged; else they are read again).
constexpr int PRESPLIT_THREADS = 256, PRESPLIT_SMEM = 96 * 1024;
__global__ void __launch_bounds__(PRESPLIT_THREADS)
f32_conv_presplit_kernel(const float *filter, uint8_t *dst, float *unscale, int C_in, int O, int taps, int blocks, int staged) {
  extern __shared__ float row[];
  __shared__ float warp_most[PRESPLIT_THREADS / 32];
  mb_grid_dep_launch();
  mb_grid_dep_wait();
  const int o = blockIdx.x, total = C_in * taps;
  const float *src = filter + static_cast<int64_t>(o) * total;
  float most = 0.f;
#pragma unroll 8
  for (int i = threadIdx.x; i < total; i += PRESPLIT_THREADS) {
    const float v = mb_load(src + i);
    if (staged) row[i] = v;
    most = fmaxf(most, fabsf(v));
  }
#pragma unroll
  for (int d = 1; d < 32; d *= 2) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, d));
  if ((threadIdx.x & 31) == 0) warp_most[threadIdx.x >> 5] = most;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < PRESPLIT_THREADS / 32; ++w) most = fmaxf(most, warp_most[w]);
  const float s = most > 0.f ? f32_row_scale(most) : 0.f;
  if (threadIdx.x == 0) unscale[o] = f32_row_unscale(s);
  const uint64_t scales = f32_pair(s, s);
  if (staged) src = row;
  // (two channels of a tap at a time)
  const int pairs = blocks * taps * 16;
#pragma unroll 4
  for (int i = threadIdx.x; i < pairs; i += PRESPLIT_THREADS) {
    const int pair = i & 15, step = i >> 4, block = step / taps, tap = step - block * taps;
    const int c = block * KC + pair * 2;
    const float x = c < C_in ? mb_load(src + c * taps + tap) : 0.f, y = c + 1 < C_in ? mb_load(src + (c + 1) * taps + tap) : 0.f;
    uint32_t hi, lo;
    f32_split2(f32_pair(x, y), scales, hi, lo);
    uint8_t *to = dst + (static_cast<int64_t>(step) * 2 * O + o) * 64 + pair * 4;
    *reinterpret_cast<uint32_t *>(to) = hi;
    *reinterpret_cast<uint32_t *>(to + static_cast<int64_t>(O) * 64) = lo;
  }
}

// TAPS: filter columns, 0: any number
template <int BN, int TAPS>
__global__ void __launch_bounds__(Cfg<BN>::THREADS, 1)
conv_f32_direct_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ Params p) {
  using C = Cfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t *smem = smem_raw + (smem_base - smem_u32(smem_raw));
  // shared memory: barriers and scales, then W (w_stages filter rows), then two patches
  const uint32_t bars = smem_base;
  const uint32_t wfull_bar = bars, wempty_bar = wfull_bar + 8 * MAX_W_STAGES;
  const uint32_t pfull_bar = wempty_bar + 8 * MAX_W_STAGES, pempty_bar = pfull_bar + 8 * 2;  // [2] patches
  const uint32_t tfull_bar = pempty_bar + 8 * 2, tempty_bar = tfull_bar + 8 * C::ACCS;
  const uint32_t turn_bar = tempty_bar + 8 * C::ACCS;                                    // [2] input groups
  uint8_t *more = smem + 8 * (2 * MAX_W_STAGES + 6 + 2 * C::ACCS);
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(more);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  volatile int *again = abort_flag + 1;
  float *scales = reinterpret_cast<float *>(more + 16);     // [SCALE_SLOTS] of the patches
  float *warp_most = scales + SCALE_SLOTS;                  // [IN_GROUPS][IN_WARPS]
  const int patch_bytes = p.patch_rows * 128;
  const uint32_t w_row_bytes = p.KW * C::W_BYTES, w_stages = p.w_stages;
  const uint32_t w_base = smem_base + 1024, patch0 = w_base + w_stages * w_row_bytes;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  mb_grid_dep_launch();
  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_w);
    for (int s = 0; s < MAX_W_STAGES; ++s) {
      mbar_init(wfull_bar + 8 * s, 1);
      mbar_init(wempty_bar + 8 * s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(pfull_bar + 8 * s, IN_WARPS);  // (of one group)
      mbar_init(pempty_bar + 8 * s, 1);
      mbar_init(turn_bar + 8 * s, IN_WARPS);
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
  const int tiles = p.tiles_m * p.tiles_n;  // column tiles first: the CTAs that read one stretch of the input run side by side

  if (warp == 0) {
    // ---- W ----
    if (lane == 0) {
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      const int rows = p.blocks * p.KH;
      for (int t = blockIdx.x; ok && t < tiles && (!p.w_stays || t == blockIdx.x); t += gridDim.x) {
        const int n0 = t % p.tiles_n * BN;
        for (int i = 0; i < rows; ++i) {
          if (!mbar_wait(wempty_bar + 8 * stage, phase ^ 1, abort_flag, WAIT_BUDGET)) {
            fail(MB_DEV_TIMEOUT_PRODUCER);
            ok = false;
            break;
          }
          mbar_arrive_expect_tx(wfull_bar + 8 * stage, w_row_bytes);
          tma_load_3d(w_base + stage * w_row_bytes, &map_w, wfull_bar + 8 * stage, 0, n0, 2 * i * p.KW);
          if (++stage == w_stages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---- MMAs: the warp runs the role, one of its threads issues ----
    {
      constexpr uint32_t idesc_wide = make_idesc(/*c f32*/ 1, /*a f16*/ 0, /*b f16*/ 0, false, false, BM, 2 * BN);
      constexpr uint32_t idesc = make_idesc(1, 0, 0, false, false, BM, BN);
      const uint64_t w0 = make_smem_desc(w_base, 16, 512, 4);  // rows of 64 bytes, 64-byte swizzle
      // rows of 128 bytes, hi then lo, 128-byte swizzle (which goes by the address: a tile may begin at any row)
      const uint64_t a0 = make_smem_desc(patch0, 16, 1024, 2);
      constexpr uint32_t to_lo = 64 >> 4, half = 32 >> 4, row = 128 >> 4;  // (descriptors count 16 bytes)
      const int taps_w = TAPS != 0 ? TAPS : p.KW, taps_h = p.KH, pitch = p.pitch, w_stays = p.w_stays, blocks = p.blocks, run = p.run;
      uint32_t stage = 0, phase = 0, patch = 0, patch_phase = 0, acc = 0, acc_phase = 0;
      bool ok = true, ready = false;
      for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
        uint32_t d = 0;
        int left = 0;                          // filter rows of this run still to come
        const bool here = w_stays && t != blockIdx.x;  // the whole filter
        for (int blk = 0; ok && blk < blocks; ++blk) {
          if (!mbar_wait_warp(pfull_bar + 8 * patch, patch_phase, abort_flag, WAIT_BUDGET)) {
            fail(MB_DEV_TIMEOUT_MMA);
            ok = false;
            break;
          }
          const uint64_t a_block = a0 + patch * (patch_bytes >> 4);
          for (int i = 0; ok && i < taps_h; ++i) {
            uint32_t add = 1u;
            if (left == 0) {
              if (!mbar_wait_warp(tempty_bar + 8 * acc, acc_phase ^ 1, abort_flag, WAIT_BUDGET)) {
                fail(MB_DEV_TIMEOUT_MMA);
                ok = false;
                break;
              }
              d = tmem + acc * C::ACC_COLS;
              left = min(run, taps_h - i);
              add = 0u;
            }
            // (a barrier per filter row: what the thread does around one takes as long as four MMAs)
            if (!ready && !mbar_wait_warp(wfull_bar + 8 * stage, phase, abort_flag, WAIT_BUDGET)) {
              fail(MB_DEV_TIMEOUT_MMA);
              ok = false;
              break;
            }
            tc_fence_after_sync();
            // whether the next row is there is asked before this one's MMAs are issued and looked at after them
            const uint32_t next = stage + 1 == w_stages ? 0 : stage + 1, next_phase = next == 0 && !w_stays ? phase ^ 1 : phase;
            ready = here || __all_sync(0xffffffffu, mbar_test_wait(wfull_bar + 8 * next, next_phase));
            uint64_t a_hi = a_block + i * pitch * row, w = w0 + stage * (w_row_bytes >> 4);
#pragma unroll
            for (int j = 0; j < taps_w; ++j) {
              mma_f16_ss_elect(d, a_hi, w, idesc_wide, add);
              mma_f16_ss_elect(d + BN, a_hi + to_lo, w, idesc, 1u);
              mma_f16_ss_elect(d, a_hi + half, w + 2, idesc_wide, 1u);
              mma_f16_ss_elect(d + BN, a_hi + to_lo + half, w + 2, idesc, 1u);
              a_hi += row;
              w += C::W_BYTES >> 4;
              add = 1u;
            }
            if (!w_stays) mma_commit_elect(wempty_bar + 8 * stage);
            stage = next;
            phase = next_phase;
            if (--left == 0) {
              mma_commit_elect(tfull_bar + 8 * acc);
              if ((acc ^= 1) == 0) acc_phase ^= 1;
            }
          }
          if (!ok) break;
          mma_commit_elect(pempty_bar + 8 * patch);
          if ((patch ^= 1) == 0) patch_phase ^= 1;
        }
      }
    }
    __syncwarp();
  } else if (warp < C::FIRST_OUT) {
    // ---- input: tensor -> registers -> hi / lo planes ----
    const int w8 = (warp - FIRST_IN) % IN_WARPS, group = (warp - FIRST_IN) / IN_WARPS;
    float *group_most = warp_most + group * IN_WARPS;
    const int row_blocks = p.patch_rows / 32;
    const int64_t hw = static_cast<int64_t>(p.H) * p.W;
    float scale = 0.f;  // of the patch before, which the next one tries first
    // (A wait that gives up ends none of these warps, which meet at a barrier: the waits that follow it return at once.)
    for (int tile = group, t = blockIdx.x + group * gridDim.x; t < tiles; t += C::IN_GROUPS * gridDim.x, tile += C::IN_GROUPS) {
      const int64_t f0 = static_cast<int64_t>(t / p.tiles_n) * BM - static_cast<int64_t>(p.ph) * p.pitch - p.pw + lane;
      for (int blk = 0; blk < p.blocks; ++blk) {
        const uint32_t nth = static_cast<uint32_t>(tile) * p.blocks + blk, patch = nth & 1, phase = (nth >> 1) & 1;
        uint8_t *to = smem + (patch0 - smem_base) + patch * patch_bytes;
        float v[KC];
        auto load = [&](int rb) {
          const int64_t at = rb < row_blocks ? value_at(p, f0 + rb * 32) : -1;
          const float *src = p.X + max(at, static_cast<int64_t>(0)) + static_cast<int64_t>(blk) * KC * hw;
          const int channels = at >= 0 ? p.C_in - blk * KC : 0;
#pragma unroll
          for (int c = 0; c < KC; ++c) v[c] = c < channels ? mb_load(src + c * hw) : 0.f;
        };
        load(w8);
        // The groups write in turn, tile by tile (and load ahead of it): a patch's barrier tells its last use from the one
        // before, not from two before, so its uses have to be waited for one after the other.
        if (C::IN_GROUPS > 1 && blk == 0 && tile > 0 &&
            !mbar_wait_warp(turn_bar + 8 * group, ((tile - 1) >> 1) & 1, abort_flag, WAIT_BUDGET))
          fail(MB_DEV_TIMEOUT_PRODUCER);
        if (!mbar_wait_warp(pempty_bar + 8 * patch, phase ^ 1, abort_flag, WAIT_BUDGET)) fail(MB_DEV_TIMEOUT_PRODUCER);
        float most = 0.f;
        auto split = [&]() {
          most = 0.f;
          const uint64_t ss = f32_pair(scale, scale);
#pragma unroll 1
          for (int rb = w8; rb < row_blocks; rb += IN_WARPS) {
            if (rb != w8) load(rb);
#pragma unroll
            for (int c = 0; c < KC; ++c) most = fmaxf(most, fabsf(v[c]));
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              uint4 hi, lo;
              f32_split2(f32_pair(v[8 * g], v[8 * g + 1]), ss, hi.x, lo.x);
              f32_split2(f32_pair(v[8 * g + 2], v[8 * g + 3]), ss, hi.y, lo.y);
              f32_split2(f32_pair(v[8 * g + 4], v[8 * g + 5]), ss, hi.z, lo.z);
              f32_split2(f32_pair(v[8 * g + 6], v[8 * g + 7]), ss, hi.w, lo.w);
              uint8_t *row = to + (rb * 32 + lane) * 128;
              *reinterpret_cast<uint4 *>(row + ((g ^ (lane & 7)) << 4)) = hi;
              *reinterpret_cast<uint4 *>(row + (((g + 4) ^ (lane & 7)) << 4)) = lo;
            }
          }
        };
        const bool first = scale == 0.f;  // (the same for all warps of the group)
        uint32_t votes = 0;
        if (!first) {
          split();
          // Whether the scale was right: how many warps have values beyond what hi holds (16 each), how many have one that is large
          // enough for a patch's largest (1 each).
          const bool high = __any_sync(0xffffffffu, most * scale >= F32_HIGH), fair = __any_sync(0xffffffffu, most * scale >= F32_LOW);
          votes = named_bar_popc(1 + group, IN_WARPS * 32, lane < 16 ? high : lane == 16 && fair);
        }
        if (votes >= 16 || votes == 0) {
          // its own, and once more if that is another one
          float finite = 0.f;
#pragma unroll 1
          for (int rb = w8; rb < row_blocks; rb += IN_WARPS) {
            if (!first || rb != w8) load(rb);
#pragma unroll
            for (int c = 0; c < KC; ++c) finite = fmaxf(finite, f32_finite_abs(v[c]));
          }
#pragma unroll
          for (int d = 1; d < 32; d *= 2) finite = fmaxf(finite, __shfl_xor_sync(0xffffffffu, finite, d));
          if (lane == 0) group_most[w8] = finite;
          named_bar_sync(1 + group, IN_WARPS * 32);
          const float own = f32_shared_scale<IN_WARPS>(group_most);
          named_bar_sync(1 + group, IN_WARPS * 32);
          if (first || (own != 0.f && own != scale)) {
            scale = own;
            if (row_blocks > IN_WARPS) load(w8);
            split();
          }
        }
        if (w8 == 0 && lane == 0) scales[nth % SCALE_SLOTS] = f32_row_unscale(scale);
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(pfull_bar + 8 * patch);
          if (C::IN_GROUPS > 1 && blk + 1 == p.blocks) mbar_arrive(turn_bar + 8 * (group ^ 1));
        }
      }
    }
  } else {
    // ---- results: a lane per place, 32 channels per thread ----
    const int quarter = warp & 3, c0 = (warp - C::FIRST_OUT) / 4 * 32;
    const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
    const int64_t hw = static_cast<int64_t>(p.H) * p.W;
    const int runs = (p.KH + p.run - 1) / p.run;  // of a block
    uint32_t acc = 0, acc_phase = 0, nth = 0;
    bool ok = true;
    for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
      const int64_t f = static_cast<int64_t>(t / p.tiles_n) * BM + quarter * 32 + lane;
      const int n0 = t % p.tiles_n * BN + c0;
      // this lane's channel: what its results are multiplied by, its bias
      const float w_mine = n0 + lane < p.O ? mb_load(p.w_unscale + n0 + lane) : 0.f;
      const float b_mine = p.bias != nullptr && n0 + lane < p.O ? mb_load(p.bias + n0 + lane) : 0.f;
      float *dst = nullptr;
      if (f < p.places) {
        const uint32_t img = fast_div(static_cast<uint32_t>(f), p.image_mul, p.image_shift);
        const uint32_t in = static_cast<uint32_t>(f) - img * p.image;
        const uint32_t y = fast_div(in, p.pitch_mul, p.pitch_shift), x = in - y * p.pitch;
        if (static_cast<int>(y) < p.H && static_cast<int>(x) < p.W)
          dst = p.C + (static_cast<int64_t>(img) * p.O + n0) * hw + static_cast<int64_t>(y) * p.W + x;
      }
      uint64_t sums[16];  // of two channels each
#pragma unroll
      for (int j = 0; j < 16; ++j) sums[j] = 0;
#pragma unroll 1
      for (int i = 0; i < p.blocks * runs; ++i) {
        if (!mbar_wait_warp(tfull_bar + 8 * acc, acc_phase, abort_flag, WAIT_BUDGET)) {
          fail(MB_DEV_TIMEOUT_EPILOGUE);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const uint32_t src = tmem + lanes + acc * C::ACC_COLS + c0;
        const uint32_t patch = nth + static_cast<uint32_t>(runs == 1 ? i : i / runs);
        const uint64_t unscale = f32_pair(scales[patch % SCALE_SLOTS], scales[patch % SCALE_SLOTS]);
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
          uint32_t r[8], s[8];
          tmem_ld_32x32b_x8(src + j, r);
          tmem_ld_32x32b_x8(src + BN + j, s);
          tmem_ld_wait_x8(r);
          tmem_ld_wait_x8(s);
#pragma unroll
          for (int k = 0; k < 8; k += 2) {
            const uint64_t x = f32_fma2(f32_pair(__uint_as_float(s[k]), __uint_as_float(s[k + 1])), f32_pair(F32_LO, F32_LO),
                                        f32_pair(__uint_as_float(r[k]), __uint_as_float(r[k + 1])));
            sums[(j + k) / 2] = f32_fma2(x, unscale, sums[(j + k) / 2]);
          }
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty_bar + 8 * acc);
        if ((acc ^= 1) == 0) acc_phase ^= 1;
      }
      nth += p.blocks;
      float z = 0.f, sum[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const float2 both = f32_parts(sums[j / 2]);
        const float x = (j % 2 == 0 ? both.x : both.y) * __shfl_sync(0xffffffffu, w_mine, j);
        z = fmaf(x, 0.f, z);
        sum[j] = x + __shfl_sync(0xffffffffu, b_mine, j);
      }
      mb_activate_n(sum, p.act, p.max_limit, p.coef);
      if (z != 0.f) {
        *again = 1;
#pragma unroll
        for (int j = 0; j < 32; ++j) sum[j] = __uint_as_float(F32_AGAIN);
      }
      if (dst != nullptr) {
        if (n0 + 32 <= p.O) {
#pragma unroll
          for (int j = 0; j < 32; ++j) dst[j * hw] = sum[j];
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (n0 + j < p.O) dst[j * hw] = sum[j];
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
    for (int i = threadIdx.x; i < BM * BN; i += blockDim.x) {
      // (a warp: one channel, 32 places)
      const int64_t first = static_cast<int64_t>(t / p.tiles_n) * BM + (i & (BM - 32));
      const int o = t % p.tiles_n * BN + i / BM;
      // (the place's result lies where its input does, with O channels instead of C_in)
      const int64_t at = o < p.O ? value_at(p, first + lane) : -1;
      const int64_t hw = static_cast<int64_t>(p.H) * p.W, img = at / (p.C_in * hw), pix = at - img * p.C_in * hw;
      f32_each_again(at >= 0 && __float_as_uint(p.C[(img * p.O + o) * hw + pix]) == F32_AGAIN,
                     [&](int of) { store_exact(p, first + of, o); });
    }
}

template <int BN, int TAPS>
int launch(mb_context *ctx, Params &p, const void *split) {
  using Cf = Cfg<BN>;
  CUtensorMap map;
  const cuuint64_t dims[3] = {32, static_cast<cuuint64_t>(p.O), static_cast<cuuint64_t>(2) * p.blocks * p.taps};
  const cuuint64_t strides[2] = {64, static_cast<cuuint64_t>(p.O) * 64};
  const cuuint32_t box[3] = {32, BN, static_cast<cuuint32_t>(2 * p.KW)};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = reinterpret_cast<EncodeTiledFn>(ctx->encode_tiled)(
      &map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void *>(split), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
      CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return mb_fail(ctx, MB_RUNTIME_ERROR, "cuTensorMapEncodeTiled (fp32 filter) failed (%d)", static_cast<int>(r));
  const int around = 2 * 1024 + 2 * p.patch_rows * 128, row = p.KW * Cf::W_BYTES;
  p.w_stages = std::min(MAX_W_STAGES, (227 * 1024 - around) / row);
  // A filter that fits stays (64 -> 64 channels, 3x3: its barriers and copies were a sixth of a row's time).
  p.w_stays = p.tiles_n == 1 && p.blocks * p.KH <= p.w_stages;
  if (p.w_stays) p.w_stages = p.blocks * p.KH;
  const int smem = around + p.w_stages * row;
  auto kern = conv_f32_direct_kernel<BN, TAPS>;
  // (the limit is the device's, not this context's: the largest for all, or a context's small call would take room from another's)
  bool &raised = ctx->f32_direct_smem[(BN == 128) * 2 + (TAPS != 0)];
  if (!raised) {
    MB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    raised = true;
  }
  const int grid = std::min<int64_t>(static_cast<int64_t>(p.tiles_m) * p.tiles_n, ctx->num_sms);
  MB_CUDA(ctx, mb_launch_chained(ctx, kern, dim3(grid), dim3(Cf::THREADS), smem, map, p));
  ctx->launches++;
  ctx->launches_tc++;
  return MB_SUCCESS;
}

int patch_rows(int64_t W, int KH, int KW) {
  return static_cast<int>((BM + (KH - 1) * (W + KW / 2) + KW - 1 + 31) / 32 * 32);
}

}  // namespace

bool mb_conv_f32_direct_supported(const mb_context *ctx, const mb_f32_conv &g) {
  if (!ctx->use_tensor_cores || ctx->encode_tiled == nullptr) return false;
  if (g.KH % 2 == 0 || g.KW % 2 == 0 || g.KH > 7 || g.KW > 7) return false;
  const int64_t image = (g.H + g.KH / 2) * (g.W + g.KW / 2);
  if (g.W >= (1 << 14) || g.H >= (1 << 14) || g.N * image >= (1ll << 31) - 4096) return false;
  if (g.C >= (1 << 20) || g.O >= (1 << 20) || ceil_div64(g.C, KC) * KC * g.O * g.KH * g.KW * 4 > static_cast<int64_t>(WEIGHT_SCRATCH_BYTES))
    return false;
  const int bn = g.O > 64 ? 128 : 64;
  if (ceil_div64(g.N * image, BM) * ceil_div64(g.O, bn) >= (1ll << 30)) return false;
  return 2 * 1024 + 2 * patch_rows(g.W, g.KH, g.KW) * 128 + 2 * g.KW * bn * 128 <= 227 * 1024;
}

// (cycles of 1.9 GHz; a step of 32 channels and a tap takes fewer, of a slower clock)
int64_t mb_conv_f32_direct_cost(const mb_context *ctx, const mb_f32_conv &g) {
  const int bn = g.O > 64 ? 128 : 64;
  const int64_t tiles = ceil_div64(g.N * (g.H + g.KH / 2) * (g.W + g.KW / 2), BM) * ceil_div64(g.O, bn);
  const int64_t blocks = ceil_div64(g.C, KC), rounds = ceil_div64(tiles, ctx->num_sms);
  // the MMAs, or the input: two blocks' worth of time for the first block of a tile, which wide images read in more than one pass
  const int64_t steps = blocks * g.KH * g.KW * (bn == 128 ? 650 : g.run == 1 ? 520 : 480);
  const int64_t passes = ceil_div64(patch_rows(g.W, g.KH, g.KW), 32 * IN_WARPS);
  const int64_t input = (blocks + 2) * passes * 3000 / (bn == 64 ? 2 : 1);
  return 15000 + g.C * g.O * g.KH * g.KW / 200 + rounds * std::max(steps, input);
}

// *done is false where the filter's split has no room (see mb_weight_scratch): nothing has been launched then.
int mb_conv_f32_direct_launch(mb_context *ctx, const mb_f32_conv &g, bool *done) {
  *done = false;
  Params p = {};
  p.X = g.X; p.filter = g.filter; p.bias = g.bias; p.C = g.out;
  p.N = static_cast<int>(g.N); p.C_in = static_cast<int>(g.C); p.H = static_cast<int>(g.H); p.W = static_cast<int>(g.W);
  p.O = static_cast<int>(g.O); p.KH = g.KH; p.KW = g.KW; p.ph = g.KH / 2; p.pw = g.KW / 2;
  p.pitch = p.W + p.pw;
  p.image = p.pitch * (p.H + p.ph);
  p.places = static_cast<int64_t>(p.N) * p.image;
  const int bn = p.O > 64 ? 128 : 64;
  p.tiles_m = static_cast<int>(ceil_div64(p.places, BM));
  p.tiles_n = static_cast<int>(ceil_div64(p.O, bn));
  p.blocks = static_cast<int>(ceil_div64(p.C_in, KC));
  p.taps = p.KH * p.KW;
  p.run = std::max(1, std::min(g.run, p.KH));
  p.patch_rows = patch_rows(p.W, p.KH, p.KW);
  p.act = g.act; p.max_limit = g.max_limit; p.coef = g.coef;
  p.status = ctx->dev_status;
  fast_div_make(static_cast<uint32_t>(p.image), &p.image_mul, &p.image_shift);
  fast_div_make(static_cast<uint32_t>(p.pitch), &p.pitch_mul, &p.pitch_shift);
  const size_t split_bytes = static_cast<size_t>(p.blocks) * p.taps * 2 * p.O * 64;
  uint8_t *split = nullptr;
  MB_RETURN_IF_ERROR(mb_weight_scratch(ctx, align_up(split_bytes, 256) + p.O * 4, reinterpret_cast<void **>(&split)));
  if (split == nullptr) return MB_SUCCESS;
  float *unscale = reinterpret_cast<float *>(split + align_up(split_bytes, 256));
  p.w_unscale = unscale;
  const size_t row_bytes = static_cast<size_t>(p.C_in) * p.taps * 4;
  const int staged = row_bytes <= PRESPLIT_SMEM;
  if (staged && row_bytes > 48 * 1024 && !ctx->f32_conv_presplit_smem) {
    MB_CUDA(ctx, cudaFuncSetAttribute(f32_conv_presplit_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PRESPLIT_SMEM));
    ctx->f32_conv_presplit_smem = true;
  }
  MB_CUDA(ctx, mb_launch_chained(ctx, f32_conv_presplit_kernel, dim3(p.O), dim3(PRESPLIT_THREADS), staged ? row_bytes : 0, g.filter,
                                 split, unscale, p.C_in, p.O, p.taps, p.blocks, staged));
  ctx->launches++;
  *done = true;
  if (p.KW == 3) return bn == 128 ? launch<128, 3>(ctx, p, split) : launch<64, 3>(ctx, p, split);
  return bn == 128 ? launch<128, 0>(ctx, p, split) : launch<64, 0>(ctx, p, split);
}
