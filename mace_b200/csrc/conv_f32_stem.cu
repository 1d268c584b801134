// fp32 convolutions of an image's few channels as a direct product on the tensor cores (kind::f16 on pairs of halves, see
// f32_split.cuh): up to 4 channels, a stride of two columns, a filter of up to 8 rows and 8 columns (7 if the padding on the left
// is odd), up to 64 output channels; bias and activation fused.
// What it serves: the first convolution of an image network (arm::Conv2dGeneral, mace/ops/arm/fp32/conv_2d.h:30-60).
//
// A chunk is what a filter row of a channel multiplies: eight columns from an even one on (those without a tap have a weight of
// zero).  Tensor memory holds, for the input rows that are at work, per lane (an output column) and channel the chunk's hi
// and lo halves, so that an output row is the product of the KH rows where they lie, each of which serves KH / stride output
// rows.  A lane loads and splits two columns and has the other six from its neighbours, so that an input value is split once,
// not once per tap; a quarter of the lanes covers up to 29 output columns.  Per filter row, an MMA per two chunks for the small
// products (hi times the filter's lo, lo times its hi) and one per two for the large ones (hi * hi), of 16 of the depth; each
// kind has an accumulator: an error of 3.1e-7 (2-norm against float64, depth 147) against the self-fetching kernel's 4.0e-7.
//
// Input is scaled by strips of output rows (see f32_shared_scale); three warps look for the largest value of the strips ahead.
//
// What bounds it: the input warps' instructions and waits, 2900 cycles per output row of three channels and 7 x 7 taps, of which the
// MMAs (48 cycles each with 64 columns) are busy 1760.  With the input in shared memory the MMAs' reads left little of its
// bandwidth to the other warps (5000 cycles).  Against the self-fetching kernel, which fetches and splits every value once per tap
// (3 -> 64 channels, 7x7, stride 2, 224 x 224, us): batch 256 718 -> 345, 96 274 -> 146, 24 72 -> 47, 8 30 -> 22, 2 12.8 -> 13.6;
// 96 of 160 x 160 142 -> 103.
//
// Roles: 8 warps input, 8 results, one MMAs, 3 look ahead.  Persistent over strips of up to 116 output columns.
#include <algorithm>

#include "conv_f32_direct.cuh"
#include "f32_split.cuh"
#include "sm100_ptx.cuh"

namespace {

using namespace sm100;

constexpr int BM = 128, BN = 64, TILE = 4 * 29;  // the last three lanes of a quarter have no neighbours for their chunks
constexpr int IN_WARPS = 8, FIRST_OUT = 8, OUT_WARPS = 8, MMA_WARP = 16, FIRST_SCAN = 17, SCAN_WARPS = 3;
constexpr int THREADS = (FIRST_SCAN + SCAN_WARPS) * 32;
constexpr int CHUNK = 4;                      // columns of tensor memory: eight halves of each lane
constexpr int W_MMA = 2 * BN * 16;            // an MMA's share of W: two chunks
constexpr int ACCS = 2, ACC_COLS = 2 * BN;    // an output row's large products, its small ones
constexpr int A_COL0 = ACCS * ACC_COLS, TMEM_COLS = 512;
constexpr int MAX_SLOTS = 16, UNITS_AHEAD = 4;
constexpr int DEPTH = 8, ITEM_BYTES = 32 * 8;  // input items on their way per warp, two columns per lane each
constexpr int HEAD = 2048;                    // barriers, scales, channel table
constexpr long long WAIT_BUDGET = 1ll << 31;  // ~1 s of SM clocks per wait

__host__ __device__ constexpr int mmas(int channels) { return channels + (channels + 1) / 2; }  // per filter row

struct Params {
  const float *X, *filter, *bias;
  float *C;
  int N, H, W, O, KH, KW, sh, pt, pl, Ho, Wo;
  int strip, strips, tiles_x, units;  // output rows per unit, units per column of an image, columns of units, all units
  int slots;                          // input rows in tensor memory
  int per, tile;                      // output columns per quarter of the lanes, and of a unit: four times as many
  int vec;                            // rows are 16-byte aligned
  int shift;                          // chunks begin so many columns ahead of the filter's, at an even one
  int act;
  float max_limit, coef;
  int *status;
};

struct Unit {
  int img, y0, x0, rows, in_rows, top, left;  // output rows, input rows, first input row and column
  __device__ __forceinline__ Unit(const Params &p, int u) {
    const int s = u / p.tiles_x;
    img = s / p.strips;
    y0 = (s - img * p.strips) * p.strip;
    x0 = (u - s * p.tiles_x) * p.tile;
    rows = min(p.strip, p.Ho - y0);
    in_rows = (rows - 1) * p.sh + p.KH;
    top = y0 * p.sh - p.pt;
    left = x0 * 2 - p.pl - p.shift;
  }
};

// A result by fp32 FMAs, by a warp.
__device__ __noinline__ void store_exact(const Params &p, int channels, float *dst, int img, int o, int y, int x) {
  const int64_t hw = static_cast<int64_t>(p.H) * p.W;
  float sum = f32_warp_window(p.X + img * channels * hw, p.filter + o * channels * p.KH * p.KW, channels, p.H, p.W, p.KH, p.KW,
                               y * p.sh - p.pt, x * 2 - p.pl);
  if ((threadIdx.x & 31) != 0) return;
  if (p.bias != nullptr) sum += p.bias[o];
  *dst = mb_activate(sum, p.act, p.max_limit, p.coef);
}

template <int CI>
__global__ void __launch_bounds__(THREADS, 1) conv_f32_stem_kernel(const __grid_constant__ Params p) {
  constexpr int MM = mmas(CI), SLOT = CI * 2 * CHUNK;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 127u) & ~127u;
  uint8_t *smem = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t full_bar = smem_base, empty_bar = full_bar + 8 * MAX_SLOTS;             // input rows
  const uint32_t tfull_bar = empty_bar + 8 * MAX_SLOTS, tempty_bar = tfull_bar + 8 * ACCS;  // accumulators
  const uint32_t sfull_bar = tempty_bar + 8 * ACCS, sempty_bar = sfull_bar + 8 * UNITS_AHEAD;
  uint8_t *more = smem + 8 * (2 * MAX_SLOTS + 2 * ACCS + 2 * UNITS_AHEAD);
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(more);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  volatile int *again = abort_flag + 1;
  volatile float *most_of = reinterpret_cast<float *>(more + 16);       // [UNITS_AHEAD][SCAN_WARPS]
  float2 *table = reinterpret_cast<float2 *>(smem + HEAD - BN * 8);      // (1 / scale, bias) of the channels
  uint8_t *w_smem = smem + HEAD;
  const uint32_t w_base = smem_base + HEAD;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  mb_grid_dep_launch();
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.slots; ++s) {
      mbar_init(full_bar + 8 * s, IN_WARPS);
      mbar_init(empty_bar + 8 * s, 1);
    }
    for (int s = 0; s < ACCS; ++s) {
      mbar_init(tfull_bar + 8 * s, 1);
      mbar_init(tempty_bar + 8 * s, OUT_WARPS);
    }
    for (int s = 0; s < UNITS_AHEAD; ++s) {
      mbar_init(sfull_bar + 8 * s, SCAN_WARPS);
      mbar_init(sempty_bar + 8 * s, OUT_WARPS);
    }
    *abort_flag = 0;
    *again = 0;
    fence_barrier_init();
  }
  if (warp == MMA_WARP) {
    tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
    tmem_relinquish();
  }
  if (threadIdx.x < BN) table[threadIdx.x] = make_float2(0.f, 0.f);
  for (int i = threadIdx.x; i < p.KH * MM * W_MMA / 16; i += THREADS) reinterpret_cast<uint4 *>(w_smem)[i] = make_uint4(0, 0, 0, 0);
  auto fail = [&](int code) {
    *abort_flag = 1;
    atomicCAS(p.status, 0, code);
  };
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  mb_grid_dep_wait();

  if (warp >= FIRST_SCAN) {
    // ---- the largest value of the units' input ----
    const int first = (warp - FIRST_SCAN) * 32 + lane;
    uint32_t slot = 0, phase = 0;
    for (int u = blockIdx.x; u < p.units; u += gridDim.x) {
      const Unit t(p, u);
      if (!mbar_wait_warp(sempty_bar + 8 * slot, phase ^ 1, abort_flag, WAIT_BUDGET)) {
        fail(MB_DEV_TIMEOUT_PRODUCER);
        break;
      }
      const int r0 = max(t.top, 0), r1 = min(t.top + t.in_rows, p.H);
      int c0 = max(t.left, 0);
      const int c1 = min(t.left + (min(p.tile, p.Wo - t.x0) - 1) * 2 + p.shift + p.KW, p.W);
      if (p.vec) c0 &= ~3;
      const int per = p.vec ? 4 : 1, across = max(c1 - c0 + per - 1, 0) / per, lines = max(r1 - r0, 0);
      float most = 0.f;
      // (eight loads in flight per thread; a position beyond the last is the last again)
      auto look = [&](const float *src, auto get) {
        int r = first / max(across, 1), x = first - r * across;
        while (r < lines) {
          float v[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            v[k] = get(src + static_cast<int64_t>(min(r, lines - 1)) * p.W + x * per);
            for (x += SCAN_WARPS * 32; x >= across; x -= across) ++r;
          }
#pragma unroll
          for (int k = 0; k < 8; ++k) most = fmaxf(most, v[k]);
        }
      };
      for (int c = 0; across > 0 && c < CI; ++c) {
        const float *src = p.X + ((static_cast<int64_t>(t.img) * CI + c) * p.H + r0) * p.W + c0;
        if (p.vec)  // (rows are whole groups of four)
          look(src, [](const float *at) {
            const float4 v = mb_load(reinterpret_cast<const float4 *>(at));
            return fmaxf(fmaxf(f32_finite_abs(v.x), f32_finite_abs(v.y)), fmaxf(f32_finite_abs(v.z), f32_finite_abs(v.w)));
          });
        else
          look(src, [](const float *at) { return f32_finite_abs(mb_load(at)); });
      }
#pragma unroll
      for (int d = 1; d < 32; d *= 2) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, d));
      if (lane == 0) {
        most_of[slot * SCAN_WARPS + warp - FIRST_SCAN] = most;
        mbar_arrive(sfull_bar + 8 * slot);
      }
      __syncwarp();
      if (++slot == UNITS_AHEAD) {
        slot = 0;
        phase ^= 1;
      }
    }
  } else if (warp < IN_WARPS) {
    // ---- input rows: two warps per quarter of the output columns, which take the channels of the rows in turn ----
    const int quarter = warp & 3, column = quarter * p.per + lane;
    // (by way of shared memory, each thread its own: loads to registers share their scoreboards, and the oldest of six waited for the
    // newest, 600 cycles per item)
    const uint32_t mine = w_base + p.KH * MM * W_MMA + warp * DEPTH * ITEM_BYTES + lane * 8;
    const uint8_t *my = smem + (mine - smem_base);
    const uint32_t ring = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + A_COL0;
    uint32_t slot = 0, phase = 0, uslot = 0, uphase = 0;
    bool ok = true;
    for (int u = blockIdx.x; ok && u < p.units; u += gridDim.x) {
      const Unit t(p, u);
      const int col = t.left + column * 2;
      const float *image = p.X + static_cast<int64_t>(t.img) * CI * p.H * p.W + col;
      int at_row = 0, at = warp >> 2;  // row and channel to be loaded next
      auto load = [&](int i, int &row, int &item) {  // into the i-th place
        if (at >= CI) {
          at -= CI;
          ++at_row;
          if (CI == 1 && at >= CI) {
            at -= CI;
            ++at_row;
          }
        }
        const int y = t.top + at_row;
        const float *src = image + (static_cast<int64_t>(at) * p.H + y) * p.W;
        const uint32_t width = at_row < t.in_rows && static_cast<uint32_t>(y) < static_cast<uint32_t>(p.H) ? p.W : 0;
        const bool in = static_cast<uint32_t>(col) < width;  // (columns without a tap are read too)
        cp_async<8>(mine + i * ITEM_BYTES, in ? src : p.X, in ? 8 : 0);
        cp_async_commit();
        row = at_row;
        item = at;
        at += IN_WARPS / 4;
      };
      int row_of[DEPTH], item_of[DEPTH];  // of the items on their way
      cp_async_wait<0>();                 // (the last ones of the unit before were beyond its end)
#pragma unroll
      for (int i = 0; i < DEPTH; ++i) load(i, row_of[i], item_of[i]);
      if (!mbar_wait_warp(sfull_bar + 8 * uslot, uphase, abort_flag, WAIT_BUDGET)) {
        fail(MB_DEV_TIMEOUT_EPILOGUE);
        break;
      }
      const float scale = f32_shared_scale<SCAN_WARPS>(most_of + uslot * SCAN_WARPS);
      const uint64_t scales = f32_pair(scale, scale);
      int open = -1;  // the row whose slot is this warp's to write
      auto advance = [&](int row) {  // ... becomes this one
        while (ok && open < row) {
          if (open >= 0) {
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(full_bar + 8 * slot);
            if (++slot == static_cast<uint32_t>(p.slots)) {
              slot = 0;
              phase ^= 1;
            }
          }
          if (++open < t.in_rows && !mbar_wait_warp(empty_bar + 8 * slot, phase ^ 1, abort_flag, WAIT_BUDGET)) {
            fail(MB_DEV_TIMEOUT_PRODUCER);
            ok = false;
          }
        }
        tc_fence_after_sync();  // (the MMAs that read the slot's previous row have completed)
      };
      auto step = [&](int i, int &row, int &item) {
        advance(min(row, t.in_rows));
        if (!ok || row >= t.in_rows) return;
        cp_async_wait<DEPTH - 1>();
        uint32_t hi[4], lo[4];
        const float2 v = *reinterpret_cast<const float2 *>(my + i * ITEM_BYTES);
        f32_split2(f32_pair(v.x, v.y), scales, hi[0], lo[0]);
#pragma unroll
        for (int j = 1; j < 4; ++j) {
          hi[j] = __shfl_down_sync(0xffffffffu, hi[0], j);
          lo[j] = __shfl_down_sync(0xffffffffu, lo[0], j);
        }
        const uint32_t to = ring + slot * SLOT + item * CHUNK;
        tmem_st_32x32b_x4(to, hi);
        tmem_st_32x32b_x4(to + CI * CHUNK, lo);
        load(i, row, item);
      };
      while (ok && open < t.in_rows) {
#pragma unroll
        for (int i = 0; i < DEPTH; ++i) step(i, row_of[i], item_of[i]);
      }
      if (++uslot == UNITS_AHEAD) {
        uslot = 0;
        uphase ^= 1;
      }
    }
  } else {
    // W: a warp per output channel
    const int taps = p.KH * p.KW, total = CI * taps;
    int hi_small[8], lo_small[8];  // where a lane's values go
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int e = i * 32 + lane, c = e / taps, ky = (e - c * taps) / p.KW, kx = e - c * taps - ky * p.KW + p.shift;
      const int row = ky * MM * W_MMA + kx * 2, h = c, l = CI + c;
      hi_small[i] = row + l / 2 * W_MMA + (l & 1) * BN * 16;
      lo_small[i] = row + h / 2 * W_MMA + (h & 1) * BN * 16;
    }
#pragma unroll 2
    for (int n = warp - FIRST_OUT; n < p.O; n += FIRST_SCAN - FIRST_OUT) {
      float v[8], most = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = i * 32 + lane < total ? mb_load(p.filter + n * total + i * 32 + lane) : 0.f;
      const float bias = p.bias != nullptr ? mb_load(p.bias + n) : 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) most = fmaxf(most, fabsf(v[i]));
#pragma unroll
      for (int d = 1; d < 32; d *= 2) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, d));
      const float s = most > 0.f ? f32_row_scale(most) : 0.f;
      if (lane == 0) table[n] = make_float2(f32_row_unscale(s), bias);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (i * 32 + lane >= total) break;
        uint32_t hi, lo;
        f32_split2(f32_pair(v[i], 0.f), f32_pair(s, s), hi, lo);
        uint8_t *row = w_smem + n * 16;
        *reinterpret_cast<uint16_t *>(row + lo_small[i]) = static_cast<uint16_t>(lo);               // times hi
        *reinterpret_cast<uint16_t *>(row + hi_small[i]) = static_cast<uint16_t>(hi);               // times lo
        *reinterpret_cast<uint16_t *>(row + lo_small[i] + CI * W_MMA) = static_cast<uint16_t>(hi);  // times hi
      }
    }
    fence_proxy_async();
    asm volatile("bar.sync 1, %0;" ::"n"((FIRST_SCAN - FIRST_OUT) * 32) : "memory");
    if (warp == MMA_WARP) {
      // ---- MMAs: the warp runs the role, one of its threads issues ----
      constexpr uint32_t idesc = make_idesc(/*c f32*/ 1, /*a f16*/ 0, /*b f16*/ 0, false, false, BM, BN);
      // (W: 8 rows of 16 bytes are 128 bytes, the next eight of the depth lie a chunk further on)
      const uint64_t w0 = make_smem_desc(w_base, BN * 16, 128, 0);
      const uint32_t slots = p.slots, tmem_u = __shfl_sync(0xffffffffu, tmem, 0);
      uint32_t first = 0;                      // the slot of an output row's first input row
      uint32_t filled = 0, filled_phase = 0;   // the next one to wait for
      uint32_t acc = 0, acc_phase = 0;
      bool ok = true;
      for (int u = blockIdx.x; ok && u < p.units; u += gridDim.x) {
        const Unit t(p, u);
        int have = 0;
        for (int y = 0; ok && y < t.rows; ++y) {
          if (!mbar_wait_warp(tempty_bar + 8 * acc, acc_phase ^ 1, abort_flag, WAIT_BUDGET)) {
            fail(MB_DEV_TIMEOUT_MMA);
            ok = false;
            break;
          }
          for (const int need = y * p.sh + p.KH; have < need; ++have) {
            if (!mbar_wait_warp(full_bar + 8 * filled, filled_phase, abort_flag, WAIT_BUDGET)) {
              fail(MB_DEV_TIMEOUT_MMA);
              ok = false;
              break;
            }
            if (++filled == slots) {
              filled = 0;
              filled_phase ^= 1;
            }
          }
          if (!ok) break;
          tc_fence_after_sync();
          // (uniform over the warp, and the compiler is to know it: the descriptors are then in uniform registers)
          const uint32_t large = tmem_u + __shfl_sync(0xffffffffu, acc, 0) * ACC_COLS, small = large + BN;
          uint32_t slot = __shfl_sync(0xffffffffu, first, 0);
#pragma unroll 1
          for (int ky = 0; ky < p.KH; ++ky) {
            const uint32_t x = tmem_u + A_COL0 + slot * SLOT;
            const uint64_t w = w0 + ky * (MM * W_MMA >> 4);
            const uint32_t more_of = ky > 0 ? 1u : 0u;
#pragma unroll
            for (int i = 0; i < CI; ++i) mma_f16_ts_elect(small, x + i * 2 * CHUNK, w + i * (W_MMA >> 4), idesc, i > 0 ? 1u : more_of);
#pragma unroll
            for (int i = 0; i < MM - CI; ++i)  // (the last one of an odd number of channels has a lo, times zero)
              mma_f16_ts_elect(large, x + i * 2 * CHUNK, w + (CI + i) * (W_MMA >> 4), idesc, i > 0 ? 1u : more_of);
            if (++slot == slots) slot = 0;
          }
          mma_commit_elect(tfull_bar + 8 * acc);
          if (++acc == ACCS) {
            acc = 0;
            acc_phase ^= 1;
          }
          // input rows that no later output row of the unit needs
          for (int i = y + 1 < t.rows ? p.sh : p.KH; i > 0; --i) {
            mma_commit_elect(empty_bar + 8 * first);
            if (++first == slots) first = 0;
          }
        }
      }
    } else {
      // ---- results: two warps per quarter of the columns, 32 channels each ----
      const int quarter = warp & 3, n0 = (warp - FIRST_OUT) / 4 * 32;
      const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
      const int64_t plane = static_cast<int64_t>(p.Ho) * p.Wo;
      uint32_t acc = 0, acc_phase = 0, uslot = 0, uphase = 0;
      bool ok = true;
      for (int u = blockIdx.x; ok && u < p.units; u += gridDim.x) {
        const Unit t(p, u);
        if (!mbar_wait_warp(sfull_bar + 8 * uslot, uphase, abort_flag, WAIT_BUDGET)) {
          fail(MB_DEV_TIMEOUT_EPILOGUE);
          break;
        }
        const float unscale = f32_row_unscale(f32_shared_scale<SCAN_WARPS>(most_of + uslot * SCAN_WARPS));
        const int x = t.x0 + quarter * p.per + lane;
        float *dst = p.C + ((static_cast<int64_t>(t.img) * p.O + n0) * p.Ho + t.y0) * p.Wo + x;
        for (int y = 0; y < t.rows; ++y, dst += p.Wo) {
          if (!mbar_wait_warp(tfull_bar + 8 * acc, acc_phase, abort_flag, WAIT_BUDGET)) {
            fail(MB_DEV_TIMEOUT_EPILOGUE);
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t src = tmem + lanes + acc * ACC_COLS + n0;
          float sum[32];
#pragma unroll
          for (int j = 0; j < 32; j += 16) {
            uint32_t r[16], s[16];
            tmem_ld_32x32b_x16(src + j, r);
            tmem_ld_32x32b_x16(src + BN + j, s);
            tmem_ld_wait_x16(r);
            tmem_ld_wait_x16(s);
#pragma unroll
            for (int k = 0; k < 16; ++k) sum[j + k] = fmaf(__uint_as_float(s[k]), F32_LO, __uint_as_float(r[k]));
          }
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(tempty_bar + 8 * acc);
          if (++acc == ACCS) {
            acc = 0;
            acc_phase ^= 1;
          }
          float z = 0.f;
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            // (the products are exact, so the sum with the bias rounds once)
            const float4 ub = *reinterpret_cast<const float4 *>(table + n0 + j);
            sum[j] = fmaf(sum[j] * unscale, ub.x, ub.y);
            sum[j + 1] = fmaf(sum[j + 1] * unscale, ub.z, ub.w);
            z = fmaf(sum[j], 0.f, z);
            z = fmaf(sum[j + 1], 0.f, z);
          }
          mb_activate_n(sum, p.act, p.max_limit, p.coef);
          if (lane < p.per && x < p.Wo) {
            if (z != 0.f) {
              *again = 1;
#pragma unroll
              for (int j = 0; j < 32; ++j) sum[j] = __uint_as_float(F32_AGAIN);
            }
            if (n0 + 32 <= p.O) {
#pragma unroll
              for (int j = 0; j < 32; ++j) dst[j * plane] = sum[j];
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (n0 + j < p.O) dst[j * plane] = sum[j];
            }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(sempty_bar + 8 * uslot);
        if (++uslot == UNITS_AHEAD) {
          uslot = 0;
          uphase ^= 1;
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (*abort_flag != 0) {
    // MMAs in flight must not outlive the memory they use (bounded: about 2 ms)
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == MMA_WARP) tmem_dealloc(tmem, TMEM_COLS);
  if (*again == 0 || *abort_flag != 0) return;
  for (int u = blockIdx.x; u < p.units; u += gridDim.x) {
    const Unit t(p, u);
    const int width = min(p.tile, p.Wo - t.x0), count = p.O * t.rows * width;
    for (int first = warp * 32; first < count; first += THREADS) {
      auto place = [&](int i, int &o, int &y, int &x) {
        const int in = i % (t.rows * width);
        o = i / (t.rows * width);
        y = t.y0 + in / width;
        x = t.x0 + in % width;
        return p.C + ((static_cast<int64_t>(t.img) * p.O + o) * p.Ho + y) * p.Wo + x;
      };
      int o, y, x;
      const bool mine = first + lane < count &&
                        __float_as_uint(*reinterpret_cast<volatile float *>(place(first + lane, o, y, x))) == F32_AGAIN;
      f32_each_again(mine, [&](int of) {
        float *dst = place(first + of, o, y, x);
        store_exact(p, CI, dst, t.img, o, y, x);
      });
    }
  }
}

template <int CI>
int launch(mb_context *ctx, Params &p, int smem) {
  auto kern = conv_f32_stem_kernel<CI>;
  // (the limit is the device's, not this context's: the largest for all, or a context's small call would take room from another's)
  bool &raised = ctx->f32_stem_smem[CI - 1];
  if (!raised) {
    MB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    raised = true;
  }
  MB_CUDA(ctx, mb_launch_chained(ctx, kern, dim3(std::min(p.units, ctx->num_sms)), dim3(THREADS), smem, p));
  ctx->launches++;
  ctx->launches_tc++;
  return MB_SUCCESS;
}

int smem_of(const mb_f32_conv &g) { return 128 + HEAD + g.KH * mmas(static_cast<int>(g.C)) * W_MMA + IN_WARPS * DEPTH * ITEM_BYTES; }
int slots_of(const mb_f32_conv &g) { return std::min(MAX_SLOTS, (TMEM_COLS - A_COL0) / (static_cast<int>(g.C) * 2 * CHUNK)); }

// Rows per strip with the smallest estimate, and that in SM cycles, from the figures above: per row the MMAs, the results of 64
// channels or the input; around it filter, first rows and last results; per further strip of a CTA its first rows.
int64_t cost_of(const mb_context *ctx, const mb_f32_conv &g, int sh, int64_t Ho, int64_t Wo, int *strip) {
  const int64_t columns = g.N * ceil_div64(Wo, TILE);
  const int64_t row = std::max<int64_t>(std::max<int64_t>(g.KH * mmas(static_cast<int>(g.C)) * 52, 2400), sh * g.C * 480);
  int64_t best = -1;
  for (int64_t k = 1; k <= Ho; ++k) {
    const int64_t rows = ceil_div64(Ho, k), strips = ceil_div64(Ho, rows), rounds = ceil_div64(columns * strips, ctx->num_sms);
    const int64_t cost = rounds * rows * row + (rounds - 1) * g.KH * g.C * 270;
    if (best < 0 || cost < best) {
      best = cost;
      *strip = static_cast<int>(rows);
    }
    if (columns * strips >= 16 * static_cast<int64_t>(ctx->num_sms)) break;
  }
  return 21000 + best;
}

}  // namespace

bool mb_conv_f32_stem_supported(const mb_context *ctx, const mb_f32_conv &g, int sh, int sw, int pl, int64_t Ho, int64_t Wo) {
  if (!ctx->use_tensor_cores || g.C > 4 || g.O > BN || g.KH > 8 || sh > g.KH) return false;
  if (sw != 2 || g.KW + pl % 2 > 8 || g.W % 2 != 0 || (reinterpret_cast<uintptr_t>(g.X) & 7u) != 0) return false;
  if (g.H >= (1 << 15) || g.W >= (1 << 15) || Ho >= (1 << 15) || Wo >= (1 << 15) || pl >= (1 << 15)) return false;
  return g.N * Ho * ceil_div64(Wo, TILE) < (1ll << 30) && slots_of(g) > g.KH;
}

int64_t mb_conv_f32_stem_cost(const mb_context *ctx, const mb_f32_conv &g, int sh, int64_t Ho, int64_t Wo) {
  int strip;
  return cost_of(ctx, g, sh, Ho, Wo, &strip);
}

int mb_conv_f32_stem_launch(mb_context *ctx, const mb_f32_conv &g, int sh, int pt, int pl, int64_t Ho, int64_t Wo) {
  Params p = {};
  p.X = g.X; p.filter = g.filter; p.bias = g.bias; p.C = g.out;
  p.N = static_cast<int>(g.N); p.H = static_cast<int>(g.H); p.W = static_cast<int>(g.W); p.O = static_cast<int>(g.O);
  p.KH = g.KH; p.KW = g.KW; p.sh = sh; p.pt = pt; p.pl = pl;
  p.Ho = static_cast<int>(Ho); p.Wo = static_cast<int>(Wo);
  p.shift = pl % 2;
  p.tiles_x = static_cast<int>(ceil_div64(Wo, TILE));
  p.per = static_cast<int>(ceil_div64(Wo, 4 * p.tiles_x));
  p.tile = 4 * p.per;
  cost_of(ctx, g, sh, Ho, Wo, &p.strip);
  p.strips = static_cast<int>(ceil_div64(Ho, p.strip));
  p.units = p.N * p.strips * p.tiles_x;
  p.slots = slots_of(g);
  p.vec = g.W % 4 == 0 && (reinterpret_cast<uintptr_t>(g.X) & 15u) == 0;
  p.act = g.act; p.max_limit = g.max_limit; p.coef = g.coef;
  p.status = ctx->dev_status;
  const int smem = smem_of(g);
  switch (g.C) {
    case 1: return launch<1>(ctx, p, smem);
    case 2: return launch<2>(ctx, p, smem);
    case 3: return launch<3>(ctx, p, smem);
    default: return launch<4>(ctx, p, smem);
  }
}
