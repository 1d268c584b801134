// fp32 GEMM on tcgen05 (kind::tf32, split operands as in gemm_f32_tc.cu) whose warps fetch X from where it lies: no
// column matrix for a convolution, no transposes, no 16-byte alignment.
//
// What it serves: the general Conv2D (mace/ops/arm/base/conv_2d_general.cc:26-197, ref/conv_2d.cc:36-122), the 3x3
// Conv2D where a direct convolution beats Winograd (arm/base/conv_2d_3x3_winograd.cc:31-787), the 1x1 one of any stride
// (conv_2d_1x1.cc:27-72), MatMul / Gemm of every transposition (arm/base/gemm.cc:520-683), FullyConnected on a batch.
//
// X (the MMA's A: 128 pixels = 128 TMEM lanes) never touches shared memory: lane i of a warp owns pixel i and loads its
// 32 values of a depth step straight from the tensor (neighbouring lanes are neighbouring pixels of a row:
// coalesced), splits them in registers and writes hi and lo to tensor memory, where the MMA takes A from.  Which
// element a depth index k means -- channel, filter row, filter column -- is the same for all lanes: lane j works out
// the offset and the row / column bits of k = 32 * step + j once per step and shares them through shared memory; a lane
// holds its pixel's valid filter rows and columns as bit masks, so padding costs one logic instruction per value.
// W comes by TMA where its rows are 16-byte aligned, else through registers, and is split in shared memory.
//
// Roles (18 or 22 warps): two groups of four load X, taking the steps in turn (two steps of loads in flight; a third group
// gained nothing and cost 0.5 us per launch; fetching with 4-byte asynchronous copies through shared memory instead took
// twice as long, 128 of them per step), four split W, four or eight store results, one thread issues the MMAs, one
// requests W.  Persistent over the tiles; where these do not fill the SMs, one tile per cluster of 2 .. 8 CTAs with the
// depth cut between them, the partial tiles added up through distributed shared memory.
//
// Accuracy.  tf32 products of split operands lose the last bit of some values, and the tensor core cuts its accumulator off
// after every MMA (8 of k), so that an error of 2e-8 (values of either sign) to 5e-8 (of one sign) per MMA piles up with the
// depth; a chain of fp32 FMAs rounds, and ends at 1.4e-7 / 1.2e-7 at k = 64, 5.7e-7 / 4.3e-7 at 1024.  (Relative errors in
// the 2-norm against float64, normal / uniform [0, 1) operands.)  Three forms:
//   WHOLE   one accumulator over the depth, hi cut off: what the TMA-fed kernel does, bit for bit (4.9e-7 / 5.1e-7 at k =
//           64, 2.7e-6 / 6.7e-6 at 1024, three times that with 128 channels).
//   RUNS    hi rounded; every `run` steps the result warps take the accumulator and carry the sum on in fp32, in shared
//           memory; small products in columns of their own (64 channels) or first (128).  run = 1: 1.4e-7 / 1.3e-7, 2:
//           2.1e-7 / 2.7e-7, 4: 3.5e-7 / 6.1e-7, whatever the depth.
//   SPREAD  for up to two steps: three accumulators of at most three MMAs, handed over together: 1.2e-7 / 9.3e-8 at 64.
// mb_f32_gather_run picks the run whose error is below the FMA chain's, for products that would otherwise run on CUDA cores;
// none is up to k = 47 and from 65 to 71.  A 3x3 convolution in place of Winograd kernels takes the run whose error is below
// theirs (F(2,3): 3.1e-8 times the root of the channels, F(6,3): 2e-6 and more).  The sums cost 384 x 384 x 64, batch
// 12, 1.1 us of 6.7 (SPREAD, with the check of its results), the 3x3 layers of ResNet-50 at batch 1 0.2 to 1.5 us each, and the largest products, whose
// shared memory is busy with W already, a half (1536 x 1536 x 1024: 33 -> 50 us; 136 us on CUDA cores).  Sums in registers
// instead spilled: 96 registers for four result warps, 80 for eight.
//
// What bounds it: the tensor pipe at three tf32 MMAs per product for long depths (12 MMAs x 92 cycles per step of
// 128 x 128 x 32; a convolution's loads bring the step to 1400), the launch, first loads and results for small shapes.
// Measured, before -> now: 7x7 stride 2 of 3 -> 64 channels, 224 x 224, batch 256, 1360 us (column matrix) -> 688;
// 5x5 stride 2 of 48 -> 32, 112 x 112, batch 24, 341 -> 116; 3x3 of 512 channels, 7 x 7, batch 1, 39 (Winograd) -> 18;
// 384 x 384 x 64 times a transposed matrix, batch 12, 10.9 (CUDA cores) -> 7.7; 736 x 176 x 384, batch 24, 76 -> 39.
#include <algorithm>

#include "f32_split.cuh"
#include "gemm_f32_gather.cuh"
#include "gemm_u8_cut.cuh"  // mb_launch_clusters
#include "sm100_ptx.cuh"

int mb_make_map_w_f32(mb_context *ctx, CUtensorMap *map, const float *W, int64_t K, int64_t N, int64_t batch, int64_t w_ns,
                      int64_t w_bs, int bn);

namespace {

using namespace sm100;

constexpr int BM = 128;         // pixels (m) per tile == TMEM lanes
constexpr int KB = 32;          // depth per step
constexpr int XGROUPS = 2;      // of four warps each, taking the steps in turn
constexpr int FIRST_W = 4 * XGROUPS, FIRST_E = FIRST_W + 4;
// EW warps for results: four, or eight where a tile's results take longer than its steps (see make_plan); then the MMA
// warp and the one that requests W
constexpr int threads(int ew) { return (FIRST_E + ew + 2) * 32; }
constexpr long long WAIT_BUDGET = 1ll << 31;        // ~1 s of SM clocks per wait
enum { W_TMA = 0, W_ROWS = 1, W_COLS = 2 };         // k contiguous and 16-byte aligned; k contiguous; n contiguous
enum { WHOLE = 0, RUNS = 1, SPREAD = 2 };           // see "Accuracy" above
enum { X_CONV = 0, X_ROWS = 1, X_COLS = 2 };        // convolution; m contiguous; k contiguous

struct Params {
  const float *X, *W, *bias, *residual;
  float *C;
  int M, N, K, batch;
  int tiles_m, tiles_n, k_blocks, splits;
  int step_m, step_n, step_b;  // gridDim.x in tile coordinates
  int64_t x_ks, x_ms, x_bs, w_ns, w_ks, w_bs, c_ns, c_ms, c_bs;
  int x_vec;                   // K-contiguous rows are 16-byte aligned
  int run;                     // RUNS: steps per run
  int exact;                   // results that are not finite are worked out again in fp32 (see store_exact4)
  int act;
  float max_limit, coef;
  int H, Wd, KW, taps, sh, sw, dh, dw, pad_t, pad_l, Wo, hw, KH;
  int64_t image;               // C_in * H * Wd
  uint32_t taps_mul, taps_shift, kw_mul, kw_shift, hw_mul, hw_shift, wo_mul, wo_shift;
  int *status;
};

template <int BN, int MODE>
struct Cfg {
  static constexpr int W_BYTES = BN * KB * 4;            // hi (or lo) of a step
  static constexpr int STAGE_BYTES = 2 * W_BYTES;
  // 64 channels: hi x [w_hi | w_lo] is one MMA of 128 columns (see the MMA role)
  static constexpr bool WIDE = BN == 64;
  static constexpr int ACC_COLS = WIDE ? 2 * BN : BN;
  // TMEM: accumulators, one or three of a tile and two or one tiles at a time, then STAGES x 64 columns of A
  static constexpr int TILE_ACCS = MODE == SPREAD ? 3 : 1, ACCS = MODE == SPREAD ? 1 : 2;
  static constexpr int A_COL0 = TILE_ACCS * ACCS * ACC_COLS;
  static constexpr int STAGES = (512 - A_COL0) / (2 * KB);
  static constexpr int RING = STAGES * STAGE_BYTES;
  static constexpr int TABLE_BYTES = FIRST_W * KB * 8;
  static constexpr int PART_BYTES = BN * BM * 4;         // the runs' shares of this CTA's channels: [rank][channel][128 m]
  // (PART_BYTES only where the depth is cut: what shared memory does not take is L1, which a convolution's windows live in)
  static constexpr int SMEM_BYTES = RING + 1024 /*align*/ + TABLE_BYTES + 256 /*barriers*/;
  // (twice where a depth that is cut has short runs as well, for the runs' sums, which no 128-channel tile has room for)
  static constexpr int MAX_SMEM_BYTES = SMEM_BYTES + (BN == 64 ? 2 : 1) * PART_BYTES;
  static_assert(MAX_SMEM_BYTES <= 227 * 1024, "shared memory budget");
};

struct TileIter {
  int tm, tn, b;
  __device__ __forceinline__ TileIter(const Params &p) {
    const unsigned t = blockIdx.x / static_cast<unsigned>(p.splits);
    tm = t % p.tiles_m;
    const unsigned q = t / p.tiles_m;
    tn = q % p.tiles_n;
    b = q / p.tiles_n;
  }
  __device__ __forceinline__ bool valid(const Params &p) const { return b < p.batch; }
  __device__ __forceinline__ void next(const Params &p) {
    tm += p.step_m;
    tn += p.step_n;
    b += p.step_b;
    if (tm >= p.tiles_m) { tm -= p.tiles_m; ++tn; }
    if (tn >= p.tiles_n) { tn -= p.tiles_n; ++b; }
  }
};

// hi + lo == v; the MMA reads the upper 11 bits of each.  With hi rounded (half = 0x1000), lo has 12 bits of either sign, of
// which at most the last is lost; with hi cut off (half = 0) lo has 13 bits and the sign of v.
__device__ __forceinline__ uint32_t tf32_hi(float v, uint32_t half) { return (__float_as_uint(v) + half) & 0xffffe000u; }
__device__ __forceinline__ uint32_t tf32_lo(float v, uint32_t half) { return __float_as_uint(v - __uint_as_float(tf32_hi(v, half))); }

__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

// Rows of 32 k, 128 bytes, the 16-byte chunks of a row permuted by its low three bits (the tensor core's 128-byte swizzle).
__device__ __forceinline__ uint32_t swz_at(int row, int chunk) { return static_cast<uint32_t>(row * 128 + ((chunk ^ (row & 7)) << 4)); }

// Where pixel m of the result lies (channel 0).
template <int XK>
__device__ __forceinline__ int64_t out_offset(const Params &p, int m, int b) {
  if (XK == X_CONV) {
    const uint32_t img = fast_div(static_cast<uint32_t>(m), p.hw_mul, p.hw_shift);
    return static_cast<int64_t>(img) * p.N * p.hw + (m - static_cast<int>(img) * p.hw);
  }
  return b * p.c_bs + m * p.c_ms;
}

// Four results of a pixel by fp32 FMAs in the order of k, padding left out.  An infinity has no split (inf - inf) and neither
// has a value that rounds beyond the largest tf32 one, so whatever they meet comes out of the tensor core as a NaN.  Results
// that are not finite are stored as F32_AGAIN, and when its tiles are done a CTA that stored one works those out again here,
// which gives what the CUDA cores give.  (Results that are finite pay one FMA each for the check.  Called from the result
// warps, tile by tile, the same code cost every launch 0.8 us, in registers that it never used; so it costs 0.2.)
template <int XK>
__device__ __noinline__ void store_exact4(const Params &p, int m, int b, int n, int n_end) {
  const float *x = p.X, *w[4];
  float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int q = 0; q < 4; ++q) w[q] = p.W + b * p.w_bs + static_cast<int64_t>(min(n + q, n_end - 1)) * p.w_ns;
  if (XK == X_CONV) {
    const uint32_t img = fast_div(static_cast<uint32_t>(m), p.hw_mul, p.hw_shift);
    const int pix = m - static_cast<int>(img) * p.hw;
    const int ho = static_cast<int>(fast_div(static_cast<uint32_t>(pix), p.wo_mul, p.wo_shift));
    const int h0 = ho * p.sh - p.pad_t, w0 = (pix - ho * p.Wo) * p.sw - p.pad_l;
    x += static_cast<int64_t>(img) * p.image;
    const int channels = p.K / p.taps;
    int64_t k = 0;
    for (int c = 0; c < channels; ++c, x += static_cast<int64_t>(p.H) * p.Wd)
      for (int i = 0; i < p.KH; ++i)
        for (int j = 0; j < p.KW; ++j, ++k) {
          const int h = h0 + i * p.dh, col = w0 + j * p.dw;
          if (h < 0 || h >= p.H || col < 0 || col >= p.Wd) continue;
          const float v = x[static_cast<int64_t>(h) * p.Wd + col];
#pragma unroll
          for (int q = 0; q < 4; ++q) sum[q] = fmaf(v, w[q][k], sum[q]);
        }
  } else {
    x += b * p.x_bs + m * p.x_ms;
#pragma unroll 1
    for (int k = 0; k < p.K; ++k) {
      const float v = x[k * p.x_ks];
#pragma unroll
      for (int q = 0; q < 4; ++q) sum[q] = fmaf(v, w[q][k * p.w_ks], sum[q]);
    }
  }
  const int64_t at = out_offset<XK>(p, m, b);
  for (int q = 0; q < 4; ++q) {
    const int c = n + q;
    if (c >= n_end) return;
    float v = sum[q];
    if (p.bias != nullptr) v += p.bias[c];
    if (p.residual != nullptr) v += p.residual[at + c * p.c_ns];
    p.C[at + c * p.c_ns] = mb_activate(v, p.act, p.max_limit, p.coef);
  }
}
template <int COUNT>
__device__ __forceinline__ bool all_finite(const float (&x)[COUNT]) {
  float z = 0.f;
#pragma unroll
  for (int j = 0; j < COUNT; ++j) z = fmaf(x[j], 0.f, z);
  return z == 0.f;
}

template <int BN, int XK, int WK, int EW, int MODE>
__global__ void __launch_bounds__(threads(EW), 1)
gemm_f32_gather_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ Params p) {
  using C = Cfg<BN, MODE>;
  constexpr int STAGES = C::STAGES, ACCS = C::ACCS, MMA_WARP = FIRST_E + EW, TMA_WARP = MMA_WARP + 1;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t *smem = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bars = smem_base + C::RING + C::TABLE_BYTES;
  const uint32_t full_bar = bars, empty_bar = bars + 8 * STAGES;          // [STAGES]
  const uint32_t wfull_bar = empty_bar + 8 * STAGES;                      // [STAGES] W landed (by TMA)
  const uint32_t tfull_bar = wfull_bar + 8 * STAGES, tempty_bar = tfull_bar + 8 * ACCS;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + C::RING + C::TABLE_BYTES + 24 * STAGES + 16 * ACCS);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  volatile int *again = abort_flag + 1;  // a result is not finite
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr uint32_t half = MODE != WHOLE ? 0x1000u : 0u;
  mb_grid_dep_launch();

  if (threadIdx.x == MMA_WARP * 32) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar + 8 * s, 8);  // four X warps and four W warps
      mbar_init(empty_bar + 8 * s, 1);
      mbar_init(wfull_bar + 8 * s, 1);
    }
    if (WK == W_TMA) prefetch_tensormap(&map_w);
    for (int a = 0; a < ACCS; ++a) {
      mbar_init(tfull_bar + 8 * a, 1);
      mbar_init(tempty_bar + 8 * a, EW);
    }
    *abort_flag = 0;
    *again = 0;
    fence_barrier_init();
  }
  if (warp == FIRST_E) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  const int rank = p.splits > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int kb_begin = static_cast<int>(static_cast<int64_t>(p.k_blocks) * rank / p.splits);
  const int steps = static_cast<int>(static_cast<int64_t>(p.k_blocks) * (rank + 1) / p.splits) - kb_begin;
  auto fail = [&](int code) {
    *abort_flag = 1;
    atomicCAS(p.status, 0, code);
  };
  tc_fence_before_sync();
  __syncthreads();
  if (p.splits > 1) cluster_sync_all();  // every CTA of the cluster runs before one writes into another's memory
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  // The X warps wait for the kernel in front only where they first read the tensor: tile coordinates and the first table
  // are worked out while that kernel still runs.
  const uint32_t part = bars + 256;

  if (warp < FIRST_W) {
    // ---- X: tensor -> registers -> hi / lo in tensor memory ----
    const int group = warp >> 2, quarter = warp & 3;
    const uint32_t a_lane = static_cast<uint32_t>(quarter * 32) << 16;
    int2 *table = reinterpret_cast<int2 *>(smem + C::RING) + warp * KB;
    int it = 0;  // steps of this CTA so far, all tiles
    bool ok = true, waited = false;
    for (TileIter t(p); ok && t.valid(p); t.next(p)) {
      const int m = t.tm * BM + quarter * 32 + lane;
      const float *base = p.X;
      uint32_t valid = 0;  // filter rows (bits 0 ..) and columns (bits 16 ..) of this pixel that lie inside the image
      if (XK == X_CONV) {
        const uint32_t img = fast_div(static_cast<uint32_t>(m), p.hw_mul, p.hw_shift);
        const int pix = m - static_cast<int>(img) * p.hw;
        const int ho = static_cast<int>(fast_div(static_cast<uint32_t>(pix), p.wo_mul, p.wo_shift));
        const int h0 = ho * p.sh - p.pad_t, w0 = (pix - ho * p.Wo) * p.sw - p.pad_l;
        base += static_cast<int64_t>(img) * p.image + static_cast<int64_t>(h0) * p.Wd + w0;
        if (m < p.M) {
          for (int i = 0; i < p.KH; ++i) valid |= (h0 + i * p.dh >= 0 && h0 + i * p.dh < p.H ? 1u : 0u) << i;
          for (int i = 0; i < p.KW; ++i) valid |= (w0 + i * p.dw >= 0 && w0 + i * p.dw < p.Wd ? 1u : 0u) << (16 + i);
        }
      } else {
        base += t.b * p.x_bs + m * p.x_ms;
        valid = m < p.M ? 1u : 0u;
      }
      for (int i = 0; i < steps; ++i, ++it) {
        if (it % XGROUPS != group) continue;
        const int stage = it % STAGES;
        const int k0 = (kb_begin + i) * KB;
        float v[KB];
        if (XK == X_COLS) {
          if (!waited) mb_grid_dep_wait();
          waited = true;
          const float *row = base + k0;
          if (p.x_vec) {
#pragma unroll
            for (int j = 0; j < KB; j += 4) {
              const bool in = valid != 0 && k0 + j < p.K;
              const float4 x = in ? mb_load(reinterpret_cast<const float4 *>(row + j)) : make_float4(0.f, 0.f, 0.f, 0.f);
              v[j] = x.x; v[j + 1] = x.y; v[j + 2] = x.z; v[j + 3] = x.w;
            }
          } else {
#pragma unroll
            for (int j = 0; j < KB; ++j) v[j] = valid != 0 && k0 + j < p.K ? mb_load(row + j) : 0.f;
          }
        } else {
          const int k = k0 + lane;
          int2 e;
          if (XK == X_CONV) {
            const int c = static_cast<int>(fast_div(static_cast<uint32_t>(k), p.taps_mul, p.taps_shift));
            const int tap = k - c * p.taps;
            const int kh = static_cast<int>(fast_div(static_cast<uint32_t>(tap), p.kw_mul, p.kw_shift));
            const int kw = tap - kh * p.KW;
            e.x = (c * p.H + kh * p.dh) * p.Wd + kw * p.dw;
            e.y = static_cast<int>((1u << kh) | (0x10000u << kw));
          } else {
            e.x = static_cast<int>(k * p.x_ks);
            e.y = 1;
          }
          if (k >= p.K) e = make_int2(0, static_cast<int>(0x80000000u));  // (no pixel has bit 31)
          __syncwarp();  // the table of the previous step has been read
          table[lane] = e;
          __syncwarp();
          if (!waited) mb_grid_dep_wait();
          waited = true;
#pragma unroll
          for (int j = 0; j < KB; j += 2) {
            const int4 t2 = *reinterpret_cast<const int4 *>(table + j);
            v[j] = (valid & t2.y) == static_cast<uint32_t>(t2.y) ? mb_load(base + t2.x) : 0.f;
            v[j + 1] = (valid & t2.w) == static_cast<uint32_t>(t2.w) ? mb_load(base + t2.z) : 0.f;
          }
        }
        if (it >= STAGES && !mbar_wait_warp(empty_bar + 8 * stage, ((it / STAGES) & 1) ^ 1, abort_flag, WAIT_BUDGET)) {
          fail(MB_DEV_TIMEOUT_PRODUCER);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const uint32_t slot = tmem + a_lane + C::A_COL0 + stage * (2 * KB);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t r[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) r[j] = tf32_hi(v[h * 16 + j], half);
          tmem_st_32x32b_x16(slot + h * 16, r);
#pragma unroll
          for (int j = 0; j < 16; ++j) r[j] = tf32_lo(v[h * 16 + j], half);
          tmem_st_32x32b_x16(slot + KB + h * 16, r);
        }
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(full_bar + 8 * stage);
      }
    }
  } else if (warp < FIRST_E) {
    // ---- W: (matrix -> registers ->) hi / lo in shared memory, rows of 32 k, 128-byte swizzle ----
    const int w4 = warp - FIRST_W;
    mb_grid_dep_wait();
    int it = 0;
    bool ok = true;
    for (TileIter t(p); ok && t.valid(p); t.next(p)) {
      const int n0 = t.tn * BN;
      const float *W = p.W + t.b * p.w_bs;
      for (int i = 0; i < steps; ++i, ++it) {
        const int stage = it % STAGES;
        uint8_t *tile = smem + stage * C::STAGE_BYTES;
        if (WK == W_TMA) {
          if (!mbar_wait_warp(wfull_bar + 8 * stage, (it / STAGES) & 1, abort_flag, WAIT_BUDGET)) {
            fail(MB_DEV_TIMEOUT_EPILOGUE);
            ok = false;
            break;
          }
#pragma unroll
          for (int c = 0; c < C::W_BYTES / 2048; ++c) {
            const int at = (c * 128 + w4 * 32 + lane) * 16;
            const float4 v = *reinterpret_cast<const float4 *>(tile + at);
            *reinterpret_cast<uint4 *>(tile + at) = make_uint4(tf32_hi(v.x, half), tf32_hi(v.y, half), tf32_hi(v.z, half), tf32_hi(v.w, half));
            *reinterpret_cast<uint4 *>(tile + C::W_BYTES + at) = make_uint4(tf32_lo(v.x, half), tf32_lo(v.y, half), tf32_lo(v.z, half), tf32_lo(v.w, half));
          }
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) mbar_arrive(full_bar + 8 * stage);
          continue;
        }
        const int k0 = (kb_begin + i) * KB;
        constexpr int CH = BN / 16;  // 16-byte chunks per thread
        float4 v[CH];
        int row[CH], chunk[CH];
        if (WK == W_COLS) {
          // lane = row, a chunk is four depth rows of the matrix
          constexpr int WARPS_N = BN / 32;  // warps along n; the others take other depth rows
          const int n = (w4 % WARPS_N) * 32 + lane;
          const bool in = n0 + n < p.N;
#pragma unroll
          for (int c = 0; c < CH; ++c) {
            row[c] = n;
            chunk[c] = (w4 / WARPS_N) * CH + c;
            const int k = k0 + chunk[c] * 4;
            const float *src = W + n0 + n + static_cast<int64_t>(k) * p.w_ks;
            v[c].x = in && k < p.K ? mb_load(src) : 0.f;
            v[c].y = in && k + 1 < p.K ? mb_load(src + p.w_ks) : 0.f;
            v[c].z = in && k + 2 < p.K ? mb_load(src + 2 * p.w_ks) : 0.f;
            v[c].w = in && k + 3 < p.K ? mb_load(src + 3 * p.w_ks) : 0.f;
          }
        } else {
          const int c8 = lane & 7, k = k0 + c8 * 4;
#pragma unroll
          for (int c = 0; c < CH; ++c) {
            row[c] = w4 * (BN / 4) + c * 4 + (lane >> 3);
            chunk[c] = c8;
            const float *src = W + static_cast<int64_t>(n0 + row[c]) * p.w_ns + k;
            const bool in = n0 + row[c] < p.N;
            v[c].x = in && k < p.K ? mb_load(src) : 0.f;
            v[c].y = in && k + 1 < p.K ? mb_load(src + 1) : 0.f;
            v[c].z = in && k + 2 < p.K ? mb_load(src + 2) : 0.f;
            v[c].w = in && k + 3 < p.K ? mb_load(src + 3) : 0.f;
          }
        }
        if (it >= STAGES && !mbar_wait_warp(empty_bar + 8 * stage, ((it / STAGES) & 1) ^ 1, abort_flag, WAIT_BUDGET)) {
          fail(MB_DEV_TIMEOUT_PRODUCER);
          ok = false;
          break;
        }
#pragma unroll
        for (int c = 0; c < CH; ++c) {
          const uint32_t at = swz_at(row[c], chunk[c]);
          *reinterpret_cast<uint4 *>(tile + at) = make_uint4(tf32_hi(v[c].x, half), tf32_hi(v[c].y, half), tf32_hi(v[c].z, half), tf32_hi(v[c].w, half));
          *reinterpret_cast<uint4 *>(tile + C::W_BYTES + at) = make_uint4(tf32_lo(v[c].x, half), tf32_lo(v[c].y, half), tf32_lo(v[c].z, half), tf32_lo(v[c].w, half));
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(full_bar + 8 * stage);
      }
    }
  } else if (warp == TMA_WARP) {
    if (WK == W_TMA && lane == 0) {
      mb_grid_dep_wait();
      int it = 0;
      bool ok = true;
      for (TileIter t(p); ok && t.valid(p); t.next(p)) {
        for (int i = 0; i < steps; ++i, ++it) {
          const int stage = it % STAGES;
          if (it >= STAGES && !mbar_wait(empty_bar + 8 * stage, ((it / STAGES) & 1) ^ 1, abort_flag, WAIT_BUDGET)) {
            fail(MB_DEV_TIMEOUT_PRODUCER);
            ok = false;
            break;
          }
          mbar_arrive_expect_tx(wfull_bar + 8 * stage, C::W_BYTES);
          tma_load_3d(smem_base + stage * C::STAGE_BYTES, &map_w, wfull_bar + 8 * stage, (kb_begin + i) * KB, t.tn * BN,
                      p.w_bs != 0 ? t.b : 0);
        }
      }
    }
    __syncwarp();
  } else if (warp == MMA_WARP) {
    // ---- MMA: one thread ----
    mb_grid_dep_wait();  // (its waits below are bounded: they must not count the time of the kernel in front)
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc(/*c f32*/ 1, /*a tf32*/ 2, /*b tf32*/ 2, false, false, BM, BN);
      constexpr uint32_t idesc_wide = make_idesc(1, 2, 2, false, false, BM, C::WIDE ? 2 * BN : BN);
      const uint64_t wdesc = make_smem_desc(0, 16, 1024, 2);
      const int run = MODE == RUNS ? p.run : steps;
      const int third = steps == 1 ? 2 : 3;  // SPREAD: MMA depths per accumulator
      int it = 0, filled = 0;  // steps, and accumulators handed to the result warps
      bool ok = true;
      uint32_t d = 0;
      // the next accumulator, once its last contents have been read
      auto next_acc = [&]() {
        const int acc = filled % ACCS;
        if (filled >= ACCS && !mbar_wait(tempty_bar + 8 * acc, ((filled / ACCS) & 1) ^ 1, abort_flag, WAIT_BUDGET)) {
          fail(MB_DEV_TIMEOUT_MMA);
          return false;
        }
        tc_fence_after_sync();
        d = tmem + acc * C::ACC_COLS;
        return true;
      };
      for (TileIter t(p); ok && t.valid(p); t.next(p)) {
        for (int i0 = 0; ok && i0 < steps; i0 += run) {
          if (!(ok = next_acc())) break;
          const int count = min(run, steps - i0);
          // 128 channels in short runs: the small products first, while they do not cost the accumulator its last bits
          constexpr bool small_first = MODE != WHOLE && !C::WIDE;
          for (int i = 0; i < count; ++i) {
            const int stage = (it + i) % STAGES;
            if (!mbar_wait(full_bar + 8 * stage, ((it + i) / STAGES) & 1, abort_flag, WAIT_BUDGET)) {
              fail(MB_DEV_TIMEOUT_MMA);
              ok = false;
              break;
            }
            tc_fence_after_sync();
            const uint32_t a_hi = tmem + C::A_COL0 + stage * (2 * KB), a_lo = a_hi + KB;
            const uint32_t sw = smem_base + stage * C::STAGE_BYTES;
            const uint64_t w_hi = wdesc | static_cast<uint64_t>((sw >> 4) & 0x3FFFu);
            const uint64_t w_lo = wdesc | static_cast<uint64_t>(((sw + C::W_BYTES) >> 4) & 0x3FFFu);
            // With A from tensor memory an MMA takes 92 cycles for 64 columns as for 128, so 64 channels take hi from
            // there once for both halves of W, whose tiles lie one behind the other: 2 MMAs per 8 of k instead of 3, and
            // hi * lo + lo * hi in columns of their own, which the result warps add.
#pragma unroll
            for (int j = 0; j < KB / 8; ++j) {
              const uint32_t add = (i > 0 || j > 0) ? 1u : 0u;
              if (C::WIDE) {
                const int at = MODE == SPREAD ? (i * 4 + j) / third : 0;
                const bool first = MODE == SPREAD ? (i * 4 + j) % third == 0 : add == 0;
                const uint32_t da = d + at * C::ACC_COLS;
                mma_tf32_ts(da, a_hi + j * 8, w_hi + 2 * j, idesc_wide, first ? 0u : 1u);
                mma_tf32_ts(da + BN, a_lo + j * 8, w_hi + 2 * j, idesc, 1u);
                continue;
              }
              mma_tf32_ts(d, a_lo + j * 8, w_hi + 2 * j, idesc, add);
              mma_tf32_ts(d, a_hi + j * 8, w_lo + 2 * j, idesc, 1u);
              if (!small_first) mma_tf32_ts(d, a_hi + j * 8, w_hi + 2 * j, idesc, 1u);
            }
            if (!small_first) mma_commit(empty_bar + 8 * stage);
          }
          if (small_first && ok) {
            for (int i = 0; i < count; ++i) {
              const int stage = (it + i) % STAGES;
              const uint32_t a_hi = tmem + C::A_COL0 + stage * (2 * KB);
              const uint64_t w_hi = wdesc | static_cast<uint64_t>(((smem_base + stage * C::STAGE_BYTES) >> 4) & 0x3FFFu);
#pragma unroll
              for (int j = 0; j < KB / 8; ++j) {
                const int at = MODE == SPREAD ? (i * 4 + j) / third : 0;
                mma_tf32_ts(d + at * C::ACC_COLS, a_hi + j * 8, w_hi + 2 * j, idesc,
                            at > 0 && (i * 4 + j) % third == 0 ? 0u : 1u);
              }
              mma_commit(empty_bar + 8 * stage);
            }
          }
          if (ok) mma_commit(tfull_bar + 8 * (filled++ % ACCS));
          it += count;
        }
      }
    }
    __syncwarp();
  } else {
    // ---- results: a lane per pixel, one channel after the other, 32 adjacent pixels per store ----
    const int quarter = warp & 3;
    constexpr int CW = BN * 4 / EW;                  // channels per warp: of eight warps, half the channels each
    const int c_begin = (warp - FIRST_E) / 4 * CW, c_end = c_begin + CW;
    const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
    int filled = 0;
    mb_grid_dep_wait();
    auto wait_acc = [&]() {
      const int acc = filled % ACCS;
      if (!mbar_wait_warp(tfull_bar + 8 * acc, (filled / ACCS) & 1, abort_flag, WAIT_BUDGET)) {
        fail(MB_DEV_TIMEOUT_EPILOGUE);
        return false;
      }
      tc_fence_after_sync();
      return true;
    };
    auto release_acc = [&]() {
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty_bar + 8 * (filled % ACCS));
      ++filled;
    };
    // this CTA's run of the depth, each channel to the CTA that adds it up (writing it there takes nobody's time; read
    // from there, one peer after the other, it took 2.1 us)
    const int share = BN / p.splits;  // channels per CTA: 8 .. 64
    auto push8 = [&](const float *x, int c) {
      const int owner = c / share;
      const uint32_t dst = mapa_shared(part, owner) + ((rank * share + c - owner * share) * BM + quarter * 32 + lane) * 4;
#pragma unroll
      for (int j = 0; j < 8; ++j) st_cluster_f32(dst + j * (BM * 4), x[j]);
    };
    // the sums of the runs so far, each thread's own
    float *sums = reinterpret_cast<float *>(smem + (part - smem_base) + (p.splits > 1 ? C::PART_BYTES : 0)) + quarter * 32 + lane;
    const int runs = MODE == RUNS ? (steps + p.run - 1) / p.run : 1;
    bool ok = true;
    for (TileIter t(p); ok && t.valid(p); t.next(p)) {
      const int m = t.tm * BM + quarter * 32 + lane;
      const int64_t at = out_offset<XK>(p, m, t.b);
      const int n0 = t.tn * BN;
      const int c_stop = MODE == WHOLE ? c_end : min(c_end, p.N - n0);  // (runs: no sums of channels that do not exist)
#pragma unroll 1
      for (int i = 0; i < runs; ++i) {
        if (!(ok = wait_acc())) break;
        const uint32_t src = tmem + lanes + (filled % ACCS) * C::ACC_COLS;
        // the next chunk's accumulators are on their way while this one is stored
        uint32_t r[16], r2[16];
        if (MODE != WHOLE && c_begin >= c_stop) {
          release_acc();
          continue;
        }
        tmem_ld_32x32b_x16(src + c_begin, r);
        if (C::WIDE) tmem_ld_32x32b_x16(src + BN + c_begin, r2);
#pragma unroll 1
        for (int c = c_begin; c < c_stop; c += 16) {
          tmem_ld_wait_x16(r);
          if (C::WIDE) tmem_ld_wait_x16(r2);
          // (everything is loaded before the first store: the compiler may not move a load above a store, and one load
          // latency per channel made a 128 x 128 tile take 19 us)
          float x[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) x[j] = C::WIDE ? __uint_as_float(r[j]) + __uint_as_float(r2[j]) : __uint_as_float(r[j]);
          if (MODE == SPREAD) {
#pragma unroll
            for (int a = 1; a < C::TILE_ACCS; ++a) {
              if (a == 2 && steps == 1) break;
              tmem_ld_32x32b_x16(src + a * C::ACC_COLS + c, r);
              if (C::WIDE) tmem_ld_32x32b_x16(src + a * C::ACC_COLS + BN + c, r2);
              tmem_ld_wait_x16(r);
              if (C::WIDE) tmem_ld_wait_x16(r2);
#pragma unroll
              for (int j = 0; j < 16; ++j) x[j] += C::WIDE ? __uint_as_float(r[j]) + __uint_as_float(r2[j]) : __uint_as_float(r[j]);
            }
          }
          if (c + 16 < c_stop) {
            tmem_ld_32x32b_x16(src + c + 16, r);
            if (C::WIDE) tmem_ld_32x32b_x16(src + BN + c + 16, r2);
          } else {
            release_acc();
          }
          if (MODE == RUNS && i > 0) {
#pragma unroll
            for (int j = 0; j < 16; ++j) x[j] += sums[(c + j) * BM];
          }
          if (MODE == RUNS && i + 1 < runs) {
#pragma unroll
            for (int j = 0; j < 16; ++j) sums[(c + j) * BM] = x[j];
            continue;
          }
          if (p.splits > 1) {
            push8(x, c);
            push8(x + 8, c + 8);
            continue;
          }
          const bool finite = MODE == WHOLE || !p.exact || all_finite(x);
          if (p.bias != nullptr) {
            const float mine = n0 + c + (lane & 15) < p.N ? mb_load(p.bias + n0 + c + (lane & 15)) : 0.f;
#pragma unroll
            for (int j = 0; j < 16; ++j) x[j] += __shfl_sync(0xffffffffu, mine, j);
          }
          if (p.residual != nullptr && m < p.M) {
            const float *src_r = p.residual + at + static_cast<int64_t>(n0 + c) * p.c_ns;
            float res[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) res[j] = n0 + c + j < p.N ? mb_load(src_r + j * p.c_ns) : 0.f;
#pragma unroll
            for (int j = 0; j < 16; ++j) x[j] += res[j];
          }
          mb_activate_n(x, p.act, p.max_limit, p.coef);
          if (MODE != WHOLE && !finite) {
            *again = 1;
#pragma unroll
            for (int j = 0; j < 16; ++j) x[j] = __uint_as_float(F32_AGAIN);
          }
          float *dst = p.C + at + static_cast<int64_t>(n0 + c) * p.c_ns;
          if (n0 + c + 16 <= p.N) {
            if (m < p.M) {
#pragma unroll
              for (int j = 0; j < 16; ++j) dst[j * p.c_ns] = x[j];
            }
          } else if (m < p.M) {
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (n0 + c + j < p.N) dst[j * p.c_ns] = x[j];
          }
        }
      }
      if (p.splits > 1) break;
    }
  }
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (*abort_flag != 0) {
    // MMAs in flight must not outlive the memory they use (bounded: about 2 ms)
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  if (p.splits > 1) {
    cluster_sync_all();
    mb_grid_dep_wait();  // (some of these warps had nothing to wait for so far)
    // every CTA of the cluster adds up its share of the channels, all runs in the order of their rank
    const TileIter t(p);
    const int m = t.tm * BM + (threadIdx.x & 127);
    const int64_t at = out_offset<XK>(p, m, t.b);
    const int share = BN / p.splits, n0 = t.tn * BN + rank * share;
    const float *mine = reinterpret_cast<const float *>(smem + C::RING + C::TABLE_BYTES + 256) + (threadIdx.x & 127);
    if (warp < 16 && m < p.M) {
      // up to four channels per round, all loads before the first store (see above)
      for (int c0 = warp >> 2; c0 < share; c0 += 16) {
        float x[4], bias[4], add[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int c = c0 + q * 4, n = n0 + c;
          x[q] = bias[q] = add[q] = 0.f;
          if (c < share && n < p.N) {
            if (p.residual != nullptr) add[q] = mb_load(p.residual + at + static_cast<int64_t>(n) * p.c_ns);
            if (p.bias != nullptr) bias[q] = mb_load(p.bias + n);
            for (int s = 0; s < p.splits; ++s) x[q] += mine[(s * share + c) * BM];
          }
        }
        const bool finite = MODE == WHOLE || !p.exact || all_finite(x);
#pragma unroll
        for (int q = 0; q < 4; ++q) x[q] = (x[q] + bias[q]) + add[q];
        if (MODE != WHOLE && !finite) *again = 1;
        mb_activate_n(x, p.act, p.max_limit, p.coef);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int c = c0 + q * 4, n = n0 + c;
          if (c < share && n < p.N) p.C[at + static_cast<int64_t>(n) * p.c_ns] = finite ? x[q] : __uint_as_float(F32_AGAIN);
        }
      }
    }
  }
  if (warp == FIRST_E) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
  if (MODE != WHOLE && p.exact) {
    if (p.splits > 1) __syncthreads();
    if (*again == 0 || *abort_flag != 0) return;
    mb_grid_dep_wait();  // (one of the warps may have had nothing to wait for so far)
    const int width = BN / p.splits;
    for (TileIter t(p); t.valid(p); t.next(p)) {
      const int n_begin = t.tn * BN + rank * width, n_end = min(p.N, n_begin + width);
      for (int i = threadIdx.x; i < BM * (width / 4); i += blockDim.x) {
        const int m = t.tm * BM + (i & (BM - 1)), n = n_begin + (i / BM) * 4;
        if (m >= p.M || n >= n_end) continue;
        const float *stored = p.C + out_offset<XK>(p, m, t.b) + n * p.c_ns;
        bool found = false;
        for (int q = 0; q < 4 && n + q < n_end; ++q) found |= __float_as_uint(stored[q * p.c_ns]) == F32_AGAIN;
        if (found) store_exact4<XK>(p, m, t.b, n, n_end);
      }
      if (p.splits > 1) break;
    }
  }
}

template <int BN, int XK, int WK, int EW, int MODE>
int launch_cfg(mb_context *ctx, Params &p) {
  using C = Cfg<BN, MODE>;
  auto kern = gemm_f32_gather_kernel<BN, XK, WK, EW, MODE>;
  constexpr int bit = (MODE == SPREAD ? 54 : MODE == RUNS ? 36 : EW == 8 ? 18 : 0) + (BN == 128 ? 9 : 0) + XK * 3 + WK;
  CUtensorMap map;
  if (WK == W_TMA) MB_RETURN_IF_ERROR(mb_make_map_w_f32(ctx, &map, p.W, p.K, p.N, p.w_bs != 0 ? p.batch : 1, p.w_ns, p.w_bs, BN));
  else memset(&map, 0, sizeof(map));
  uint64_t &mask = ctx->f32_gather_attr_mask[bit >> 6];
  if (!(mask & (1ull << (bit & 63)))) {
    MB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::MAX_SMEM_BYTES));
    mask |= 1ull << (bit & 63);
  }
  const int64_t tiles = static_cast<int64_t>(p.batch) * p.tiles_m * p.tiles_n;
  const int slots = p.splits > 1 ? static_cast<int>(tiles) : static_cast<int>(std::min<int64_t>(tiles, ctx->num_sms));
  p.step_m = slots % p.tiles_m;
  p.step_n = (slots / p.tiles_m) % p.tiles_n;
  p.step_b = (slots / p.tiles_m) / p.tiles_n;
  const bool sums = MODE == RUNS && p.run < ceil_div64(p.k_blocks, p.splits);  // (some CTA has more than one run)
  MB_CUDA(ctx, mb_launch_clusters(ctx, kern, static_cast<unsigned>(slots * p.splits), threads(EW),
                                  C::SMEM_BYTES + ((p.splits > 1) + sums) * C::PART_BYTES,
                                  p.splits, map, p));
  ctx->launches++;
  ctx->launches_tc++;
  return MB_SUCCESS;
}

struct Plan {
  int bn = 64, splits = 1, warps = 4;
  int64_t cost = -1, steps = 0;  // (steps of a CTA beyond the first two of a tile)
};

// Tile width and depth runs with the smallest estimate, in SM cycles.  Measured: a step is bound by the MMAs, whose A
// operand comes from tensor memory at the same rate for either width (0.6 us for the 12 of 128 channels), or by a
// convolution's loads (0.72 us); a tile's stores take 2.7 us per 64 channels, twice that with a residual; 5.5 us around the
// steps, 6.3 us with the exchange between the CTAs of a cluster.
Plan make_plan(mb_context *ctx, const mb_f32_gemm &g) {
  const int64_t tiles_m = ceil_div64(g.M, BM), k_blocks = ceil_div64(g.K, KB);
  Plan best;
  int asked = ctx->f32_splits;
  while (asked > k_blocks) asked /= 2;
  for (int w : {128, 64}) {
    if (ctx->f32_bn != 0 ? w != ctx->f32_bn : (w == 128 && g.N <= 64)) continue;
    const int64_t tiles = g.batch * tiles_m * ceil_div64(g.N, w);
    for (int s : {1, 2, 4, 8}) {
      if (asked != 0 ? s != asked : s > k_blocks) continue;
      if (w == 128 && s > 1 && g.run != 0) continue;  // (no room for the runs' sums)
      const int64_t rounds = ceil_div64(tiles * s, s == 1 ? ctx->num_sms : mb_resident_cluster_ctas(ctx, s));
      if (s > 1 && rounds > 1 && asked == 0) continue;  // (one tile per CTA: a second round would start from nothing)
      const int64_t steps = ceil_div64(k_blocks, s);
      const int64_t step = g.conv ? (w == 128 ? 1450 : g.run != 0 ? 1280 : 1200) : (w == 128 ? 1250 : 1100);
      const bool res = g.residual != nullptr;
      int64_t results = (w == 128 ? 10600 : 5400) * (res ? 2 : 1);
      // eight warps for results: where they bound a 128-wide tile (at 64 eight are no faster), or the launch is one round of
      // few steps; not elsewhere, as the warps that load X then have too few registers
      const bool eight = s == 1 && steps * step <= results && (w == 128 || rounds == 1);
      if (eight && w == 128) results = res ? 16000 : 7000;
      const int64_t last = (w == 128 ? 4000 : 1500) + (res ? 2000 : 0) - (eight ? 700 : 0);
      // products in TMA's layout: 64 channels undivided take 13.6 us for 16 of 512 x 48 x 512 and 8.6 for 16 of 256 x 48 x 256, 128
      // with the depth cut 16.4 and 10.3, the TMA-fed kernel 13.9 and 9.2
      const int64_t product = g.conv || g.run != 0 ? 0 : w == 64 && s == 1 ? -1500 : w == 128 && s > 1 ? 3500 : 0;
      const int64_t cost = product + (s == 1 ? 8000 + (rounds - 1) * std::max<int64_t>(steps * step, results) + steps * step + last
                           : w == 128 ? 10500 + steps * 1350 + last
                                      : (s == 2 ? 11500 : s == 4 ? 10500 : 11000) + steps * (s == 2 ? 1150 : 1050) + last);
      if (best.cost < 0 || cost < best.cost) {
        best.bn = w; best.splits = s; best.warps = eight ? 8 : 4; best.cost = cost; best.steps = rounds * std::max<int64_t>(0, steps - 2);
      }
    }
  }
  return best;
}

}  // namespace

bool mb_gemm_f32_gather_supported(const mb_context *ctx, const mb_f32_gemm &g) {
  if (!ctx->use_tensor_cores || g.M < 1 || g.N < 1 || g.K < 1 || g.batch < 1) return false;
  if (g.M >= (1ll << 31) - 128 || g.N >= (1ll << 31) - 128 || g.K >= (1ll << 30) || g.batch >= (1ll << 31)) return false;
  if (g.batch * ceil_div64(g.M, BM) * ceil_div64(g.N, 64) * 8 >= (1ll << 31)) return false;
  if (g.conv)
    return g.KH <= 16 && g.KW <= 15 && static_cast<int64_t>(g.C_in) * g.H * g.Wd < (1ll << 30) &&
           g.C_in * static_cast<int64_t>(g.KH) * g.KW == g.K;
  if ((g.x_ms != 1 && g.x_ks != 1) || (g.w_ns != 1 && g.w_ks != 1)) return false;
  return g.x_ms != 1 || g.K * g.x_ks < (1ll << 31);
}

int64_t mb_gemm_f32_gather_cost(mb_context *ctx, const mb_f32_gemm &g) {
  const Plan plan = make_plan(ctx, g);
  // (X with its depth contiguous is a lane per row, 32 lines per load: 2550 cycles per step of 128 columns, 1950 of 64)
  return plan.cost + (!g.conv && g.x_ms != 1 ? plan.steps * (plan.bn == 128 ? 1300 : 850) : 0);
}

int mb_gemm_f32_gather_launch(mb_context *ctx, const mb_f32_gemm &g) {
  const Plan plan = make_plan(ctx, g);
  Params p = {};
  p.X = g.X; p.W = g.W; p.bias = g.bias; p.residual = g.residual; p.C = g.C;
  p.M = static_cast<int>(g.M); p.N = static_cast<int>(g.N); p.K = static_cast<int>(g.K); p.batch = static_cast<int>(g.batch);
  p.tiles_m = static_cast<int>(ceil_div64(g.M, BM));
  p.tiles_n = static_cast<int>(ceil_div64(g.N, plan.bn));
  p.k_blocks = static_cast<int>(ceil_div64(g.K, KB));
  p.splits = plan.splits;
  p.run = plan.bn == 128 ? std::min(g.run, 2) : g.run;  // (of the four steps that its ring holds)
  // (a residual that lies where the results do is gone by then)
  p.exact = g.run != 0 && !mb_ranges_meet(g.residual, g.C, g.batch * g.M * g.N * 4);
  p.x_ks = g.x_ks; p.x_ms = g.x_ms; p.x_bs = g.x_bs;
  p.w_ns = g.w_ns; p.w_ks = g.w_ks; p.w_bs = g.w_bs;
  p.c_ns = g.c_ns; p.c_ms = g.c_ms; p.c_bs = g.c_bs;
  p.act = g.act; p.max_limit = g.max_limit; p.coef = g.coef;
  p.status = ctx->dev_status;
  const bool w_nc = !g.conv && g.w_ks != 1;
  const bool w_tma = !w_nc && ctx->encode_tiled != nullptr && (reinterpret_cast<uintptr_t>(g.W) & 15u) == 0 &&
                     (g.conv ? g.K : g.w_ns) % 4 == 0 && g.w_bs % 4 == 0;
  if (g.conv) {
    p.H = g.H; p.Wd = g.Wd; p.KH = g.KH; p.KW = g.KW; p.taps = g.KH * g.KW;
    p.sh = g.sh; p.sw = g.sw; p.dh = g.dh; p.dw = g.dw; p.pad_t = g.pad_t; p.pad_l = g.pad_l;
    p.Wo = g.Wo; p.hw = g.Ho * g.Wo;
    p.image = static_cast<int64_t>(g.C_in) * g.H * g.Wd;
    p.w_ns = g.K; p.w_ks = 1;
    p.c_ns = p.hw;
    fast_div_make(static_cast<uint32_t>(p.taps), &p.taps_mul, &p.taps_shift);
    fast_div_make(static_cast<uint32_t>(p.KW), &p.kw_mul, &p.kw_shift);
    fast_div_make(static_cast<uint32_t>(p.hw), &p.hw_mul, &p.hw_shift);
    fast_div_make(static_cast<uint32_t>(p.Wo), &p.wo_mul, &p.wo_shift);
#define MB_F32_CONV(BN_, EW_, MODE_) \
  return w_tma ? launch_cfg<BN_, X_CONV, W_TMA, EW_, MODE_>(ctx, p) : launch_cfg<BN_, X_CONV, W_ROWS, EW_, MODE_>(ctx, p);
    if (p.run == 1 && p.k_blocks <= 2) {
      if (plan.bn == 128) { MB_F32_CONV(128, 8, SPREAD) }
      MB_F32_CONV(64, 4, SPREAD)
    }
    if (p.run != 0 && plan.bn == 128) { MB_F32_CONV(128, 8, RUNS) }
    if (plan.bn == 64 && (p.run != 0 || plan.warps == 4)) {
      // (one kernel for 64 channels with short runs or without: where a network's 1x1 and 3x3 layers took two in turn, every
      // launch began with the other's instructions in the caches, 30 us of ResNet-50's 570 at batch 1)
      if (p.run == 0) p.run = p.k_blocks;
      MB_F32_CONV(64, 4, RUNS)
    }
    if (plan.bn == 64) { MB_F32_CONV(64, 8, WHOLE) }
    if (plan.warps == 8) { MB_F32_CONV(128, 8, WHOLE) }
    MB_F32_CONV(128, 4, WHOLE)
#undef MB_F32_CONV
  }
  const bool cols = g.x_ms != 1;
  p.x_vec = cols && (reinterpret_cast<uintptr_t>(g.X) & 15u) == 0 && g.x_ms % 4 == 0 && g.x_bs % 4 == 0 && g.K % 4 == 0;
#define MB_F32_W(BN_, XK_, EW_, MODE_)                                           \
  if (w_nc) return launch_cfg<BN_, XK_, W_COLS, EW_, MODE_>(ctx, p);              \
  return w_tma ? launch_cfg<BN_, XK_, W_TMA, EW_, MODE_>(ctx, p) : launch_cfg<BN_, XK_, W_ROWS, EW_, MODE_>(ctx, p);
#define MB_F32(BN_, EW_, MODE_)                   \
  if (cols) { MB_F32_W(BN_, X_COLS, EW_, MODE_) } \
  MB_F32_W(BN_, X_ROWS, EW_, MODE_)
  if (p.run == 1 && p.k_blocks <= 2) {
    if (plan.bn == 128) { MB_F32(128, 8, SPREAD) }
    MB_F32(64, 4, SPREAD)
  }
  if (p.run != 0) {
    if (plan.bn == 128) { MB_F32(128, 8, RUNS) }
    MB_F32(64, 8, RUNS)
  }
  if (plan.warps == 8) {
    if (plan.bn == 128) { MB_F32(128, 8, WHOLE) }
    MB_F32(64, 8, WHOLE)
  }
  if (plan.bn == 128) { MB_F32(128, 4, WHOLE) }
  MB_F32(64, 4, WHOLE)
#undef MB_F32
#undef MB_F32_W
}
