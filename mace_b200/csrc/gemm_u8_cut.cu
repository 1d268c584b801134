// uint8 x uint8 -> int32 GEMM on tcgen05, one tile per CTA, the depth cut over a cluster of up to eight
// CTAs: a few rows against a large matrix, k x k convolutions, FullyConnected on a batch.
//
// What it replaces: gemmlowp's GEMM and the Im2col in front of it as MACE's quantized MatMul, Conv2D and
// FullyConnected call them (mace/ops/matmul.cc:283-301, mace/ops/conv_2d.cc:301-412,
// mace/ops/arm/q8/gemv.cc:36-171).
//
// Roles (ten warps): one thread requests the tiles by TMA -- a convolution's windows in im2col mode, one
// channel run of one filter tap per step, straight from the NHWC input --, one issues the MMAs, four
// warps look after A and four after B: they add up the operand bytes for the zero-point terms from
// the tiles in shared memory, and, for a padded convolution, write the input zero point over the pixels
// outside the image (TMA fills them with zeros) before the MMA may read the tile.
//
// Why a cut, and why this way.  A persistent CTA per 128 x 256 tile (gemm_u8_tc.cu) leaves most SMs without
// work when there are few tiles and walks the whole depth with the rest.  Here every CTA of a cluster
// takes a run of the depth, leaves its exact int32 tile in its own shared memory, and after a cluster
// barrier every CTA adds up and requantizes its share of the tile out of all of them: no workspace in global
// memory, no second kernel, no counters.  The barrier costs 0.2 us.  What bounds it: the chain launch ->
// first tile -> MMAs -> epilogue (about 5 us back to back) for the small shapes, the bytes a CTA can pull
// for the long ones.  16 rows against 4096 x 4096: 10.9 us with the
// depth cut through global memory (gemm_u8.cu), 7.7 here.  41 vectors through 5696 -> 1200: 41.4 us on CUDA cores,
// 7.0 here.  3x3 over 14 x 14 x 240 -> 48: 32.8 us with the patches written out, 6.4 here.
#include <algorithm>

#include "gemm_u8_cut.cuh"
#include "gemm_u8_tail.cuh"

int mb_make_map_u8(mb_context *ctx, CUtensorMap *map, const void *base, uint64_t inner, uint64_t rows, uint64_t batch,
                   uint64_t batch_stride_bytes, uint32_t box_inner, uint32_t box_rows, CUtensorMapSwizzle swizzle,
                   uint64_t row_pitch);
int mb_gemm_u8_tc_launch_conv(mb_context *ctx, const mb_cut_gemm &g, const CUtensorMap &map_a, const CUtensorMap &map_b,
                              int bn, int kbt, int c_blocks, int patch);

namespace {

using namespace sm100;

constexpr int WORK_WARPS = 8;                 // 0..3 look after A, 4..7 after B, all of them store the result
constexpr int MMA_WARP = 8, TMA_WARP = 9;
constexpr int THREADS = 320;
constexpr long long WAIT_BUDGET = 1ll << 31;  // ~1 s of SM clocks per wait
enum { A_KMAJOR = 0, A_MN = 1, A_CONV = 2 };

struct Params {
  TailParams tail;
  int tiles_m, tiles_n, k_blocks;
  int a_batched, b_batched;
  uint32_t a_tx;      // bytes of an A box
  int patch;          // convolution windows reach outside the image and the zero point is not 0
  int H, W, Cin, KW, sh, sw, pad_t, pad_l, Ho, Wo, c_blocks;
  uint32_t wo_mul, wo_shift, ho_mul, ho_shift;
  int *status;
};

// KBT: depth bytes per step and operand row (128; a convolution of few channels: 64 or 32)
template <int BN, bool B_MN, int KBT, int CTAS>
struct Cfg {
  static_assert(!B_MN || KBT == 128, "row-major B: 128 depth rows per step");
  static constexpr int A_BYTES = 128 * KBT;
  static constexpr int B_BYTES = BN * KBT;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int FIT = (CTAS == 2 ? 104 : 208) * 1024 / STAGE_BYTES;
  static constexpr int STAGES = FIT > 12 ? 12 : FIT;
  static constexpr int RING = STAGES * STAGE_BYTES;
  static_assert(128 * TAIL_PITCH<BN> * 4 <= RING, "the int32 tile reuses the ring");
  static constexpr int SMEM_BYTES = RING + 1024 /*align*/ + 512 /*barriers*/ + (128 + BN) * 4;
  static_assert(CTAS * (SMEM_BYTES + 1024) <= 227 * 1024, "shared memory");
};

// Byte sum of row r of a K-major tile (the swizzle permutes 16-byte chunks inside a row, which a sum does
// not see; starting at chunk r spreads a quarter warp over the banks).  Four chains: one would be 32
// dependent instructions per step.
template <int KBT>
__device__ __forceinline__ uint32_t row_sum(const uint8_t *tile, int r, uint32_t s) {
  uint32_t s1 = 0, s2 = 0, s3 = 0;
#pragma unroll
  for (int i = 0; i < KBT / 16; ++i) {
    const uint4 v = *reinterpret_cast<const uint4 *>(tile + r * KBT + ((i + r) & (KBT / 16 - 1)) * 16);
    s = __dp4a(v.x, 0x01010101u, s);
    s1 = __dp4a(v.y, 0x01010101u, s1);
    s2 = __dp4a(v.z, 0x01010101u, s2);
    s3 = __dp4a(v.w, 0x01010101u, s3);
  }
  return (s + s1) + (s2 + s3);
}

// Column sums of an MN-major tile [128 depth rows][PANEL bytes]: warp q takes depth rows 32 q .. 32 q + 31, a lane
// one word of a row (128 bytes: a row per load, 64: two), as pairs of 16-bit counts.
template <int PANEL>
__device__ __forceinline__ void col_sums(const uint8_t *tile, int q, int lane, uint32_t (&s)[4]) {
  constexpr int RPP = 128 / PANEL;  // rows per pass
  const int word = lane % (PANEL / 4), k0 = q * 32 + lane / (PANEL / 4);
  const int c = word >> 2;
  const uint8_t *p = tile + k0 * PANEL + (word & 3) * 4;
  uint32_t ev = 0, od = 0;
#pragma unroll
  for (int i = 0; i < 32; i += RPP) {
    const int swz = PANEL == 128 ? (i & 7) : ((k0 + i) >> 1) & 3;
    const uint32_t w = *reinterpret_cast<const uint32_t *>(p + i * PANEL + ((c ^ swz) << 4));
    ev += w & 0x00ff00ffu;
    od += __byte_perm(w, 0, 0x4341);
  }
  s[0] += ev & 0xffffu;
  s[1] += od & 0xffffu;
  s[2] += ev >> 16;
  s[3] += od >> 16;
}

template <int BN, int A_KIND, bool B_MN, int KBT, int CTAS>
__global__ void __launch_bounds__(THREADS, CTAS)
gemm_u8_cut_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                   const __grid_constant__ Params p) {
  using C = Cfg<BN, B_MN, KBT, CTAS>;
  constexpr int STAGES = C::STAGES;
  constexpr bool A_IS_MN = A_KIND == A_MN;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t *smem = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t full_bar = smem_base + C::RING;             // tile landed
  const uint32_t ready_bar = full_bar + 8 * STAGES;          // ... and its outside pixels overwritten
  const uint32_t empty_bar = ready_bar + 8 * STAGES;         // tile consumed
  const uint32_t done_bar = empty_bar + 8 * STAGES;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + C::RING + 24 * STAGES + 8);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  uint32_t *row_sums = reinterpret_cast<uint32_t *>(smem + C::RING + 512);  // [128]
  uint32_t *column_sums = row_sums + 128;                                   // [BN]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool patch = A_KIND == A_CONV && p.patch;
  const bool want_a = p.tail.zp_b != 0, want_b = p.tail.zp_a != 0;
  mb_grid_dep_launch();

  if (threadIdx.x == MMA_WARP * 32) {
    prefetch_tensormap(&map_a);
    prefetch_tensormap(&map_b);
    const int users = 1 + ((want_a || patch) ? 4 : 0) + (want_b ? 4 : 0);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar + 8 * s, 1);
      mbar_init(ready_bar + 8 * s, 4);
      mbar_init(empty_bar + 8 * s, users);
    }
    mbar_init(done_bar, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == TMA_WARP) {
    tmem_alloc(smem_u32(tmem_slot), BN);
    tmem_relinquish();
  }
  for (int i = threadIdx.x; i < 128 + BN; i += THREADS) row_sums[i] = 0;

  // which tile, and which run of its depth
  const int rank = p.tail.splits > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const unsigned t = blockIdx.x / static_cast<unsigned>(p.tail.splits);
  const int tm = t % p.tiles_m;
  const unsigned q = t / p.tiles_m;
  const int tn = q % p.tiles_n, b = q / p.tiles_n;
  const int m0 = tm * 128, n0 = tn * BN;
  const int kb_begin = static_cast<int>(static_cast<int64_t>(p.k_blocks) * rank / p.tail.splits);
  const int steps = static_cast<int>(static_cast<int64_t>(p.k_blocks) * (rank + 1) / p.tail.splits) - kb_begin;
  // convolution: the tap and channel run of the first step, and the window of a pixel
  int tap_h = 0, tap_w = 0, cb = 0;
  if (A_KIND == A_CONV) {
    const int tap = kb_begin / p.c_blocks;
    cb = kb_begin - tap * p.c_blocks;
    tap_h = tap / p.KW;
    tap_w = tap - tap_h * p.KW;
  }
  auto next_tap = [&] {
    if (++cb == p.c_blocks) {
      cb = 0;
      if (++tap_w == p.KW) {
        tap_w = 0;
        ++tap_h;
      }
    }
  };
  auto corner = [&](int pix, int &n, int &h, int &w) {
    const uint32_t r = fast_div(static_cast<uint32_t>(pix), p.wo_mul, p.wo_shift);
    const uint32_t img = fast_div(r, p.ho_mul, p.ho_shift);
    n = static_cast<int>(img);
    h = static_cast<int>(r - img * static_cast<uint32_t>(p.Ho)) * p.sh - p.pad_t;
    w = (pix - static_cast<int>(r) * p.Wo) * p.sw - p.pad_l;
  };
  auto fail = [&](int code) {
    *abort_flag = 1;
    atomicCAS(p.status, 0, code);
  };

  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  mb_grid_dep_wait();

  if (warp == TMA_WARP) {
    if (lane == 0) {
      int img = 0, h0 = 0, w0 = 0;
      if (A_KIND == A_CONV) corner(m0, img, h0, w0);
      const int ab = p.a_batched ? b : 0, bb = p.b_batched ? b : 0;
      int stage = 0;
      uint32_t phase = 1;
      for (int i = 0; i < steps; ++i) {
        if (!mbar_wait(empty_bar + 8 * stage, phase, abort_flag, WAIT_BUDGET)) {
          fail(MB_DEV_TIMEOUT_PRODUCER);
          break;
        }
        const uint32_t fb = full_bar + 8 * stage, sa = smem_base + stage * C::STAGE_BYTES, sb = sa + C::A_BYTES;
        const int k = (kb_begin + i) * KBT;
        mbar_arrive_expect_tx(fb, p.a_tx + C::B_BYTES);
        if (A_KIND == A_CONV) {
          tma_load_im2col_4d(sa, &map_a, fb, cb * KBT, w0, h0, img, static_cast<uint16_t>(tap_w), static_cast<uint16_t>(tap_h));
          tma_load_3d(sb, &map_b, fb, cb * KBT, n0, tap_h * p.KW + tap_w);
          next_tap();
        } else {
          if (A_IS_MN) tma_load_3d(sa, &map_a, fb, m0, k, ab);
          else tma_load_3d(sa, &map_a, fb, k, m0, ab);
          if (B_MN) tma_load_3d(sb, &map_b, fb, n0, k, bb);
          else tma_load_3d(sb, &map_b, fb, k, n0, bb);
        }
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
    __syncwarp();
  } else if (warp == MMA_WARP) {
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc(/*c s32*/ 2, /*a u8*/ 0, /*b u8*/ 0, A_IS_MN, B_MN, 128, BN);
      // (operand layouts as in gemm_u8_tc.cu)
      constexpr uint32_t SWZ = KBT == 128 ? 2u : KBT == 64 ? 4u : 6u;
      const uint64_t a_base = A_IS_MN ? make_smem_desc(0, 128 * 128, 1024, 2) : make_smem_desc(0, 16, 8 * KBT, SWZ);
      const uint64_t b_base = B_MN ? make_smem_desc(0, BN * 128, 8 * BN, BN == 128 ? 2 : 4) : make_smem_desc(0, 16, 8 * KBT, SWZ);
      constexpr uint32_t a_step = (A_IS_MN ? 32 * 128 : 32) >> 4, b_step = (B_MN ? 32 * BN : 32) >> 4;
      const uint32_t landed = patch ? ready_bar : full_bar;
      int stage = 0;
      uint32_t phase = 0;
      for (int i = 0; i < steps; ++i) {
        if (!mbar_wait(landed + 8 * stage, phase, abort_flag, WAIT_BUDGET)) {
          fail(MB_DEV_TIMEOUT_MMA);
          break;
        }
        tc_fence_after_sync();
        const uint32_t sa = smem_base + stage * C::STAGE_BYTES;
        const uint64_t a_desc = a_base | static_cast<uint64_t>((sa >> 4) & 0x3FFFu);
        const uint64_t b_desc = b_base | static_cast<uint64_t>(((sa + C::A_BYTES) >> 4) & 0x3FFFu);
#pragma unroll
        for (int j = 0; j < KBT / 32; ++j)
          mma_i8_ss(tmem, a_desc + j * a_step, b_desc + j * b_step, idesc, (i > 0 || j > 0) ? 1u : 0u);
        mma_commit(empty_bar + 8 * stage);
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
      mma_commit(done_bar);
    }
    __syncwarp();
  } else {
    const bool for_a = warp < 4;
    const int r = threadIdx.x & 127;  // tile row of a K-major operand
    if (for_a ? (want_a || patch) : want_b) {
      int img, h0 = 0, w0 = 0;
      if (A_KIND == A_CONV && for_a) corner(m0 + r, img, h0, w0);
      uint32_t sum = 0, cs[4] = {0, 0, 0, 0};
      int stage = 0;
      uint32_t phase = 0;
      for (int i = 0; i < steps; ++i) {
        if (!mbar_wait_warp(full_bar + 8 * stage, phase, abort_flag, WAIT_BUDGET)) {
          fail(MB_DEV_TIMEOUT_EPILOGUE);
          break;
        }
        uint8_t *tile = smem + stage * C::STAGE_BYTES + (for_a ? 0 : C::A_BYTES);
        if (for_a && patch) {
          const int h = h0 + tap_h, w = w0 + tap_w;
          const bool outside = h < 0 || h >= p.H || w < 0 || w >= p.W;
          if (outside) {
            // this pixel's channel run lies outside the image: the zero point, in the real channels
            const uint32_t z = static_cast<uint32_t>(p.tail.zp_a) * 0x01010101u;
            const int chunks = min(KBT, p.Cin - cb * KBT) / 16;
            const int swz = KBT == 128 ? (r & 7) : KBT == 64 ? ((r >> 1) & 3) : ((r >> 2) & 1);
            for (int c = 0; c < chunks; ++c)
              *reinterpret_cast<uint4 *>(tile + r * KBT + ((c ^ swz) << 4)) = make_uint4(z, z, z, z);
          }
          next_tap();
          if (__any_sync(0xffffffffu, outside)) {
            fence_proxy_async();
            __syncwarp();
          }
          if (lane == 0) mbar_arrive(ready_bar + 8 * stage);
        }
        if (for_a) {
          if (want_a) {
            if (A_IS_MN) col_sums<128>(tile, warp, lane, cs);
            else sum = row_sum<KBT>(tile, r, sum);
          }
        } else if (B_MN) {
          col_sums<BN>(tile, warp - 4, lane, cs);
        } else if (r < BN) {
          sum = row_sum<KBT>(tile, r, sum);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty_bar + 8 * stage);
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
      uint32_t *sums = for_a ? row_sums : column_sums;
      if (for_a ? A_IS_MN : B_MN) {
#pragma unroll
        for (int j = 0; j < 4; ++j) atomicAdd(sums + 4 * (for_a || BN == 128 ? lane : lane & 15) + j, cs[j]);
      } else if (for_a || r < BN) {
        sums[r] = sum;
      }
    }
    if (!mbar_wait_warp(done_bar, 0, abort_flag, WAIT_BUDGET)) fail(MB_DEV_TIMEOUT_EPILOGUE);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (*abort_flag != 0) {
    // copies and MMAs in flight must not outlive the memory they write (bounded: about 2 ms)
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }

  finish_tile<BN, WORK_WARPS>(p.tail, reinterpret_cast<int32_t *>(smem), tmem, row_sums, column_sums, m0, n0, b, rank, warp, lane);
  // no CTA of a cluster may leave while another still reads its tile
  if (p.tail.splits > 1) cluster_sync_all();
  else __syncthreads();
  if (warp == TMA_WARP) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, BN);
  }
}

template <int BN, int A_KIND, bool B_MN, int KBT, int CTAS>
int launch_cfg(mb_context *ctx, const CUtensorMap &ma, const CUtensorMap &mb, const Params &p, int64_t batch) {
  using C = Cfg<BN, B_MN, KBT, CTAS>;
  auto kern = gemm_u8_cut_kernel<BN, A_KIND, B_MN, KBT, CTAS>;
  constexpr uint64_t bit = 8 + (CTAS == 2 ? 24 : 0) + (BN == 128 ? 12 : 0) +
                           (A_KIND == A_CONV ? (KBT == 128 ? 8 : KBT == 64 ? 9 : 10) : A_KIND * 2 + (B_MN ? 1 : 0));
  if (!(ctx->cut_attr_mask & (1ull << bit))) {
    MB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
    ctx->cut_attr_mask |= 1ull << bit;
  }
  const unsigned grid = static_cast<unsigned>(batch * p.tiles_m * p.tiles_n * p.tail.splits);
  MB_CUDA(ctx, mb_launch_clusters(ctx, kern, grid, THREADS, C::SMEM_BYTES, p.tail.splits, ma, mb, p));
  ctx->launches++;
  ctx->launches_tc++;
  return MB_SUCCESS;
}

// Depth bytes per step of a convolution with C channels: whole swizzled rows unless more than a third of
// one would lie beyond the last channel.
int conv_kbt(int64_t C) {
  for (int k : {128, 64})
    if (3 * static_cast<int64_t>(align_up(static_cast<size_t>(C), k)) <= 4 * C) return k;
  return 32;
}

typedef CUresult (*EncodeIm2colFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const int *, const int *, cuuint32_t, cuuint32_t,
                                   const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// Right / bottom end of the box that the windows' top-left corners run over, relative to the image's.
int upper_corner(int extent, int out, int stride, int pad) { return (out - 1) * stride - pad - (extent - 1); }

bool conv_map_possible(const mb_context *ctx, const mb_cut_gemm &g) {
  auto byte = [](int v) { return v >= -128 && v <= 127; };
  return ctx->encode_im2col != nullptr && g.sh <= 8 && g.sw <= 8 && byte(-g.pad_t) && byte(-g.pad_l) && g.KH <= 256 &&
         g.KW <= 256 && byte(upper_corner(g.H, g.Ho, g.sh, g.pad_t)) && byte(upper_corner(g.W, g.Wo, g.sw, g.pad_l));
}

}  // namespace

// CTAs of clusters of `s` that the device holds at once with one CTA per SM (a cluster lies inside a
// GPC, and not every GPC has a whole number of clusters' SMs).
int64_t mb_resident_cluster_ctas(mb_context *ctx, int s) {
  if (s == 1) return ctx->num_sms;
  const int slot = s == 2 ? 1 : s == 4 ? 2 : 3;
  if (ctx->cut_clusters[slot] == 0) {
    using C = Cfg<128, false, 128, 1>;
    auto kern = gemm_u8_cut_kernel<128, A_KMAJOR, false, 128, 1>;
    cudaLaunchConfig_t probe = {};
    probe.gridDim = dim3(static_cast<unsigned>(ctx->num_sms / s * s));
    probe.blockDim = dim3(THREADS);
    probe.dynamicSmemBytes = C::SMEM_BYTES;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(s);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    probe.attrs = attr;
    probe.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &probe) != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = std::max(1, (ctx->num_sms - 20) / s);
    }
    ctx->cut_clusters[slot] = n * s;
  }
  return ctx->cut_clusters[slot];
}

mb_cut_plan mb_gemm_u8_cut_plan(mb_context *ctx, const mb_cut_gemm &g) {
  mb_cut_plan best;
  // 255 * 255 * K must stay below 2^31
  if (g.M < 1 || g.N < 1 || g.K < 1 || g.K > 33000 || g.M >= (1ll << 31) - 128 || g.N >= (1ll << 31) - 128) return best;
  const int64_t lda = g.lda != 0 ? g.lda : g.a_mn ? g.M : g.K, ldb = g.ldb != 0 ? g.ldb : g.b_mn ? g.N : g.K;
  const bool aligned = ((reinterpret_cast<uintptr_t>(g.A) | reinterpret_cast<uintptr_t>(g.B)) & 15u) == 0 &&
                       (g.conv ? g.C_in % 16 == 0 : (lda | ldb) % 16 == 0);
  const bool by_tma = aligned && ctx->encode_tiled != nullptr && (!g.conv || conv_map_possible(ctx, g));
  if (g.conv && !by_tma) return best;
  // the 16-bit column counts of gemm_u8_gather.cu hold 64 steps of each of its two groups
  if (!by_tma && (g.a_mn || g.b_mn) && g.K > 16384) return best;
  const int64_t tiles_m = ceil_div64(g.M, 128);
  const int kbt = g.conv ? conv_kbt(g.C_in) : 128;
  const int64_t k_blocks = g.conv ? static_cast<int64_t>(g.KH) * g.KW * ceil_div64(g.C_in, kbt) : ceil_div64(g.K, 128);
  if (g.batch * tiles_m * ceil_div64(g.N, 64) * 8 >= (1ll << 31)) return best;
  int asked = ctx->cut_splits;
  while (asked > k_blocks) asked /= 2;
  // the combination with the smallest estimate, in SM cycles, of rounds of CTAs x (start and end of a
  // CTA + its steps).  Measured: 5 us around the steps of the first round, 4.5 us around those of a further
  // one; 0.35 us per step of 128 + 128 rows by TMA (0.26 us at 64), 0.55 us where one operand is a
  // convolution's windows (128 pixels in im2col mode and their outside ones overwritten; 0.45 us on the
  // persistent kernel, which hides the start and the end of its tiles)
  for (int w : {128, 64}) {
    if (ctx->cut_bn != 0 ? w != ctx->cut_bn : (w == 128 && g.N <= 64)) continue;
    const int64_t tiles = g.batch * tiles_m * ceil_div64(g.N, w);
    if (g.conv && ctx->cut_two != 1 && ctx->cut_two != 2 && asked == 0) {
      const int64_t cost = 8500 + ceil_div64(tiles, ctx->num_sms) * std::max<int64_t>(k_blocks * (w == 128 ? 900 : 800), w == 128 ? 1500 : 1000);
      if (best.cost < 0 || cost < best.cost) {
        best.bn = w; best.splits = 1; best.by_tma = true; best.persistent = true; best.cost = cost;
      }
    }
    if (ctx->cut_two == 3 && g.conv) continue;
    for (int s : {1, 2, 4, 8}) {
      if (asked != 0 ? s != asked : (s > 1 && s * 2 > k_blocks)) continue;
      const int64_t sms = mb_resident_cluster_ctas(ctx, s);
      const int64_t steps = ceil_div64(k_blocks, s);
      for (int two : {0, 1}) {
        if ((two && !g.conv) || ((ctx->cut_two == 1 || ctx->cut_two == 2) && by_tma && two != ctx->cut_two - 1)) continue;
        const int64_t rounds = ceil_div64(tiles * s, sms * (two ? 2 : 1));
        int64_t step = !by_tma ? (w == 128 ? 2300 : 1750) : g.conv ? (w == 128 ? 1050 : 980) : g.b_mn ? (w == 128 ? 660 : 560) : (w == 128 ? 520 : 430);
        if (two && tiles * s > sms) step = step * 8 / 5;
        // what follows the steps: up to 128 x w values through shared memory, shared by the cluster
        const int64_t tail = std::min<int64_t>(128, g.M) * w * 7 / 16 / s;
        const int64_t cost = 9500 + (s > 1 ? 300 : 0) + (rounds - 1) * 8500 + rounds * steps * step + tail;
        if (best.cost < 0 || cost < best.cost) {
          best.bn = w; best.splits = s; best.by_tma = by_tma; best.two_per_sm = two != 0;
          best.persistent = false; best.cost = cost;
        }
      }
    }
  }
  return best;
}

int mb_gemm_u8_cut_launch(mb_context *ctx, const mb_cut_gemm &g, const mb_cut_plan &plan) {
  if (!plan.by_tma) return mb_gemm_u8_gather_launch(ctx, g, plan.bn, plan.splits);
  Params p = {};
  p.tail = make_tail(g, plan.splits);
  p.a_batched = g.a_batched; p.b_batched = g.b_batched;
  p.tiles_m = static_cast<int>(ceil_div64(g.M, 128));
  p.tiles_n = static_cast<int>(ceil_div64(g.N, plan.bn));
  p.status = ctx->dev_status;
  const int kbt = g.conv ? conv_kbt(g.C_in) : 128;
  CUtensorMap ma, mb;
  if (g.conv) {
    p.c_blocks = static_cast<int>(ceil_div64(g.C_in, kbt));
    p.k_blocks = g.KH * g.KW * p.c_blocks;
    p.H = g.H; p.W = g.W; p.Cin = g.C_in; p.KW = g.KW; p.sh = g.sh; p.sw = g.sw;
    p.pad_t = g.pad_t; p.pad_l = g.pad_l; p.Ho = g.Ho; p.Wo = g.Wo;
    fast_div_make(static_cast<uint32_t>(g.Wo), &p.wo_mul, &p.wo_shift);
    fast_div_make(static_cast<uint32_t>(g.Ho), &p.ho_mul, &p.ho_shift);
    p.patch = g.zp_a != 0 && (g.pad_t > 0 || g.pad_l > 0 || (g.Ho - 1) * g.sh - g.pad_t + g.KH > g.H ||
                              (g.Wo - 1) * g.sw - g.pad_l + g.KW > g.W);
    p.a_tx = 128 * kbt;
    const CUtensorMapSwizzle swz = kbt == 32   ? CU_TENSOR_MAP_SWIZZLE_32B
                                   : kbt == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                                               : CU_TENSOR_MAP_SWIZZLE_128B;
    const int64_t C = g.C_in, images = g.M / (static_cast<int64_t>(g.Ho) * g.Wo);
    const cuuint64_t dims[4] = {static_cast<cuuint64_t>(C), static_cast<cuuint64_t>(g.W), static_cast<cuuint64_t>(g.H),
                                static_cast<cuuint64_t>(images)};
    const cuuint64_t strides[3] = {static_cast<cuuint64_t>(C), static_cast<cuuint64_t>(C * g.W),
                                   static_cast<cuuint64_t>(C * g.W * g.H)};
    const int lower[2] = {-g.pad_l, -g.pad_t};
    const int upper[2] = {upper_corner(g.W, g.Wo, g.sw, g.pad_l), upper_corner(g.H, g.Ho, g.sh, g.pad_t)};
    const cuuint32_t estr[4] = {1, static_cast<cuuint32_t>(g.sw), static_cast<cuuint32_t>(g.sh), 1};
    const CUresult r = reinterpret_cast<EncodeIm2colFn>(ctx->encode_im2col)(
        &ma, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<uint8_t *>(g.A), dims, strides, lower, upper,
        static_cast<cuuint32_t>(kbt), 128, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
      return mb_fail(ctx, MB_RUNTIME_ERROR, "cuTensorMapEncodeIm2col failed (%d)", static_cast<int>(r));
    // the filter as [taps][O][C]: channels beyond the last arrive as zeros, like those of the windows
    MB_RETURN_IF_ERROR(mb_make_map_u8(ctx, &mb, g.B, C, g.N, static_cast<uint64_t>(g.KH) * g.KW, C, kbt, plan.bn, swz,
                                      static_cast<uint64_t>(g.KH) * g.KW * C));
    if (plan.persistent) return mb_gemm_u8_tc_launch_conv(ctx, g, ma, mb, plan.bn, kbt, p.c_blocks, p.patch);
  } else {
    p.k_blocks = static_cast<int>(ceil_div64(g.K, 128));
    const int64_t lda = g.lda != 0 ? g.lda : g.a_mn ? g.M : g.K, ldb = g.ldb != 0 ? g.ldb : g.b_mn ? g.N : g.K;
    const uint64_t nb_a = g.a_batched ? g.batch : 1, nb_b = g.b_batched ? g.batch : 1;
    // (few rows: the box holds no more than they need)
    const uint32_t a_rows = g.a_mn ? 128 : static_cast<uint32_t>(std::min<int64_t>(128, align_up(static_cast<size_t>(g.M), 8)));
    p.a_tx = a_rows * 128;
    if (g.a_mn)
      MB_RETURN_IF_ERROR(mb_make_map_u8(ctx, &ma, g.A, g.M, g.K, nb_a, g.K * lda, 128, 128, CU_TENSOR_MAP_SWIZZLE_128B, lda));
    else
      MB_RETURN_IF_ERROR(mb_make_map_u8(ctx, &ma, g.A, g.K, g.M, nb_a, g.M * lda, 128, a_rows, CU_TENSOR_MAP_SWIZZLE_128B, lda));
    if (g.b_mn)
      MB_RETURN_IF_ERROR(mb_make_map_u8(ctx, &mb, g.B, g.N, g.K, nb_b, g.K * ldb, plan.bn, 128,
                                        plan.bn == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, ldb));
    else
      MB_RETURN_IF_ERROR(mb_make_map_u8(ctx, &mb, g.B, g.K, g.N, nb_b, g.N * ldb, 128, plan.bn, CU_TENSOR_MAP_SWIZZLE_128B, ldb));
  }
#define MB_CUT_CONV(BN_, CTAS_)                                                                     \
  if (kbt == 128) return launch_cfg<BN_, A_CONV, false, 128, CTAS_>(ctx, ma, mb, p, 1);             \
  if (kbt == 64) return launch_cfg<BN_, A_CONV, false, 64, CTAS_>(ctx, ma, mb, p, 1);               \
  return launch_cfg<BN_, A_CONV, false, 32, CTAS_>(ctx, ma, mb, p, 1);
#define MB_CUT(BN_)                                                                                 \
  if (g.b_mn)                                                                                       \
    return g.a_mn ? launch_cfg<BN_, A_MN, true, 128, 1>(ctx, ma, mb, p, g.batch)                    \
                  : launch_cfg<BN_, A_KMAJOR, true, 128, 1>(ctx, ma, mb, p, g.batch);               \
  return g.a_mn ? launch_cfg<BN_, A_MN, false, 128, 1>(ctx, ma, mb, p, g.batch)                     \
                : launch_cfg<BN_, A_KMAJOR, false, 128, 1>(ctx, ma, mb, p, g.batch);
  if (g.conv) {
    if (plan.two_per_sm) {
      if (plan.bn == 64) { MB_CUT_CONV(64, 2) }
      MB_CUT_CONV(128, 2)
    }
    if (plan.bn == 64) { MB_CUT_CONV(64, 1) }
    MB_CUT_CONV(128, 1)
  }
  if (plan.bn == 64) { MB_CUT(64) }
  MB_CUT(128)
#undef MB_CUT_CONV
#undef MB_CUT
}
