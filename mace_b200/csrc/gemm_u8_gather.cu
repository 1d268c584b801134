// uint8 x uint8 -> int32 GEMM on tcgen05 for operands whose rows lie at any byte alignment, which TMA
// cannot fetch.
//
// What it replaces: gemmlowp's packing of unaligned operands as MACE's quantized MatMul and
// FullyConnected call it (mace/ops/matmul.cc:283-301, mace/ops/arm/q8/gemv.cc:36-171), in ONE launch:
// sixteen warps load the bytes of a 128 x BN x 128 step into registers, shift them into place,
// store them in the swizzled layout the tensor core reads, and add up the operand bytes for the
// zero-point terms as they pass; one thread issues the MMAs.
//
// What bounds it: the loads.  Five words per 16 bytes, four rows per instruction, make a step about 1300
// L1 wavefronts (1.2 us at width 128, 0.9 us at 64, against 0.3 us for aligned rows by TMA); around the steps
// lie about 5.5 us of launch, first load and epilogue.  It is the way for products of few steps: a copy that
// makes the rows addressable costs a launch of its own.  Two groups of eight warps take alternate
// steps, which keeps two steps (64 KB) of loads in flight per SM.  132 x 126 x 417: 65.6 us on the CUDA cores, one
// multiply-add per value, 7.6 us here.
#include <algorithm>

#include "gemm_u8_cut.cuh"
#include "gemm_u8_tail.cuh"

namespace {

using namespace sm100;

constexpr int KB = 128;              // depth per step: one 128-byte swizzled row
constexpr int GROUP_WARPS = 8;       // warps that load one step
constexpr int GROUPS = 2;
constexpr int LOAD_WARPS = GROUP_WARPS * GROUPS;
constexpr int THREADS = (LOAD_WARPS + 1) * 32;
constexpr int STAGES = 4;
constexpr long long WAIT_BUDGET = 1ll << 31;  // ~1 s of SM clocks per wait

struct Params {
  TailParams tail;
  const uint8_t *A, *B;
  int K;
  int64_t lda, ldb;         // bytes from row to row
  int64_t a_bs, b_bs;       // bytes from matrix to matrix of a batch (0: shared)
  int tiles_m, tiles_n, k_blocks;
  int *status;
};

template <int BN, bool B_MN>
struct Cfg {
  static constexpr int A_BYTES = 128 * KB;
  static constexpr int B_BYTES = B_MN ? 128 * KB : BN * KB;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int RING = STAGES * STAGE_BYTES;
  static_assert(128 * TAIL_PITCH<BN> * 4 <= RING, "the int32 tile reuses the ring");
  static constexpr int SMEM_BYTES = RING + 1024 /*align*/ + 256 /*barriers*/ + (128 + BN) * 4;
};

// Sixteen bytes at any address as five aligned words, of which only those that hold one of the
// `valid` bytes are read.
__device__ __forceinline__ void load_bytes(const uint8_t *q, int valid, uint32_t (&w)[5]) {
  const int off = static_cast<int>(reinterpret_cast<uintptr_t>(q) & 3u);
  const uint32_t *a = reinterpret_cast<const uint32_t *>(q - off);
  if (valid >= 16) {
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = mb_load(a + j);
    w[4] = mb_load(a + (off != 0 ? 4 : 3));
  } else {
    const int need = valid > 0 ? valid + off : 0;
#pragma unroll
    for (int j = 0; j < 5; ++j) w[j] = 4 * j < need ? mb_load(a + j) : 0u;
  }
}

// The words shifted into place, bytes from `valid` on cleared.
__device__ __forceinline__ uint4 place(const uint32_t (&w)[5], int off, int valid) {
  uint32_t v[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) v[j] = __funnelshift_r(w[j], w[j + 1], off * 8);
  if (valid < 16) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int left = valid - 4 * j;
      v[j] = left >= 4 ? v[j] : left <= 0 ? 0u : v[j] & ((1u << (8 * left)) - 1u);
    }
  }
  return make_uint4(v[0], v[1], v[2], v[3]);
}

__device__ __forceinline__ uint32_t sum16(const uint4 v, uint32_t s) {
  s = __dp4a(v.x, 0x01010101u, s);
  s = __dp4a(v.y, 0x01010101u, s);
  s = __dp4a(v.z, 0x01010101u, s);
  return __dp4a(v.w, 0x01010101u, s);
}

// One thread's share of an operand's tile: CHUNKS chunks of 16 bytes per step.
//   K-major: row i * 32 + warp * 4 + lane / 8 of the tile, chunk lane % 8 of its 128 depth bytes
//   MN:      depth row (the same expression), chunk of the 128 (64) values along M or N
template <bool MN, int WIDTH>
struct Loader {
  static constexpr int PER_ROW = MN ? WIDTH / 16 : 8;       // chunks of a row
  static constexpr int ROWS = MN ? KB : WIDTH;
  static constexpr int LANE_ROWS = 32 / PER_ROW;            // rows per warp and pass
  static constexpr int STEP = LANE_ROWS * GROUP_WARPS;      // rows per pass of a group
  static constexpr int CHUNKS = ROWS / STEP;
  const uint8_t *base;   // first row of this thread, first step
  int64_t ld;
  int row0, chunk;       // of this thread in the tile
  int row_limit;         // K-major: rows of the tile inside the matrix; MN: depth
  int inner_limit;       // K-major: depth; MN: values of the tile along M / N inside the matrix
  int offs;              // byte offsets of the chunks inside their words, two bits each
  uint32_t w[CHUNKS][5];
  uint32_t sum[MN ? 8 : CHUNKS];  // K-major: a sum per row; MN: 16-bit counts of 16 columns, even and odd

  __device__ __forceinline__ void init(const uint8_t *matrix, int extent, int K, int64_t pitch, int first, int gwarp, int lane) {
    row0 = gwarp * LANE_ROWS + lane / PER_ROW;
    chunk = lane % PER_ROW;
    ld = pitch;
    row_limit = MN ? K : extent - first;
    inner_limit = MN ? extent - first : K;
    base = MN ? matrix + static_cast<int64_t>(row0) * ld + first + chunk * 16
              : matrix + static_cast<int64_t>(first + row0) * ld + chunk * 16;
    offs = 0;
#pragma unroll
    for (int i = 0; i < CHUNKS; ++i)
      offs |= static_cast<int>((reinterpret_cast<uintptr_t>(base) + static_cast<uint32_t>(i * STEP) * static_cast<uint32_t>(ld)) & 3u) << (2 * i);
#pragma unroll
    for (int i = 0; i < (MN ? 8 : CHUNKS); ++i) sum[i] = 0;
  }
  __device__ __forceinline__ int valid(int i, int kb) const {
    const int row = row0 + i * STEP + (MN ? kb * KB : 0);
    const int at = chunk * 16 + (MN ? 0 : kb * KB);
    return row < row_limit ? max(0, min(16, inner_limit - at)) : 0;
  }
  __device__ __forceinline__ void load(int kb) {
    const uint8_t *p = base + static_cast<int64_t>(kb) * (MN ? KB * ld : KB);
#pragma unroll
    for (int i = 0; i < CHUNKS; ++i) {
      const uint8_t *q = p + static_cast<int64_t>(i * STEP) * ld;
      const int v = valid(i, kb);
      load_bytes(q, v, w[i]);
    }
  }
  __device__ __forceinline__ void store(uint8_t *tile, int kb, bool want_sum) {
#pragma unroll
    for (int i = 0; i < CHUNKS; ++i) {
      const int row = row0 + i * STEP;
      const int v = valid(i, kb);
      // (rows of the tile outside the matrix, and values along M / N outside it, meet only results
      // that are not stored: they may hold anything.  Depth beyond K must be zero.)
      if (!MN && row >= row_limit) continue;
      const uint4 x = place(w[i], (offs >> (2 * i)) & 3, v);
      *reinterpret_cast<uint4 *>(tile + row * 128 + ((chunk ^ (row & 7)) << 4)) = x;
      if (want_sum) count(x, i);
    }
  }
  __device__ __forceinline__ void count(const uint4 x, int i) {
    if (MN) {
      const uint32_t ww[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        sum[(MN ? j : 0)] += ww[j] & 0x00ff00ffu;
        sum[(MN ? 4 + j : 0)] += __byte_perm(ww[j], 0, 0x4341);
      }
    } else {
      sum[MN ? 0 : i] = sum16(x, sum[MN ? 0 : i]);
    }
  }
  // this thread's sums into the tile's sums in shared memory
  __device__ __forceinline__ void flush(uint32_t *sums, int lane) {
    if (MN) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t s[4] = {sum[MN ? j : 0] & 0xffffu, sum[MN ? 4 + j : 0] & 0xffffu, sum[MN ? j : 0] >> 16,
                               sum[MN ? 4 + j : 0] >> 16};
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          uint32_t t = s[b];
#pragma unroll
          for (int o = PER_ROW; o < 32; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
          if (lane < PER_ROW) atomicAdd(sums + chunk * 16 + j * 4 + b, t);
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < CHUNKS; ++i) {
        uint32_t t = sum[MN ? 0 : i];
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (chunk == 0) atomicAdd(sums + row0 + i * STEP, t);
      }
    }
  }
};

template <int BN, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(THREADS, 1) gemm_u8_gather_kernel(const __grid_constant__ Params p) {
  using C = Cfg<BN, B_MN>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t *smem = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bars = smem_base + C::RING;
  const uint32_t full_bar = bars, empty_bar = bars + 8 * STAGES, done_bar = bars + 16 * STAGES;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + C::RING + 16 * STAGES + 8);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  uint32_t *row_sums = reinterpret_cast<uint32_t *>(smem + C::RING + 256);  // [128]
  uint32_t *col_sums = row_sums + 128;                                      // [BN]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  mb_grid_dep_launch();

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar + 8 * s, GROUP_WARPS);
      mbar_init(empty_bar + 8 * s, 1);
    }
    mbar_init(done_bar, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == LOAD_WARPS) {
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

  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  mb_grid_dep_wait();

  if (warp == LOAD_WARPS) {
    // ---- MMA: one thread ----
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc(/*c s32*/ 2, /*a u8*/ 0, /*b u8*/ 0, A_MN, B_MN, 128, BN);
      // (operand layouts as in gemm_u8_tc.cu)
      const uint64_t a_base = A_MN ? make_smem_desc(0, 128 * KB, 1024, 2) : make_smem_desc(0, 16, 1024, 2);
      const uint64_t b_base = B_MN ? make_smem_desc(0, 128 * KB, 1024, 2) : make_smem_desc(0, 16, 1024, 2);
      constexpr uint32_t a_step = (A_MN ? 32 * 128 : 32) >> 4, b_step = (B_MN ? 32 * 128 : 32) >> 4;
      for (int i = 0; i < steps; ++i) {
        const int stage = i % STAGES;
        if (!mbar_wait(full_bar + 8 * stage, (i / STAGES) & 1, abort_flag, WAIT_BUDGET)) {
          *abort_flag = 1;
          atomicCAS(p.status, 0, MB_DEV_TIMEOUT_MMA);
          break;
        }
        tc_fence_after_sync();
        const uint32_t sa = smem_base + stage * C::STAGE_BYTES;
        const uint64_t a_desc = a_base | static_cast<uint64_t>((sa >> 4) & 0x3FFFu);
        const uint64_t b_desc = b_base | static_cast<uint64_t>(((sa + C::A_BYTES) >> 4) & 0x3FFFu);
#pragma unroll
        for (int j = 0; j < KB / 32; ++j)
          mma_i8_ss(tmem, a_desc + j * a_step, b_desc + j * b_step, idesc, (i > 0 || j > 0) ? 1u : 0u);
        mma_commit(empty_bar + 8 * stage);
      }
      mma_commit(done_bar);
    }
    __syncwarp();
  } else {
    // ---- loads ----
    Loader<A_MN, 128> la;
    Loader<B_MN, BN> lb;
    const int group = warp / GROUP_WARPS, gwarp = warp % GROUP_WARPS;
    const bool want_a = p.tail.zp_b != 0, want_b = p.tail.zp_a != 0;
    auto wait_free = [&](int i) {  // the stage of step i
      if (i < STAGES || mbar_wait_warp(empty_bar + 8 * (i % STAGES), ((i / STAGES) & 1) ^ 1, abort_flag, WAIT_BUDGET)) return true;
      *abort_flag = 1;
      atomicCAS(p.status, 0, MB_DEV_TIMEOUT_PRODUCER);
      return false;
    };
    la.init(p.A + b * p.a_bs, p.tail.M, p.K, p.lda, m0, gwarp, lane);
    lb.init(p.B + b * p.b_bs, p.tail.N, p.K, p.ldb, n0, gwarp, lane);
    auto load = [&](int i) {
      la.load(kb_begin + i);
      lb.load(kb_begin + i);
    };
    if (group < steps) load(group);
    for (int i = group; i < steps; i += GROUPS) {
      if (!wait_free(i)) break;
      uint8_t *ta = smem + (i % STAGES) * C::STAGE_BYTES;
      la.store(ta, kb_begin + i, want_a);
      lb.store(ta + C::A_BYTES, kb_begin + i, want_b);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(full_bar + 8 * (i % STAGES));
      if (i + GROUPS < steps) load(i + GROUPS);
    }
    __syncwarp();
    if (want_a) la.flush(row_sums, lane);
    if (want_b) lb.flush(col_sums, lane);
    if (!mbar_wait_warp(done_bar, 0, abort_flag, WAIT_BUDGET)) {
      *abort_flag = 1;
      atomicCAS(p.status, 0, MB_DEV_TIMEOUT_EPILOGUE);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (*abort_flag != 0) {
    // MMAs in flight must not outlive the tensor memory they write (bounded: about 2 ms)
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }

  finish_tile<BN, LOAD_WARPS>(p.tail, reinterpret_cast<int32_t *>(smem), tmem, row_sums, col_sums, m0, n0, b, rank, warp, lane);
  // no CTA of a cluster may leave while another still reads its tile
  if (p.tail.splits > 1) cluster_sync_all();
  else __syncthreads();
  if (warp == LOAD_WARPS) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, BN);
  }
}

template <int BN, bool A_MN, bool B_MN>
int launch_cfg(mb_context *ctx, Params &p, int64_t batch) {
  using C = Cfg<BN, B_MN>;
  constexpr uint64_t bit = (BN == 128 ? 4 : 0) + (A_MN ? 2 : 0) + (B_MN ? 1 : 0);
  auto kern = gemm_u8_gather_kernel<BN, A_MN, B_MN>;
  if (!(ctx->cut_attr_mask & (1ull << bit))) {
    MB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
    ctx->cut_attr_mask |= 1ull << bit;
  }
  const unsigned grid = static_cast<unsigned>(batch * p.tiles_m * p.tiles_n * p.tail.splits);
  MB_CUDA(ctx, mb_launch_clusters(ctx, kern, grid, THREADS, C::SMEM_BYTES, p.tail.splits, p));
  ctx->launches++;
  ctx->launches_tc++;
  return MB_SUCCESS;
}

}  // namespace

int mb_gemm_u8_gather_launch(mb_context *ctx, const mb_cut_gemm &g, int bn, int splits) {
  Params p = {};
  p.tail = make_tail(g, splits);
  p.A = g.A; p.B = g.B;
  p.K = static_cast<int>(g.K);
  p.lda = g.lda != 0 ? g.lda : g.a_mn ? g.M : g.K;
  p.ldb = g.ldb != 0 ? g.ldb : g.b_mn ? g.N : g.K;
  p.a_bs = g.a_batched ? (g.a_mn ? g.K : g.M) * p.lda : 0;
  p.b_bs = g.b_batched ? (g.b_mn ? g.K : g.N) * p.ldb : 0;
  p.tiles_m = static_cast<int>(ceil_div64(g.M, 128));
  p.tiles_n = static_cast<int>(ceil_div64(g.N, bn));
  p.k_blocks = static_cast<int>(ceil_div64(g.K, KB));
  p.status = ctx->dev_status;
  if (bn == 128) {
    if (g.a_mn) return g.b_mn ? launch_cfg<128, true, true>(ctx, p, g.batch) : launch_cfg<128, true, false>(ctx, p, g.batch);
    return g.b_mn ? launch_cfg<128, false, true>(ctx, p, g.batch) : launch_cfg<128, false, false>(ctx, p, g.batch);
  }
  if (g.a_mn) return g.b_mn ? launch_cfg<64, true, true>(ctx, p, g.batch) : launch_cfg<64, true, false>(ctx, p, g.batch);
  return g.b_mn ? launch_cfg<64, false, true>(ctx, p, g.batch) : launch_cfg<64, false, false>(ctx, p, g.batch);
}
