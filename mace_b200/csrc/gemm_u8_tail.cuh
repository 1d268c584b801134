// The end that the cluster-cut uint8 GEMM kernels share: accumulator -> exact int32 partial tile in
// shared memory -> the runs of a cluster added up, bias, requantization, store.
#pragma once

#include "gemm_u8_cut.cuh"
#include "sm100_ptx.cuh"

namespace {

struct TailParams {
  const int32_t *bias;
  void *C;
  int M, N, splits;
  int32_t zp_a, zp_b, kzz;
  int bias_per_row, out_is_int32, words_ok;  // words_ok: rows of the uint8 output start word-aligned
  mb_requant_params rq;
  int rq_variant;  // mb_requant_variant(), or 8 for the Gemv delegators' float rule
  float mult_f, zp_f;
};

inline TailParams make_tail(const mb_cut_gemm &g, int splits) {
  TailParams t = {};
  t.bias = g.bias; t.C = g.C;
  t.M = static_cast<int>(g.M); t.N = static_cast<int>(g.N);
  t.splits = splits;
  t.zp_a = g.zp_a; t.zp_b = g.zp_b;
  t.kzz = static_cast<int32_t>(static_cast<uint32_t>(g.K) * static_cast<uint32_t>(g.zp_a) * static_cast<uint32_t>(g.zp_b));
  t.bias_per_row = g.bias_per_row; t.out_is_int32 = g.out_is_int32;
  t.words_ok = ((static_cast<uintptr_t>(g.N) | reinterpret_cast<uintptr_t>(g.C)) & 3u) == 0;
  t.rq = g.rq; t.rq_variant = g.rq_variant; t.mult_f = g.mult_f; t.zp_f = g.zp_f;
  return t;
}

// int32 tile: rows 16-byte aligned, lane-per-row 16-byte accesses without bank conflicts
template <int BN>
constexpr int TAIL_PITCH = BN + 4;

__device__ __forceinline__ int4 ld_cluster_v4(uint32_t addr) {
  int4 v;
  asm volatile("ld.shared::cluster.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}

// Called by every thread of the CTA after the accumulator is complete; the first WARPS warps (a multiple of
// four) do the work.  `tile` holds 128 x TAIL_PITCH<BN> values.  After it the caller must keep the shared
// memory alive until the whole cluster is through (cluster_sync_all).
template <int BN, int WARPS>
__device__ __forceinline__ void finish_tile(const TailParams &p, int32_t *tile, uint32_t tmem, const uint32_t *row_sums,
                                            const uint32_t *col_sums, int m0, int n0, int b, int rank, int warp,
                                            int lane) {
  using namespace sm100;
  // ---- this CTA's exact int32 partial result, zero-point terms of its run of the depth included
  // (they are linear in the depth), into shared memory ----
  const int rows = min(128, p.M - m0);
  if (warp < WARPS) {
    const int quarter = warp & 3, slice = warp >> 2;
    constexpr int COLS = BN / (WARPS / 4);  // columns per warp
    const int row = quarter * 32 + lane;
    const int32_t row_term = -p.zp_b * static_cast<int32_t>(row_sums[row]);
    if (quarter * 32 < rows) {
      constexpr int CHUNKS = COLS / 16;
      uint32_t rr[CHUNKS][16];
#pragma unroll
      for (int h = 0; h < CHUNKS; ++h)
        tmem_ld_32x32b_x16(tmem + (static_cast<uint32_t>(quarter * 32) << 16) + slice * COLS + h * 16, rr[h]);
#pragma unroll
      for (int h = 0; h < CHUNKS; ++h) {
        uint32_t (&r)[16] = rr[h];
        tmem_ld_wait_x16(r);
        const int c0 = slice * COLS + h * 16;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 cs = *reinterpret_cast<const uint4 *>(col_sums + c0 + 4 * j);
          *reinterpret_cast<int4 *>(tile + row * TAIL_PITCH<BN> + c0 + 4 * j) =
              make_int4(static_cast<int32_t>(r[4 * j + 0]) + row_term - p.zp_a * static_cast<int32_t>(cs.x),
                        static_cast<int32_t>(r[4 * j + 1]) + row_term - p.zp_a * static_cast<int32_t>(cs.y),
                        static_cast<int32_t>(r[4 * j + 2]) + row_term - p.zp_a * static_cast<int32_t>(cs.z),
                        static_cast<int32_t>(r[4 * j + 3]) + row_term - p.zp_a * static_cast<int32_t>(cs.w));
        }
      }
    }
  }
  tc_fence_before_sync();
  if (p.splits > 1) cluster_sync_all();
  else __syncthreads();

  // ---- four columns per thread, row after row: add the runs, bias, requantize, store ----
  if (warp < WARPS) {
    constexpr int LANES = BN / 4, ROWS = 32 / LANES;  // lanes per row, rows per warp and pass
    const int n = n0 + (lane % LANES) * 4;
    const int left = p.N - n;
    if (left > 0) {
      const int row0 = (warp * p.splits + rank) * ROWS + lane / LANES, stride = WARPS * p.splits * ROWS;
      int32_t add[4] = {p.kzz, p.kzz, p.kzz, p.kzz};
      if (p.bias != nullptr && !p.bias_per_row) {
#pragma unroll
        for (int j = 0; j < 4; ++j) add[j] += j < left ? mb_load(p.bias + n + j) : 0;
      }
      const int32_t *mine = tile + (lane % LANES) * 4;
      uint32_t peer[7];
#pragma unroll
      for (int s = 1; s < 8; ++s) {
        int r = rank + s;
        if (r >= p.splits) r -= p.splits;
        peer[s - 1] = s < p.splits ? mapa_shared(smem_u32(mine), static_cast<uint32_t>(r)) : 0u;
      }
#pragma unroll 4
      for (int row = row0; row < rows; row += stride) {
        const int4 x = *reinterpret_cast<const int4 *>(mine + row * TAIL_PITCH<BN>);
        int32_t v[4] = {x.x + add[0], x.y + add[1], x.z + add[2], x.w + add[3]};
#pragma unroll
        for (int s = 1; s < 8; ++s) {
          if (s < p.splits) {
            const int4 y = ld_cluster_v4(peer[s - 1] + row * (TAIL_PITCH<BN> * 4));
            v[0] += y.x; v[1] += y.y; v[2] += y.z; v[3] += y.w;
          }
        }
        const int m = m0 + row;
        if (p.bias_per_row && p.bias != nullptr) {
          const int32_t rb = mb_load(p.bias + m);
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] += rb;
        }
        const int64_t at = (static_cast<int64_t>(b) * p.M + m) * p.N + n;
        if (p.out_is_int32) {
          int32_t *out = static_cast<int32_t *>(p.C) + at;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (j < left) out[j] = v[j];
          continue;
        }
        uint32_t word;
        if (p.rq_variant == 4) {
          word = mb_requant_pack4<false>(v[0], v[1], v[2], v[3], p.rq);
        } else if (p.rq_variant == 5) {
          word = mb_requant_pack4<true>(v[0], v[1], v[2], v[3], p.rq);
        } else if (p.rq_variant == 8) {
          uint32_t u[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            u[j] = mb_saturate_round_u8(__fadd_rn(__fmul_rn(static_cast<float>(v[j]), p.mult_f), p.zp_f));
          word = u[0] | (u[1] << 8) | (u[2] << 16) | (u[3] << 24);
        } else {
          word = mb_requant_fast(v[0], p.rq) | (mb_requant_fast(v[1], p.rq) << 8) |
                 (mb_requant_fast(v[2], p.rq) << 16) | (mb_requant_fast(v[3], p.rq) << 24);
        }
        uint8_t *out = static_cast<uint8_t *>(p.C) + at;
        if (p.words_ok) {
          *reinterpret_cast<uint32_t *>(out) = word;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (j < left) out[j] = static_cast<uint8_t>(word >> (8 * j));
        }
      }
    }
  }
}

}  // namespace
