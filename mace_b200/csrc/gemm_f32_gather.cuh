// The fp32 tensor-core GEMM whose warps fetch the X operand themselves (gemm_f32_gather.cu): convolutions of any
// filter, stride and dilation without a column matrix, and matrix products of any layout and size.
#pragma once

#include "common.cuh"

// C[b][n][m] = act(bias[n] + sum_k X[b][k][m] * W[b][n][k] [+ R[b][n][m]])
struct mb_f32_gemm {
  const float *X = nullptr, *W = nullptr, *bias = nullptr, *residual = nullptr;
  float *C = nullptr;
  int64_t batch = 1, M = 0, N = 0, K = 0;
  // element strides: X(k, m) at k * x_ks + m * x_ms (one of them 1), W(n, k) at n * w_ns + k * w_ks (one of
  // them 1), C(n, m) at n * c_ns + m * c_ms
  int64_t x_ks = 0, x_ms = 1, x_bs = 0, w_ns = 0, w_ks = 1, w_bs = 0, c_ns = 0, c_ms = 1, c_bs = 0;
  int act = 0;
  float max_limit = 0.f, coef = 0.f;
  // conv: X is an NCHW tensor, M its output pixels over all images, k = (c * KH + kh) * KW + kw, and C an NCHW
  // tensor of N channels (x_*, c_* and the W strides unused)
  bool conv = false;
  // How many steps of 32 of the depth the tensor core adds up before the sum is carried on in fp32; 0: all of them, as
  // the TMA-fed kernel does.
  int run = 0;
  int C_in = 0, H = 0, Wd = 0, KH = 1, KW = 1, sh = 1, sw = 1, dh = 1, dw = 1, pad_t = 0, pad_l = 0, Ho = 0, Wo = 0;
};

// The run that keeps the error of a product of this depth below that of a chain of fp32 FMAs, 0 where none does (see
// "Accuracy" in gemm_f32_gather.cu).
static inline int mb_f32_gather_run(int64_t K) { return K < 48 || (K > 64 && K < 72) ? 0 : K < 384 ? 1 : 2; }

bool mb_gemm_f32_gather_supported(const mb_context *ctx, const mb_f32_gemm &g);
// Estimated time of the launch in SM cycles.
int64_t mb_gemm_f32_gather_cost(mb_context *ctx, const mb_f32_gemm &g);
int mb_gemm_f32_gather_launch(mb_context *ctx, const mb_f32_gemm &g);
// The same where both operands have their depth contiguous and lie as TMA wants them (gemm_f32_rows.cu).
bool mb_gemm_f32_rows_supported(const mb_context *ctx, const mb_f32_gemm &g);
int64_t mb_gemm_f32_rows_cost(const mb_context *ctx, const mb_f32_gemm &g);
int mb_gemm_f32_rows_launch(mb_context *ctx, const mb_f32_gemm &g);
