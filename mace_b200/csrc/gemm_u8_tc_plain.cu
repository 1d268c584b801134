// The instances of the tensor-core uint8 GEMM whose results do not go through TMA stores: int32 outputs, and uint8
// outputs whose rows are not 16-byte aligned.
#include "gemm_u8_tc.cuh"

int mb_tc_dispatch_plain(mb_context *ctx, const mb_tc::TcChoice &c, const CUtensorMap &ta, const CUtensorMap &tb,
                         const CUtensorMap &tc, mb_tc::TcParams &p) {
  return mb_tc::dispatch<true>(ctx, c, ta, tb, tc, p);
}

int mb_tc_dispatch_conv_plain(mb_context *ctx, int bn, int kb, const CUtensorMap &ta, const CUtensorMap &tb,
                              const CUtensorMap &tc, mb_tc::ConvTcParams &p) {
  return mb_tc::dispatch_conv<true>(ctx, bn, kb, ta, tb, tc, p);
}
