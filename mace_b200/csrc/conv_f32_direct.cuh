// fp32 convolutions as direct products on the tensor cores: stride 1 with SAME padding (conv_f32_direct.cu) ...
#pragma once

#include "common.cuh"

struct mb_f32_conv {
  const float *X = nullptr, *filter = nullptr, *bias = nullptr;  // NCHW, OIHW, null or one per output channel
  float *out = nullptr;
  int64_t N = 0, C = 0, H = 0, W = 0, O = 0;
  int KH = 3, KW = 3;  // (conv_f32_direct.cu: odd; the output is as large as the input)
  int act = 0;
  float max_limit = 0.f, coef = 0.f;
  int run = 1;         // filter rows of 32 channels, KH at most, that the tensor core adds up before the sum is carried on in fp32
};

// ... and few input channels with a stride of two columns (conv_f32_stem.cu); the geometry of g plus stride, padding and output.
bool mb_conv_f32_stem_supported(const mb_context *ctx, const mb_f32_conv &g, int sh, int sw, int pl, int64_t Ho, int64_t Wo);
int64_t mb_conv_f32_stem_cost(const mb_context *ctx, const mb_f32_conv &g, int sh, int64_t Ho, int64_t Wo);
int mb_conv_f32_stem_launch(mb_context *ctx, const mb_f32_conv &g, int sh, int pt, int pl, int64_t Ho, int64_t Wo);

bool mb_conv_f32_direct_supported(const mb_context *ctx, const mb_f32_conv &g);
// Estimated time in SM cycles.
int64_t mb_conv_f32_direct_cost(const mb_context *ctx, const mb_f32_conv &g);
// *done is false where nothing was launched, for want of room for the split filter (see mb_weight_scratch).
int mb_conv_f32_direct_launch(mb_context *ctx, const mb_f32_conv &g, bool *done);
