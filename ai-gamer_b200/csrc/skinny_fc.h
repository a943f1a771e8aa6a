// skinny_fc.h -- internal interface of the fully connected product for few rows (skinny_fc.cu), used by the FC plans
// (igemm_tcgen05.cu) and by the reference network's fused inference (host/layers/Layers.cpp).
#pragma once
#include <cuda_fp16.h>

#include "aig_b200.h"

// What may follow the product and the bias: per-output BatchNorm (read as the layer keeps it), ReLU, sigmoid on the
// first n_sigmoid outputs.  Each of them rounds to fp16, as the layers one after another do.
struct FcTail {
  const float *gamma = nullptr, *beta = nullptr, *mean = nullptr, *var = nullptr;
  float eps = 0.f;
  int relu = 0, n_sigmoid = 0;
};
struct SkinnyFc {
  int rows, in_c, out_c;
  const __half *w, *x;            // [out_c rounded up to 16][in_c], [rows][in_c]
  const float *scale, *shift;     // two_step: shift is the bias
  int two_step, act;
  float slope;
  __half* y;                      // [rows][out_c], or null
  float* y32;
  FcTail tail;
};
// Rows up to which an FC plan takes it: 6.2 us for 64 rows at K = 1024, N = 1024, 8.7 for 111 rows at K = 256, N = 768, where
// the tiled GEMM takes 7.3.
constexpr int kSkinnyRows = 64;
int skinny_fc_forward(aig_ctx* ctx, const SkinnyFc& p);

// igemm_tcgen05.cu:
// Whether an FC plan takes it, where the number of rows must not decide (the two products add in different orders).
void fc_plan_use_skinny(aig_conv_plan* plan, bool enable);
// An FC plan's product with a tail; the plan must be in two-step mode and have few enough rows.
int fc_plan_forward_tail(aig_conv_plan* plan, const aig_half* x, aig_half* y, const FcTail& tail);
// Its weights from [in_c][n] columns, as output columns first .. first + n - 1 of the plan (the affine is left alone).
int fc_plan_pack_columns(aig_conv_plan* plan, const aig_half* w_in_out, int n, int first);
// Its weights from [c * hw][out] rows in the order (channel, position), for inputs in the order (position, channel), and
// the bias.
int fc_plan_set_weights_nhwc(aig_conv_plan* plan, const aig_half* w_in_out, const aig_half* bias, int c, int hw);
