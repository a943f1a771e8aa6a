// res_chain.h -- internal interface between the frame encoder (host/cnn_encoder.cpp), the convolution plans
// (igemm_tcgen05.cu) and the one-kernel chain of residual blocks for small batches (res_chain.cu).
#pragma once
#include <cuda_fp16.h>

#include <vector>

#include "aig_b200.h"

// What the chain reads of a patch-resident plan with a flat input: geometry of the flattened position space, the packed
// weights [rows][k] and the folded affine (both stay where the plan keeps them).
struct ConvPlanView {
  bool is_down;
  int batch, in_c, out_c, Ho, Wo;
  int P, RP, pad, kw, kh, taps, cblocks, sub_cblocks;
  int act;
  float slope;
  int s2d, Hb, Wb;
  const __half* w;
  int w_rows, w_k;
  const float *scale, *shift;
};
// False unless the plan is patch-resident with a flat input (and, for a down-sampling pair, padded outputs).
bool conv_plan_view(const aig_conv_plan* plan, ConvPlanView* out);

struct ResChainBlock {
  aig_conv_plan *down, *conv1;
  aig_half *in, *t, *r, *y;  // block input (space-to-depth), the pair's outputs (padded layout), block output
};
struct ResChainHead {        // as aig_cnn_head_forward; hw = 0: no head
  const aig_half *mask_w, *fc_w, *fc_b;
  float mask_b;
  aig_half *feat, *out_half;
  float* out_f32;
  int hw, c, n_out, n_sigmoid;
};
struct ResChain;
// *out stays null (and the call succeeds) where the per-layer launches are the better or the only choice.
// hw, c_last, n_out: positions and channels of the last block's output, outputs of the head (0: none).
int res_chain_create(aig_ctx* ctx, const std::vector<ResChainBlock>& blocks, int hw, int c_last, int n_out, ResChain** out);
void res_chain_destroy(ResChain* c);
int res_chain_forward(ResChain* c, const ResChainHead& head);
