// clip_conv.h -- internal interface between the clip encoder (host/conv3d_encoder.cpp), the first layer's plan
// (conv_first.cu) and the depth-walking 3-D convolution (clip_conv.cu): 3x3x3, stride 1x2x2, pad 1, 32 or 64 input channels.
#pragma once
#include <stddef.h>

#include "aig_b200.h"

// Input: blocks [d][n][Hb][Wb][4][c] of 2x2 pixels, block ((y+1)>>1, (x+1)>>1), sub-position ((y+1)&1)*2 + ((x+1)&1), the
// sub-positions outside the image zero.
static inline int clip_block_extent(int v) { return (v + 1) / 2 + 1; }
static inline size_t clip_block_elems(int batch, int d, int h, int w, int c) {
  return (size_t)batch * d * clip_block_extent(h) * clip_block_extent(w) * 4 * c;
}
struct ClipConvGeom {
  int batch, D, H, W;  // input extents in pixels
  int C, K;            // input and output channels
  float slope;         // leaky ReLU behind the folded BatchNorm
  int out_blocks;      // 1: the output in such blocks too (the next layer's input); 0: [n][d][h][w][K]
};
struct ClipConv;
bool clip_conv_supported(const aig_ctx* ctx, const ClipConvGeom& g);
int clip_conv_create(aig_ctx* ctx, const ClipConvGeom& g, ClipConv** out);
void clip_conv_destroy(ClipConv* c);
int clip_conv_set_weights(ClipConv* c, const aig_half* w_kcx, const aig_half* bias, const float* gamma, const float* beta, const float* mean,
                          const float* var, float eps);
int clip_conv_forward(ClipConv* c, const aig_half* x, aig_half* y);

// The first layer of a clip (3-D plan) writes such blocks.  False: its kernels cannot.
bool conv0_plan_set_output_clip_blocks(aig_conv0_plan* plan);
