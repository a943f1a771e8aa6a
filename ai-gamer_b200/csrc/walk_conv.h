// walk_conv.h -- internal interface between the model runners (host/conv3d_encoder.cpp, host/cnn_encoder.cpp), the first
// layers' plan (conv_first.cu) and the convolutions that walk along one axis (walk_conv.cu).
#pragma once
#include <stddef.h>

#include "aig_b200.h"

struct WalkConv;
void walk_conv_destroy(WalkConv* c);

// ---- 3-D, 3x3x3, stride 1x2x2, pad 1, 32 or 64 input channels: along the depth
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
bool clip_conv_supported(const aig_ctx* ctx, const ClipConvGeom& g);
int clip_conv_create(aig_ctx* ctx, const ClipConvGeom& g, WalkConv** out);
int clip_conv_set_weights(WalkConv* c, const aig_half* w_kcx, const aig_half* bias, const float* gamma, const float* beta, const float* mean,
                          const float* var, float eps);
int clip_conv_forward(WalkConv* c, const aig_half* x, aig_half* y);
int clip_blocks_to_ndhwc(aig_ctx* ctx, const aig_half* blocks, aig_half* y, int batch, int d, int h, int w, int c);

// ---- a residual block of the frame encoder (main k4 s2 p1, then k3 s1 p1; shortcut k2 s2 p0): along the rows
// Input: blocks [yb][n][xb][4][c] (extents as of aig_nhwc_to_s2d, rows outermost).  Between the two launches: [y][n][x][K]
// with one column behind every image row that stays zero (res_walk_rows rows of K channels).
enum ResWalkOut { RES_OUT_NHWC, RES_OUT_BLOCKS, RES_OUT_ROW_BLOCKS };  // channels-last; blocks [n][yb][xb][4][K]; blocks [yb][n][xb][4][K]
struct ResWalkGeom {
  int batch, H, W;     // input extents in pixels
  int C, K;            // 32 -> 64, 64 -> 128 channels
  int act;
  float slope;
  ResWalkOut out;
};
bool res_walk_supported(const aig_ctx* ctx, const ResWalkGeom& g);
size_t res_walk_rows(const ResWalkGeom& g);
int res_walk_create(aig_ctx* ctx, const ResWalkGeom& g, WalkConv** down, WalkConv** conv1);
int res_walk_set_down(WalkConv* down, const aig_half* w_main, const aig_half* b_main, const float* gamma, const float* beta, const float* mean,
                      const float* var, float eps, const aig_half* w_short, const aig_half* b_short);
int res_walk_set_conv1(WalkConv* conv1, const aig_half* w, const aig_half* bias, const float* gamma, const float* beta, const float* mean, const float* var,
                       float eps);
int res_walk_down(WalkConv* down, const aig_half* x, aig_half* t, aig_half* r);
int res_walk_conv1(WalkConv* conv1, const aig_half* t, const aig_half* r, aig_half* y);

// ---- its 3x3 convolution alone, 256 channels, on the padded position layout [n][h+1][w+1][256]; weights and forward as of conv1
struct ConvWalkGeom {
  int batch, h, w, C;
  int act;
  float slope;
  ResWalkOut out;      // channels-last or blocks [n][yb][xb]
};
bool conv_walk_supported(const aig_ctx* ctx, const ConvWalkGeom& g);
int conv_walk_create(aig_ctx* ctx, const ConvWalkGeom& g, WalkConv** out);
int row_blocks_to_nhwc(aig_ctx* ctx, const aig_half* blocks, aig_half* y, int batch, int h, int w, int c);

// ---- the first layer's output in the layouts above; false: its kernels cannot
bool conv0_plan_set_output_clip_blocks(aig_conv0_plan* plan);
bool conv0_plan_set_output_row_blocks(aig_conv0_plan* plan);
