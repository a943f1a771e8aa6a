// seq_step.h -- internal interface between the sequence-head and agent runners (host/seq_head.cpp, host/agent.cpp) and
// the fused streaming step (csrc/seq_step.cu).
#pragma once
#include <stddef.h>

#include "aig_b200.h"
#include "aig_host.h"

struct SeqStepFused;

struct SeqStepConfig {
  int batch, in_c, hidden, layers, heads, window, n_out, n_sigmoid;
  float rope_base, clip;
  int double_bias;
  int features;  // input width of the FC in front of the head (the agent's bridge); 0: the head's own input only
};

// True when the fused step covers this configuration (up to 128 sequences, head size 64, bounded window).
bool seq_step_fused_supported(const SeqStepConfig& c);
int seq_step_fused_create(aig_ctx* ctx, const SeqStepConfig& c, SeqStepFused** out);
void seq_step_fused_destroy(SeqStepFused* s);
// Device pointers to the parameters as loaded (reference layouts): LSTM blob, MHA matrices [in][out],
// LayerNorm gamma/beta, FC W [in][out] and bias.  Makes the transposed copies the kernel reads.
int seq_step_fused_set_weights(SeqStepFused* s, const aig_half* lstm_blob, const aig_half* wq, const aig_half* wk,
                               const aig_half* wv, const aig_half* wo, const float* ln_g, const float* ln_b,
                               const aig_half* fcw, const aig_half* fcb);
// The bridge FC W [features][in_c] and its bias (device memory).
int seq_step_fused_set_bridge(SeqStepFused* s, const aig_half* w_in_out, const aig_half* bias);
// One streaming step from emb [B][in_c] or, with emb null, from features [B][features] through the bridge;
// h_state/c_state [layers][B][hidden] are read and updated; y [B][hidden] = top LSTM output; logits [B][n_out] fp16 and
// out_f32 [B][n_out] = the head outputs.  The step's number is kept on the device: 0 after create and reset.
// after_encoder: the launch follows the frame encoder's on the stream, whose first kernel waited for everything before
// it, so this kernel may start (and read the carried state) under the encoder's tail.
int seq_step_fused_run(SeqStepFused* s, const aig_half* emb, const aig_half* features, aig_half* h_state, aig_half* c_state, aig_half* y,
                       aig_half* logits, float* out_f32, bool after_encoder);
int seq_step_fused_reset(SeqStepFused* s);

// The end of the full-sequence forward in one launch (elementwise.cu): row LayerNorm, FC (weights [n_out][c], two-step
// rounding), sigmoid on the first n_sigmoid outputs and tanh on the rest, as fp16 and fp32.
bool seq_tail_supported(int c, int n_out);
int seq_tail_forward(aig_ctx* ctx, const aig_half* x, const float* gamma, const float* beta, const aig_half* fc_w, const aig_half* fc_b, aig_half* out_half,
                     float* out_f32, int rows, int c, int n_out, int n_sigmoid, float eps);

// Internal entry points of the sequence-head runner for the agent: a head whose fused step starts at the frame
// encoder's features.
int seq_create_with_bridge(aig_ctx* ctx, const aig_seq_config* cfg, int features, aig_seq** out);
bool seq_has_fused_step(const aig_seq* m);
int seq_set_bridge(aig_seq* m, const aig_half* w_in_out, const aig_half* bias);
int seq_step_from_features(aig_seq* m, const aig_half* features);
