// cnn_stream.h -- internal interface between the frame encoder (cnn_encoder.cpp) and the offline inference over
// recordings (recording.cpp): the pipelined host step of aig_cnn_submit_host in its parts, so that a batch can arrive
// in several pieces while it is still being read, and the pinned staging memory those pieces pass through.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include "aig_host.h"

// Pinned ring of `slots` pieces of `piece_bytes` each, one event per piece (recorded after its copy), and output
// buffers of [batch][n_out] floats for the two frame slots.  Belongs to the encoder and goes with it.
struct CnnStaging {
  unsigned char* ring = nullptr;
  size_t piece_bytes = 0;
  int slots = 0;
  cudaEvent_t copied[16] = {};
  float* out[2] = {nullptr, nullptr};
};
// At least `slots` (2 to 16) pieces of at least `piece_bytes`: allocated on first use, again when a call needs more.
int cnn_staging(aig_cnn* m, size_t piece_bytes, int slots, CnnStaging** out);

const aig_cnn_config& cnn_config(const aig_cnn* m);
int cnn_stream_begin(aig_cnn* m, int slot);  // the copy stream waits until the slot's frames have been consumed
int cnn_stream_copy(aig_cnn* m, int slot, size_t offset, const void* host, size_t bytes, cudaEvent_t copied);  // copied may be null
int cnn_stream_submit(aig_cnn* m, int slot, float* out_host, bool planar);  // forward once the copies have landed, outputs to the host
int cnn_stream_drain(aig_cnn* m);            // nothing of the encoder's is in flight afterwards
