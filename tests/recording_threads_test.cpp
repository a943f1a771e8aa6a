// recording_threads_test.cpp -- offline inference over a recording on a host that refuses threads or memory.  Built by
// test_recording_cpu.py together with recording.cpp, without the CUDA runtime: the encoder below keeps its frames in host
// memory and its "outputs" are sums over a frame's bytes, pthread_create starts as many threads as it is told to, and
// operator new fails when it is told to.
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <unistd.h>

#include <atomic>
#include <new>
#include <string>
#include <vector>

#include "cnn_stream.h"

// ---------------------------------------------------------------- what the host gives
static std::atomic<int> g_threads_left{1000}, g_news_left{-1};
extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg) {
  using Fn = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  static const Fn real = reinterpret_cast<Fn>(dlsym(RTLD_NEXT, "pthread_create"));
  return g_threads_left.fetch_sub(1) > 0 ? real(t, a, f, arg) : EAGAIN;
}
void* operator new(size_t n) {
  if (g_news_left.load() >= 0 && g_news_left.fetch_sub(1) == 0) throw std::bad_alloc();
  if (void* p = malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }

// ---------------------------------------------------------------- the encoder's side of cnn_stream.h
struct aig_cnn {
  aig_cnn_config cfg{};
  std::vector<unsigned char> slot[2], ring;
  std::vector<float> out[2];
  CnnStaging st;
};
extern "C" {
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
const char* aig_cnn_last_error(aig_cnn*) { return "encoder"; }
int aig_cnn_wait(aig_cnn*, int) { return AIG_OK; }
}
const aig_cnn_config& cnn_config(const aig_cnn* m) { return m->cfg; }
int cnn_staging(aig_cnn* m, size_t piece_bytes, int slots, CnnStaging** out) {
  m->ring.resize(piece_bytes * slots);
  m->st.ring = m->ring.data();
  m->st.piece_bytes = piece_bytes;
  m->st.slots = slots;
  for (int s = 0; s < 2; ++s) m->st.out[s] = m->out[s].data();
  *out = &m->st;
  return AIG_OK;
}
int cnn_stream_begin(aig_cnn*, int) { return AIG_OK; }
int cnn_stream_copy(aig_cnn* m, int slot, size_t offset, const void* host, size_t bytes, cudaEvent_t) {
  memcpy(m->slot[slot].data() + offset, host, bytes);
  return AIG_OK;
}
static float frame_sum(const unsigned char* f, size_t n, int o) {
  unsigned s = 0;
  for (size_t i = 0; i < n; ++i) s = s * 31u + f[i] + (unsigned)o;
  return (float)(s & 0xFFFFF);
}
int cnn_stream_submit(aig_cnn* m, int slot, float* out, bool) {
  const size_t n = (size_t)3 * m->cfg.height * m->cfg.width;
  for (int b = 0; b < m->cfg.batch; ++b)
    for (int o = 0; o < m->cfg.n_out; ++o) out[b * m->cfg.n_out + o] = frame_sum(m->slot[slot].data() + b * n, n, o);
  return AIG_OK;
}
int cnn_stream_drain(aig_cnn*) { return AIG_OK; }

// ---------------------------------------------------------------- the cases
int main(int argc, char** argv) {
  if (argc != 2) return 2;
  const int W = 100, H = 60, batch = 64, n_out = 3, count = 64 * 3 + 5;   // 58 and 6 frames a batch in pieces
  const size_t fb = (size_t)3 * W * H;
  std::vector<unsigned char> frames(fb * count);
  for (size_t i = 0; i < frames.size(); ++i) frames[i] = (unsigned char)((i * 2654435761u) >> 13);
  FILE* f = fopen(argv[1], "wb");
  const int wh[2] = {W, H};
  fwrite(wh, 4, 2, f);
  for (int i = 0; i < count; ++i) {
    fwrite("\0\0\0\0\0\0\0\0\0", 1, 10, f);
    fwrite(frames.data() + i * fb, 1, fb, f);
  }
  fclose(f);
  std::vector<float> want((size_t)count * n_out), got(want.size());
  for (int i = 0; i < count; ++i)
    for (int o = 0; o < n_out; ++o) want[(size_t)i * n_out + o] = frame_sum(frames.data() + i * fb, fb, o);

  aig_cnn m;
  m.cfg.batch = batch; m.cfg.width = W; m.cfg.height = H; m.cfg.n_out = n_out;
  for (int s = 0; s < 2; ++s) {
    m.slot[s].resize(fb * batch);
    m.out[s].resize((size_t)batch * n_out);
  }
  aig_recording* r = nullptr;
  if (aig_recording_open(argv[1], &r) != AIG_OK) return 3;
  int failed = 0;
  auto run = [&] {
    std::fill(got.begin(), got.end(), -1.0f);
    return aig_cnn_infer_recording(&m, r, 0, count, batch, n_out, got.data());
  };
  // fewer threads than wanted, down to none: the calling thread reads what nobody else does
  for (int threads : {1000, 0, 1, 2, 3, 0, 1000}) {
    g_threads_left = threads;
    const int rc = run();
    if (rc != AIG_OK || got != want) failed += printf("FAILED: %d threads: status %d, outputs %s\n", threads, rc, got == want ? "right" : "wrong") > 0;
  }
  // memory refused at each allocation of a call in turn: an error, and the next call is right again
  g_threads_left = 1000;
  int refused = 0;
  for (int k = 0; k < 64; ++k) {
    g_news_left = k;
    const int rc = run();
    const bool hit = g_news_left.load() < 0;
    g_news_left = -1;
    if (!hit) break;
    ++refused;
    if (rc == AIG_OK && got != want) failed += printf("FAILED: allocation %d refused: wrong outputs\n", k) > 0;
    if (run() != AIG_OK || got != want) failed += printf("FAILED: call after allocation %d was refused\n", k) > 0;
  }
  if (refused == 0 || refused == 64) failed += printf("FAILED: %d allocations met\n", refused) > 0;
  // a file that has become shorter: an error from every number of threads
  if (truncate(argv[1], (off_t)(8 + (fb + 10) * 100)) != 0) return 4;
  for (int threads : {1000, 1, 0}) {
    g_threads_left = threads;
    const int rc = run();
    if (rc != AIG_ERR_IO) failed += printf("FAILED: short file, %d threads: status %d\n", threads, rc) > 0;
  }
  aig_recording_close(r);
  if (failed == 0) printf("all as expected\n");
  return failed ? 1 : 0;
}
