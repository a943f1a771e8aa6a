// recording.cpp -- reader for the recording files the reference's input recorder writes, and batched offline
// inference over them.
//
// File layout (little endian, no padding; input_recorder.cpp:24-27 writes the header, :122-133 every record):
//   int32 width, int32 height
//   per frame:  uint16 keyStates, int32 mouseDeltaX, int32 mouseDeltaY        (10 bytes)
//               uint8 planar RGB frame: plane R, plane G, plane B, width*height bytes each
// Records are indexed the way ReadStateData does (main.cpp:41-92): only whole records count, a partial one at
// the end of the file is ignored.  Targets follow Train.cpp:70-76: button j = bit j of keyStates (14 buttons),
// axes = mouse deltas / 256.
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
#include <unistd.h>

#include <algorithm>
#include <condition_variable>
#include <exception>
#include <mutex>
#include <string>
#include <system_error>
#include <thread>
#include <vector>

#include "aig_b200.h"
#include "aig_host.h"
#include "cnn_stream.h"

struct aig_recording {
  FILE* f = nullptr;
  int width = 0, height = 0;
  long long n_records = 0;
  size_t frame_bytes = 0, stride = 0;
  std::string err;
};

namespace {
constexpr long long kHeaderBytes = 8, kRecordHeader = 10;
constexpr size_t kPieceBytes = 1 << 20, kRingBytes = 16 << 20;
std::string g_open_error;
int rfail(aig_recording* r, int code, const std::string& msg) {
  r->err = msg;
  return code;
}

// The threads that read pieces, and what they share with the one that issues the copies.  Whichever way a scope that
// holds them is left, none of them runs on.
struct Readers {
  std::mutex mu;
  std::condition_variable cv;
  long long next = 0, issued = 0;   // next piece to read; pieces whose copy has been issued
  bool stop = false;
  std::vector<std::thread> threads;

  void finish() {
    {
      std::lock_guard<std::mutex> lk(mu);
      stop = true;
    }
    cv.notify_all();
    for (std::thread& t : threads) t.join();
    threads.clear();
  }
  ~Readers() { finish(); }
};
}  // namespace

extern "C" {

const char* aig_recording_last_error(aig_recording* r) { return r ? r->err.c_str() : g_open_error.c_str(); }

int aig_recording_open(const char* path, aig_recording** out) {
  if (!path || !out) return AIG_ERR_INVALID;
  *out = nullptr;
  FILE* f = fopen(path, "rb");
  if (!f) {
    g_open_error = std::string("cannot open ") + path;
    return AIG_ERR_IO;
  }
  int32_t wh[2] = {0, 0};
  if (fread(wh, 4, 2, f) != 2 || wh[0] <= 0 || wh[1] <= 0 || (long long)wh[0] * wh[1] > (1ll << 28)) {
    fclose(f);
    g_open_error = std::string("no valid width/height header in ") + path;
    return AIG_ERR_IO;
  }
  aig_recording* r = new aig_recording();
  r->f = f;
  r->width = wh[0];
  r->height = wh[1];
  r->frame_bytes = (size_t)3 * wh[0] * wh[1];
  r->stride = (size_t)kRecordHeader + r->frame_bytes;
  fseeko(f, 0, SEEK_END);
  const long long size = (long long)ftello(f);
  r->n_records = (size - kHeaderBytes) / (long long)r->stride;  // whole records only
  *out = r;
  return AIG_OK;
}

int aig_recording_close(aig_recording* r) {
  if (!r) return AIG_OK;
  if (r->f) fclose(r->f);
  delete r;
  return AIG_OK;
}

int aig_recording_info(const aig_recording* r, int* width, int* height, long long* n_records) {
  if (!r) return AIG_ERR_INVALID;
  if (width) *width = r->width;
  if (height) *height = r->height;
  if (n_records) *n_records = r->n_records;
  return AIG_OK;
}

// `count` consecutive records from `first`: frames [count][3][height][width] as stored, key_states [count],
// mouse_dxdy [count][2]; any of the three may be null
int aig_recording_read(aig_recording* r, long long first, int count, uint8_t* frames, uint16_t* key_states, int32_t* mouse_dxdy) {
  if (!r || count < 0) return AIG_ERR_INVALID;
  if (first < 0 || first + count > r->n_records) return rfail(r, AIG_ERR_INVALID, "record range outside the file");
  for (int i = 0; i < count; ++i) {
    if (fseeko(r->f, (off_t)(kHeaderBytes + (first + i) * (long long)r->stride), SEEK_SET) != 0) return rfail(r, AIG_ERR_IO, "seek failed");
    unsigned char hdr[kRecordHeader];
    if (fread(hdr, 1, kRecordHeader, r->f) != (size_t)kRecordHeader) return rfail(r, AIG_ERR_IO, "short read of a record header");
    if (key_states) memcpy(&key_states[i], hdr, 2);
    if (mouse_dxdy) {
      memcpy(&mouse_dxdy[2 * i], hdr + 2, 4);
      memcpy(&mouse_dxdy[2 * i + 1], hdr + 6, 4);
    }
    if (frames && fread(frames + (size_t)i * r->frame_bytes, 1, r->frame_bytes, r->f) != r->frame_bytes)
      return rfail(r, AIG_ERR_IO, "short read of a frame");
  }
  return AIG_OK;
}

// Train.cpp:70-76: targets [count][16]
int aig_recording_targets(const uint16_t* key_states, const int32_t* mouse_dxdy, int count, float* targets) {
  if (!key_states || !mouse_dxdy || !targets || count < 0) return AIG_ERR_INVALID;
  for (int i = 0; i < count; ++i) {
    for (int j = 0; j < 14; ++j) targets[i * 16 + j] = (float)((key_states[i] >> j) & 1);
    targets[i * 16 + 14] = (float)mouse_dxdy[2 * i] / 256.0f;
    targets[i * 16 + 15] = (float)mouse_dxdy[2 * i + 1] / 256.0f;
  }
  return AIG_OK;
}

}  // extern "C"

// Offline inference over records [first, first + count): batches of the encoder's batch size as planar RGB (the bytes
// of the file, untouched), two batches in flight; in the last one the frames past `count` are whatever the slot held,
// their outputs are dropped.  out_host [count][n_out] fp32 (host memory).  n_out is the encoder's.
//
// Bound by the host: the forward of 256 frames takes 0.53 ms and their PCIe copy 0.55 ms, one thread reads them from
// the page cache in about 4 ms, and allocating and freeing pinned memory for two batches took longer than all of it.
// So the file is read by several threads, in pieces of about 1 MB that go to the GPU as they come (the first batch
// starts after one piece's read, not one batch's), through a pinned ring that the encoder keeps.  600 frames of
// 256x144 in batches of 256: 42 ms before, 3.3 after; an encoder's first call, which allocates the ring and captures the
// two slots' graphs, takes 22 to 25.
static int infer_recording(aig_cnn* m, aig_recording* r, long long first, long long count, int batch, int n_out, float* out_host) {
  // pieces: whole frames, none of them across two batches
  const int per_piece = (int)std::min<size_t>(std::max<size_t>(1, kPieceBytes / r->frame_bytes), (size_t)batch);
  const int per_batch = (batch + per_piece - 1) / per_piece;
  const long long n_batches = (count + batch - 1) / batch;
  const int last_n = (int)(count - (n_batches - 1) * batch);
  const long long n_pieces = (n_batches - 1) * per_batch + (last_n + per_piece - 1) / per_piece;
  const size_t piece_bytes = (size_t)per_piece * r->frame_bytes;
  const int slots = (int)std::min<size_t>(16, std::max<size_t>(4, kRingBytes / piece_bytes));
  CnnStaging* st = nullptr;
  int rc = cnn_staging(m, piece_bytes, slots, &st);
  if (rc != AIG_OK) return rfail(r, rc, aig_cnn_last_error(m));
  int device = 0;
  cudaGetDevice(&device);

  // piece i goes through ring slot i % slots: read once the copy of piece i - slots has left it, copied in order
  std::vector<char> ready(n_pieces, 0);
  const int fd = fileno(r->f);
  auto piece_frames = [&](long long i, long long* lo) {
    const long long b = i / per_batch, k = i % per_batch;
    *lo = b * batch + k * per_piece;
    const long long end = std::min(std::min(*lo + per_piece, (b + 1) * batch), count);
    return (int)(end - *lo);
  };
  auto read_piece = [&](long long i) {  // (the copy of piece i - slots has been issued)
    bool ok = i < slots || cudaEventSynchronize(st->copied[i % slots]) == cudaSuccess;
    long long lo;
    const int n = piece_frames(i, &lo);
    uint8_t* dst = st->ring + (size_t)(i % slots) * st->piece_bytes;
    for (int k = 0; k < n && ok; ++k) {
      const off_t at = (off_t)(kHeaderBytes + (first + lo + k) * (long long)r->stride + kRecordHeader);
      size_t got = 0;
      while (got < r->frame_bytes) {
        const ssize_t x = pread(fd, dst + (size_t)k * r->frame_bytes + got, r->frame_bytes - got, at + (off_t)got);
        if (x <= 0) break;
        got += (size_t)x;
      }
      ok = got == r->frame_bytes;
    }
    return ok;
  };
  Readers rd;  // (declared after all that its threads use)
  auto reader = [&]() {
    cudaSetDevice(device);
    for (;;) {
      long long i;
      {
        std::unique_lock<std::mutex> lk(rd.mu);
        if (rd.stop || rd.next == n_pieces) return;
        i = rd.next++;
        rd.cv.wait(lk, [&] { return rd.stop || rd.issued > i - slots; });
        if (rd.stop) return;
      }
      const bool ok = read_piece(i);
      std::lock_guard<std::mutex> lk(rd.mu);
      ready[i] = ok ? 1 : 2;
      rd.cv.notify_all();
    }
  };
  // A core copies about 6 GB/s out of the page cache and PCIe takes 52: eight readers about keep up with it.  Where the host
  // gives fewer threads, those read; where it gives none, this one does.
  const long long n_readers = std::min<long long>(n_pieces, std::min(8u, std::max(1u, std::thread::hardware_concurrency())));
  rd.threads.reserve((size_t)n_readers);
  try {
    for (long long i = 0; i < n_readers; ++i) rd.threads.emplace_back(reader);
  } catch (const std::system_error&) {
  }

  auto collect = [&](long long b) {
    const int s = (int)(b & 1);
    const int w = aig_cnn_wait(m, s);
    if (w != AIG_OK) return w;
    const long long lo = b * batch, n = std::min<long long>(batch, count - lo);
    memcpy(out_host + (size_t)lo * n_out, st->out[s], (size_t)n * n_out * sizeof(float));
    return (int)AIG_OK;
  };
  bool io_ok = true;
  for (long long i = 0; i < n_pieces && rc == AIG_OK; ++i) {
    const long long b = i / per_batch;
    const int s = (int)(b & 1);
    if (rd.threads.empty()) {
      io_ok = read_piece(i);
    } else {
      std::unique_lock<std::mutex> lk(rd.mu);
      rd.cv.wait(lk, [&] { return ready[i] != 0; });
      io_ok = ready[i] == 1;
    }
    if (!io_ok) break;
    if (i % per_batch == 0) rc = cnn_stream_begin(m, s);
    long long lo;
    const int n = piece_frames(i, &lo);
    if (rc == AIG_OK)
      rc = cnn_stream_copy(m, s, (size_t)(lo - b * batch) * r->frame_bytes, st->ring + (size_t)(i % slots) * st->piece_bytes,
                           (size_t)n * r->frame_bytes, st->copied[i % slots]);
    {
      std::lock_guard<std::mutex> lk(rd.mu);
      rd.issued = i + 1;
      rd.cv.notify_all();
    }
    if (rc == AIG_OK && (i + 1 == n_pieces || (i + 1) % per_batch == 0)) {
      // the slot's output buffer is free once the batch before the last has been taken from it
      if (b >= 2) rc = collect(b - 2);
      if (rc == AIG_OK) rc = cnn_stream_submit(m, s, st->out[s], true);
    }
  }
  rd.finish();
  for (long long b = (n_batches >= 2 ? n_batches - 2 : 0); b < n_batches && rc == AIG_OK && io_ok; ++b) rc = collect(b);
  if (rc == AIG_OK && io_ok) return AIG_OK;
  cnn_stream_drain(m);  // the ring and the output buffers are not in use any more
  return rc != AIG_OK ? rfail(r, rc, aig_cnn_last_error(m)) : rfail(r, AIG_ERR_IO, "short read of a frame");
}

extern "C" int aig_cnn_infer_recording(aig_cnn* m, aig_recording* r, long long first, long long count, int batch, int n_out, float* out_host) {
  if (!m || !r || !out_host || batch <= 0 || n_out <= 0 || count < 0) return AIG_ERR_INVALID;
  try {
    if (first < 0 || first + count > r->n_records) return rfail(r, AIG_ERR_INVALID, "record range outside the file");
    const aig_cnn_config& c = cnn_config(m);
    if (batch != c.batch || n_out != c.n_out || r->width != c.width || r->height != c.height)
      return rfail(r, AIG_ERR_INVALID, "the encoder's batch, outputs or frame size differ from the call's");
    return count == 0 ? AIG_OK : infer_recording(m, r, first, count, batch, n_out, out_host);
  } catch (const std::exception&) {
    // host memory or threads ran out; the threads have ended, and copies that were issued end here
    try {
      cnn_stream_drain(m);
      r->err = "out of host memory or threads";
    } catch (const std::exception&) {
      r->err.clear();
    }
    return AIG_ERR_IO;
  }
}
