// res_chain.cu -- the residual blocks and the head of the 2-D frame encoder as ONE cooperative kernel for small batches.
//
// At batch 1 a layer is one to 19 tiles of 128 positions, and what a launch of its own costs is not its work (1.2 GFLOP
// a frame, 7 MB of weights) but start and end: eight residual-block launches and the head took 12 to 21 us each, most
// of it pipeline fill, drain and, on the deep layers, one CTA walking 36 to 64 blocks of K alone.  Here the layers are
// stages of one launch:
//  - a stage is (tile of 128 positions, 64 output columns) jobs; clusters of four CTAs take them, one CTA a job or, on
//    the deep layers, two or four CTAs a job with a share of K each, whose fp32 sums meet through distributed shared
//    memory (every CTA finishes a share of the rows, always in the same order of addition);
//  - the weights of a CTA's next jobs are fetched ahead of the stage barrier (they depend on nothing); activations are
//    fetched as in the patch-resident kernel: one run of rows per 64 channels, every filter tap a row offset into it;
//  - a stage's barrier counts only the CTAs that had jobs in it, and a CTA without further jobs leaves, so that the
//    next launch finds room while the last, small stages run.
// Bound by the latency of the nine stages at batch 1 (about 9500 clk each: 1200 to hear of the stage before, 1700 for the
// first patch, 2050 for nine blocks of K, 2000 for the exchange of partial sums, 900 to finish the rows, 1250 for the stores
// to be seen; clock64), by the tensor pipe's rate with 64 columns (50 clk an instruction, shared-memory reads) from batch 6
// on.  Before the second MMA issuer, the second set of epilogue warps and the third and fourth patch buffer: 11000 a stage;
// 19 frames of 107x189 82 us, now 66.
#include "res_chain.h"

#include <limits.h>
#include <stdlib.h>

#include "aig_common.cuh"

namespace {

constexpr int kThreads = 384;       // patch producer, MMA issuer, weight producer, second issuer and TMEM owner, eight epilogue warps
constexpr int kCluster = 4;
constexpr int kTileM = 128, kTileN = 64;
constexpr int kWBlock = kTileN * 128;
constexpr int kMaxStages = 14;
constexpr int kAcc = 4;             // accumulator buffers of two times 64 TMEM columns (see the MMA issuer)
constexpr int kAccCols = 2 * kTileN;
constexpr int kPartBytes = kTileM * kTileN * 4;
constexpr int kMaxRing = 12;
constexpr int kMaxBufs = 4;
constexpr int kStageBytes = 2560;
constexpr int kEpi0 = 128;          // first epilogue thread
constexpr int kEpi = kThreads - kEpi0;
// Tiles of the first stage up to which the chain is the faster way.  Measured per frame batch, the whole encoder, chain / launches
// per layer (by rows where they can be): 144x256 x 1 (19 tiles) 57 / 82 us, x 6 (113) 66 / 82, x 10 (188) 78 / 86, 180x320 x 6 (175)
// 79 / 89, 107x189 x 19 (200) 78 / 85, 64x96 x 60 (200) 85 / 85, 360x640 x 2 (229) 90 / 106; beyond, the launches of wider tiles win:
// 144x256 x 13 (245) 88 / 87, 107x189 x 24 (252) 84 / 87, 180x320 x 9 (262) 95 / 92, 144x256 x 16 (301) 99 / 94, 107x189 x 32 (336)
// 100 / 94.
constexpr long long kMaxChainTiles = 240;

struct Walk {                       // what the loops over jobs and K need of a stage
  int P, pad, n_tiles, jobs;
  int taps, kw, cblocks;
  int sparse0, sub;                 // first column tile of a shortcut whose K is one space-to-depth position per tap
  int split;                        // CTAs per job: 1, 2 or 4
  int boxes, box_rows;
  int bufs, buf_bytes;              // patch buffers: as many of this stage's patches as the room for two of the largest holds
};
struct Stage : Walk {
  int RP, Ho, Wo, rows;             // flattened position space of the stage (rows = batch * RP * P)
  int co, c_split;                  // columns >= c_split go to y1
  int act0, act1, padded, s2d, Hb, Wb;
  int arrivals;                     // CTAs with jobs in this stage
  __half *y0, *y1;
  const __half* res;                // residual, rows as the stage's positions
  const float *scale, *shift;
};
static_assert(sizeof(Stage) * kMaxStages <= kStageBytes && sizeof(Stage) % 8 == 0, "stage table");
struct ChainParams {
  int n_stages, clusters, batch;
  int head_bytes;                   // FC weights, mask weights, FC bias
  int patch_bytes, ring;
  float slope;
  unsigned int* words;              // two sets of kMaxStages barrier counters, then the epoch
  int* gerr;
  ResChainHead head;
  Stage st[kMaxStages];
};
struct ChainMaps {
  CUtensorMap a[kMaxStages], b[kMaxStages];
};

__device__ __forceinline__ unsigned int ld_acquire_gpu(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_gpu_add(unsigned int* p, unsigned int v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
// own shared memory -> a cluster CTA's, the bytes counted on that CTA's barrier
__device__ __forceinline__ void bulk_to_cluster(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "r"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// the epilogue warps meet; true if all of them say so
__device__ __forceinline__ bool epilogue_and(bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 q, %1, 0;\n\t"
      "bar.red.and.pred p, 1, %2, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r)
      : "r"(v ? 1u : 0u), "n"(kEpi)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ bool wait_stage(const unsigned int* counter, unsigned int target, volatile int* abort_flag, int* gerr, int code) {
  if (ld_acquire_gpu(counter) >= target) return true;
  const long long t0 = clock64();
  while (ld_acquire_gpu(counter) < target) {
    if (*abort_flag) return false;
    if (clock64() - t0 > AIG_WAIT_CYCLES) {
      *abort_flag = 1;
      atomicCAS(gerr, 0, code);
      return false;
    }
  }
  return true;
}

// The same in every lane, and known to be: the loops that issue TMA and MMA instructions keep their arithmetic in uniform
// registers, where those take their operands from.
__device__ __forceinline__ int uniform(int v) { return __shfl_sync(0xffffffffu, v, 0); }
__device__ __forceinline__ Walk uniform_walk(const Stage& s) {
  Walk w;
  w.P = uniform(s.P); w.pad = uniform(s.pad); w.n_tiles = uniform(s.n_tiles); w.jobs = uniform(s.jobs);
  w.taps = uniform(s.taps); w.kw = uniform(s.kw); w.cblocks = uniform(s.cblocks);
  w.sparse0 = uniform(s.sparse0); w.sub = uniform(s.sub); w.split = uniform(s.split);
  w.boxes = uniform(s.boxes); w.box_rows = uniform(s.box_rows); w.bufs = uniform(s.bufs); w.buf_bytes = uniform(s.buf_bytes);
  return w;
}

// The jobs of a CTA in one stage: job, job + step, ...; `part` is its share of K.
struct JobIter {
  int job, step, part;
};
__device__ __forceinline__ JobIter jobs_of(const Walk& s, int clusters, int cluster, int rank) {
  const int per = kCluster / s.split;
  return JobIter{cluster * per + rank / s.split, clusters * per, rank % s.split};
}
// Its K: dense column tiles take whole blocks of 64 channels with all taps, sparse ones a (tap, block) at a time.
struct KRange {
  bool sparse;
  int lo, hi;
};
__device__ __forceinline__ KRange k_range(const Walk& s, int n_tile, int part) {
  KRange k;
  k.sparse = n_tile >= s.sparse0;
  const int units = k.sparse ? s.taps * s.sub : s.cblocks;
  k.lo = units * part / s.split;
  k.hi = units * (part + 1) / s.split;
  return k;
}
__device__ __forceinline__ void unit_of(const Walk& s, const KRange& k, int u, int& cb, int& tap0, int& tap1) {
  if (k.sparse) {
    tap0 = u / s.sub;
    tap1 = tap0 + 1;
    cb = ((1 - tap0 / s.kw) * 2 + (1 - tap0 % s.kw)) * s.sub + u % s.sub;
  } else {
    cb = u;
    tap0 = 0;
    tap1 = s.taps;
  }
}

// Where one position (a row of a job's tile) goes.
struct RowDst {
  bool store, valid;   // padding positions of a padded destination are stored as zeros
  size_t row;          // row of the destination
};
__device__ __forceinline__ RowDst row_dst(const Stage& s, int q) {
  RowDst r;
  const int vr = q / s.P, vc = q - vr * s.P, n = vr / s.RP, yy = vr - n * s.RP;
  r.valid = q < s.rows && yy < s.Ho && vc < s.Wo;
  r.store = q < s.rows && (r.valid || s.padded);
  r.row = q;
  if (s.s2d) r.row = (((size_t)n * s.Hb + ((yy + 1) >> 1)) * s.Wb + ((vc + 1) >> 1)) * 4 + ((yy + 1) & 1) * 2 + ((vc + 1) & 1);
  else if (!s.padded) r.row = ((size_t)n * s.Ho + yy) * s.Wo + vc;
  return r;
}
// Eight columns of it: affine, residual, activation, store.  aff: scale[64], shift[64] of the job's columns.
template <int ACT>
__device__ __forceinline__ void finish8(const float* aff, const float (&v)[8], bool res, const uint4& rv, const RowDst& r, __half* dst, float slope) {
  const __half2* rh = reinterpret_cast<const __half2*>(&rv);
  uint4 o;
  __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float4 a = *reinterpret_cast<const float4*>(aff + 4 * i), b = *reinterpret_cast<const float4*>(aff + kTileN + 4 * i);
    float2 x = make_float2(fmaf(v[4 * i], a.x, b.x), fmaf(v[4 * i + 1], a.y, b.y));
    float2 y = make_float2(fmaf(v[4 * i + 2], a.z, b.z), fmaf(v[4 * i + 3], a.w, b.w));
    if (res) {
      // the reference stores fp16 after BatchNorm and again after the add (ResConvLayer.cpp:35-36)
      x = __half22float2(__hadd2(__floats2half2_rn(x.x, x.y), rh[2 * i]));
      y = __half22float2(__hadd2(__floats2half2_rn(y.x, y.y), rh[2 * i + 1]));
    }
    oh[2 * i] = __floats2half2_rn(act_apply_fast(x.x, ACT, slope), act_apply_fast(x.y, ACT, slope));
    oh[2 * i + 1] = __floats2half2_rn(act_apply_fast(y.x, ACT, slope), act_apply_fast(y.y, ACT, slope));
  }
  if (!r.valid) o = make_uint4(0, 0, 0, 0);
  if (r.store) *reinterpret_cast<uint4*>(dst) = o;
}
// N groups of eight columns of one row, the first at aff and dst.
template <int N>
__device__ __forceinline__ void finish_row(int act, const float* aff, const float (&v)[N][8], bool res, const uint4* rv, const RowDst& r, __half* dst,
                                           float slope) {
#define AIG_FINISH(ACT) \
  _Pragma("unroll") for (int g = 0; g < N; ++g) finish8<ACT>(aff + 8 * g, v[g], res, rv[g], r, dst + 8 * g, slope)
  switch (act) {
    case AIG_ACT_RELU: AIG_FINISH(AIG_ACT_RELU); break;
    case AIG_ACT_SWISH: AIG_FINISH(AIG_ACT_SWISH); break;
    case AIG_ACT_LEAKY: AIG_FINISH(AIG_ACT_LEAKY); break;
    default: AIG_FINISH(AIG_ACT_NONE); break;
  }
#undef AIG_FINISH
}
// Partial sums of a split job in shared memory: [half of the columns][share of K][R rows][128 bytes], 16-byte chunk c of
// row r at this place of it, so that the writers (a lane per row, one chunk at a time) and the readers (two or four
// neighbouring lanes per row) both meet eight different bank groups.
__device__ __forceinline__ int part_slot(int row, int c) { return row * 128 + ((c ^ (row & 7)) << 4); }
// 8 N columns of row `row`, from chunk c0 of its half on.
template <int S, int N>
__device__ __forceinline__ void sum_parts(const uint8_t* part, int half, int row, int c0, float (&v)[N][8]) {
  constexpr int R = kTileM / S;
  float4 x[S][2 * N];
#pragma unroll
  for (int k = 0; k < S; ++k)
#pragma unroll
    for (int c = 0; c < 2 * N; ++c) x[k][c] = *reinterpret_cast<const float4*>(part + (half * S + k) * R * 128 + part_slot(row, c0 + c));
#pragma unroll
  for (int c = 0; c < 2 * N; ++c) {
    float4 s = x[0][c];
#pragma unroll
    for (int k = 1; k < S; ++k) {
      s.x += x[k][c].x;
      s.y += x[k][c].y;
      s.z += x[k][c].z;
      s.w += x[k][c].w;
    }
    float* o = v[c >> 1] + 4 * (c & 1);
    o[0] = s.x;
    o[1] = s.y;
    o[2] = s.z;
    o[3] = s.w;
  }
}

// Mask attention, pool, FC and outputs of one frame by the epilogue warps (the arithmetic of cnn_head_kernel).
// sx: [HW][C] in shared memory; w: the FC's weights, the mask's, the FC's bias, there already.
__device__ void head_frame(const ResChainHead& h, const __half* x, int b, __half* sx, const __half* w, float* s_mask, float* s_pool, int tid) {
  const int warp = tid >> 5, lane = tid & 31, HW = h.hw, C = h.c, nvec = HW * C / 8;
  const uint4* xb = reinterpret_cast<const uint4*>(x + (size_t)b * HW * C);
  for (int i0 = tid; i0 < nvec; i0 += kEpi * 4) {
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = i0 + u * kEpi < nvec ? __ldcg(xb + i0 + u * kEpi) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i0 + u * kEpi < nvec) reinterpret_cast<uint4*>(sx)[i0 + u * kEpi] = v[u];
  }
  named_bar_sync(1, kEpi);
  const __half* w1 = w + C * h.n_out;
  constexpr int kAtOnce = 4, kWarps = kEpi / 32;
  for (int p0 = warp; p0 < HW; p0 += kWarps * kAtOnce) {
    float s[kAtOnce];
#pragma unroll
    for (int u = 0; u < kAtOnce; ++u) s[u] = 0.f;
    for (int c = lane * 8; c < C; c += 256) {
      const uint4 wv = *reinterpret_cast<const uint4*>(w1 + c);
      const __half2* wh = reinterpret_cast<const __half2*>(&wv);
#pragma unroll
      for (int u = 0; u < kAtOnce; ++u) {
        const uint4 xv = p0 + kWarps * u < HW ? *reinterpret_cast<const uint4*>(sx + (p0 + kWarps * u) * C + c) : make_uint4(0, 0, 0, 0);
        const __half2* xh = reinterpret_cast<const __half2*>(&xv);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 a = __half22float2(xh[e]), m = __half22float2(wh[e]);
          s[u] = fmaf(a.x, m.x, s[u]);
          s[u] = fmaf(a.y, m.y, s[u]);
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int u = 0; u < kAtOnce; ++u) s[u] += __shfl_xor_sync(0xffffffffu, s[u], o);
    float mine = s[0];
#pragma unroll
    for (int u = 1; u < kAtOnce; ++u) mine = lane == u ? s[u] : mine;
    if (lane < kAtOnce && p0 + kWarps * lane < HW) s_mask[p0 + kWarps * lane] = 1.0f / (1.0f + expf(-(mine + h.mask_b)));
  }
  named_bar_sync(1, kEpi);
  for (int c = tid * 2; c < C; c += 2 * kEpi) {
    float s0 = 0.f, s1 = 0.f;
#pragma unroll 16
    for (int p = 0; p < HW; ++p) {
      const float2 v = __half22float2(*reinterpret_cast<const __half2*>(sx + (size_t)p * C + c));
      const float2 m = __half22float2(__floats2half2_rn(v.x * s_mask[p], v.y * s_mask[p]));
      s0 += m.x;
      s1 += m.y;
    }
    const __half2 f = __floats2half2_rn(s0 / (float)HW, s1 / (float)HW);
    *reinterpret_cast<__half2*>(reinterpret_cast<__half*>(h.feat) + (size_t)b * C + c) = f;
    s_pool[c] = __low2float(f);
    s_pool[c + 1] = __high2float(f);
  }
  named_bar_sync(1, kEpi);
  for (int o = tid >> 3; o < (h.n_out + 31) / 32 * 32; o += 32) {  // eight lanes an output
    const bool on = o < h.n_out;
    float acc = 0.f;
    if (on) {
#pragma unroll 16
      for (int c = tid & 7; c < C; c += 8) acc = fmaf(s_pool[c], __half2float(w[(size_t)c * h.n_out + o]), acc);
    }
    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
    acc += __shfl_xor_sync(0xffffffffu, acc, 2);
    acc += __shfl_xor_sync(0xffffffffu, acc, 4);
    if (on && (tid & 7) == 0) {
      const float t = __half2float(__float2half(acc));
      const float y = __half2float(__float2half(t + __half2float(w1[C + o])));
      const __half v = o < h.n_sigmoid ? __float2half(1.0f / (1.0f + expf(-y))) : __float2half(tanhf(y));
      reinterpret_cast<__half*>(h.out_half)[(size_t)b * h.n_out + o] = v;
      h.out_f32[(size_t)b * h.n_out + o] = __half2float(v);
    }
  }
  named_bar_sync(1, kEpi);
}

__global__ void __launch_bounds__(kThreads, 1) res_chain_kernel(const __grid_constant__ ChainMaps maps, const __grid_constant__ ChainParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - raw);
  const uint32_t sPatch = base, sW = base + 2 * p.patch_bytes, sPart = sW + p.ring * kWBlock;
  uint8_t* part = sm + 2 * p.patch_bytes + p.ring * kWBlock;    // partial sums received from the CTAs of a split job
  uint8_t* sent = part + kPartBytes;                            // and sent to them
  float* s_aff = reinterpret_cast<float*>(sent + kPartBytes);   // [2][128]: scale and shift of a job's columns
  // the stages' descriptions: indexed in the parameter block every field was a constant-cache miss of its own
  const Stage* st = reinterpret_cast<const Stage*>(s_aff + 256);
  __half* s_head = reinterpret_cast<__half*>(sm + 2 * p.patch_bytes + p.ring * kWBlock + 2 * kPartBytes + 1024 + kStageBytes);  // the head's weights
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(s_head) + p.head_bytes);
  const uint32_t bar_pfull = smem_u32(bars), bar_pempty = bar_pfull + 8 * kMaxBufs, bar_tfull = bar_pempty + 8 * kMaxBufs, bar_tempty = bar_tfull + 8 * kAcc;
  const uint32_t bar_wfull = bar_tempty + 8 * kAcc, bar_wempty = bar_wfull + 8 * kMaxRing;
  const uint32_t bar_part = bar_wempty + 8 * kMaxRing;  // partial sums of a split job have arrived
  const uint32_t bar_free = bar_part + 8;               // [2]: the other CTAs of a job split in two / four have read theirs
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(bars + 2 * kMaxBufs + 2 * kAcc + 2 * kMaxRing + 3);
  volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int rank = uniform((int)cluster_ctarank()), cluster = blockIdx.x / kCluster;
  griddep_launch_dependents();
  for (int i = threadIdx.x; i < (int)(sizeof(Stage) / 8) * p.n_stages; i += kThreads)
    const_cast<uint64_t*>(reinterpret_cast<const uint64_t*>(st))[i] = reinterpret_cast<const uint64_t*>(p.st)[i];
  if (threadIdx.x == 0) {
    for (int i = 0; i < kMaxBufs; ++i) {
      mbar_init(bar_pfull + 8 * i, 1);
      mbar_init(bar_pempty + 8 * i, 2);
    }
    for (int i = 0; i < kAcc; ++i) {
      mbar_init(bar_tfull + 8 * i, 2);
      mbar_init(bar_tempty + 8 * i, kEpi / 32);
    }
    for (int i = 0; i < p.ring; ++i) {
      mbar_init(bar_wfull + 8 * i, 1);
      mbar_init(bar_wempty + 8 * i, 2);
    }
    mbar_init(bar_part, 1);
    mbar_init(bar_free, 2);
    mbar_init(bar_free + 8, 4);
    *s_abort = 0;
    fence_mbar_init();
  }
  if (warp == 2 && lane < p.n_stages) {
    tma_prefetch_desc(&maps.a[lane]);
    tma_prefetch_desc(&maps.b[lane]);
  }
  if (warp == 3) {
    tmem_alloc(smem_u32(s_tmem), kAcc * kAccCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // every CTA's barriers are there before anything crosses
  tc_fence_after();
  const uint32_t tmem_base = *s_tmem;
  // (written by the launch before this one on the stream, which the first layer's ordinary launch waited for)
  unsigned int* const epoch_word = p.words + 2 * kMaxStages;
  const unsigned int epoch = *reinterpret_cast<volatile unsigned int*>(epoch_word);
  unsigned int* counters = p.words + (epoch & 1u) * kMaxStages;

  if (warp == 0) {
    // ------------------------------------------------------------------ patch producer
    const bool leader = elect_one();
    uint32_t ph = 0;  // a bit per buffer
    bool ok = true;
    griddep_wait();
    for (int si = 0; si < p.n_stages && ok; ++si) {
      const Walk s = uniform_walk(st[si]);
      const JobIter it = jobs_of(s, p.clusters, cluster, rank);
      if (it.job >= s.jobs) continue;
      if (si > 0) {
        ok = wait_stage(counters + si - 1, (unsigned int)st[si - 1].arrivals, s_abort, p.gerr, 810 + si);
        if (!ok) break;
        fence_proxy_async_global();  // written with ordinary stores, read by the TMA unit
      }
      int buf = 0;  // (every MMA of the stage before has been done: its buffers are free, however large they were)
      for (int job = it.job; job < s.jobs && ok; job += it.step) {
        const int n_tile = job % s.n_tiles, m_tile = job / s.n_tiles;
        const KRange k = k_range(s, n_tile, it.part);
        const int row0 = m_tile * kTileM - s.pad * (s.P + 1);  // (rows before the tensor read as zeros)
        for (int u = k.lo; u < k.hi; ++u) {
          int cb, t0, t1;
          unit_of(s, k, u, cb, t0, t1);
          if (!mbar_wait_bounded(bar_pempty + 8 * buf, (ph >> buf & 1u) ^ 1u, s_abort, p.gerr, 801)) { ok = false; break; }
          if (leader) {
            mbar_expect_tx(bar_pfull + 8 * buf, (uint32_t)(s.boxes * s.box_rows * 128));
            for (int b = 0; b < s.boxes; ++b)
              tma_load_2d(sPatch + buf * s.buf_bytes + b * s.box_rows * 128, &maps.a[si], bar_pfull + 8 * buf, cb * 64, row0 + b * s.box_rows);
          }
          ph ^= 1u << buf;
          if (++buf == s.bufs) buf = 0;
        }
      }
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------------ weight producer (waits for no stage)
    const bool leader = elect_one();
    int slot = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int si = 0; si < p.n_stages && ok; ++si) {
      const Walk s = uniform_walk(st[si]);
      const JobIter it = jobs_of(s, p.clusters, cluster, rank);
      for (int job = it.job; job < s.jobs && ok; job += it.step) {
        const int n_tile = job % s.n_tiles;
        const KRange k = k_range(s, n_tile, it.part);
        for (int u = k.lo; u < k.hi && ok; ++u) {
          int cb, t0, t1;
          unit_of(s, k, u, cb, t0, t1);
          for (int tap = t0; tap < t1; ++tap) {
            if (!mbar_wait_bounded(bar_wempty + 8 * slot, ph ^ 1u, s_abort, p.gerr, 802)) { ok = false; break; }
            if (leader) {
              mbar_expect_tx(bar_wfull + 8 * slot, (uint32_t)kWBlock);
              tma_load_2d(sW + slot * kWBlock, &maps.b[si], bar_wfull + 8 * slot, (tap * s.cblocks + cb) * 64, n_tile * kTileN);
            }
            if (++slot == p.ring) { slot = 0; ph ^= 1u; }
          }
        }
      }
    }
  } else if (warp == 1 || warp == 3) {
    // ------------------------------------------------------------------ MMA issuers (all lanes run it, one issues: see elect_one)
    // Two warps issue every second instruction each, into an accumulator of its own (the epilogue adds them): a block of K
    // costs one warp 300 to 340 clk, the wait for its weights 75 and every instruction 38 of them, where the tensor pipe needs
    // 210 for its four instructions.
    constexpr uint32_t idesc = umma_idesc_f16(kTileM, kTileN);
    const bool leader = elect_one();
    const int mine = warp >> 1;
    int slot = 0, acc = 0;
    uint32_t pph = 0, wph = 0, aph = 0;  // pph: a bit per buffer
    bool ok = true;
    for (int si = 0; si < p.n_stages && ok; ++si) {
      const Walk s = uniform_walk(st[si]);
      const JobIter it = jobs_of(s, p.clusters, cluster, rank);
      int buf = 0;
      for (int job = it.job; job < s.jobs && ok; job += it.step) {
        const KRange k = k_range(s, job % s.n_tiles, it.part);
        if (!mbar_wait_bounded(bar_tempty + 8 * acc, aph ^ 1u, s_abort, p.gerr, 803)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d = tmem_base + (uint32_t)(acc * kAccCols + mine * kTileN);
        uint32_t first = 0;
        for (int u = k.lo; u < k.hi && ok; ++u) {
          int cb, t0, t1;
          unit_of(s, k, u, cb, t0, t1);
          if (!mbar_wait_bounded(bar_pfull + 8 * buf, pph >> buf & 1u, s_abort, p.gerr, 804)) { ok = false; break; }
          int fs = t0 % s.kw;
          uint32_t a_lo = umma_desc_lo(sPatch + buf * s.buf_bytes) + (uint32_t)(t0 / s.kw * s.P + fs) * 8u + mine * 2u;
          for (int tap = t0; tap < t1; ++tap) {
            if (!mbar_wait_bounded(bar_wfull + 8 * slot, wph, s_abort, p.gerr, 805)) { ok = false; break; }
            const uint32_t b_lo = umma_desc_lo(sW + slot * kWBlock) + mine * 2u;
#pragma unroll
            for (int kk = 0; kk < 2; ++kk)
              if (leader) umma_f16_ss_lo(d, a_lo + (uint32_t)(kk * 4), b_lo + (uint32_t)(kk * 4), umma_desc_hi(128), idesc, kk == 0 ? first : 1u);
            first = 1u;
            if (leader) umma_commit(bar_wempty + 8 * slot);
            if (++slot == p.ring) { slot = 0; wph ^= 1u; }
            a_lo += 8u;
            if (++fs == s.kw) { fs = 0; a_lo += (uint32_t)(s.P - s.kw) * 8u; }
          }
          if (ok && leader) umma_commit(bar_pempty + 8 * buf);
          pph ^= 1u << buf;
          if (++buf == s.bufs) buf = 0;
        }
        if (ok && leader) umma_commit(bar_tfull + 8 * acc);
        if (++acc == kAcc) { acc = 0; aph ^= 1u; }
      }
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ epilogue
    const int tid = threadIdx.x - kEpi0, q4 = warp & 3, half = tid >> 7, tl = tid & 127;
    int acc = 0, split_jobs = 0, free_jobs[2] = {0, 0}, jobs = 0;
    uint32_t aph = 0;
    bool ok = true;
    const bool with_head = p.head.hw > 0;
    if (with_head && (int)blockIdx.x < p.batch) {
      const int n_fc = p.head.c * p.head.n_out;
      for (int i = tid; i < n_fc / 8; i += kEpi) reinterpret_cast<uint4*>(s_head)[i] = __ldg(reinterpret_cast<const uint4*>(p.head.fc_w) + i);
      for (int i = tid; i < p.head.c; i += kEpi) s_head[n_fc + i] = reinterpret_cast<const __half*>(p.head.mask_w)[i];
      for (int i = tid; i < p.head.n_out; i += kEpi) s_head[n_fc + p.head.c + i] = p.head.fc_b ? reinterpret_cast<const __half*>(p.head.fc_b)[i] : __float2half(0.f);
    }
    for (int si = 0; si < p.n_stages && ok; ++si) {
      const Stage s = st[si];
      const JobIter it = jobs_of(s, p.clusters, cluster, rank);
      if (it.job >= s.jobs) continue;
      const int S = s.split, R = kTileM / S, which = S == 4 ? 1 : 0, rank0 = rank - it.part;
      const bool res = s.res != nullptr;
      // what this thread finishes: 32 columns of its TMEM lane or, in a split job, S neighbouring threads share 32 columns of
      // one of this CTA's rows
      const int lrow = S == 1 ? tl : tl / S, row = (S == 1 ? 0 : it.part * R) + lrow, part_cols = 32 / S, c0 = half * 32 + tl % S * part_cols;
      if (res) {  // residual rows come from the stage before
        if (tid == 0) ok = wait_stage(counters + si - 1, (unsigned int)st[si - 1].arrivals, s_abort, p.gerr, 840 + si);
        ok = epilogue_and(ok);
      }
      // (after a wait that ran out a warp goes on with the rest, whose waits return at once, so that all warps meet at every barrier)
      for (int job = it.job; job < s.jobs; job += it.step, ++jobs) {
        const int n_tile = job % s.n_tiles, m_tile = job / s.n_tiles, col0 = n_tile * kTileN;
        const bool second = col0 >= s.c_split;
        const int ch0 = second ? col0 - s.c_split : col0, act = second ? s.act1 : s.act0;
        // everything that does not depend on the accumulator, while it is being computed
        float* aff = s_aff + (jobs & 1) * 128;
        if (tid < 2 * kTileN) aff[tid] = tid < kTileN ? __ldg(s.scale + col0 + tid) : __ldg(s.shift + col0 + tid - kTileN);
        const RowDst rd = row_dst(s, m_tile * kTileM + row);
        __half* dst = (second ? s.y1 : s.y0) + rd.row * s.co + ch0 + c0;
        uint4 rv[4];
#pragma unroll
        for (int g = 0; g < 4; ++g)
          rv[g] = res && rd.valid && g * 8 < part_cols ? __ldcg(reinterpret_cast<const uint4*>(s.res + (size_t)(m_tile * kTileM + row) * s.co + ch0 + c0) + g)
                                                       : make_uint4(0, 0, 0, 0);
        named_bar_sync(1, kEpi);  // scale and shift are there
        ok = mbar_wait_bounded(bar_tfull + 8 * acc, aph, s_abort, p.gerr, 806) && ok;
        if (S > 1 && job != it.job) ok = ok && mbar_wait_bounded_cl(bar_free + 8 * which, (uint32_t)(free_jobs[which] - 1) & 1u, s_abort, p.gerr, 807);
        tc_fence_after();
        const uint32_t t_addr = tmem_base + (uint32_t)(acc * kAccCols + half * 32) + ((uint32_t)(q4 * 32) << 16);
        float v[4][8];
        uint32_t w[32];
        tmem_ld_32x32(t_addr, reinterpret_cast<uint32_t (&)[32]>(v));
        tmem_ld_32x32(t_addr + kTileN, w);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i >> 3][i & 7] += __uint_as_float(w[i]);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_tempty + 8 * acc);
        if (S == 1) {
          finish_row<4>(act, aff + c0, v, res, rv, rd, dst, p.slope);
        } else {
          // this warp's 32 rows go to the CTA that finishes them
          const int target = q4 * 32 / R, r0 = q4 * 32 % R, block = (half * S + it.part) * R * 128;
          uint8_t* mine = target == it.part ? part + block + r0 * 128 : sent + (half * 4 + q4) * 4096;
#pragma unroll
          for (int c = 0; c < 8; ++c)
            *reinterpret_cast<float4*>(mine + part_slot(lane, c)) = make_float4(v[c >> 1][(c & 1) * 4], v[c >> 1][(c & 1) * 4 + 1], v[c >> 1][(c & 1) * 4 + 2], v[c >> 1][(c & 1) * 4 + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0 && target != it.part)
            bulk_to_cluster(mapa_shared(sPart, (uint32_t)(rank0 + target)) + (uint32_t)(block + r0 * 128), smem_u32(mine), 4096,
                            mapa_shared(bar_part, (uint32_t)(rank0 + target)));
          if (tid == 0) mbar_expect_tx(bar_part, kPartBytes - kPartBytes / S);
          ok = mbar_wait_bounded_cl(bar_part, (uint32_t)split_jobs & 1u, s_abort, p.gerr, 808) && ok;
          ++split_jobs;
          named_bar_sync(1, kEpi);  // this CTA's own share is there as well
          float (&v2)[2][8] = reinterpret_cast<float (&)[2][8]>(v);
          float (&v1)[1][8] = reinterpret_cast<float (&)[1][8]>(v);
          if (S == 4) sum_parts<4, 1>(part, half, lrow, tl % 4 * 2, v1);
          else sum_parts<2, 2>(part, half, lrow, tl % 2 * 4, v2);
          if (job + it.step < s.jobs) {  // (between stages the stage barrier says as much; the arrival waits for all this thread has in flight)
            named_bar_sync(1, kEpi);  // all have read
            if (tid < S) mbar_arrive_cluster(mapa_shared(bar_free + 8 * which, (uint32_t)(rank0 + tid)));
            ++free_jobs[which];
          }
          if (S == 4) finish_row<1>(act, aff + c0, v1, res, rv, rd, dst, p.slope);
          else finish_row<2>(act, aff + c0, v2, res, rv, rd, dst, p.slope);
        }
        if (++acc == kAcc) { acc = 0; aph ^= 1u; }
      }
      fence_proxy_async_global();  // the next stage's TMA loads read these rows
      ok = epilogue_and(ok);
      if (!ok) break;
      if (tid == 0) red_release_gpu_add(counters + si, 1u);
    }
    if (ok && with_head && (int)blockIdx.x < p.batch) {
      // ---------------------------------------------------------------- head (patches and ring are free by now)
      const int last = p.n_stages - 1;
      __half* sx = reinterpret_cast<__half*>(sm);
      float* s_mask = reinterpret_cast<float*>(part);
      if (tid == 0) ok = wait_stage(counters + last, (unsigned int)st[last].arrivals, s_abort, p.gerr, 830);
      ok = epilogue_and(ok);
      for (int b = blockIdx.x; b < p.batch && ok; b += gridDim.x) head_frame(p.head, st[last].y0, b, sx, s_head, s_mask, s_mask + p.head.hw, tid);
    }
    if (blockIdx.x == 0 && tid == 0) {
      // the next launch's counters: their last user was the launch before this one
      for (int i = 0; i < kMaxStages; ++i) p.words[((epoch + 1u) & 1u) * kMaxStages + i] = 0u;
      *epoch_word = epoch + 1u;
    }
  }

  if (*s_abort) {
    // give copies and MMAs still in flight time to land before shared memory and TMEM go away
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // no CTA leaves while another of its cluster may still write to it
  if (warp == 3) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kAcc * kAccCols);
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
int encode_rows(aig_ctx* ctx, CUtensorMap* m, const void* ptr, uint64_t cols, uint64_t rows, uint32_t box_rows) {
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
    return aig_fail(ctx, AIG_ERR_CUDA, "cuTensorMapEncodeTiled entry point not available");
  cuuint64_t dims[2] = {cols, rows}, strides[1] = {cols * 2};
  cuuint32_t box[2] = {64, box_rows}, es[2] = {1, 1};
  const CUresult r = reinterpret_cast<EncodeTiledFn>(fn)(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, es,
                                                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? AIG_OK : aig_fail(ctx, AIG_ERR_CUDA, "cuTensorMapEncodeTiled(rows) failed: %d", (int)r);
}

}  // namespace

struct ResChain {
  aig_ctx* ctx = nullptr;
  ChainParams prm{};
  ChainMaps maps{};
  int smem = 0;
};

namespace {

cudaLaunchConfig_t chain_config(const ResChain* c, int clusters, cudaLaunchAttribute (&attr)[3]) {
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kCluster;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeCooperative;
  attr[1].val.cooperative = 1;
  attr[2] = pdl_attribute(c->ctx);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(clusters * kCluster);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = c->smem;
  cfg.stream = c->ctx->stream;
  cfg.attrs = attr;
  cfg.numAttrs = 3;
  return cfg;
}

}  // namespace

int res_chain_create(aig_ctx* ctx, const std::vector<ResChainBlock>& blocks, int hw, int c_last, int n_out, ResChain** out) {
  *out = nullptr;
  if (const char* e = getenv("AIG_CNN_NO_CHAIN")) if (atoi(e)) return AIG_OK;
  if (blocks.empty() || 2 * blocks.size() > kMaxStages) return AIG_OK;
  DeviceGuard guard(ctx->device);
  ResChain* c = new ResChain();
  c->ctx = ctx;
  ChainParams& p = c->prm;
  auto decline = [&]() {
    cudaGetLastError();
    res_chain_destroy(c);
    return (int)AIG_OK;
  };
  std::vector<ConvPlanView> views;
  int patch_rows = 0;
  for (const ResChainBlock& b : blocks)
    for (const aig_conv_plan* plan : {b.down, b.conv1}) {
      ConvPlanView v;
      if (!plan || !conv_plan_view(plan, &v) || v.out_c % 64 != 0 || v.is_down != (plan == b.down)) return decline();
      views.push_back(v);
      Stage& s = p.st[p.n_stages++];
      s.P = v.P; s.RP = v.RP; s.pad = v.pad; s.Ho = v.Ho; s.Wo = v.Wo;
      const long long rows = (long long)v.batch * v.RP * v.P;
      if (rows > kMaxChainTiles * kTileM) return decline();
      s.rows = (int)rows;
      s.n_tiles = (v.is_down ? 2 : 1) * v.out_c / kTileN;
      s.jobs = (int)ceil_div_ll(rows, kTileM) * s.n_tiles;
      s.taps = v.taps; s.kw = v.kw; s.cblocks = v.cblocks;
      s.sub = v.sub_cblocks;
      s.sparse0 = v.sub_cblocks ? v.out_c / kTileN : INT_MAX;
      const int need = kTileM + (v.kh - 1) * v.P + v.kw - 1;
      s.boxes = (need + 255) / 256;
      s.box_rows = ((need + s.boxes - 1) / s.boxes + 7) / 8 * 8;
      if (s.boxes * s.box_rows > patch_rows) patch_rows = s.boxes * s.box_rows;
      s.co = v.out_c;
      s.c_split = v.is_down ? v.out_c : INT_MAX;
      s.act0 = v.act; s.act1 = AIG_ACT_NONE;
      s.padded = v.is_down ? 1 : 0;
      s.s2d = v.s2d; s.Hb = v.Hb; s.Wb = v.Wb;
      s.y0 = (__half*)(v.is_down ? b.t : b.y);
      s.y1 = (__half*)b.r;
      s.res = v.is_down ? nullptr : (const __half*)b.r;
      s.scale = v.scale; s.shift = v.shift;
      p.batch = v.batch;
      p.slope = v.slope;
    }
  p.patch_bytes = (patch_rows * 128 + 1023) / 1024 * 1024;
  for (int i = 0; i < p.n_stages; ++i) {
    Stage& s = p.st[i];
    s.buf_bytes = (s.boxes * s.box_rows * 128 + 1023) / 1024 * 1024;
    s.bufs = 2 * p.patch_bytes / s.buf_bytes;
    if (s.bufs > kMaxBufs) s.bufs = kMaxBufs;
  }
  p.head_bytes = ((n_out + 1) * c_last + n_out) * 2;
  p.head_bytes = (p.head_bytes + 127) / 128 * 128;
  const int fixed = 1024 + 2 * kPartBytes + 1024 + kStageBytes + p.head_bytes + 512;
  p.ring = (227 * 1024 - fixed - 2 * p.patch_bytes) / kWBlock;
  if (p.ring > kMaxRing) p.ring = kMaxRing;
  if (p.ring < 4) return decline();
  // the head keeps a frame's last feature map where patches and weights were
  if (c_last % 8 != 0 || (size_t)hw * c_last * 2 > (size_t)2 * p.patch_bytes + p.ring * kWBlock || (hw + c_last) * 4 > kPartBytes) return decline();
  c->smem = fixed + 2 * p.patch_bytes + p.ring * kWBlock;
  cudaLaunchAttribute attr[3];
  cudaLaunchConfig_t cfg = chain_config(c, ctx->sm_count / kCluster, attr);
  int n = 0;
  if (cudaFuncSetAttribute(res_chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, res_chain_kernel, &cfg) != cudaSuccess)
    return decline();
  p.clusters = n < ctx->sm_count / kCluster ? n : ctx->sm_count / kCluster;
  if (p.clusters < 8) return decline();
  for (int i = 0; i < p.n_stages; ++i) {
    Stage& s = p.st[i];
    // CTAs per job: the busiest CTA's blocks of K (0.17 us each, measured with one MMA issuer; 0.12 with two) and hand-overs
    // (1 us a job, 2 with the exchange)
    double best = 0.0;
    const int units = s.sub ? (s.cblocks < s.taps * s.sub ? s.cblocks : s.taps * s.sub) : s.cblocks;
    for (int split = 1; split <= kCluster && split <= units; split *= 2) {
      const int rounds = ceil_div(s.jobs, p.clusters * (kCluster / split));
      const double t = rounds * (ceil_div(s.cblocks, split) * s.taps * 0.17 + (split == 1 ? 1.0 : 2.0));
      if (best == 0.0 || t < best) {
        best = t;
        s.split = split;
      }
    }
    const int groups = p.clusters * (kCluster / s.split);
    s.arrivals = (s.jobs < groups ? s.jobs : groups) * s.split;
  }
  int rc = AIG_OK;
  for (int i = 0; i < p.n_stages && rc == AIG_OK; ++i) {
    const ConvPlanView& v = views[i];
    const ResChainBlock& b = blocks[i / 2];
    rc = encode_rows(ctx, &c->maps.a[i], v.is_down ? b.in : b.t, v.in_c, (uint64_t)p.st[i].rows, (uint32_t)p.st[i].box_rows);
    if (rc == AIG_OK) rc = encode_rows(ctx, &c->maps.b[i], v.w, (uint64_t)v.w_k, (uint64_t)v.w_rows, kTileN);
  }
  const size_t words = (2 * kMaxStages + 1) * sizeof(unsigned int);
  if (rc == AIG_OK && (cudaMalloc(&p.words, words) != cudaSuccess || cudaMemsetAsync(p.words, 0, words, ctx->stream) != cudaSuccess))
    rc = aig_fail(ctx, AIG_ERR_CUDA, "residual block chain: allocation failed");
  if (rc != AIG_OK) {
    res_chain_destroy(c);
    return rc;
  }
  p.gerr = ctx->d_err;
  *out = c;
  return AIG_OK;
}

void res_chain_destroy(ResChain* c) {
  if (!c) return;
  cudaFree(c->prm.words);
  delete c;
}

int res_chain_forward(ResChain* c, const ResChainHead& head) {
  aig_ctx* ctx = c->ctx;
  DeviceGuard guard(ctx->device);
  c->prm.head = head;
  cudaLaunchAttribute attr[3];
  const cudaLaunchConfig_t cfg = chain_config(c, c->prm.clusters, attr);
  AIG_CUDA_OK(ctx, cudaLaunchKernelEx(&cfg, res_chain_kernel, c->maps, c->prm));
  return AIG_OK;
}
