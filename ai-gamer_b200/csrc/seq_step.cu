// seq_step.cu -- the streaming step of the sequence head ([bridge FC ->] LSTM layers -> attention over the ring cache
// -> LayerNorm -> FC -> sigmoid/tanh) as ONE cooperative kernel for up to 128 sequences.
//
// A step multiplies 10.5 MB of fp16 weights (two layers of 512) with one column per sequence.  What bounds it is the
// chain of dependent stages, not bandwidth: as launches it was 15 of them at 9 to 19 us (a GEMM of one M tile walks its
// K extent in 4 to 32 CTAs), and as one kernel that streamed the weights from L2 after each stage's barrier 57 us.  Here
//  - the weights of a CTA (4 hidden units: their 16 gate rows of every layer's W and R, 4 rows each of Wq, Wk, Wv, Wo,
//    the FC: 95 KB at 512) go to shared memory by bulk copies that are issued at once, before the kernel waits for its
//    predecessor (programmatic launch), so they arrive under the last kernels of the frame encoder;
//  - R.h of every layer needs the previous step only and is done while the first weights are the only ones there;
//  - a stage is a [16 rows x K] x [K x batch] product on mma.sync m16n8k16: with 16 weight rows per CTA the stage is
//    bound by latency and by L2 (every CTA reads all activations), which tcgen05's 128-row tiles would only worsen.
//    The eight warps split the sequences in tiles of eight and, where there are fewer tiles than warps, K;
//  - stages are separated by grid barriers on a global counter (bounded spin, cooperative launch):
//    [bridge] | LSTM 0 | LSTM 1 | ... | q,k,v | attention per (sequence, head) | output projection | LayerNorm, FC.
// The step's position and the barrier's epoch live in device memory, so that a captured graph replays the step.
//
// Arithmetic: fp32 accumulation, fp16 where the per-operator launches store fp16 (embedding before and after the bias,
// h, c, q, k, v, context, attention output, LayerNorm output, FC output before and after the bias).
#include <math.h>

#include "aig_common.cuh"
#include "seq_step.h"

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxLayers = 4;
constexpr int kMaxWindow = 128;
constexpr int kHeadDim = 64;
constexpr int kUnits = 4;         // hidden units (and rows of every other matrix) per CTA
constexpr int kAttnFloats = 3 * kHeadDim + 16;  // a warp's q, k, v and partial context
constexpr int kRows = 16;         // rows of an mma tile: four gates of kUnits units
constexpr int kMaxBatch = 128;
constexpr int kMaxBars = 2 + kMaxLayers + 3;
constexpr size_t kMaxSmem = 220 * 1024;

enum { kCount0 = 0, kCount1 = 1, kEpoch = 2, kPosition = 3, kWords = 4 };

struct StepParams {
  int B, nt, kw;                  // sequences, tiles of eight of them, warps along K
  int in_c, H, layers, heads, window, n_out, n_sig, feat, bridge_rows;
  float rope_base, scale, clip;
  const __half* features;         // [B][feat], or null: emb is the input
  const __half *bw_t, *bb;        // bridge [in_c][feat], bias
  __half* emb_out;
  const __half* emb;
  const __half* lstm;
  unsigned long long w_off[kMaxLayers], r_off[kMaxLayers], bw_off[kMaxLayers], br_off[kMaxLayers];
  int double_bias;
  const __half *wq_t, *wk_t, *wv_t, *wo_t, *fcw_t, *fcb;  // [out][in]
  const float *ln_g, *ln_b;
  __half *h_state, *c_state, *h_new;
  __half *q, *k, *v, *ctx, *a;
  __half *kcache, *vcache;
  __half *y, *logits;
  float* out_f32;
  unsigned int* words;
  int* gerr;
  // shared memory, bytes from the start
  int o_r[kMaxLayers], o_w[kMaxLayers], o_bridge, o_qkv, o_wo, o_fc, o_pre, o_red, o_cell, o_hid, o_bias, o_attn;
};

// rows of `k` halfs in shared memory: whole 64-byte blocks, and an odd number of them, so that the eight rows a warp
// reads at once (16 bytes a lane) fall on different banks
__host__ __device__ constexpr int row_stride(int k) { return (((k * 2 + 63) / 64) | 1) * 64; }

__device__ __forceinline__ unsigned int ld_acquire_gpu(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_gpu_add(unsigned int* p, unsigned int v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float sigmoidf_(float x) { return 1.0f / (1.0f + expf(-x)); }

struct StepCta {
  const StepParams& p;
  uint8_t* sm;
  uint32_t bars;
  volatile int* abort_flag;
  int* s_flag;
  unsigned int* counter;
  unsigned int arrived;

  // Grid-wide barrier.  Every CTA arrives once; the wait is bounded.
  __device__ bool barrier(int code) {
    __syncthreads();
    arrived += gridDim.x;
    if (threadIdx.x == 0) {
      red_release_gpu_add(counter, 1u);  // (releases what the block wrote before the __syncthreads)
      const long long t0 = clock64();
      int ok = 1;
      while ((int)(ld_acquire_gpu(counter) - arrived) < 0) {
        if (clock64() - t0 > AIG_WAIT_CYCLES) {
          atomicCAS(p.gerr, 0, code);
          ok = 0;
          break;
        }
      }
      *s_flag = ok;
    }
    __syncthreads();
    return *s_flag != 0;
  }
  // the same answer for every thread
  __device__ bool weights(int i) { return __syncthreads_and(mbar_wait_bounded(bars + 8 * i, 0, abort_flag, p.gerr, 720 + i)) != 0; }
  __device__ float* red() const { return reinterpret_cast<float*>(sm + p.o_red); }
  // element (row, b) of the product that `multiply` left behind, its parts along K added up
  __device__ float value(int row, int b) const {
    const float* r = red() + ((b >> 3) * kRows + row) * 8 + (b & 7);
    float s = r[0];
    for (int w = 1; w < p.kw; ++w) s += r[(size_t)w * p.nt * kRows * 8];
    return s;
  }
  // [16 rows of `a` in shared memory] x [K x B], x [b][K] in global memory.  A lane takes 16 bytes of a row and of a
  // column at the same place, which the two mma steps of a 32-deep block use as their k: the order of k is free.
  template <int TPW>
  __device__ void multiply(const uint8_t* a, const __half* x, int x_stride, int K) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const int wk = warp % p.kw, wn = warp / p.kw, groups = kWarps / p.kw;
    const int nkb = (K + 31) >> 5, stride = row_stride(K);
    const uint8_t* a0 = a + g * stride + q * 16;
    const uint8_t* a1 = a0 + 8 * stride;
    constexpr int U = 4;  // blocks in flight
    float acc[TPW][4];
    const __half* xr[TPW];
    bool on[TPW];
#pragma unroll
    for (int j = 0; j < TPW; ++j) {
      const int b = (wn + j * groups) * 8 + g;
      on[j] = b < p.B;
      xr[j] = x + (size_t)(on[j] ? b : 0) * x_stride + q * 8;
      acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    }
    for (int kb0 = wk; kb0 < nkb; kb0 += p.kw * U) {
      uint4 xv[U][TPW];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int kb = kb0 + u * p.kw;
#pragma unroll
        for (int j = 0; j < TPW; ++j)
          xv[u][j] = on[j] && kb * 32 + q * 8 < K ? __ldcg(reinterpret_cast<const uint4*>(xr[j] + kb * 32)) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int kb = kb0 + u * p.kw;
        if (kb >= nkb) break;
        const uint4 w0 = *reinterpret_cast<const uint4*>(a0 + kb * 64), w1 = *reinterpret_cast<const uint4*>(a1 + kb * 64);
#pragma unroll
        for (int j = 0; j < TPW; ++j) {
          mma_16816(acc[j], w0.x, w1.x, w0.y, w1.y, xv[u][j].x, xv[u][j].y);
          mma_16816(acc[j], w0.z, w1.z, w0.w, w1.w, xv[u][j].z, xv[u][j].w);
        }
      }
    }
    float* r = red();
#pragma unroll
    for (int j = 0; j < TPW; ++j) {
      const int t = wn + j * groups;
      if (t < p.nt) {
        float* d = r + ((size_t)(wk * p.nt + t) * kRows + g) * 8 + 2 * q;
        *reinterpret_cast<float2*>(d) = make_float2(acc[j][0], acc[j][1]);
        *reinterpret_cast<float2*>(d + 8 * 8) = make_float2(acc[j][2], acc[j][3]);
      }
    }
    __syncthreads();
  }
};

// Attention of one (sequence, head) by `warps` warps of a CTA, this one being number `sub`: rotate q and k at `position`,
// append k and v to the ring (warp 0), attend to the slots of this warp's share.  A lane takes eight dimensions of every
// fourth slot; all of a block's k and v rows are in flight together, because the stage is bound by that latency.  The
// share's running maximum, sum and context go to `part` where an item has several warps, else to the context itself.
__device__ void attend(const StepParams& p, int item, int position, int n_valid, float cs, float sn, float* sq, float* part, int warps, int sub,
                       int lane) {
  constexpr int d = kHeadDim, half_d = d / 2, kBlock = 8;  // slots a lane has in flight (32 per warp)
  const int b = item / p.heads, h = item - b * p.heads, E = p.H, slot = position % p.window;
  const size_t row = (size_t)b * E + (size_t)h * d, ring = (size_t)b * p.window * E + (size_t)h * d;
  const int grp = lane >> 3, dim = (lane & 7) * 8;
  const int share = ((n_valid + warps - 1) / warps + 3) & ~3, lo = sub * share, hi = min(n_valid, lo + share);
  __half* sk = reinterpret_cast<__half*>(sq + d);  // this step's k and v
  __half* sv = sk + d;
  {
    const int j = lane;  // half_d == 32
    const float qa = __half2float(__ldcg(p.q + row + j)), qb = __half2float(__ldcg(p.q + row + j + half_d));
    const float ka = __half2float(__ldcg(p.k + row + j)), kb = __half2float(__ldcg(p.k + row + j + half_d));
    const __half va = __ldcg(p.v + row + j), vb = __ldcg(p.v + row + j + half_d);
    const __half k0 = __float2half(ka * cs - kb * sn), k1 = __float2half(kb * cs + ka * sn);
    sq[j] = __half2float(__float2half(qa * cs - qb * sn));
    sq[j + half_d] = __half2float(__float2half(qb * cs + qa * sn));
    sk[j] = k0; sk[j + half_d] = k1;
    sv[j] = va; sv[j + half_d] = vb;
    if (sub == 0) {
      __half* kslot = p.kcache + ring + (size_t)slot * E;
      __half* vslot = p.vcache + ring + (size_t)slot * E;
      kslot[j] = k0; kslot[j + half_d] = k1;
      vslot[j] = va; vslot[j + half_d] = vb;
    }
  }
  __syncwarp();
  float q[8], acc[8], mx = -INFINITY, sum = 0.f;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    q[e] = sq[dim + e] * p.scale;
    acc[e] = 0.f;
  }
  for (int i0 = lo; i0 < hi; i0 += 4 * kBlock) {
    uint4 kv[kBlock], vv[kBlock];
#pragma unroll
    for (int u = 0; u < kBlock; ++u) {
      const int i = i0 + 4 * u + grp;
      kv[u] = vv[u] = make_uint4(0, 0, 0, 0);
      if (i < hi && i != slot) {
        kv[u] = *reinterpret_cast<const uint4*>(p.kcache + ring + (size_t)i * E + dim);
        vv[u] = *reinterpret_cast<const uint4*>(p.vcache + ring + (size_t)i * E + dim);
      } else if (i < hi) {
        kv[u] = *reinterpret_cast<const uint4*>(sk + dim);
        vv[u] = *reinterpret_cast<const uint4*>(sv + dim);
      }
    }
    float s[kBlock], top = mx;
#pragma unroll
    for (int u = 0; u < kBlock; ++u) {
      const __half2* kh = reinterpret_cast<const __half2*>(&kv[u]);
      float t = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = __half22float2(kh[e]);
        t = fmaf(q[2 * e], f.x, t);
        t = fmaf(q[2 * e + 1], f.y, t);
      }
      t += __shfl_xor_sync(0xffffffffu, t, 1);
      t += __shfl_xor_sync(0xffffffffu, t, 2);
      t += __shfl_xor_sync(0xffffffffu, t, 4);
      s[u] = i0 + 4 * u + grp < hi ? t : -INFINITY;
      top = fmaxf(top, s[u]);
    }
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 8));
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 16));
    const float keep = expf(mx - top);  // (0 in the first block)
    mx = top;
    sum *= keep;
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] *= keep;
#pragma unroll
    for (int u = 0; u < kBlock; ++u) {
      const float w = expf(s[u] - mx);
      const __half2* vh = reinterpret_cast<const __half2*>(&vv[u]);
      sum += w;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = __half22float2(vh[e]);
        acc[2 * e] = fmaf(w, f.x, acc[2 * e]);
        acc[2 * e + 1] = fmaf(w, f.y, acc[2 * e + 1]);
      }
    }
  }
  sum += __shfl_xor_sync(0xffffffffu, sum, 8);
  sum += __shfl_xor_sync(0xffffffffu, sum, 16);
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], 8);
    acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], 16);
  }
  if (grp != 0) return;
  if (warps == 1) {
    __align__(16) __half out[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) out[e] = __float2half(acc[e] / sum);
    *reinterpret_cast<uint4*>(p.ctx + row + dim) = *reinterpret_cast<const uint4*>(out);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) part[dim + e] = acc[e];
    if (dim == 0) {
      part[d] = mx;
      part[d + 1] = sum;
    }
  }
}

// TPW = tiles of eight sequences per warp: 1 up to 64 sequences, 2 up to 128
template <int TPW>
__global__ void __launch_bounds__(kThreads, 1) seq_step_kernel(const StepParams p) {
  extern __shared__ __align__(128) uint8_t sm[];
  __shared__ uint64_t s_bars[kMaxBars];
  __shared__ int s_flag;
  __shared__ int s_abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int H = p.H, B = p.B, L = p.layers, unit0 = blockIdx.x * kUnits, n_bars = 2 + L + 3;
  const uint32_t base = smem_u32(sm), bars = smem_u32(s_bars);
  const int b_bridge = 1, b_qkv = 2 + L, b_wo = 3 + L, b_fc = 4 + L;
  const int bridge0 = blockIdx.x * p.bridge_rows, n_bridge = p.features ? max(0, min(p.bridge_rows, p.in_c - bridge0)) : 0;

  // ---- weights to shared memory, in the order of their use
  if (warp == 0) {
    if (lane == 0) {
      for (int i = 0; i < n_bars; ++i) mbar_init(bars + 8 * i, 1);
      s_abort = 0;
      fence_mbar_init();
      mbar_expect_tx(bars, (uint32_t)(L * kRows * H * 2));
      mbar_expect_tx(bars + 8 * b_bridge, (uint32_t)(n_bridge * p.feat * 2));
      for (int l = 0; l < L; ++l) mbar_expect_tx(bars + 8 * (2 + l), (uint32_t)(kRows * (l == 0 ? p.in_c : H) * 2));
      mbar_expect_tx(bars + 8 * b_qkv, (uint32_t)(3 * kUnits * H * 2));
      mbar_expect_tx(bars + 8 * b_wo, (uint32_t)(kUnits * H * 2));
      mbar_expect_tx(bars + 8 * b_fc, (uint32_t)(p.n_out * H * 2));
    }
    __syncwarp();
    const uint32_t hb = (uint32_t)H * 2;
    const int hs = row_stride(H);
    for (int i = lane; i < L * kRows; i += 32) {
      const int l = i / kRows, r = i % kRows;
      bulk_load(base + p.o_r[l] + r * hs, p.lstm + p.r_off[l] + ((size_t)(r >> 2) * H + unit0 + (r & 3)) * H, hb, bars);
    }
    for (int r = lane; r < n_bridge; r += 32)
      bulk_load(base + p.o_bridge + r * row_stride(p.feat), p.bw_t + (size_t)(bridge0 + r) * p.feat, (uint32_t)p.feat * 2, bars + 8 * b_bridge);
    for (int i = lane; i < L * kRows; i += 32) {
      const int l = i / kRows, r = i % kRows, in = l == 0 ? p.in_c : H;
      bulk_load(base + p.o_w[l] + r * row_stride(in), p.lstm + p.w_off[l] + ((size_t)(r >> 2) * H + unit0 + (r & 3)) * in, (uint32_t)in * 2,
                bars + 8 * (2 + l));
    }
    for (int r = lane; r < 3 * kUnits; r += 32) {
      const __half* m = (r >> 2) == 0 ? p.wq_t : ((r >> 2) == 1 ? p.wk_t : p.wv_t);
      bulk_load(base + p.o_qkv + r * hs, m + (size_t)(unit0 + (r & 3)) * H, hb, bars + 8 * b_qkv);
    }
    for (int r = lane; r < kUnits; r += 32) bulk_load(base + p.o_wo + r * hs, p.wo_t + (size_t)(unit0 + r) * H, hb, bars + 8 * b_wo);
    for (int r = lane; r < p.n_out; r += 32) bulk_load(base + p.o_fc + r * hb, p.fcw_t + (size_t)r * H, hb, bars + 8 * b_fc);
  }
  // a K that is an odd multiple of 16 leaves half a block per row: zero, not whatever was there
  if (p.in_c % 32 != 0)
#pragma unroll 1
    for (int i = tid; i < kRows * 8; i += kThreads)
      *reinterpret_cast<uint32_t*>(sm + p.o_w[0] + (i >> 3) * row_stride(p.in_c) + p.in_c * 2 + (i & 7) * 4) = 0u;
  if (n_bridge && p.feat % 32 != 0)
#pragma unroll 1
    for (int i = tid; i < n_bridge * 8; i += kThreads)
      *reinterpret_cast<uint32_t*>(sm + p.o_bridge + (i >> 3) * row_stride(p.feat) + p.feat * 2 + (i & 7) * 4) = 0u;
  float* s_bias = reinterpret_cast<float*>(sm + p.o_bias);  // [L][16]
#pragma unroll 1
  for (int i = tid; i < L * kRows; i += kThreads) {
    const int l = i / kRows, r = i % kRows;
    const size_t at = (size_t)(r >> 2) * H + unit0 + (r & 3);
    s_bias[i] = __half2float(p.lstm[p.bw_off[l] + at]) + (p.double_bias ? __half2float(p.lstm[p.br_off[l] + at]) : 0.f);
  }

  // ---- carried state.  Its last writer is the step before, which had finished before the first kernel of this step's
  // encoder started (that one is an ordinary launch), so it need not wait for this kernel's direct predecessor.
  const unsigned int epoch = p.words[kEpoch];
  const int position = (int)p.words[kPosition], n_valid = min(position + 1, p.window);
  float* s_cell = reinterpret_cast<float*>(sm + p.o_cell);    // [L][B][4]
  __half* s_hid = reinterpret_cast<__half*>(sm + p.o_hid);    // [L][B][4], this step's
#pragma unroll 1
  for (int i = tid; i < L * B * kUnits; i += kThreads) {
    const int l = i / (B * kUnits), b = i / kUnits % B, u = i % kUnits;
    s_cell[i] = __half2float(p.c_state[((size_t)l * B + b) * H + unit0 + u]);
  }
  float cs = 1.f, sn = 0.f;
  if (p.rope_base > 0.f) {
    const float ang = (float)position * powf(p.rope_base, -2.0f * (float)lane / (float)kHeadDim);
    cs = cosf(ang);
    sn = sinf(ang);
  }
  const bool item_per_cta = B * p.heads <= (int)gridDim.x;
  for (int item = item_per_cta ? blockIdx.x : blockIdx.x * kWarps + warp; item < B * p.heads; item += item_per_cta ? gridDim.x : gridDim.x * kWarps) {
    const size_t ring = (size_t)(item / p.heads) * p.window * H + (size_t)(item % p.heads) * kHeadDim;
#pragma unroll 1
    for (int i = item_per_cta ? tid : lane; i < n_valid; i += item_per_cta ? kThreads : 32) {
      prefetch_l2(p.kcache + ring + (size_t)i * H);
      prefetch_l2(p.vcache + ring + (size_t)i * H);
    }
  }
  __syncthreads();
  StepCta c{p, sm, bars, &s_abort, &s_flag, p.words + (epoch & 1u), 0u};
  float* s_pre = reinterpret_cast<float*>(sm + p.o_pre);      // [L][16][nt*8]: R.h
  const int pre_n = p.nt * 8;
  // ---- the products, one after another through the same code: the kernel runs once through everything else it has, and its
  // time at few sequences is that of fetching instructions.  With a copy of the product per stage, eight blocks in flight and
  // unrolled loops around it a frame of one player took 112 us, a step of 6 sequences 94.7, of 128 292; now 107, 92.8 and 281.
  enum { kPre, kBridge, kLayer, kQkv, kOut };
  const int bridge_tiles = p.features ? (p.bridge_rows + kRows - 1) / kRows : 0;
  auto after_predecessor = [&]() {
    griddep_wait();
    // Two counters alternate between launches: each launch clears the one that its successor will use, whose last user,
    // the launch before this one, has finished; so a launch starts from zero even after one that gave up on a barrier.
    if (blockIdx.x == 0 && tid == 0) p.words[(epoch + 1u) & 1u] = 0u;
  };
  bool ok = true, waited = false;
#pragma unroll 1
  for (int st = 0; ok; ++st) {
    int kind = kPre, l = st, wait = 0, K = H, stride = H;
    const uint8_t* a = sm + p.o_r[st < L ? st : 0];
    const __half* x = p.h_state + (size_t)st * B * H;           // R.h of every layer needs the step before only
    if (st >= L) {
      if (!waited) after_predecessor();
      waited = true;
      l = st - L;                                               // bridge FC's tile of rows
      kind = kBridge;
      wait = b_bridge;
      a = sm + p.o_bridge + l * kRows * row_stride(p.feat);
      x = p.features;
      K = stride = p.feat;
      if (l >= bridge_tiles) {
        l -= bridge_tiles;                                      // LSTM layer
        kind = kLayer;
        wait = 2 + l;
        a = sm + p.o_w[l < L ? l : 0];
        x = p.h_new + (size_t)(l - 1) * B * H;
        K = stride = H;
        if (l == 0) {
          x = p.features ? p.emb_out : p.emb;
          K = stride = p.in_c;
        } else if (l == L) {
          kind = kQkv;
          wait = b_qkv;
          a = sm + p.o_qkv;
        } else if (l > L) {
          kind = kOut;
          wait = b_wo;
          a = sm + p.o_wo;
          x = p.ctx;
        }
      }
    }
    ok = c.weights(wait);
    if (!ok) break;
    if (kind != kBridge || l * kRows < n_bridge) c.template multiply<TPW>(a, x, stride, K);
    if (kind == kPre) {
#pragma unroll 1
      for (int i = tid; i < kRows * B; i += kThreads) s_pre[((size_t)l * kRows + i / B) * pre_n + i % B] = c.value(i / B, i % B);
      __syncthreads();
    } else if (kind == kBridge) {
      // features -> embedding, rounded before and after the bias
      const int n = min(kRows, n_bridge - l * kRows);
#pragma unroll 1
      for (int i = tid; i < n * B; i += kThreads) {
        const int r = i % n, b = i / n, o = bridge0 + l * kRows + r;
        const float t = __half2float(__float2half(c.value(r, b)));
        p.emb_out[(size_t)b * p.in_c + o] = __float2half(t + __half2float(p.bb[o]));
      }
      if (l + 1 < bridge_tiles) __syncthreads();
      else ok = c.barrier(701);
    } else if (kind == kLayer) {
      // a lane per gate, four lanes per (unit, sequence)
#pragma unroll 1
      for (int i = tid; i < (B * kRows + 31) / 32 * 32; i += kThreads) {
        const int g = i & 3, cell = i >> 2, u = cell & 3, b = cell >> 2, r = g * kUnits + u;
        const bool on = b < B;
        float act = 0.f;
        if (on) {
          const float pre = s_pre[((size_t)l * kRows + r) * pre_n + b] + (c.value(r, b) + s_bias[l * kRows + r]);
          act = sigmoidf_(g == 2 ? 2.0f * pre : pre);
          if (g == 2) act = 2.0f * act - 1.0f;
        }
        const float fg = __shfl_down_sync(0xffffffffu, act, 1), gg = __shfl_down_sync(0xffffffffu, act, 2), og = __shfl_down_sync(0xffffffffu, act, 3);
        if (on && g == 0) {
          float cn = fg * s_cell[l * B * kUnits + cell] + act * gg;
          if (p.clip > 0.f) cn = fminf(p.clip, fmaxf(-p.clip, cn));
          const __half ch = __float2half(cn), hn = __float2half(og * tanhf(__half2float(ch)));
          const size_t si = ((size_t)l * B + b) * H + unit0 + u;
          p.c_state[si] = ch;
          p.h_new[si] = hn;
          s_hid[l * B * kUnits + cell] = hn;
          if (l == L - 1) p.y[(size_t)b * H + unit0 + u] = hn;
        }
      }
      ok = c.barrier(702 + l);
    } else if (kind == kQkv) {
#pragma unroll 1
      for (int i = tid; i < 3 * B * kUnits; i += kThreads) {
        const int m = i / (B * kUnits), b = i / kUnits % B, u = i % kUnits;
        (m == 0 ? p.q : (m == 1 ? p.k : p.v))[(size_t)b * H + unit0 + u] = __float2half(c.value(m * kUnits + u, b));
      }
      // every CTA has read the previous hidden state by now: publish the new one
#pragma unroll 1
      for (int i = tid; i < L * B * kUnits; i += kThreads) {
        const int k = i / (B * kUnits), b = i / kUnits % B, u = i % kUnits;
        p.h_state[((size_t)k * B + b) * H + unit0 + u] = s_hid[i];
      }
      ok = c.barrier(707);
      if (!ok) break;
      // ---- attention: an item per warp, or per CTA where every item can have one of its own
      float* sq = reinterpret_cast<float*>(sm + p.o_attn) + warp * kAttnFloats;
      const int items = B * p.heads, first = item_per_cta ? blockIdx.x : blockIdx.x * kWarps + warp, step = item_per_cta ? items : gridDim.x * kWarps;
#pragma unroll 1
      for (int item = first; item < items; item += step)
        attend(p, item, position, n_valid, cs, sn, sq, sq + 2 * kHeadDim, item_per_cta ? kWarps : 1, item_per_cta ? warp : 0, lane);
      if (item_per_cta && (int)blockIdx.x < items) {
        __syncthreads();
        if (tid < kHeadDim) {
          const float* all = reinterpret_cast<float*>(sm + p.o_attn) + 2 * kHeadDim;
          float mx = -INFINITY, sum = 0.f, acc = 0.f;
#pragma unroll 1
          for (int w = 0; w < kWarps; ++w) mx = fmaxf(mx, all[w * kAttnFloats + kHeadDim]);
#pragma unroll 1
          for (int w = 0; w < kWarps; ++w) {
            const float f = expf(all[w * kAttnFloats + kHeadDim] - mx);  // (0 for a warp without a share)
            sum = fmaf(f, all[w * kAttnFloats + kHeadDim + 1], sum);
            acc = fmaf(f, all[w * kAttnFloats + tid], acc);
          }
          p.ctx[(size_t)(blockIdx.x / p.heads) * H + (size_t)(blockIdx.x % p.heads) * kHeadDim + tid] = __float2half(acc / sum);
        }
      }
      ok = c.barrier(708);
    } else {
#pragma unroll 1
      for (int i = tid; i < B * kUnits; i += kThreads) p.a[(size_t)(i / kUnits) * H + unit0 + i % kUnits] = __float2half(c.value(i % kUnits, i / kUnits));
      ok = c.barrier(709);
      break;
    }
  }
  if (!waited) after_predecessor();                             // (gave up before)
  // ---- per sequence: row LayerNorm (eps 1e-5; every warp for itself), FC with the two-step rounding, sigmoid / tanh
  if (ok && (ok = c.weights(b_fc))) {
    constexpr int kPairs = 512 / 64;  // half2 a lane holds at most
    for (int b = blockIdx.x; b < B; b += gridDim.x) {
      const __half2* src = reinterpret_cast<const __half2*>(p.a + (size_t)b * H);
      float2 v[kPairs];
      float s = 0.f, ss = 0.f;
#pragma unroll
      for (int j = 0; j < kPairs; ++j) {
        v[j] = j * 64 < H ? __half22float2(__ldcg(src + lane + 32 * j)) : make_float2(0.f, 0.f);
        s += v[j].x + v[j].y;
      }
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      const float mu = s / (float)H;
#pragma unroll
      for (int j = 0; j < kPairs; ++j)
        if (j * 64 < H) ss += (v[j].x - mu) * (v[j].x - mu) + (v[j].y - mu) * (v[j].y - mu);
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      const float rstd = rsqrtf(ss / (float)H + 1e-5f);
#pragma unroll
      for (int j = 0; j < kPairs; ++j)
        if (j * 64 < H) {
          const float2 gm = reinterpret_cast<const float2*>(p.ln_g)[lane + 32 * j], bt = reinterpret_cast<const float2*>(p.ln_b)[lane + 32 * j];
          v[j] = __half22float2(__floats2half2_rn((v[j].x - mu) * rstd * gm.x + bt.x, (v[j].y - mu) * rstd * gm.y + bt.y));
        }
      for (int o = warp; o < p.n_out; o += kWarps) {
        const __half2* w = reinterpret_cast<const __half2*>(sm + p.o_fc + (size_t)o * H * 2);
        float acc = 0.f;
#pragma unroll
        for (int j = 0; j < kPairs; ++j)
          if (j * 64 < H) {
            const float2 f = __half22float2(w[lane + 32 * j]);
            acc = fmaf(f.x, v[j].x, acc);
            acc = fmaf(f.y, v[j].y, acc);
          }
        for (int k = 16; k > 0; k >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, k);
        if (lane == 0) {
          const float t = __half2float(__float2half(acc));                           // FCLayer: GEMM result stored as half,
          float r = __half2float(__float2half(t + __half2float(p.fcb[o])));          // then bias added and stored again
          r = o < p.n_sig ? sigmoidf_(r) : tanhf(r);
          const __half hv = __float2half(r);
          p.logits[(size_t)b * p.n_out + o] = hv;
          p.out_f32[(size_t)b * p.n_out + o] = __half2float(hv);
        }
      }
    }
  }
  // no CTA leaves with copies into its shared memory still under way
  if (!ok)
    for (int i = 0; i < n_bars; ++i) c.weights(i);
  if (blockIdx.x == 0 && tid == 0) {
    p.words[kEpoch] = epoch + 1u;
    if (ok) p.words[kPosition] = (unsigned int)position + 1u;
  }
}

__global__ void transpose_kernel(const __half* __restrict__ in_out, __half* __restrict__ out_in, int in_c, int out_c) {
  const long long total = (long long)in_c * out_c;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(i % in_c), o = (int)(i / in_c);
    out_in[i] = in_out[(size_t)k * out_c + o];
  }
}

}  // namespace

struct SeqStepFused {
  aig_ctx* ctx = nullptr;
  SeqStepConfig cfg{};
  StepParams prm{};
  __half* buf = nullptr;        // transposed weights + scratch
  unsigned int* words = nullptr;
  int grid = 1;
  size_t smem = 0;
  bool weights_set = false;
};

namespace {

using StepKernel = void (*)(const StepParams);
StepKernel step_kernel(int batch) { return batch <= 64 ? seq_step_kernel<1> : seq_step_kernel<2>; }

// shared memory of one CTA; sets the offsets
size_t lay_out(StepParams& p) {
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off = (off + bytes + 127) & ~(size_t)127;
    return (int)at;
  };
  const size_t hs = row_stride(p.H);
  size_t tile_end = 0;  // a multiply reads 16 rows, also where fewer are kept
  auto tile = [&](size_t rows, size_t stride) {
    const int at = take(rows * stride);
    const size_t last = (rows + kRows - 1) / kRows * kRows;
    tile_end = tile_end > at + last * stride ? tile_end : at + last * stride;
    return at;
  };
  for (int l = 0; l < p.layers; ++l) p.o_r[l] = tile(kRows, hs);
  p.o_bridge = p.bridge_rows ? tile(p.bridge_rows, row_stride(p.feat)) : 0;
  for (int l = 0; l < p.layers; ++l) p.o_w[l] = tile(kRows, l == 0 ? row_stride(p.in_c) : hs);
  p.o_qkv = tile(3 * kUnits, hs);
  p.o_wo = tile(kUnits, hs);
  p.o_fc = take((size_t)p.n_out * p.H * 2);
  p.o_pre = take((size_t)p.layers * kRows * p.nt * 8 * 4);
  p.o_red = take((size_t)p.kw * p.nt * kRows * 8 * 4);
  p.o_cell = take((size_t)p.layers * p.B * kUnits * 4);
  p.o_hid = take((size_t)p.layers * p.B * kUnits * 2);
  p.o_bias = take((size_t)p.layers * kRows * 4);
  p.o_attn = take((size_t)kWarps * kAttnFloats * 4);
  return off > tile_end ? off : tile_end;
}

StepParams step_shape(const SeqStepConfig& c) {
  StepParams p{};
  p.B = c.batch; p.in_c = c.in_c; p.H = c.hidden; p.layers = c.layers; p.heads = c.heads; p.window = c.window;
  p.n_out = c.n_out; p.n_sig = c.n_sigmoid; p.double_bias = c.double_bias; p.rope_base = c.rope_base;
  p.scale = 1.0f / sqrtf((float)kHeadDim); p.clip = c.clip;
  p.nt = (c.batch + 7) / 8;
  p.kw = p.nt == 1 ? 8 : (p.nt == 2 ? 4 : (p.nt <= 4 ? 2 : 1));  // as many warps along K as the tiles leave free
  p.feat = c.features;
  if (c.features) p.bridge_rows = (c.in_c + c.hidden / kUnits - 1) / (c.hidden / kUnits);
  return p;
}

}  // namespace

bool seq_step_fused_supported(const SeqStepConfig& c) {
  if (!(c.batch >= 1 && c.batch <= kMaxBatch && c.layers >= 1 && c.layers <= kMaxLayers && c.hidden % 64 == 0 && c.hidden <= 512 &&
        c.in_c % 16 == 0 && c.features % 16 == 0 && c.heads * kHeadDim == c.hidden && c.window >= 1 && c.window <= kMaxWindow && c.n_out >= 1 &&
        c.n_out <= 64))
    return false;
  StepParams p = step_shape(c);
  return lay_out(p) <= kMaxSmem;
}

int seq_step_fused_create(aig_ctx* ctx, const SeqStepConfig& c, SeqStepFused** out) {
  *out = nullptr;
  if (!seq_step_fused_supported(c)) return aig_fail(ctx, AIG_ERR_UNSUPPORTED, "fused sequence step: configuration not covered");
  DeviceGuard g(ctx->device);
  SeqStepFused* s = new SeqStepFused();
  s->ctx = ctx;
  s->cfg = c;
  StepParams& p = s->prm;
  p = step_shape(c);
  s->smem = lay_out(p);
  s->grid = c.hidden / kUnits;
  const size_t E = c.hidden, BE = (size_t)c.batch * E;
  // layout of buf (halfs): wq_t wk_t wv_t wo_t fcw_t bw_t | h_new q k v ctx a emb | kcache vcache
  const size_t n_w = 4 * E * E + (size_t)c.n_out * E + (size_t)c.features * c.in_c;
  const size_t n_s = (size_t)c.layers * BE + 5 * BE + (size_t)c.batch * c.in_c;
  const size_t n_c = 2 * (size_t)c.batch * c.window * E;
  int per_sm = 0;
  if (cudaMalloc(&s->buf, (n_w + n_s + n_c) * sizeof(__half)) != cudaSuccess || cudaMalloc(&s->words, kWords * sizeof(unsigned int)) != cudaSuccess ||
      cudaMemsetAsync(s->buf, 0, (n_w + n_s + n_c) * sizeof(__half), ctx->stream) != cudaSuccess ||
      cudaMemsetAsync(s->words, 0, kWords * sizeof(unsigned int), ctx->stream) != cudaSuccess ||
      cudaFuncSetAttribute(step_kernel(c.batch), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, step_kernel(c.batch), kThreads, s->smem) != cudaSuccess) {
    seq_step_fused_destroy(s);
    return aig_fail(ctx, AIG_ERR_CUDA, "fused sequence step: allocation failed");
  }
  if (per_sm * ctx->sm_count < s->grid) {
    seq_step_fused_destroy(s);
    return aig_fail(ctx, AIG_ERR_UNSUPPORTED, "fused sequence step: %d CTAs cannot be co-resident", s->grid);
  }
  __half* w = s->buf;
  p.wq_t = w; p.wk_t = w + E * E; p.wv_t = w + 2 * E * E; p.wo_t = w + 3 * E * E; p.fcw_t = w + 4 * E * E;
  p.bw_t = p.fcw_t + (size_t)c.n_out * E;
  __half* sc = s->buf + n_w;
  p.h_new = sc; sc += (size_t)c.layers * BE;
  p.q = sc; p.k = sc + BE; p.v = sc + 2 * BE; p.ctx = sc + 3 * BE; p.a = sc + 4 * BE; p.emb_out = sc + 5 * BE;
  p.kcache = s->buf + n_w + n_s;
  p.vcache = p.kcache + (size_t)c.batch * c.window * E;
  p.words = s->words;
  p.gerr = ctx->d_err;
  // blob offsets (halfs): per layer W then R, then per layer bW [and bR]
  size_t off = 0;
  for (int l = 0; l < c.layers; ++l) {
    const size_t in_l = l == 0 ? c.in_c : c.hidden;
    p.w_off[l] = off; off += 4 * E * in_l;
    p.r_off[l] = off; off += 4 * E * E;
  }
  for (int l = 0; l < c.layers; ++l) {
    p.bw_off[l] = off; off += 4 * E;
    if (c.double_bias) { p.br_off[l] = off; off += 4 * E; }
  }
  *out = s;
  return AIG_OK;
}

void seq_step_fused_destroy(SeqStepFused* s) {
  if (!s) return;
  cudaFree(s->buf);
  cudaFree(s->words);
  delete s;
}

int seq_step_fused_set_weights(SeqStepFused* s, const aig_half* lstm_blob, const aig_half* wq, const aig_half* wk, const aig_half* wv,
                               const aig_half* wo, const float* ln_g, const float* ln_b, const aig_half* fcw, const aig_half* fcb) {
  aig_ctx* ctx = s->ctx;
  DeviceGuard g(ctx->device);
  AIG_REQUIRE(ctx, lstm_blob && wq && wk && wv && wo && ln_g && ln_b && fcw && fcb, "fused sequence step: null parameter");
  StepParams& p = s->prm;
  const int E = s->cfg.hidden;
  const aig_half* src[4] = {wq, wk, wv, wo};
  __half* dst[4] = {(__half*)p.wq_t, (__half*)p.wk_t, (__half*)p.wv_t, (__half*)p.wo_t};
  for (int i = 0; i < 4; ++i) {
    transpose_kernel<<<ctx->sm_count * 4, 256, 0, ctx->stream>>>((const __half*)src[i], dst[i], E, E);
    AIG_LAUNCH_OK(ctx);
  }
  transpose_kernel<<<ctx->sm_count, 256, 0, ctx->stream>>>((const __half*)fcw, (__half*)p.fcw_t, E, s->cfg.n_out);
  AIG_LAUNCH_OK(ctx);
  p.lstm = (const __half*)lstm_blob;
  p.ln_g = ln_g;
  p.ln_b = ln_b;
  p.fcb = (const __half*)fcb;
  s->weights_set = true;
  return AIG_OK;
}

int seq_step_fused_set_bridge(SeqStepFused* s, const aig_half* w_in_out, const aig_half* bias) {
  aig_ctx* ctx = s->ctx;
  DeviceGuard g(ctx->device);
  AIG_REQUIRE(ctx, s->cfg.features > 0 && w_in_out && bias, "fused sequence step: no bridge in this configuration");
  transpose_kernel<<<ctx->sm_count, 256, 0, ctx->stream>>>((const __half*)w_in_out, (__half*)s->prm.bw_t, s->cfg.features, s->cfg.in_c);
  AIG_LAUNCH_OK(ctx);
  s->prm.bb = (const __half*)bias;
  return AIG_OK;
}

int seq_step_fused_reset(SeqStepFused* s) {
  aig_ctx* ctx = s->ctx;
  AIG_CUDA_OK(ctx, cudaMemsetAsync(s->words, 0, kWords * sizeof(unsigned int), ctx->stream));
  return AIG_OK;
}

int seq_step_fused_run(SeqStepFused* s, const aig_half* emb, const aig_half* features, aig_half* h_state, aig_half* c_state, aig_half* y,
                       aig_half* logits, float* out_f32, bool after_encoder) {
  aig_ctx* ctx = s->ctx;
  DeviceGuard g(ctx->device);
  AIG_REQUIRE(ctx, s->weights_set && (emb || (features && s->prm.bb)) && h_state && c_state && y && logits && out_f32,
              "fused sequence step: bad arguments");
  StepParams p = s->prm;
  p.emb = (const __half*)emb;
  p.features = (const __half*)features;
  p.h_state = (__half*)h_state;
  p.c_state = (__half*)c_state;
  p.y = (__half*)y;
  p.logits = (__half*)logits;
  p.out_f32 = out_f32;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(s->grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = s->smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  attr[1] = pdl_attribute(ctx);
  cfg.attrs = attr;
  cfg.numAttrs = after_encoder ? 2 : 1;
  AIG_CUDA_OK(ctx, cudaLaunchKernelEx(&cfg, step_kernel(s->cfg.batch), p));
  return AIG_OK;
}
