// clip_conv.cu -- 3-D convolution of the clip encoder behind its first layer (ConvLayer3D.cpp:106-111 + BatchNorm.cpp:55-63 +
// LeakyReLU.cpp:9-13: 3x3x3, stride 1x2x2, pad 1) for sm_100a, walking along the depth.
//
// The streamed GEMM fetches an activation tile once for each of 27 taps.  Here the input lies in 2x2 space-to-depth blocks,
// so the nine taps of a plane are row shifts of four (64 channels) or two (32) patches of 128 positions and a halo, and a
// plane's patches are fetched once per output tile:
//  - an input plane contributes to three output planes, whose accumulators lie side by side in TMEM: ONE instruction
//    multiplies a patch with the weights of its three depth taps, N = 3 x 64 (or 3 x 32) columns, instead of three of N = 64
//    that would each read the patch again;
//  - the weights of all 27 taps stay in shared memory: 64 output channels of 32 input channels in one CTA, or 32 of 64, the
//    output channels being split over the CTAs;
//  - a CTA takes a run of (tile of positions, depth) outputs; at either end of a run in the middle of a tile one plane is read
//    by two CTAs.  Planes before the first and behind the last are not multiplied.
// Positions are those of all clips' blocks at one depth, one after another; the last row and column of blocks of an image give
// no output (4 to 8 % of the rows at 36x64 and 18x32 outputs).
// Bound by shared-memory bandwidth: a plane of a tile takes about 2200 clk for 18 products of 10 KB of operands, 41 KB of
// patches written and 32 KB of staging (64 channels: 2750 for 36 of 7 KB, 77 KB and 16 KB), near 128 bytes a clk.  16 clips of
// 8x144x256, the two layers: 61 and 38 us by the streamed GEMM, now 31 and 35; smaller clips gain more (9 of 5x98x305, the whole
// encoder: 143 -> 72 us).  Five patch buffers instead of four for 64 channels: 3340 -> 2660 clk a plane (a patch takes over
// 2000 clk to come).
#include "clip_conv.h"

#include <type_traits>
#include <utility>

#include "aig_common.cuh"

namespace {

constexpr int kFirstEpi = 4;       // warps: patch producer, MMA issuer, TMEM owner, one idle, then the epilogue's
constexpr int kStage = 2048;       // staging of one epilogue warp: 32 rows x 32 channels
constexpr int kMaxUnits = 4, kMaxPatches = 8, kMaxSlots = 16;

struct Entry {                     // a run of K against one row shift of a patch
  int unit, shift, block, k0, nk;  // shift: 0, 1, Wb, Wb + 1; k0: first 16 of the weight block's 64
  bool first, last;                // of the unit
};
template <int C>
struct Cfg;
template <>
struct Cfg<32> {                   // unit u: the two sub-positions of sub-row u
  static constexpr int kNC = 64, kUnits = 2, kBlocks = 5, kEntries = 6;
  // weight blocks: filter rows 0, 2, 1 with columns 0 and 1; column 2 of rows 0 and 2; column 2 of row 1
  __host__ __device__ static constexpr Entry entry(int e) {
    constexpr Entry t[kEntries] = {{0, 0, 0, 0, 4, true, false}, {0, 1, 3, 0, 2, false, false}, {0, 2, 1, 0, 4, false, false},
                                   {0, 3, 3, 2, 2, false, true}, {1, 0, 2, 0, 4, true, false},  {1, 1, 4, 0, 2, false, true}};
    return t[e];
  }
  static constexpr int kHalo[kUnits] = {3, 1};        // largest shift of the unit
  static constexpr bool kEqualPatches = false;        // patch buffers: two planes', of the units' own sizes
};
template <>
struct Cfg<64> {                   // unit u: sub-position u
  static constexpr int kNC = 32, kUnits = 4, kBlocks = 9, kEntries = 9;
  // weight blocks: (filter row, column) = (0,0) (0,2) (2,0) (2,2) | (0,1) (2,1) | (1,0) (1,2) | (1,1)
  __host__ __device__ static constexpr Entry entry(int e) {
    constexpr Entry t[kEntries] = {{0, 0, 0, 0, 4, true, false}, {0, 1, 1, 0, 4, false, false}, {0, 2, 2, 0, 4, false, false},
                                   {0, 3, 3, 0, 4, false, true}, {1, 0, 4, 0, 4, true, false},  {1, 2, 5, 0, 4, false, true},
                                   {2, 0, 6, 0, 4, true, false}, {2, 1, 7, 0, 4, false, true},  {3, 0, 8, 0, 4, true, true}};
    return t[e];
  }
  static constexpr int kHalo[kUnits] = {3, 2, 1, 0};
  static constexpr bool kEqualPatches = true;         // any unit in any buffer: five fit, four would be one plane's
};

struct ClipParams {
  int batch, D, Ho, Wo, Hb, Wb;
  int P;                           // positions of one depth: batch * Hb * Wb
  int outs, parts, ctas;           // tiles * D, channel shares, CTAs per share
  int patches, patch_bytes[2];     // buffers; sizes of the even and the odd ones
  int unit_rows[kMaxUnits];
  int blocks_out, Hb2, Wb2;
  uint32_t row16, d_stride16;      // a pixel's channels and a depth's step in the output, in 16-byte pieces
  float slope;
  const __half* wimg;              // [part][block][3 * NC rows][64], rows swizzled as they lie in shared memory
  const float *scale, *shift;      // [K]
  uint4* y;
  int* gerr;
};
struct ClipMaps {
  CUtensorMap u[kMaxUnits];
};

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// has the phase ended? (does not wait)
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// The same in every lane, and known to be: the issuing loop keeps its arithmetic in uniform registers, where tcgen05.mma takes
// its operands from.
__device__ __forceinline__ uint32_t uniform(uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); }
__device__ __forceinline__ bool uniform(bool v) { return __shfl_sync(0xffffffffu, v ? 1 : 0, 0) != 0; }

// The outputs of a CTA, [g, end), in runs of one tile each: depths [da, db) of tile t.  A run's accumulators take consecutive
// slots of the ring from `slot` on; one that fits goes back to slot 0 rather than turn over in the middle, which would make
// two instructions of each of a plane's products.
template <int SLOTS>
struct Runs {
  int g, end, D;
  int t, da, db, slot, next_slot;
  __device__ __forceinline__ bool next() {
    if (g >= end) return false;
    t = g / D;
    da = g - t * D;
    db = min(D, da + end - g);
    const int n = db - da;
    g += n;
    slot = next_slot + n > SLOTS && n <= SLOTS ? 0 : next_slot;
    next_slot = (slot + n) % SLOTS;
    return true;
  }
  __device__ __forceinline__ int f0() const { return max(da - 1, 0); }
  __device__ __forceinline__ int f1() const { return min(db, D - 1); }
  __device__ __forceinline__ int slot_of(int d) const { return (slot + d - da) % SLOTS; }
};

template <class F, int... E>
__device__ __forceinline__ void for_each_entry(F&& f, std::integer_sequence<int, E...>) {
  (f(std::integral_constant<int, E>()), ...);
}

// The ring of patch buffers.
struct PatchRing {
  int i;
  uint32_t phase;
  __device__ __forceinline__ void advance(int count) {
    if (++i == count) {
      i = 0;
      phase ^= 1u;
    }
  }
};
template <int C>
__device__ __forceinline__ uint32_t patch_offset(const ClipParams& p, int i) {
  return Cfg<C>::kEqualPatches ? (uint32_t)(i * p.patch_bytes[0]) : (uint32_t)((i >> 1) * (p.patch_bytes[0] + p.patch_bytes[1]) + (i & 1) * p.patch_bytes[0]);
}
template <int C>
__host__ __device__ constexpr int clip_threads() { return 32 * (kFirstEpi + Cfg<C>::kNC / 8); }  // four epilogue warps per 32 channels

template <int C>
__global__ void __launch_bounds__(clip_threads<C>(), 1) clip_conv_kernel(const __grid_constant__ ClipMaps maps, const __grid_constant__ ClipParams p) {
  using G = Cfg<C>;
  constexpr int NC = G::kNC, U = G::kUnits;
  constexpr int kBlockBytes = 3 * NC * 128, kWBytes = G::kBlocks * kBlockBytes;
  constexpr int kCols = 512, kSlots = kCols / NC, kThreads = clip_threads<C>();
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - raw);
  const uint32_t sW = base, sPatch = base + kWBytes;
  uint8_t* s_stage = sm + kWBytes + patch_offset<C>(p, p.patches);
  float* s_scale = reinterpret_cast<float*>(s_stage + NC / 8 * kStage);
  float* s_shift = s_scale + NC;
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_shift + NC);
  const uint32_t bar_w = smem_u32(bars), bar_tfull = bar_w + 8, bar_tempty = bar_tfull + 8 * kMaxSlots;
  const uint32_t bar_ufull = bar_tempty + 8 * kMaxSlots, bar_uempty = bar_ufull + 8 * kMaxPatches;
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(bars + 1 + 2 * kMaxSlots + 2 * kMaxPatches);
  volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

  const int part = (int)(blockIdx.x % (unsigned)p.parts), cta = (int)(blockIdx.x / (unsigned)p.parts);
  const Runs<kSlots> all{(int)((long long)p.outs * cta / p.ctas), (int)((long long)p.outs * (cta + 1) / p.ctas), p.D, 0, 0, 0, 0, 0};
  griddep_launch_dependents();
  for (int i = threadIdx.x; i < NC; i += kThreads) {
    s_scale[i] = p.scale[part * NC + i];
    s_shift[i] = p.shift[part * NC + i];
  }
  if (threadIdx.x == 0) {
    mbar_init(bar_w, 1);
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(bar_tfull + 8 * i, 1);
      mbar_init(bar_tempty + 8 * i, 4 * (NC / 32));
    }
    for (int i = 0; i < kMaxPatches; ++i) {
      mbar_init(bar_ufull + 8 * i, 1);
      mbar_init(bar_uempty + 8 * i, 1);
    }
    *s_abort = 0;
    fence_mbar_init();
  }
  if (warp == 2) {
    tmem_alloc(smem_u32(s_tmem), kCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *s_tmem;

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    const bool leader = elect_one();
    if (leader) {
      mbar_expect_tx(bar_w, kWBytes);
      const uint8_t* w = reinterpret_cast<const uint8_t*>(p.wimg) + (size_t)part * kWBytes;
      for (int b = 0; b < G::kBlocks; ++b) bulk_load(sW + b * kBlockBytes, w + (size_t)b * kBlockBytes, kBlockBytes, bar_w);
      for (int u = 0; u < U; ++u) tma_prefetch_desc(&maps.u[u]);
    }
    griddep_wait();
    Runs<kSlots> r = all;
    PatchRing ring{0, 0};
    bool ok = true;
    while (ok && r.next()) {
      for (int f = r.f0(); f <= r.f1() && ok; ++f) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (!mbar_wait_bounded_sleepy(bar_uempty + 8 * ring.i, ring.phase ^ 1u, s_abort, p.gerr, 901)) { ok = false; break; }
          if (leader) {
            mbar_expect_tx(bar_ufull + 8 * ring.i, (uint32_t)p.unit_rows[u] * 128u);
            tma_load_2d(sPatch + patch_offset<C>(p, ring.i), &maps.u[u], bar_ufull + 8 * ring.i, 64 * u, f * p.P + r.t * 128);
          }
          ring.advance(p.patches);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (see elect_one)
    // A barrier is looked at one step before it is needed, between products that are already on their way: the tensor pipe
    // runs little ahead of this warp, and a wait, even for something long done, costs about 180 clk, three to four products.
    constexpr uint32_t hi = umma_desc_hi(128);
    const bool leader = elect_one();
    const uint32_t tmem = uniform(tmem_base);
    Runs<kSlots> r = all;
    PatchRing ring{0, 0};
    uint32_t empty = ~0u;          // a bit per slot: the parity that says that its columns may be overwritten
    bool ok = uniform(mbar_wait_bounded(bar_w, 0, s_abort, p.gerr, 911)), unit_ready = false, slot_ready = false;
    while (ok && r.next()) {
      for (int f = r.f0(); f <= r.f1() && ok; ++f) {
        const int lo = max(f - 1, r.da), top = min(f + 1, r.db - 1), n = top - lo + 1;
        const int fresh = f == r.f0() ? lo : f + 1;       // outputs from here on get their first plane
        for (int o = fresh; o <= top; ++o) {
          const int so = r.slot_of(o);
          if (!slot_ready && !uniform(mbar_wait_bounded(bar_tempty + 8 * so, empty >> so & 1u, s_abort, p.gerr, 912))) { ok = false; break; }
          empty ^= 1u << so;
          slot_ready = false;
        }
        if (!ok) break;
        tc_fence_after();
        // the outputs' columns in TMEM, in two pieces where the ring turns over
        const int slot = r.slot_of(lo), n1 = min(n, kSlots - slot), n2 = n - n1;
        const uint32_t d1 = tmem + (uint32_t)(slot * NC), w1 = sW + (uint32_t)((lo - f + 1) * NC * 128), w2 = w1 + (uint32_t)(n1 * NC * 128);
        const uint32_t id1 = umma_idesc_f16(128, NC) + ((uint32_t)((n1 - 1) * NC / 8) << 17), id2 = umma_idesc_f16(128, NC) + ((uint32_t)((n2 - 1) * NC / 8) << 17);
        auto products = [&](auto number) {
          constexpr int e = decltype(number)::value;
          constexpr Entry T = G::entry(e);
          if (!ok) return;
          if (T.first && !unit_ready && !uniform(mbar_wait_bounded(bar_ufull + 8 * ring.i, ring.phase, s_abort, p.gerr, 913))) { ok = false; return; }
          const int rows = (T.shift & 1) + (T.shift & 2 ? p.Wb : 0);
          const uint32_t a = umma_desc_lo(sPatch + patch_offset<C>(p, ring.i) + (uint32_t)(rows * 128));
          const uint32_t b1 = umma_desc_lo(w1 + T.block * kBlockBytes + T.k0 * 32), b2 = umma_desc_lo(w2 + T.block * kBlockBytes + T.k0 * 32);
#pragma unroll
          for (int k = 0; k < T.nk; ++k) {
            if (e == 0 && k == 0) {                       // an output's first product overwrites what lies in its columns
#pragma unroll
              for (int i = 0; i < 3; ++i)
                if (i < n && leader)
                  umma_f16_ss_lo(tmem + (uint32_t)(r.slot_of(lo + i) * NC), a, b1 + (uint32_t)(i * NC * 8), hi, umma_idesc_f16(128, NC), lo + i >= fresh ? 0u : 1u);
            } else if (leader) {
              umma_f16_ss_lo(d1, a + 2 * k, b1 + 2 * k, hi, id1, 1u);
            }
            if (T.last && k == 0) {
              PatchRing next = ring;
              next.advance(p.patches);
              unit_ready = uniform(mbar_test(bar_ufull + 8 * next.i, next.phase));
            }
            if (e + 1 == G::kEntries && k == 0 && f < r.f1() && f + 2 < r.db) {
              const int sn = r.slot_of(f + 2);            // of the output that the next plane begins
              slot_ready = uniform(mbar_test(bar_tempty + 8 * sn, empty >> sn & 1u));
            }
          }
          if (n2 > 0) {
#pragma unroll
            for (int k = e == 0 ? 1 : 0; k < T.nk; ++k)
              if (leader) umma_f16_ss_lo(tmem, a + 2 * k, b2 + 2 * k, hi, id2, 1u);
          }
          if (T.last) {
            if (leader) umma_commit(bar_uempty + 8 * ring.i);
            ring.advance(p.patches);
          }
        };
        for_each_entry(products, std::make_integer_sequence<int, G::kEntries>());
        if (!ok) break;
        for (int o = lo; o <= top; ++o)
          if (f == min(o + 1, p.D - 1) && leader) umma_commit(bar_tfull + 8 * r.slot_of(o));
      }
    }
  } else if (warp >= kFirstEpi) {
    // ------------------------------------------------------------------ epilogue: 32 channels of an output by four warps
    const int q = warp & 3, chunk = (warp - kFirstEpi) >> 2;
    uint8_t* stg = s_stage + (warp - kFirstEpi) * kStage;
    const uint32_t own = (uint32_t)(lane * 64), own_x = (uint32_t)((lane >> 1) & 3);
    const int gr = lane >> 2, gc = lane & 3;
    Runs<kSlots> r = all;
    uint32_t full = 0;                                    // a bit per slot, as `empty`
    bool ok = true;
    griddep_wait();                                       // the output may still be read by an earlier launch
    while (ok && r.next()) {
      const int pos = r.t * 128 + q * 32 + lane;
      const int img = p.Hb * p.Wb, n = pos / img, rem = pos - n * img, y = rem / p.Wb, x = rem - y * p.Wb;
      const bool valid = pos < p.P && y < p.Ho && x < p.Wo;
      uint32_t off = p.blocks_out ? (((uint32_t)(n * p.Hb2 + ((y + 1) >> 1)) * p.Wb2 + ((x + 1) >> 1)) * 4 + ((y + 1) & 1) * 2 + ((x + 1) & 1)) * p.row16
                                  : ((uint32_t)(n * p.D * p.Ho + y) * p.Wo + x) * p.row16;
      off += (uint32_t)(part * (NC / 8) + chunk * 4);
      uint32_t offs[4];
      bool vs[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        offs[i] = __shfl_sync(0xffffffffu, off, 8 * i + gr) + gc;
        vs[i] = __shfl_sync(0xffffffffu, valid ? 1 : 0, 8 * i + gr) != 0;
      }
      for (int d = r.da; d < r.db; ++d) {
        const int slot = r.slot_of(d);
        if (!mbar_wait_bounded_sleepy(bar_tfull + 8 * slot, full >> slot & 1u, s_abort, p.gerr, 921)) { ok = false; break; }
        full ^= 1u << slot;
        tc_fence_after();
        uint32_t v[32];
        tmem_ld_32x32(tmem_base + (uint32_t)(slot * NC + chunk * 32) + ((uint32_t)(q * 32) << 16), v);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_tempty + 8 * slot);
        const float4 *sc = reinterpret_cast<const float4*>(s_scale + chunk * 32), *sh = reinterpret_cast<const float4*>(s_shift + chunk * 32);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t o[4];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float4 s4 = sc[2 * c + h], h4 = sh[2 * c + h];
            const float a0 = fmaf(__uint_as_float(v[8 * c + 4 * h]), s4.x, h4.x), a1 = fmaf(__uint_as_float(v[8 * c + 4 * h + 1]), s4.y, h4.y);
            const float a2 = fmaf(__uint_as_float(v[8 * c + 4 * h + 2]), s4.z, h4.z), a3 = fmaf(__uint_as_float(v[8 * c + 4 * h + 3]), s4.w, h4.w);
            const __half2 p0 = __floats2half2_rn(a0 < 0.f ? a0 * p.slope : a0, a1 < 0.f ? a1 * p.slope : a1);
            const __half2 p1 = __floats2half2_rn(a2 < 0.f ? a2 * p.slope : a2, a3 < 0.f ? a3 * p.slope : a3);
            o[2 * h] = *reinterpret_cast<const uint32_t*>(&p0);
            o[2 * h + 1] = *reinterpret_cast<const uint32_t*>(&p1);
          }
          *reinterpret_cast<uint4*>(stg + own + (((uint32_t)c ^ own_x) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
        }
        __syncwarp();
        uint4* yd = p.y + (size_t)d * p.d_stride16;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int row = 8 * i + gr;
          const uint4 o = *reinterpret_cast<const uint4*>(stg + row * 64 + ((gc ^ ((row >> 1) & 3)) << 4));
          if (vs[i]) yd[offs[i]] = o;
        }
        __syncwarp();
      }
    }
  }

  if (*s_abort) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);     // copies in flight land
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kCols);
  }
}

// w [K][C][3][3][3] -> the weight blocks as they lie in shared memory: row s * NC + n of a block is output channel n of the
// share with depth tap 2 - s; scale / shift: bias and BatchNorm folded
template <int C>
__global__ void clip_pack_kernel(const __half* __restrict__ w, const __half* __restrict__ bias, const float* gamma, const float* beta, const float* mean,
                                 const float* var, float eps, __half* __restrict__ img, float* scale, float* shift, int K) {
  constexpr int NC = Cfg<C>::kNC, blocks = Cfg<C>::kBlocks;
  const int total = K / NC * blocks * 3 * NC * 64;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int k = i & 63, r = (i >> 6) % (3 * NC), b = (i >> 6) / (3 * NC) % blocks, part = (i >> 6) / (3 * NC * blocks);
    const int out = part * NC + r % NC, kd = 2 - r / NC;
    int fr, fs, c;
    bool used = true;
    if (C == 32) {
      c = k & 31;
      if (b < 3) { fr = b == 0 ? 0 : b == 1 ? 2 : 1; fs = k >> 5; }
      else { fr = b == 4 ? 1 : k < 32 ? 0 : 2; fs = 2; used = b == 3 || k < 32; }
    } else {
      c = k;
      fr = b < 4 ? b & 2 : b < 6 ? 2 * (b - 4) : 1;
      fs = b < 4 ? 2 * (b & 1) : b < 6 ? 1 : b < 8 ? 2 * (b - 6) : 1;
    }
    const __half v = used ? w[((size_t)(out * C + c) * 3 + kd) * 9 + fr * 3 + fs] : __ushort_as_half((unsigned short)0);
    img[(size_t)(i >> 6) * 64 + (((k >> 3) ^ (r & 7)) << 3) + (k & 7)] = v;
  }
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < K; k += gridDim.x * blockDim.x) {
    const float b = bias ? __half2float(bias[k]) : 0.f, s = gamma ? gamma[k] / sqrtf(var[k] + eps) : 1.f;
    scale[k] = s;
    shift[k] = gamma ? (b - mean[k]) * s + beta[k] : b;
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

template <int C>
int clip_layout(ClipParams& p) {   // fills in the patches' rows and buffers; the shared memory that a CTA needs
  using G = Cfg<C>;
  int bytes[kMaxUnits];
  for (int u = 0; u < G::kUnits; ++u) {
    p.unit_rows[u] = 128 + (G::kHalo[u] & 1) + (G::kHalo[u] & 2 ? p.Wb : 0);
    bytes[u] = (p.unit_rows[u] * 128 + 1023) & ~1023;
  }
  const int fixed = 1024 + G::kBlocks * 3 * G::kNC * 128 + G::kNC / 8 * kStage + 2 * G::kNC * 4 + 8 * (1 + 2 * kMaxSlots + 2 * kMaxPatches) + 16;
  const int room = 227 * 1024 - fixed;
  p.patch_bytes[0] = bytes[0];     // (the largest)
  p.patch_bytes[1] = G::kEqualPatches ? bytes[0] : bytes[1];
  const int pair = p.patch_bytes[0] + p.patch_bytes[1];
  p.patches = G::kEqualPatches ? room / bytes[0] : room / pair * 2;
  if (p.patches > kMaxPatches) p.patches = kMaxPatches;
  if (p.patches < 2) return 228 * 1024;
  return fixed + (p.patches / 2) * pair + (p.patches & 1) * bytes[0];
}
ClipParams clip_params(const ClipConvGeom& g) {
  ClipParams p{};
  p.batch = g.batch; p.D = g.D;
  p.Ho = (g.H - 1) / 2 + 1; p.Wo = (g.W - 1) / 2 + 1;
  p.Hb = clip_block_extent(g.H); p.Wb = clip_block_extent(g.W);
  p.P = g.batch * p.Hb * p.Wb;
  p.outs = ceil_div(p.P, 128) * g.D;
  p.parts = g.K / (g.C == 32 ? 64 : 32);
  p.blocks_out = g.out_blocks;
  p.Hb2 = clip_block_extent(p.Ho); p.Wb2 = clip_block_extent(p.Wo);
  p.row16 = (uint32_t)g.K / 8;
  p.d_stride16 = g.out_blocks ? (uint32_t)(g.batch * p.Hb2 * p.Wb2 * 4) * p.row16 : (uint32_t)(p.Ho * p.Wo) * p.row16;
  p.slope = g.slope;
  return p;
}

}  // namespace

struct ClipConv {
  aig_ctx* ctx = nullptr;
  ClipConvGeom g{};
  ClipParams prm{};
  ClipMaps maps{};
  const void* map_x = nullptr;
  __half* wimg = nullptr;
  float* affine = nullptr;
  int smem = 0;
  bool weights_set = false;
};

bool clip_conv_supported(const aig_ctx* ctx, const ClipConvGeom& g) {
  if (!(g.C == 32 && g.K % 64 == 0) && !(g.C == 64 && g.K % 32 == 0)) return false;
  if (g.batch <= 0 || g.D <= 0 || g.H <= 0 || g.W <= 0 || g.K <= 0 || g.K > 512) return false;
  const long long rows = (long long)g.batch * g.D * clip_block_extent(g.H) * clip_block_extent(g.W);
  if (rows > (1ll << 28) / (g.C > g.K ? g.C : g.K) * 8 || clip_block_extent(g.W) > 256 - 129) return false;  // 32-bit rows and pieces; rows of a TMA box
  ClipParams p = clip_params(g);
  return p.parts <= ctx->sm_count && (g.C == 32 ? clip_layout<32>(p) : clip_layout<64>(p)) <= 227 * 1024;
}

int clip_conv_create(aig_ctx* ctx, const ClipConvGeom& g, ClipConv** out) {
  *out = nullptr;
  if (!clip_conv_supported(ctx, g)) return aig_fail(ctx, AIG_ERR_UNSUPPORTED, "clip convolution: unsupported geometry");
  ClipConv* c = new ClipConv();
  c->ctx = ctx;
  c->g = g;
  c->prm = clip_params(g);
  ClipParams& p = c->prm;
  c->smem = g.C == 32 ? clip_layout<32>(p) : clip_layout<64>(p);
  p.ctas = ctx->sm_count / p.parts;
  if (p.ctas > p.outs) p.ctas = p.outs;
  const size_t img = (size_t)p.parts * (g.C == 32 ? Cfg<32>::kBlocks * 3 * Cfg<32>::kNC : Cfg<64>::kBlocks * 3 * Cfg<64>::kNC) * 128;
  if (cudaMalloc(&c->wimg, img) != cudaSuccess || cudaMalloc(&c->affine, 2 * (size_t)g.K * sizeof(float)) != cudaSuccess) {
    clip_conv_destroy(c);
    return aig_fail(ctx, AIG_ERR_CUDA, "clip convolution: allocation failed");
  }
  p.wimg = c->wimg;
  p.scale = c->affine;
  p.shift = c->affine + g.K;
  p.gerr = ctx->d_err;
  const cudaError_t e = g.C == 32 ? cudaFuncSetAttribute(clip_conv_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024)
                                  : cudaFuncSetAttribute(clip_conv_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (e != cudaSuccess) {
    clip_conv_destroy(c);
    return aig_fail(ctx, AIG_ERR_CUDA, "clip convolution: %s", cudaGetErrorString(e));
  }
  *out = c;
  return AIG_OK;
}

void clip_conv_destroy(ClipConv* c) {
  if (!c) return;
  cudaFree(c->wimg);
  cudaFree(c->affine);
  delete c;
}

int clip_conv_set_weights(ClipConv* c, const aig_half* w, const aig_half* bias, const float* gamma, const float* beta, const float* mean, const float* var,
                          float eps) {
  const __half *wh = (const __half*)w, *bh = (const __half*)bias;
  if (c->g.C == 32) clip_pack_kernel<32><<<128, 256, 0, c->ctx->stream>>>(wh, bh, gamma, beta, mean, var, eps, c->wimg, c->affine, c->affine + c->g.K, c->g.K);
  else clip_pack_kernel<64><<<128, 256, 0, c->ctx->stream>>>(wh, bh, gamma, beta, mean, var, eps, c->wimg, c->affine, c->affine + c->g.K, c->g.K);
  AIG_LAUNCH_OK(c->ctx);
  c->weights_set = true;
  return AIG_OK;
}

int clip_conv_forward(ClipConv* c, const aig_half* x, aig_half* y) {
  aig_ctx* ctx = c->ctx;
  AIG_REQUIRE(ctx, x && y && c->weights_set, "clip convolution: null pointer or weights not set");
  AIG_REQUIRE(ctx, (((uintptr_t)x | (uintptr_t)y) & 15) == 0, "clip convolution: misaligned tensors");
  ClipParams& p = c->prm;
  if (c->map_x != x) {
    static EncodeTiledFn enc = nullptr;
    if (!enc) {
      void* fn = nullptr;
      cudaDriverEntryPointQueryResult qres;
      if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess || qres != cudaDriverEntryPointSuccess)
        return aig_fail(ctx, AIG_ERR_CUDA, "cuTensorMapEncodeTiled entry point not available");
      enc = reinterpret_cast<EncodeTiledFn>(fn);
    }
    for (int u = 0; u < (c->g.C == 32 ? Cfg<32>::kUnits : Cfg<64>::kUnits); ++u) {
      cuuint64_t dims[2] = {(cuuint64_t)4 * c->g.C, (cuuint64_t)p.D * p.P};
      cuuint64_t strides[1] = {(cuuint64_t)4 * c->g.C * 2};
      cuuint32_t box[2] = {64u, (cuuint32_t)p.unit_rows[u]};
      cuuint32_t es[2] = {1, 1};
      const CUresult r = enc(&c->maps.u[u], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<aig_half*>(x), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
      if (r != CUDA_SUCCESS) return aig_fail(ctx, AIG_ERR_CUDA, "cuTensorMapEncodeTiled(clip blocks) failed: %d", (int)r);
    }
    c->map_x = x;
  }
  p.y = reinterpret_cast<uint4*>(y);
  const dim3 grid((unsigned)(p.parts * p.ctas));
  AIG_CUDA_OK(ctx, c->g.C == 32 ? launch_pdl(ctx, clip_conv_kernel<32>, grid, dim3(clip_threads<32>()), (size_t)c->smem, c->maps, p)
                                : launch_pdl(ctx, clip_conv_kernel<64>, grid, dim3(clip_threads<64>()), (size_t)c->smem, c->maps, p));
  return AIG_OK;
}
