// walk_conv.cu -- convolutions that walk along one axis of their input, for sm_100a:
//  - the clip encoder behind its first layer (ConvLayer3D.cpp:106-111 + BatchNorm.cpp:55-63 + LeakyReLU.cpp:9-13: 3x3x3, stride
//    1x2x2, pad 1), along the depth;
//  - the frame encoder's first residual blocks (ResConvLayer.cpp:13-21: main k4 s2 p1 and shortcut k2 s2 p0 in one launch, then
//    k3 s1 p1 with the residual), along the image rows, for batches beyond the one-launch chain's.
//
// The axis walked along is the outermost of the layout, so a step of it (a plane of all clips, a row of all frames) is one run
// of positions, cut into tiles of 128:
//  - the taps within a step are row shifts of a tile's patches (128 positions and a halo; strided layers lie in 2x2
//    space-to-depth blocks), and a patch is fetched once;
//  - a step contributes to three output steps (two for k4 s2), whose accumulators lie side by side in TMEM: ONE instruction
//    multiplies a patch with the weights of all taps along the axis, N = 3 x 64 columns instead of three times 64, each of which
//    would read the patch again;
//  - the weights of all taps stay in shared memory, the output channels being split over the CTAs where they do not fit;
//  - a CTA takes a run of (tile, step) outputs; at either end of a run in the middle of a tile one step is read by two CTAs.
//    Steps before the first and behind the last are not multiplied.
// Positions between images (the last column of blocks or the zero column; of planes also the last row) give no output.
//
// Clips: bound by shared-memory bandwidth.  A plane of a tile takes 1950 clk for 18 products of 10 KB of operands and 41 KB of
// patches written (64 channels: 2470 for 36 of 7 KB and 77 KB).  16 clips of 8x144x256, the two layers: 61 and 38 us by the
// streamed GEMM, now 28 and 31; smaller clips gain more (9 of 5x98x305, the whole encoder: 143 -> 72 us).  Five patch buffers
// instead of four for 64 channels, measured with outputs that left through a staging tile: 3340 -> 2660 clk a plane (a patch takes
// over 2000 clk to come); without the staging 2470.
// Frames: the 64-channel block has no unit at its peak.  256 frames of 144x256: 261 and 194 MB of DRAM traffic in 51 and 44 us,
// 0.78 and 0.67 of the copy bandwidth; 128 frames: tensor pipe active 49 and 54 %.  The 128-channel one is bound by the products
// (3690 and 2410 clk a row of a tile).  By the patch-resident kernels, 256 frames: 89, 75, 65 and 57 us; now 51, 44, 45 and 37
// (start to start of the launches); the 256-channel 3x3 convolutions 52 and 27, now 46 and 18.  That kernel multiplies 64 columns
// at a time, reads a patch's halo rows again for every tile and, with 128 channels, streams the weights.
#include "walk_conv.h"

#include <type_traits>
#include <utility>

#include "aig_common.cuh"

namespace {

constexpr int kFirstEpi = 4;       // warps: patch producer, MMA issuer, TMEM owner, one idle, then the epilogue's
constexpr int kMaxUnits = 4, kMaxPatches = 8, kMaxSlots = 16;

enum Kind { MAIN, SHORT_HERE, SHORT_BEFORE };  // all taps along the axis; shortcut of output f; of output f - 1
struct Entry {                     // a run of K against one row shift of a patch
  int unit, shift, block;          // shift: bits 1, Wb, 2; weight block (of the shortcut's for that)
  int a0, b0, nk;                  // in pieces of 16: first of the patch's and of the block's 64, number
  Kind kind;
  bool first, last;                // of the unit
};
// kTaps: taps along the axis.  A unit is 64 channels of a position: a patch of 128 + kHalo rows that begins kStart positions
// before the tile.  Weight blocks: kTaps * kNC rows of 64, then the shortcut's of kNC rows.
struct Clip32 {                    // unit u: the two sub-positions of sub-row u
  static constexpr int kTaps = 3, kNC = 64, kUnits = 2, kBlocks = 5, kShort = 0, kEntries = 6, kStart = 0, kEpiWarps = 8;
  // weight blocks: filter rows 0, 2, 1 with columns 0 and 1; column 2 of rows 0 and 2; column 2 of row 1
  __host__ __device__ static constexpr Entry entry(int e) {
    constexpr Entry t[kEntries] = {{0, 0, 0, 0, 0, 4, MAIN, true, false}, {0, 1, 3, 0, 0, 2, MAIN, false, false}, {0, 2, 1, 0, 0, 4, MAIN, false, false},
                                   {0, 3, 3, 0, 2, 2, MAIN, false, true}, {1, 0, 2, 0, 0, 4, MAIN, true, false},  {1, 1, 4, 0, 0, 2, MAIN, false, true}};
    return t[e];
  }
  static constexpr int kHalo[kUnits] = {3, 1};        // largest shift of the unit, bits as above
  static constexpr bool kEqualPatches = false;        // patch buffers in pairs of the two units' sizes
  static constexpr bool kImages = false;              // (see Conv256)
};
struct Clip64 {                    // unit u: sub-position u
  static constexpr int kTaps = 3, kNC = 32, kUnits = 4, kBlocks = 9, kShort = 0, kEntries = 9, kStart = 0, kEpiWarps = 4;
  // weight blocks: (filter row, column) = (0,0) (0,2) (2,0) (2,2) | (0,1) (2,1) | (1,0) (1,2) | (1,1)
  __host__ __device__ static constexpr Entry entry(int e) {
    constexpr Entry t[kEntries] = {{0, 0, 0, 0, 0, 4, MAIN, true, false}, {0, 1, 1, 0, 0, 4, MAIN, false, false}, {0, 2, 2, 0, 0, 4, MAIN, false, false},
                                   {0, 3, 3, 0, 0, 4, MAIN, false, true}, {1, 0, 4, 0, 0, 4, MAIN, true, false},  {1, 2, 5, 0, 0, 4, MAIN, false, true},
                                   {2, 0, 6, 0, 0, 4, MAIN, true, false}, {2, 1, 7, 0, 0, 4, MAIN, false, true},  {3, 0, 8, 0, 0, 4, MAIN, true, true}};
    return t[e];
  }
  static constexpr int kHalo[kUnits] = {3, 2, 1, 0};
  static constexpr bool kEqualPatches = true;         // any unit in any buffer: five fit, four would be one plane's
  static constexpr bool kImages = false;
};
// k3 s1 p1 over U * 64 channels: unit u its 64 channels, weight block 3 * u + filter column
template <int U>
struct Conv1 {
  static constexpr int kTaps = 3, kNC = 64, kUnits = U, kBlocks = 3 * U, kShort = 0, kEntries = 3 * U, kStart = 1, kEpiWarps = 16;
  __host__ __device__ static constexpr Entry entry(int e) { return Entry{e / 3, e % 3 == 2 ? 4 : e % 3, e, 0, 0, 4, MAIN, e % 3 == 0, e % 3 == 2}; }
  static constexpr int kHalo[2] = {4, 4};
  static constexpr bool kEqualPatches = true, kImages = false;
};
// The same over 256 channels, 32 outputs a CTA, on images outermost ([n][y][x] with a zero column and row behind every image):
// a tile is as many whole image rows as 128 positions hold, one of each image, with a zero row of its own before them.
struct Conv256 {
  static constexpr int kTaps = 3, kNC = 32, kUnits = 4, kBlocks = 12, kShort = 0, kEntries = 12, kStart = 1, kEpiWarps = 8;
  __host__ __device__ static constexpr Entry entry(int e) { return Conv1<4>::entry(e); }
  static constexpr int kHalo[kUnits] = {4, 4, 4, 4};
  static constexpr bool kEqualPatches = true, kImages = true;
};
// k4 s2 p1 and the shortcut k2 s2 p0: over blocks, filter (2*ty + dy, 2*tx + dx) at block tap (ty, tx), sub-position (dy, dx);
// of the shortcut's filter (ty, tx) at sub-position (1 - ty, 1 - tx).  Weight block 2 * unit + tx; the shortcut's: unit
struct Down32 {                    // unit u: the two sub-positions of sub-row u
  static constexpr int kTaps = 2, kNC = 64, kUnits = 2, kBlocks = 4, kShort = 2, kEntries = 8, kStart = 0, kEpiWarps = 16;
  __host__ __device__ static constexpr Entry entry(int e) {
    const int u = e / 4, i = e % 4;
    if (i < 2) return Entry{u, i, 2 * u + i, 0, 0, 4, MAIN, i == 0, false};
    const int tx = i - 2, half = tx == 0 ? 2 : 0;     // the sub-position 1 - tx of the sub-row
    return Entry{u, tx, u, half, half, 2, u == 1 ? SHORT_HERE : SHORT_BEFORE, false, i == 3};
  }
  static constexpr int kHalo[kUnits] = {1, 1};
  static constexpr bool kEqualPatches = true, kImages = false;
};
struct Down64 {                    // unit u: sub-position u
  static constexpr int kTaps = 2, kNC = 64, kUnits = 4, kBlocks = 8, kShort = 4, kEntries = 12, kStart = 0, kEpiWarps = 16;
  __host__ __device__ static constexpr Entry entry(int e) {
    const int u = e / 3, i = e % 3;
    if (i < 2) return Entry{u, i, 2 * u + i, 0, 0, 4, MAIN, i == 0, false};
    return Entry{u, 1 - (u & 1), u, 0, 0, 4, u >= 2 ? SHORT_HERE : SHORT_BEFORE, false, true};
  }
  static constexpr int kHalo[kUnits] = {1, 1, 1, 1};
  static constexpr bool kEqualPatches = true, kImages = false;
};

struct WalkParams {
  int steps, outs_per_tile;        // input and output steps of the axis
  int P, tile;                     // positions of a step, of a tile
  uint32_t res_n, res_step;        // residual: rows from image to image and from step to step
  int img, Wb, Ho, Wo;             // positions of one image and of one of its rows; of them, rows and columns that give outputs
  int outs, parts, ctas;           // tiles * output steps, channel shares, CTAs per share
  int patches, patch_bytes[2];     // buffers; sizes of the even and the odd ones
  int unit_rows[kMaxUnits];
  int y_blocks, step_blocks;       // outputs in blocks of 2x2: of (row, column) of a position; of (step, column)
  uint32_t n16, y16, x16, step16, sub16;  // strides of an output's image, row, column, step and sub-row (of a sub-position pair), 16-byte pieces
  int act;
  float slope;
  const __half* wimg;              // [part][weight blocks], rows swizzled as they lie in shared memory
  const float *scale, *shift;      // [K], then the shortcut's
  int K;
  uint4 *y, *y_short;
  const uint4* residual;           // rows as the positions
  int* gerr;
};
struct WalkMaps {
  CUtensorMap u[kMaxUnits];
};

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const void* desc, uint32_t bar, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(desc)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// 16 lanes x 32 columns: lane l of the warp gets of rows l / 4 and l / 4 + 8 the columns 8 i + 2 (l % 4) and + 1, in registers
// 4 i, 4 i + 1 and 4 i + 2, 4 i + 3
__device__ __forceinline__ void tmem_ld_16x32(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// zeros into 32 lanes x 32 columns
__device__ __forceinline__ void tmem_zero_32x32(uint32_t taddr) {
#pragma unroll
  for (int c = 0; c < 32; c += 8)
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(taddr + c), "r"(0) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// the output channel of column n: in each 32, columns 8 i + 2 j + b are channels 8 j + 2 i + b
__device__ __forceinline__ int channel_of(int n) { return (n & ~31) + (n >> 1 & 3) * 8 + (n >> 3 & 3) * 2 + (n & 1); }
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
__device__ __forceinline__ int uniform(int v) { return __shfl_sync(0xffffffffu, v, 0); }
__device__ __forceinline__ bool uniform(bool v) { return __shfl_sync(0xffffffffu, v ? 1 : 0, 0) != 0; }

// The outputs of a CTA, [g, end), in runs of one tile each: output steps [da, db) of tile t.  A run's accumulators take consecutive
// slots of the ring from `slot` on; one that fits goes back to slot 0 rather than turn over in the middle, which would make
// two instructions of each of a step's products; not within three outputs, so that a team that takes every second output has
// waited for one of its own between two uses of a slot and cannot mistake the earlier for the later.
template <int SLOTS, int TAPS>
struct Runs {
  int g, end, D, steps;            // D: outputs of a tile, steps: of its input
  int t, da, db, slot, next_slot;
  __device__ __forceinline__ bool next() {
    if (g >= end) return false;
    t = g / D;
    da = g - t * D;
    db = min(D, da + end - g);
    const int n = db - da;
    g += n;
    slot = next_slot + n > SLOTS && n <= SLOTS && next_slot > 2 ? 0 : next_slot;
    next_slot = (slot + n) % SLOTS;
    return true;
  }
  __device__ __forceinline__ bool next_uniform() {  // (a division's result is not known to be the same in every lane)
    const bool any = uniform(next());
    t = uniform(t);
    da = uniform(da);
    db = uniform(db);
    slot = uniform(slot);
    return any;
  }
  __device__ __forceinline__ int f0() const { return max(da + 2 - TAPS, 0); }  // input steps: output o takes o + 2 - TAPS .. o + 1
  __device__ __forceinline__ int f1() const { return min(db, steps - 1); }
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
template <class G>
__device__ __forceinline__ uint32_t patch_offset(const WalkParams& p, int i) {
  return G::kEqualPatches ? (uint32_t)(i * p.patch_bytes[0]) : (uint32_t)((i >> 1) * (p.patch_bytes[0] + p.patch_bytes[1]) + (i & 1) * p.patch_bytes[0]);
}
template <class G>
__host__ __device__ constexpr int walk_threads() { return 32 * (kFirstEpi + G::kEpiWarps); }
template <class G>
__host__ __device__ constexpr int walk_weight_bytes() { return (G::kBlocks * G::kTaps + G::kShort) * G::kNC * 128; }

template <int ACT>
__device__ __forceinline__ float act_of(float v, float slope) {
  if (ACT == AIG_ACT_RELU) return fmaxf(v, 0.f);
  if (ACT == AIG_ACT_SWISH) return swish_sfu(v);
  if (ACT == AIG_ACT_LEAKY) return v < 0.f ? v * slope : v;
  return v;
}
// act(v) of two values, rounded; four pairs at a time
template <int ACT>
__device__ __forceinline__ void act_pairs(const float2 (&v)[4], float slope, uint32_t (&o)[4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const __half2 h = __floats2half2_rn(act_of<ACT>(v[e].x, slope), act_of<ACT>(v[e].y, slope));
    o[e] = *reinterpret_cast<const uint32_t*>(&h);
  }
}
__device__ __forceinline__ void act_pairs(const float2 (&v)[4], int act, float slope, uint32_t (&o)[4]) {
  switch (act) {
    case AIG_ACT_RELU: act_pairs<AIG_ACT_RELU>(v, slope, o); break;
    case AIG_ACT_SWISH: act_pairs<AIG_ACT_SWISH>(v, slope, o); break;
    case AIG_ACT_LEAKY: act_pairs<AIG_ACT_LEAKY>(v, slope, o); break;
    default: act_pairs<AIG_ACT_NONE>(v, slope, o); break;
  }
}

template <class G>
__global__ void __launch_bounds__(walk_threads<G>(), 1) walk_conv_kernel(const __grid_constant__ WalkMaps maps, const __grid_constant__ WalkParams p) {
  constexpr int NC = G::kNC, U = G::kUnits, T = G::kTaps;
  constexpr bool kShort = G::kShort > 0, kRes = G::kStart > 0;      // with a shortcut's outputs; with a residual
  constexpr int kBlockBytes = T * NC * 128, kShortBytes = NC * 128, kWBytes = walk_weight_bytes<G>(), kWPiece = 16384;
  constexpr int kCols = 512, kSlots = kCols / (kShort ? 2 * NC : NC), kColsPerOut = kShort ? 2 * NC : NC;
  constexpr int kTeams = G::kEpiWarps / 4, kChunks = kColsPerOut / 32;  // of four epilogue warps; of 32 channels of an output
  static_assert(kWBytes % 1024 == 0 && kSlots <= kMaxSlots && U <= kMaxUnits, "layout");
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - raw);
  const uint32_t sW = base, sPatch = base + kWBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + kWBytes + patch_offset<G>(p, p.patches));
  const uint32_t bar_w = smem_u32(bars), bar_tfull = bar_w + 8, bar_tempty = bar_tfull + 8 * kMaxSlots;
  const uint32_t bar_ufull = bar_tempty + 8 * kMaxSlots, bar_uempty = bar_ufull + 8 * kMaxPatches;
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(bars + 1 + 2 * kMaxSlots + 2 * kMaxPatches);
  volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

  const int part = (int)(blockIdx.x % (unsigned)p.parts), cta = (int)(blockIdx.x / (unsigned)p.parts);
  using WalkRuns = Runs<kSlots, T>;
  const WalkRuns all{(int)((long long)p.outs * cta / p.ctas), (int)((long long)p.outs * (cta + 1) / p.ctas), p.outs_per_tile, p.steps, 0, 0, 0, 0, 0};
  griddep_launch_dependents();
  if (threadIdx.x == 0) {
    mbar_init(bar_w, 1);
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(bar_tfull + 8 * i, 1);
      mbar_init(bar_tempty + 8 * i, 4 * kChunks);
    }
    for (int i = 0; i < kMaxPatches; ++i) {
      mbar_init(bar_ufull + 8 * i, 1);
      mbar_init(bar_uempty + 8 * i, 1);
    }
    *s_abort = 0;
    fence_mbar_init();
  }
  if (G::kImages) {                // the zero rows
    for (int i = threadIdx.x; i < p.patches * 8; i += walk_threads<G>())
      *reinterpret_cast<uint4*>(sm + kWBytes + patch_offset<G>(p, i >> 3) + (i & 7) * 16) = make_uint4(0, 0, 0, 0);
    fence_proxy_async_smem();
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
      for (int b = 0; b < kWBytes; b += kWPiece) bulk_load(sW + b, w + b, min(kWPiece, kWBytes - b), bar_w);
      for (int u = 0; u < U; ++u) tma_prefetch_desc(&maps.u[u]);
    }
    griddep_wait();
    WalkRuns r = all;
    PatchRing ring{0, 0};
    bool ok = true;
    while (ok && r.next_uniform()) {
      for (int f = r.f0(); f <= r.f1() && ok; ++f) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (!mbar_wait_bounded_sleepy(bar_uempty + 8 * ring.i, ring.phase ^ 1u, s_abort, p.gerr, 901)) { ok = false; break; }
          if (leader) {
            mbar_expect_tx(bar_ufull + 8 * ring.i, (uint32_t)(G::kImages ? p.tile : p.unit_rows[u]) * 128u);
            const uint32_t dst = sPatch + patch_offset<G>(p, ring.i);
            if (G::kImages) tma_load_4d(dst + 128, &maps.u[0], bar_ufull + 8 * ring.i, 64 * u, 0, f, r.t * (p.tile / p.Wb));
            else tma_load_2d(dst, &maps.u[u], bar_ufull + 8 * ring.i, 64 * u, f * p.P + r.t * 128 - G::kStart);
          }
          ring.advance(p.patches);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (see elect_one)
    // The tensor pipe runs only a product or two ahead of this warp, so what a step needs (its barriers, its columns) is looked
    // up between the last products of the step before, and nothing in the loop but the shapes depends on the kind of step.
    // With waits and completions in loops of their own a row of 128 channels (24 products) took 2840 clk, so 2490; with zeroed
    // columns instead of first products that overwrite (see the epilogue) 2410.
    constexpr uint32_t hi = umma_desc_hi(128);
    const bool leader = elect_one();
    const uint32_t tmem = uniform(tmem_base);
    WalkRuns r = all;
    PatchRing ring{0, 0};
    uint32_t empty = 0;            // a bit per slot: the parity that says that its columns are zero
    bool ok = uniform(mbar_wait_bounded(bar_w, 0, s_abort, p.gerr, 911)), unit_ready = false, slot_ready = false;
    struct Step {
      int f, lo, n, old, slot, n2; // input step; outputs lo .. lo + n - 1, the first `old` of them begun before; slot of lo
      uint32_t d1, w1, id1;        // their columns, weight rows and shape, without the last n2, which lie behind the ring's end
    };
    while (ok && r.next_uniform()) {
      const int f0 = r.f0(), f1 = r.f1();
      auto step_at = [&](int f, int slot) {
        Step c;
        c.f = f;
        c.slot = slot;
        c.lo = max(f - 1, r.da);
        c.n = min(f + T - 1, r.db) - c.lo;
        c.old = f == f0 ? 0 : f + T - 2 - c.lo;           // (all of them where the run has no more to begin)
        const int n1 = min(c.n, kSlots - slot);
        c.n2 = c.n - n1;
        c.d1 = tmem + (uint32_t)(slot * NC);
        c.w1 = sW + (uint32_t)((c.lo - f + 1) * NC * 128);
        c.id1 = umma_idesc_f16(128, NC) + ((uint32_t)((n1 - 1) * NC / 8) << 17);
        return c;
      };
      Step c = step_at(f0, r.slot), next = c;
      while (ok) {
        if (slot_ready) {
          empty ^= 1u << ((c.slot + c.old) % kSlots);
          slot_ready = false;
        } else {
          for (int i = c.old; i < c.n; ++i) {
            const int so = (c.slot + i) % kSlots;
            if (!uniform(mbar_wait_bounded(bar_tempty + 8 * so, empty >> so & 1u, s_abort, p.gerr, 912))) { ok = false; break; }
            empty ^= 1u << so;
          }
          if (!ok) break;
        }
        tc_fence_after();
        auto look_ahead = [&](bool step_ends) {
          if (step_ends && c.f < f1) {
            next = step_at(c.f + 1, (c.slot + (c.lo < c.f ? 1 : 0)) % kSlots);
            if (next.old < next.n) {
              const int so = (next.slot + next.old) % kSlots;
              slot_ready = uniform(mbar_test(bar_tempty + 8 * so, empty >> so & 1u));
            }
          }
          PatchRing after = ring;
          after.advance(p.patches);
          unit_ready = uniform(mbar_test(bar_ufull + 8 * after.i, after.phase));
        };
        auto products = [&](auto number) {
          constexpr int e = decltype(number)::value;
          constexpr Entry E = G::entry(e);
          if (!ok) return;
          if (E.first && !unit_ready && !uniform(mbar_wait_bounded(bar_ufull + 8 * ring.i, ring.phase, s_abort, p.gerr, 913))) { ok = false; return; }
          const int rows = (E.shift & 1) + (E.shift & 2 ? p.Wb : 0) + (E.shift & 4 ? 2 : 0);
          const uint32_t a = umma_desc_lo(sPatch + patch_offset<G>(p, ring.i) + (uint32_t)(rows * 128)) + 2 * E.a0;
          if constexpr (E.kind == MAIN) {
            const uint32_t b1 = umma_desc_lo(c.w1 + E.block * kBlockBytes) + 2 * E.b0;
#pragma unroll
            for (int k = 0; k < E.nk; ++k) {
              if (leader) umma_f16_ss_lo(c.d1, a + 2 * k, b1 + 2 * k, hi, c.id1, 1u);
              if (E.last && k == 0) look_ahead(e + 1 == G::kEntries);
            }
            if (c.n2 > 0) {
              const uint32_t b2 = b1 + (uint32_t)((c.n - c.n2) * NC * 8), id2 = umma_idesc_f16(128, NC) + ((uint32_t)((c.n2 - 1) * NC / 8) << 17);
#pragma unroll
              for (int k = 0; k < E.nk; ++k)
                if (leader) umma_f16_ss_lo(tmem, a + 2 * k, b2 + 2 * k, hi, id2, 1u);
            }
          } else {
            constexpr bool here = E.kind == SHORT_HERE;
            const int i = here ? c.f - c.lo : 0;          // output f - 1 is lo, unless the run begins with f
            const uint32_t b = umma_desc_lo(sW + G::kBlocks * kBlockBytes + E.block * kShortBytes) + 2 * E.b0;
            const uint32_t d = tmem + (uint32_t)(kSlots * NC + (c.slot + i) % kSlots * NC);
            const bool mine = leader && (here ? i < c.n : c.lo < c.f);
#pragma unroll
            for (int k = 0; k < E.nk; ++k) {
              if (mine) umma_f16_ss_lo(d, a + 2 * k, b + 2 * k, hi, umma_idesc_f16(128, NC), 1u);
              if (E.last && k == 0) look_ahead(e + 1 == G::kEntries);
            }
          }
          if (E.last) {
            if (leader) umma_commit(bar_uempty + 8 * ring.i);
            ring.advance(p.patches);
          }
        };
        for_each_entry(products, std::make_integer_sequence<int, G::kEntries>());
        if (!ok) break;
        // the output before this step is complete and, with the last step, this step's
        if (c.lo < c.f && leader) umma_commit(bar_tfull + 8 * c.slot);
        if (c.f == p.steps - 1 && c.lo + c.n > c.f && leader) umma_commit(bar_tfull + 8 * ((c.slot + c.f - c.lo) % kSlots));
        if (c.f == f1) break;
        c = next;
      }
    }
  } else if (warp >= kFirstEpi) {
    // ------------------------------------------------------------------ epilogue: 32 channels at a time by four warps
    // A team takes one 32 channels of every output or, with more teams than there are, of every kGroups-th.  A quad of lanes
    // holds a row's 32 columns, eight each; the weight rows are in such an order (channel_of) that a lane's are consecutive
    // channels: they leave as 64 contiguous bytes of eight rows an instruction, without a turn through shared memory.
    constexpr int kGroups = kTeams / kChunks;
    static_assert(kTeams % kChunks == 0 && kGroups <= 2, "teams");
    const int q = warp & 3, team = (warp - kFirstEpi) >> 2, c32 = team % kChunks, group = team / kChunks;
    const int gr = lane >> 2, gc = lane & 3;              // this lane's rows: gr, gr + 8, gr + 16, gr + 24 of the warp's
    const bool shortcut = kShort && c32 >= NC / 32;       // main's channels first, then the shortcut's
    const uint32_t cols = tmem_base + (uint32_t)((shortcut ? (kSlots - 1) * NC : 0) + c32 * 32) + ((uint32_t)(q * 32) << 16);
    const int ch = part * NC + (shortcut ? c32 * 32 - NC : c32 * 32) + gc * 8;
    float sc[8], sh[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      sc[i] = p.scale[(shortcut ? p.K : 0) + ch + i];
      sh[i] = p.shift[(shortcut ? p.K : 0) + ch + i];
    }
    WalkRuns r = all;
    uint32_t full = 0;                                    // a bit per slot, as `empty`
    int turn = 0;                                         // number of the output, modulo kGroups
    bool ok = true;
    // every product adds: a first one that overwrites would be a shape of its own between overlapping columns, which the tensor
    // pipe runs one after another
    auto release = [&](int slot) {
      tmem_zero_32x32(cols + (uint32_t)(slot * NC));
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_tempty + 8 * slot);
    };
    if (group == 0)
      for (int i = 0; i < kSlots; ++i) release(i);
    griddep_wait();                                       // the output may still be read by an earlier launch
    while (ok && r.next()) {
      uint32_t offs[4], res_offs[4];
      bool vs[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = q * 32 + 8 * i + gr, pos = r.t * p.tile + row;
        const int n = pos / p.img, rem = pos - n * p.img, y = rem / p.Wb, x = rem - y * p.Wb;
        vs[i] = row < p.tile && pos < p.P && y < p.Ho && x < p.Wo;
        res_offs[i] = ((uint32_t)n * p.res_n + (uint32_t)x) * (uint32_t)(p.K / 8) + (uint32_t)(ch / 8);
        // (sub16 is the step between a block's sub-rows, half of it the one between its columns)
        offs[i] = (uint32_t)n * p.n16 + (uint32_t)(ch / 8) +
                  (p.y_blocks ? (uint32_t)((y + 1) >> 1) * p.y16 + (uint32_t)((y + 1) & 1) * p.sub16 : (uint32_t)y * p.y16) +
                  (p.y_blocks | p.step_blocks ? (uint32_t)((x + 1) >> 1) * p.x16 + (uint32_t)((x + 1) & 1) * (p.sub16 / 2) : (uint32_t)x * p.x16);
      }
      uint4 res[4];                                       // the residual, fetched an output ahead
      auto fetch = [&](int d) {
        const uint4* rr = p.residual + (size_t)d * p.res_step * (p.K / 8);
#pragma unroll
        for (int i = 0; i < 4; ++i) res[i] = vs[i] ? __ldg(rr + res_offs[i]) : make_uint4(0, 0, 0, 0);
      };
      if constexpr (kRes) {
        const int d = r.da + (kGroups > 1 && turn != group ? 1 : 0);
        if (d < r.db) fetch(d);
      }
      for (int d = r.da; d < r.db; ++d) {
        const int slot = r.slot_of(d);
        if (kGroups > 1) {
          const bool mine = turn == group;
          turn ^= 1;
          if (!mine) {
            full ^= 1u << slot;
            continue;
          }
        }
        if (!mbar_wait_bounded_sleepy(bar_tfull + 8 * slot, full >> slot & 1u, s_abort, p.gerr, 921)) { ok = false; break; }
        full ^= 1u << slot;
        tc_fence_after();
        uint32_t v[2][16];
        tmem_ld_16x32(cols + (uint32_t)(slot * NC), v[0]);
        tmem_ld_16x32(cols + (uint32_t)(slot * NC) + (16u << 16), v[1]);
        tmem_ld_wait();
        release(slot);
        uint4* yd = (shortcut ? p.y_short : p.y) + (p.step_blocks ? (size_t)((d + 1) >> 1) * p.step16 + (size_t)((d + 1) & 1) * p.sub16 : (size_t)d * p.step16);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float2 a[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const uint32_t* u = &v[i >> 1][4 * e + 2 * (i & 1)];
            a[e] = make_float2(fmaf(__uint_as_float(u[0]), sc[2 * e], sh[2 * e]), fmaf(__uint_as_float(u[1]), sc[2 * e + 1], sh[2 * e + 1]));
          }
          if constexpr (kRes) {
            // the reference stores fp16 after BatchNorm and again after the add (ResConvLayer.cpp:35-36)
            const __half2* rh = reinterpret_cast<const __half2*>(&res[i]);
#pragma unroll
            for (int e = 0; e < 4; ++e) a[e] = __half22float2(__hadd2(__floats2half2_rn(a[e].x, a[e].y), rh[e]));
          }
          uint32_t o[4];
          if (shortcut) act_pairs<AIG_ACT_NONE>(a, 0.f, o);
          else act_pairs(a, p.act, p.slope, o);
          if (vs[i]) yd[offs[i]] = make_uint4(o[0], o[1], o[2], o[3]);
        }
        if constexpr (kRes) {
          if (d + kGroups < r.db) fetch(d + kGroups);
        }
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

// ---- weights as they lie in shared memory: element k of a block's row, 16-byte pieces in the 128-byte swizzle order
__device__ __forceinline__ size_t swizzled(int row, int k) { return (size_t)row * 64 + (((k >> 3) ^ (row & 7)) << 3) + (k & 7); }

// w [K][C][3][3][3]: row s * NC + n of a block is output channel n of the share with depth tap 2 - s
template <class G>
__global__ void clip_pack_kernel(const __half* __restrict__ w, __half* __restrict__ img, int K) {
  constexpr int NC = G::kNC, rows = 3 * NC, C = std::is_same<G, Clip32>::value ? 32 : 64;
  const int total = K / NC * G::kBlocks * rows * 64;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int k = i & 63, r = (i >> 6) % rows, b = (i >> 6) / rows % G::kBlocks, part = (i >> 6) / (rows * G::kBlocks);
    const int out = part * NC + channel_of(r % NC), kd = 2 - r / NC;
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
    img[(size_t)((i >> 6) - r) * 64 + swizzled(r, k)] = used ? w[((size_t)(out * C + c) * 3 + kd) * 9 + fr * 3 + fs] : __ushort_as_half((unsigned short)0);
  }
}
// w [K][64 U][3][3]: row s * NC + n is output channel n of the share with filter row 2 - s
template <class G>
__global__ void conv1_pack_kernel(const __half* __restrict__ w, __half* __restrict__ img, int K) {
  constexpr int NC = G::kNC, rows = 3 * NC, U = G::kUnits;
  const int total = K / NC * G::kBlocks * rows * 64;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int k = i & 63, r = (i >> 6) % rows, b = (i >> 6) / rows % G::kBlocks, part = (i >> 6) / (rows * G::kBlocks);
    const int out = part * NC + channel_of(r % NC), c = b / 3 * 64 + k;
    img[(size_t)((i >> 6) - r) * 64 + swizzled(r, k)] = w[(size_t)(out * 64 * U + c) * 9 + (2 - r / NC) * 3 + b % 3];
  }
}
// w_main [K][C][4][4]: row s * NC + n is output channel n of the share at block tap ty = 1 - s; w_short [K][C][2][2]
template <class G>
__global__ void down_pack_kernel(const __half* __restrict__ w_main, const __half* __restrict__ w_short, __half* __restrict__ img, int K) {
  constexpr int NC = G::kNC, C = std::is_same<G, Down32>::value ? 32 : 64, rows = G::kBlocks * 2 * NC + G::kShort * NC;  // of a share
  const int total = K / NC * rows * 64;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int k = i & 63, R = (i >> 6) % rows, part = (i >> 6) / rows;
    const bool main = R < G::kBlocks * 2 * NC;
    const int r = main ? R : R - G::kBlocks * 2 * NC, b = main ? r / (2 * NC) : r / NC, unit = main ? b >> 1 : b;
    const int out = part * NC + channel_of(r % NC), c = k % C;
    const int dy = C == 32 ? unit : unit >> 1, dx = C == 32 ? k >> 5 : unit & 1;
    const int ty = main ? 1 - r / NC % 2 : 1 - dy, tx = main ? b & 1 : 1 - dx;
    img[(size_t)part * rows * 64 + swizzled(R, k)] =
        main ? w_main[((size_t)(out * C + c) * 4 + 2 * ty + dy) * 4 + 2 * tx + dx] : w_short[((size_t)(out * C + c) * 2 + ty) * 2 + tx];
  }
}
// scale / shift: bias and BatchNorm folded
__global__ void walk_affine_kernel(const __half* bias, const float* gamma, const float* beta, const float* mean, const float* var, float eps, float* scale,
                                   float* shift, int K) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < K; k += gridDim.x * blockDim.x) {
    const float b = bias ? __half2float(bias[k]) : 0.f, s = gamma ? gamma[k] / sqrtf(var[k] + eps) : 1.f;
    scale[k] = s;
    shift[k] = gamma ? (b - mean[k]) * s + beta[k] : b;
  }
}

// blocks [yb][n][xb][4][c] -> channels-last, 8 channels per thread
__global__ void row_blocks_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst, int batch, int h, int w, int c8, int wb) {
  const long long total = (long long)batch * h * w * c8;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % c8), x = (int)(i / c8 % w), y = (int)(i / c8 / w % h), n = (int)(i / c8 / w / h);
    dst[i] = src[((((size_t)((y + 1) >> 1) * batch + n) * wb + ((x + 1) >> 1)) * 4 + ((y + 1) & 1) * 2 + ((x + 1) & 1)) * c8 + c];
  }
}

// blocks [d][n][Hb][Wb][4][c] -> [n][d][h][w][c], 8 channels per thread
__global__ void clip_blocks_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst, int batch, int d, int h, int w, int c8, int Hb, int Wb) {
  const long long total = (long long)batch * d * h * w * c8;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % c8), x = (int)(i / c8 % w), y = (int)(i / c8 / w % h), z = (int)(i / c8 / w / h % d), n = (int)(i / c8 / w / h / d);
    dst[i] = src[((((size_t)z * batch + n) * Hb + ((y + 1) >> 1)) * Wb + ((x + 1) >> 1)) * 4 * c8 + (((y + 1) & 1) * 2 + ((x + 1) & 1)) * c8 + c];
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

template <class G>
int walk_layout(WalkParams& p) {   // fills in the patches' rows and buffers; the shared memory that a CTA needs (too much: cannot be had)
  int bytes[kMaxUnits];
  for (int u = 0; u < G::kUnits; ++u) {
    p.unit_rows[u] = 128 + (G::kHalo[u] & 1) + (G::kHalo[u] & 2 ? p.Wb : 0) + (G::kHalo[u] & 4 ? 2 : 0);
    bytes[u] = p.unit_rows[u] * 128;  // (the 128-byte swizzle goes by the address, so a patch may begin at any row)
  }
  const int fixed = 1024 + walk_weight_bytes<G>() + 8 * (1 + 2 * kMaxSlots + 2 * kMaxPatches) + 16;
  const int room = 227 * 1024 - fixed;
  p.patch_bytes[0] = bytes[0];     // (the largest)
  p.patch_bytes[1] = G::kEqualPatches ? bytes[0] : bytes[1];
  const int pair = p.patch_bytes[0] + p.patch_bytes[1];
  p.patches = G::kEqualPatches ? room / bytes[0] : room / pair * 2;
  if (p.patches > kMaxPatches) p.patches = kMaxPatches;
  if (p.patches < 2) return 228 * 1024;
  return fixed + (p.patches / 2) * pair + (p.patches & 1) * bytes[0];
}

// what walk_conv_kernel is instantiated for
enum Variant { CLIP32, CLIP64, CONV64, CONV128, CONV256, DOWN32, DOWN64 };
template <class F>
auto with_variant(Variant v, F&& f) {
  switch (v) {
    case CLIP32: return f(Clip32());
    case CLIP64: return f(Clip64());
    case CONV64: return f(Conv1<1>());
    case CONV128: return f(Conv1<2>());
    case CONV256: return f(Conv256());
    case DOWN32: return f(Down32());
    default: return f(Down64());
  }
}
int variant_layout(Variant v, WalkParams& p) {
  return with_variant(v, [&](auto g) { return walk_layout<decltype(g)>(p); });
}

WalkParams clip_params(const ClipConvGeom& g) {
  WalkParams p{};
  p.steps = p.outs_per_tile = g.D;
  p.Ho = (g.H - 1) / 2 + 1; p.Wo = (g.W - 1) / 2 + 1;
  p.Wb = clip_block_extent(g.W);
  p.img = clip_block_extent(g.H) * p.Wb;
  p.P = g.batch * p.img;
  p.tile = 128;
  p.K = g.K;
  p.parts = g.K / (g.C == 32 ? Clip32::kNC : Clip64::kNC);
  const uint32_t k16 = (uint32_t)g.K / 8, Hb2 = clip_block_extent(p.Ho), Wb2 = clip_block_extent(p.Wo);
  if (g.out_blocks) {
    p.y_blocks = 1;
    p.sub16 = 2 * k16; p.x16 = 4 * k16; p.y16 = Wb2 * p.x16; p.n16 = Hb2 * p.y16; p.step16 = (uint32_t)g.batch * p.n16;
  } else {
    p.x16 = k16; p.y16 = (uint32_t)p.Wo * k16; p.step16 = (uint32_t)p.Ho * p.y16; p.n16 = (uint32_t)g.D * p.step16;
  }
  p.act = AIG_ACT_LEAKY;
  p.slope = g.slope;
  return p;
}

int res_out_h(const ResWalkGeom& g) { return (g.H - 2) / 2 + 1; }
int res_out_w(const ResWalkGeom& g) { return (g.W - 2) / 2 + 1; }
WalkParams res_params(const ResWalkGeom& g, bool down) {
  WalkParams p{};
  p.Ho = 1;                        // (positions of a step are one row)
  p.Wo = res_out_w(g);
  p.Wb = p.img = p.Wo + 1;         // blocks of an input row, or an image row with its zero column: as many
  p.P = g.batch * p.Wb;
  p.tile = 128;
  p.res_n = (uint32_t)p.Wb; p.res_step = (uint32_t)p.P;
  p.outs_per_tile = res_out_h(g);
  p.steps = down ? p.outs_per_tile + 1 : p.outs_per_tile;
  p.K = g.K;
  p.parts = g.K / 64;
  p.act = g.act;
  p.slope = g.slope;
  const uint32_t k16 = (uint32_t)g.K / 8, h = (uint32_t)res_out_h(g), w = (uint32_t)p.Wo, hb = (h - 2) / 2 + 2, wb = (w - 2) / 2 + 2;
  if (down) {
    p.x16 = k16; p.n16 = (uint32_t)p.Wb * k16; p.step16 = (uint32_t)p.P * k16;
  } else if (g.out == RES_OUT_NHWC) {
    p.x16 = k16; p.step16 = w * k16; p.n16 = h * p.step16;
  } else {
    p.step_blocks = 1;
    p.sub16 = 2 * k16; p.x16 = 4 * k16;
    p.step16 = wb * p.x16; p.n16 = hb * p.step16;
    if (g.out == RES_OUT_ROW_BLOCKS) { p.n16 = wb * p.x16; p.step16 = (uint32_t)g.batch * p.n16; }
  }
  return p;
}
Variant down_variant(const ResWalkGeom& g) { return g.C == 32 ? DOWN32 : DOWN64; }
// k3 s1 p1 alone, h x w pixels
WalkParams conv_params(const ConvWalkGeom& g) {
  WalkParams p = res_params(ResWalkGeom{g.batch, 2 * g.h, 2 * g.w, 0, g.C, g.act, g.slope, g.out}, false);  // (a block of that output)
  p.parts = g.C / Conv256::kNC;
  p.tile = 128 / p.Wb * p.Wb;
  p.res_step = (uint32_t)p.Wb; p.res_n = (uint32_t)((g.h + 1) * p.Wb);
  return p;
}
Variant conv1_variant(const ResWalkGeom& g) { return g.K == 64 ? CONV64 : CONV128; }

}  // namespace

struct WalkConv {
  aig_ctx* ctx = nullptr;
  Variant variant{};
  int in_c = 0;                    // channels of a position (of a block: four pixels')
  WalkParams prm{};
  WalkMaps maps{};
  const void* map_x = nullptr;
  __half* wimg = nullptr;
  float* affine = nullptr;
  int smem = 0;
  bool weights_set = false;
};

static int walk_create(aig_ctx* ctx, Variant v, int in_c, const WalkParams& prm, WalkConv** out) {
  *out = nullptr;
  DeviceGuard guard(ctx->device);
  WalkConv* c = new WalkConv();
  c->ctx = ctx;
  c->variant = v;
  c->in_c = in_c;
  c->prm = prm;
  WalkParams& p = c->prm;
  c->smem = variant_layout(v, p);
  p.outs = ceil_div(p.P, p.tile) * p.outs_per_tile;
  p.ctas = ctx->sm_count / p.parts;
  if (p.ctas > p.outs) p.ctas = p.outs;
  const bool shortcut = v == DOWN32 || v == DOWN64;
  const size_t img = (size_t)p.parts * with_variant(v, [](auto g) { return walk_weight_bytes<decltype(g)>(); });
  const size_t rows = (size_t)p.K * (shortcut ? 2 : 1);
  if (cudaMalloc(&c->wimg, img) != cudaSuccess || cudaMalloc(&c->affine, 2 * rows * sizeof(float)) != cudaSuccess) {
    walk_conv_destroy(c);
    return aig_fail(ctx, AIG_ERR_CUDA, "walking convolution: allocation failed");
  }
  p.wimg = c->wimg;
  p.scale = c->affine;
  p.shift = c->affine + rows;
  p.gerr = ctx->d_err;
  const cudaError_t e = with_variant(v, [](auto g) {
    return cudaFuncSetAttribute(walk_conv_kernel<decltype(g)>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  });
  if (e != cudaSuccess) {
    walk_conv_destroy(c);
    return aig_fail(ctx, AIG_ERR_CUDA, "walking convolution: %s", cudaGetErrorString(e));
  }
  *out = c;
  return AIG_OK;
}

void walk_conv_destroy(WalkConv* c) {
  if (!c) return;
  DeviceGuard guard(c->ctx->device);
  cudaFree(c->wimg);
  cudaFree(c->affine);
  delete c;
}

static int walk_launch(WalkConv* c, const aig_half* x, const aig_half* residual, aig_half* y, aig_half* y_short) {
  aig_ctx* ctx = c->ctx;
  DeviceGuard guard(ctx->device);
  AIG_REQUIRE(ctx, x && y && c->weights_set, "walking convolution: null pointer or weights not set");
  AIG_REQUIRE(ctx, (((uintptr_t)x | (uintptr_t)y | (uintptr_t)residual | (uintptr_t)y_short) & 15) == 0, "walking convolution: misaligned tensors");
  WalkParams& p = c->prm;
  if (c->map_x != x) {
    static EncodeTiledFn enc = nullptr;
    if (!enc) {
      void* fn = nullptr;
      cudaDriverEntryPointQueryResult qres;
      if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess || qres != cudaDriverEntryPointSuccess)
        return aig_fail(ctx, AIG_ERR_CUDA, "cuTensorMapEncodeTiled entry point not available");
      enc = reinterpret_cast<EncodeTiledFn>(fn);
    }
    for (int u = 0; u < with_variant(c->variant, [](auto g) { return (int)decltype(g)::kUnits; }); ++u) {
      cuuint64_t dims[2] = {(cuuint64_t)c->in_c, (cuuint64_t)p.steps * p.P};
      cuuint64_t strides[1] = {(cuuint64_t)c->in_c * 2};
      cuuint32_t box[2] = {64u, (cuuint32_t)p.unit_rows[u]};
      cuuint32_t es[2] = {1, 1};
      const cuuint64_t h1 = (cuuint64_t)p.steps + 1, w1 = (cuuint64_t)p.Wb;                     // images outermost: (channel, x, y, n)
      cuuint64_t dims4[4] = {(cuuint64_t)c->in_c, w1, h1, (cuuint64_t)p.P / w1}, strides4[3] = {strides[0], strides[0] * w1, strides[0] * w1 * h1};
      cuuint32_t box4[4] = {64u, (cuuint32_t)w1, 1, (cuuint32_t)(p.tile / p.Wb)}, es4[4] = {1, 1, 1, 1};
      const bool images = c->variant == CONV256;
      const CUresult r = enc(&c->maps.u[u], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, images ? 4 : 2, const_cast<aig_half*>(x), images ? dims4 : dims,
                             images ? strides4 : strides, images ? box4 : box, images ? es4 : es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
      if (r != CUDA_SUCCESS) return aig_fail(ctx, AIG_ERR_CUDA, "cuTensorMapEncodeTiled(walking convolution) failed: %d", (int)r);
    }
    c->map_x = x;
  }
  p.y = reinterpret_cast<uint4*>(y);
  p.y_short = reinterpret_cast<uint4*>(y_short);
  p.residual = reinterpret_cast<const uint4*>(residual);
  AIG_CUDA_OK(ctx, with_variant(c->variant, [&](auto g) {
    using G = decltype(g);
    return launch_pdl(ctx, walk_conv_kernel<G>, dim3((unsigned)(p.parts * p.ctas)), dim3(walk_threads<G>()), (size_t)c->smem, c->maps, p);
  }));
  return AIG_OK;
}

static int walk_affine(WalkConv* c, int first, const aig_half* bias, const float* gamma, const float* beta, const float* mean, const float* var, float eps) {
  walk_affine_kernel<<<ceil_div(c->prm.K, 128), 128, 0, c->ctx->stream>>>((const __half*)bias, gamma, beta, mean, var, eps, const_cast<float*>(c->prm.scale) + first,
                                                                         const_cast<float*>(c->prm.shift) + first, c->prm.K);
  AIG_LAUNCH_OK(c->ctx);
  return AIG_OK;
}

// 32-bit positions and 16-byte pieces
static bool walk_counts_fit(long long in_rows, int in_c, long long out_pixels, int K) {
  return in_rows < (1ll << 30) && in_rows * in_c < (1ll << 34) && out_pixels * K < (1ll << 34);
}

bool clip_conv_supported(const aig_ctx* ctx, const ClipConvGeom& g) {
  if (!(g.C == 32 && g.K % 64 == 0) && !(g.C == 64 && g.K % 32 == 0)) return false;
  if (g.batch <= 0 || g.D <= 0 || g.H <= 0 || g.W <= 0 || g.K <= 0 || g.K > 512) return false;
  const long long rows = (long long)g.batch * g.D * clip_block_extent(g.H) * clip_block_extent(g.W);
  if (!walk_counts_fit(rows, 4 * g.C, rows, g.K) || clip_block_extent(g.W) > 256 - 129) return false;  // (a TMA box has 256 rows)
  WalkParams p = clip_params(g);
  return p.parts <= ctx->sm_count && variant_layout(g.C == 32 ? CLIP32 : CLIP64, p) <= 227 * 1024;
}
int clip_conv_create(aig_ctx* ctx, const ClipConvGeom& g, WalkConv** out) {
  *out = nullptr;
  if (!clip_conv_supported(ctx, g)) return aig_fail(ctx, AIG_ERR_UNSUPPORTED, "clip convolution: unsupported geometry");
  return walk_create(ctx, g.C == 32 ? CLIP32 : CLIP64, 4 * g.C, clip_params(g), out);
}
int clip_conv_set_weights(WalkConv* c, const aig_half* w, const aig_half* bias, const float* gamma, const float* beta, const float* mean, const float* var,
                          float eps) {
  if (c->variant == CLIP32) clip_pack_kernel<Clip32><<<128, 256, 0, c->ctx->stream>>>((const __half*)w, c->wimg, c->prm.K);
  else clip_pack_kernel<Clip64><<<128, 256, 0, c->ctx->stream>>>((const __half*)w, c->wimg, c->prm.K);
  AIG_LAUNCH_OK(c->ctx);
  c->weights_set = true;
  return walk_affine(c, 0, bias, gamma, beta, mean, var, eps);
}
int clip_conv_forward(WalkConv* c, const aig_half* x, aig_half* y) { return walk_launch(c, x, nullptr, y, nullptr); }
int clip_blocks_to_ndhwc(aig_ctx* ctx, const aig_half* blocks, aig_half* y, int batch, int d, int h, int w, int c) {
  DeviceGuard guard(ctx->device);
  clip_blocks_kernel<<<ctx->sm_count * 8, 256, 0, ctx->stream>>>((const uint4*)blocks, (uint4*)y, batch, d, h, w, c / 8, clip_block_extent(h), clip_block_extent(w));
  AIG_LAUNCH_OK(ctx);
  return AIG_OK;
}

// No rule on sizes: against the patch-resident kernel the first block's launches gain from one frame of 320x320 (11.6 -> 10.5 us,
// the second convolution) over one of 540x960 (16.0 + 14.9 -> 12.5 + 12.0; the second block 14.7 + 14.3 -> 12.5 + 12.4), the first
// that is beyond the chain, to the largest batches (see above); one of 1400x400 is even.
bool res_walk_supported(const aig_ctx* ctx, const ResWalkGeom& g) {
  if (!(g.C == 32 && g.K == 64) && !(g.C == 64 && g.K == 128)) return false;
  if (g.batch <= 0 || g.H < 4 || g.W < 4) return false;
  const long long rows = (long long)g.batch * (res_out_h(g) + 1) * (res_out_w(g) + 1);
  if (!walk_counts_fit(rows, 4 * g.C, rows, 4 * g.K)) return false;
  WalkParams d = res_params(g, true), c = res_params(g, false);
  return d.parts <= ctx->sm_count && variant_layout(down_variant(g), d) <= 227 * 1024 && variant_layout(conv1_variant(g), c) <= 227 * 1024;
}
size_t res_walk_rows(const ResWalkGeom& g) { return (size_t)g.batch * res_out_h(g) * (res_out_w(g) + 1); }
int res_walk_create(aig_ctx* ctx, const ResWalkGeom& g, WalkConv** down, WalkConv** conv1) {
  *down = *conv1 = nullptr;
  if (!res_walk_supported(ctx, g)) return aig_fail(ctx, AIG_ERR_UNSUPPORTED, "residual block by rows: unsupported geometry");
  int rc = walk_create(ctx, down_variant(g), 4 * g.C, res_params(g, true), down);
  if (rc == AIG_OK) rc = walk_create(ctx, conv1_variant(g), g.K, res_params(g, false), conv1);
  return rc;
}
int res_walk_set_down(WalkConv* c, const aig_half* w_main, const aig_half* b_main, const float* gamma, const float* beta, const float* mean, const float* var,
                      float eps, const aig_half* w_short, const aig_half* b_short) {
  if (c->variant == DOWN32) down_pack_kernel<Down32><<<128, 256, 0, c->ctx->stream>>>((const __half*)w_main, (const __half*)w_short, c->wimg, c->prm.K);
  else down_pack_kernel<Down64><<<128, 256, 0, c->ctx->stream>>>((const __half*)w_main, (const __half*)w_short, c->wimg, c->prm.K);
  AIG_LAUNCH_OK(c->ctx);
  c->weights_set = true;
  const int rc = walk_affine(c, 0, b_main, gamma, beta, mean, var, eps);
  return rc != AIG_OK ? rc : walk_affine(c, c->prm.K, b_short, nullptr, nullptr, nullptr, nullptr, 0.f);
}
int res_walk_set_conv1(WalkConv* c, const aig_half* w, const aig_half* bias, const float* gamma, const float* beta, const float* mean, const float* var,
                       float eps) {
  if (c->variant == CONV64) conv1_pack_kernel<Conv1<1>><<<128, 256, 0, c->ctx->stream>>>((const __half*)w, c->wimg, c->prm.K);
  else if (c->variant == CONV128) conv1_pack_kernel<Conv1<2>><<<128, 256, 0, c->ctx->stream>>>((const __half*)w, c->wimg, c->prm.K);
  else conv1_pack_kernel<Conv256><<<256, 256, 0, c->ctx->stream>>>((const __half*)w, c->wimg, c->prm.K);
  AIG_LAUNCH_OK(c->ctx);
  c->weights_set = true;
  return walk_affine(c, 0, bias, gamma, beta, mean, var, eps);
}
int res_walk_down(WalkConv* down, const aig_half* x, aig_half* t, aig_half* r) {
  AIG_REQUIRE(down->ctx, r, "residual block by rows: null pointer");
  return walk_launch(down, x, nullptr, t, r);
}
int res_walk_conv1(WalkConv* conv1, const aig_half* t, const aig_half* r, aig_half* y) {
  AIG_REQUIRE(conv1->ctx, r, "residual block by rows: null pointer");
  return walk_launch(conv1, t, r, y, nullptr);
}
bool conv_walk_supported(const aig_ctx* ctx, const ConvWalkGeom& g) {
  if (g.C != 256 || g.batch <= 0 || g.h < 2 || g.w < 2 || g.w + 1 > 128) return false;
  const long long rows = (long long)g.batch * (g.h + 1) * (g.w + 1);
  if (!walk_counts_fit(rows, g.C, rows, 4 * g.C)) return false;
  WalkParams p = conv_params(g);
  if (p.parts > ctx->sm_count || variant_layout(CONV256, p) > 227 * 1024) return false;
  // Against the patch-resident kernel, which takes a round of one 128-position tile per SM (17 to 30 us for the first, 41, 57, 68-80
  // and 85-94 us for two to five), while this one takes 2.0 to 2.9 us a row of a tile on a share's CTAs, however full, and 11 for the
  // launch.  Not where rows of the images side by side fill less than 0.68 of the tiles (16 frames of 576x1024, 65 of 128: 51 us by
  // patches, 74 by rows; 8 of 720x1280, 0.63: 41, 52; 8 of 380x672, 0.67: 21.6, 22.2; one of 1400x400, 0.20: 16.8, 20.5; but 64 of
  // 72x1440, 0.71: 40.9, 39.0), unless a CTA has two rows or so (one of 576x1024, 0.51, 2.0 rows: 17.1, 15.4); and not where the rows
  // per CTA are more than the rounds make up for (144x256, 192 frames, 14 rows and 2 rounds: 41.8, 41.7; 222, 16 and 2: 45.0, 47.3;
  // 256, 18.5 and 3: 56.8, 49.4; 334, 24 and 3: 62.8, 66.7; 800 of 96x160, 24.3 and 4: 72.8, 66.8; 64 of 360x640, 27 and 4: 67.9, 74.9).
  const long long tiles = ceil_div(p.P, p.tile), outs = tiles * p.outs_per_tile, ctas = ctx->sm_count / p.parts;
  const long long rounds = ceil_div_ll(ceil_div_ll(rows, 128), ctx->sm_count);
  const bool full = 100ll * p.P >= 68ll * 128 * tiles;
  return 10 * outs <= ctas * (full ? 40 + 53 * rounds : 24);
}
int conv_walk_create(aig_ctx* ctx, const ConvWalkGeom& g, WalkConv** out) {
  *out = nullptr;
  if (!conv_walk_supported(ctx, g)) return aig_fail(ctx, AIG_ERR_UNSUPPORTED, "convolution by rows: unsupported geometry");
  return walk_create(ctx, CONV256, g.C, conv_params(g), out);
}
int row_blocks_to_nhwc(aig_ctx* ctx, const aig_half* blocks, aig_half* y, int batch, int h, int w, int c) {
  DeviceGuard guard(ctx->device);
  row_blocks_kernel<<<ctx->sm_count * 8, 256, 0, ctx->stream>>>((const uint4*)blocks, (uint4*)y, batch, h, w, c / 8, (w - 2) / 2 + 2);
  AIG_LAUNCH_OK(ctx);
  return AIG_OK;
}
