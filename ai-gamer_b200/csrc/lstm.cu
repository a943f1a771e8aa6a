// lstm.cu -- LSTM forward (LSTMLayer.cpp:75-104 / LSTMLayerv8.cpp:78-82) for sm_100a.
//
// Per layer:  (1) the input projection W.x + bW + bR for all time steps is hoisted into one
// tcgen05 GEMM (rows = T*B, fp32 output);  (2) the recurrence.  Sequences are independent, so a cluster of CTAs takes
// 16 or 32 of them through all steps: each of its H/32 CTAs keeps the 4 gate rows of 32 hidden units of R (128 rows x H
// fp16) in TMEM and every step
//    - waits until all h_{t-1} of the cluster's sequences has arrived in its own shared memory,
//    - issues tcgen05.mma  R-slice [128 x H] x h_{t-1} [H x sequences]  into TMEM (gates are the M side, so that few
//      sequences waste nothing but columns),
//    - its 128 epilogue threads (one per gate row) add the hoisted projection and apply the gate function, trade gates
//      within each quad of lanes, keep the cell state in registers (rounded to fp16 every step, like the library's cy
//      tensor) and write h_t as fp16, and
//    - one bulk copy per CTA of the cluster delivers its 32 units of h_t, already in the operand's layout.
// What bounds a step is this chain's latency.  Of its 2550 clk (H = 512, 16 sequences; clock64) the 32 MMAs take 560, the
// gate functions 560, issue and delivery of the copies 1270 (about 20 B/clk of distributed shared memory come into an SM);
// with the MMAs in a loop of four it was 3240, 1160 of them the loop.  More sequences than the clusters of one group of 16 hold
// (seven of 16 CTAs fit the device) share clusters in groups of 16, each with its own issuer and epilogue warps, so that
// one group's MMAs run under the other's gates and delivery.  Up to eight sequences deliver half of the rows.
//
// (3)  Two layers run side by side in one launch where their clusters fit the device together (lstm_pair_kernel): the
// second layer's clusters multiply W.x_t themselves, a step or two behind, W beside R in TMEM (what does not fit, in
// shared memory).  That takes out half of the dependent steps and the second layer's projection, whose 4H fp32 values
// per step and sequence went through memory.  Whole sequence head, before and after, us, sequences of 64 steps at H = 512:
// 16 of them 279 and 161, 64 (two groups a cluster) 519 and 212, 128 (three groups and two) 379 and 264; 3 of 37 steps at
// H = 256 132 and 76.  (64 took longer than 128 before because two CTAs of different clusters could share an SM, of which
// one waited for the other's TMEM: see recurrent_smem.)
// Gate order i,f,g,o; blob layout: per layer W then R, then per layer bW [and bR]  (the library's
// blob is opaque in the reference: LSTMLayer.cpp:29-35,139-146; this layout is this library's
// definition, stated in the header).
#include <vector>

#include "aig_common.cuh"
#include "skinny_fc.h"

namespace {

constexpr int kUnits = 32;        // hidden units per CTA: 128 gate rows, UMMA's M
constexpr int kGateRows = 4 * kUnits;
constexpr int kSeqs = 16;         // sequences of a group: UMMA's N
__host__ __device__ constexpr int lstm_threads(int groups) { return 32 * 5 * groups; }  // per group an MMA issuer and four epilogue warps
__host__ __device__ constexpr int pair_threads(int ga, int gb) {  // and a warp that passes h_t on, or two for W . x_t
  return lstm_threads(ga) + 32 > lstm_threads(gb) + 64 ? lstm_threads(ga) + 32 : lstm_threads(gb) + 64;
}
// TMEM columns: the groups' accumulators, [two sets of accumulators of W . x_t,] R (two values of K each) [, W]
constexpr int kColX = 32;
__host__ __device__ constexpr int col_r(bool second) { return second ? kColX + 4 * kSeqs : 48; }

struct LstmParams {
  int T, B, H, ctas;              // ctas: CTAs of the cluster that have units (the rest of a power of two only wait)
  float clip;
  const __half* R;                // [4][H][H]
  const float* gx;                // hoisted projection, element (t,b,j) at t*gx_sT + b*gx_sB + j, j < 4H
  long long gx_sT, gx_sB;
  __half* y;                      // output sequence, element (t,b,j) at t*y_sT + b*y_sB + j
  long long y_sT, y_sB;
  const __half *h0, *c0;          // [B][H] initial state (null: zero)
  __half *hT, *cT;                // [B][H] final state (may be null; may be the initial state's memory)
  int* gerr;
};
// Two layers in one launch: the first `a_clusters` clusters run layer a, the rest layer b (see lstm_pair_kernel).
struct LstmPairParams {
  LstmParams a, b;
  int a_clusters, clusters;
  const __half* W;                // layer b's input matrix [4][H][H]
  const float* bias;              // and the sum of its biases [4H]
  __half* xs;                     // h_t of layer a: [T][groups][2][H/8][8 sequences][8 units]
  unsigned int* counters;         // [groups] parts of h_t written so far by layer a's CTAs, then clusters done
};

// own shared memory -> a cluster CTA's, the bytes counted on that CTA's barrier
__device__ __forceinline__ void bulk_to_cluster(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "r"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ unsigned int ld_acquire_gpu(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_gpu_add(unsigned int* p, unsigned int v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
// Operands in shared memory: K-major without swizzle, core matrices of 8 rows x 16 bytes, `lbo` bytes between neighbours
// along K, `sbo` along the rows.
__device__ __forceinline__ uint32_t plain_lo(uint32_t saddr, uint32_t lbo) { return ((saddr & 0x3FFFFu) >> 4) | (lbo >> 4) << 16; }
__device__ __forceinline__ constexpr uint32_t plain_hi(uint32_t sbo) { return (sbo >> 4) | (1u << 14); }
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
// N instructions in a row, one step of K (16) each: every iteration of a loop of them costs its branch and the way of the
// loop's values to the uniform registers, about 75 clk, beside 20 per instruction
template <int N>
__device__ __forceinline__ void umma_ts_steps(bool leader, uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_units, uint32_t b_hi, uint32_t idesc,
                                              uint32_t accumulate_first) {
#pragma unroll
  for (int k = 0; k < N; ++k)
    if (leader) umma_f16_ts(d_tmem, a_tmem + k * 8, b_lo + (k >> 1) * b_units + (k & 1) * 16, b_hi, idesc, k == 0 ? accumulate_first : 1u);
}
// D[tmem] = A[tmem] * B[smem], `steps` (a multiple of 4) of K; b_units: from 32 units of B to the next, in 16 bytes
__device__ __forceinline__ void umma_ts_product(bool leader, uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_units, uint32_t b_hi, uint32_t idesc,
                                                int steps) {
  if (steps == 32) {
    umma_ts_steps<32>(leader, d_tmem, a_tmem, b_lo, b_units, b_hi, idesc, 0u);
    return;
  }
  int k = 0;
  for (; k + 16 <= steps; k += 16) umma_ts_steps<16>(leader, d_tmem, a_tmem + k * 8, b_lo + (k >> 1) * b_units, b_units, b_hi, idesc, k != 0 ? 1u : 0u);
  for (; k < steps; k += 4) umma_ts_steps<4>(leader, d_tmem, a_tmem + k * 8, b_lo + (k >> 1) * b_units, b_units, b_hi, idesc, k != 0 ? 1u : 0u);
}
// D[tmem] += A[smem] * B[smem]
__device__ __forceinline__ void umma_f16_ss_plain(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %2};\n\t"
      "mov.b64 db, {%3, %4};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc)
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]),
      "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]),
      "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
// Gate non-linearities through the special-function unit (ex2 and rcp approximations, relative error ~2^-22, far
// below the fp16 rounding of h and c): an exact expf, IEEE division and tanhf per gate made the 128-thread
// epilogue the longest part of a step.
__device__ __forceinline__ float sigmoid_fast(float x) {
  float e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * -1.4426950408889634f));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
  return r;
}
__device__ __forceinline__ float tanh_fast(float x) {  // 2*sigmoid(2x) - 1
  return fmaf(2.0f, sigmoid_fast(2.0f * x), -1.0f);
}
// the four epilogue warps of a group meet; true if all of them say so
__device__ __forceinline__ bool epilogue_and(int group, bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 q, %1, 0;\n\t"
      "bar.red.and.pred p, %2, 128, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r)
      : "r"(v ? 1u : 0u), "r"(1 + group)
      : "memory");
  return r != 0;
}
// x[k] of lane g of a quad -> x[g'] of lane k: every lane ends with all four gates of its own column
__device__ __forceinline__ void transpose_quad(float (&x)[4], int lane) {
  const bool b0 = lane & 1, b1 = lane & 2;
#pragma unroll
  for (int k = 0; k < 4; k += 2) {
    const float r = __shfl_xor_sync(0xffffffffu, b0 ? x[k] : x[k + 1], 1);
    if (b0) x[k] = r;
    else x[k + 1] = r;
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const float r = __shfl_xor_sync(0xffffffffu, b1 ? x[k] : x[k + 2], 2);
    if (b1) x[k] = r;
    else x[k + 2] = r;
  }
}

// What a cluster does: a layer by itself, or one of two layers that run side by side.
enum LstmRole { kAlone, kFirst, kSecond };

// Shared memory of a CTA, bytes from its start.
struct LstmSmem {
  int h_bytes, group_bytes;       // per group: h of all units [2] (a block per CTA), this CTA's part of h_t [2]
  int w, x, bars, end;            // second layer: W's columns that TMEM has no room for; layer a's steps [kXStages][groups]; barriers
};
constexpr int kXStages = 3;
// K of the second layer's W in TMEM: what the accumulators and R leave
__host__ __device__ constexpr int w_tmem_k(int H) { return H <= 512 - col_r(true) ? H : 2 * (512 - col_r(true) - H / 2); }
__host__ __device__ constexpr LstmSmem lstm_smem(int H, int groups, bool second) {
  LstmSmem l{};
  l.h_bytes = kSeqs * H * 2;
  l.group_bytes = 2 * (l.h_bytes + kSeqs * kUnits * 2);
  l.w = groups * l.group_bytes;
  l.x = l.w + (second ? (H - w_tmem_k(H)) * kGateRows * 2 : 0);
  l.bars = l.x + (second ? kXStages * groups * l.h_bytes : 0);
  l.end = l.bars + 8 * (6 * groups + 2 * kXStages + 4) + 16;
  return l;
}

// G = groups of 16 sequences per cluster.
template <int G, int ROLE>
__device__ __forceinline__ void recurrence(const LstmParams& p, const LstmPairParams* pp, int cluster) {
  constexpr int NB = kSeqs;
  constexpr int kBlock = NB * kUnits * 2;      // one CTA's units of a group: [2 x 8 sequences][4 chunks of 8 units], 8 rows x 16 bytes each
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - raw);
  const LstmSmem lay = lstm_smem(p.H, G, ROLE == kSecond);
  const int h_bytes = lay.h_bytes, group_bytes = lay.group_bytes;
  const uint32_t tmem_cols = ROLE != kAlone ? 512u : (p.H > 384 ? 512u : 256u);  // accumulators, R [, W]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + lay.bars);
  const uint32_t bar0 = smem_u32(bars);                      // per group: h arrived [2], accumulator ready, accumulator drained
  const uint32_t bar_part = bar0 + 32 * G;                   // first layer, per group: part of h_t written, taken
  const uint32_t bar_xfull = bar_part + 16 * G, bar_xempty = bar_xfull + 8 * kXStages;  // second layer: x_t there, used,
  const uint32_t bar_xready = bar_xempty + 8 * kXStages, bar_xdrained = bar_xready + 16;  // W . x_t ready, drained
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(bars + 6 * G + 2 * kXStages + 4);
  volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;  // (uniform for the compiler)
  const int rank = (int)cluster_ctarank();
  const int group0 = cluster * G, row0 = group0 * NB, unit0 = rank * kUnits, n_groups = (p.B + NB - 1) / NB;
  const int groups = min(G, n_groups - group0);
  const bool working = rank < p.ctas;
  constexpr uint32_t kColR = col_r(ROLE == kSecond);

  if (threadIdx.x == 0) {
    for (int i = 0; i < 4 * G; ++i) mbar_init(bar0 + 8 * i, i % 4 == 3 ? 4 : 1);
    for (int i = 0; i < 2 * G + 2 * kXStages + 2; ++i) mbar_init(bar_part + 8 * i, 1);
    for (int i = 0; i < 2; ++i) mbar_init(bar_xdrained + 8 * i, 4 * groups);
    *s_abort = 0;
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(s_tmem), tmem_cols);
    tmem_relinquish();
  }
  griddep_launch_dependents();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *s_tmem;
  [[maybe_unused]] const uint32_t colW = kColR + (uint32_t)p.H / 2;
  // R to TMEM: lane = row = unit * 4 + gate.  W likewise, its last columns to shared memory.
  const auto load_rows = [&](const __half* m, uint32_t col, int k_tmem) {
    const int q = warp & 3;
    const uint4* src = reinterpret_cast<const uint4*>(m + ((size_t)(lane & 3) * p.H + unit0 + q * 8 + (lane >> 2)) * p.H);
    for (int k = 0; k < p.H / 64; ++k) {
      uint4 v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = __ldg(src + k * 8 + i);
      if (k * 64 < k_tmem) {
        tmem_st_32x32(tmem_base + col + k * 32 + ((uint32_t)(q * 32) << 16), reinterpret_cast<const uint32_t (&)[32]>(v));
      } else if (ROLE == kSecond) {
#pragma unroll
        for (int i = 0; i < 8; ++i) reinterpret_cast<uint4*>(sm + lay.w)[((k * 64 - k_tmem) / 8 + i) * kGateRows + q * 32 + lane] = v[i];
      }
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  };
  constexpr int kWWarp = G == 1 ? G : G + 4;
  if (working && warp >= G && warp < G + 4) load_rows(p.R, kColR, p.H);
  if (ROLE == kSecond && working && warp >= kWWarp && warp < kWWarp + 4) load_rows(pp->W, colW, w_tmem_k(p.H));
  griddep_wait();  // (the weights are what the plan was given at load time; the rest comes from the launches before this one)
  if (working) {
    // h_{-1}, as step -1 would have delivered it (buffer 1)
    for (int i = threadIdx.x; i < G * h_bytes / 16; i += blockDim.x) {
      const int g = i / (h_bytes / 16), k = i - g * (h_bytes / 16), chunk = (k >> 6) * 4 + (k >> 3 & 3), b = row0 + g * NB + (k >> 5 & 1) * 8 + (k & 7);
      uint4 v = make_uint4(0, 0, 0, 0);
      if (p.h0 && b < p.B) v = *reinterpret_cast<const uint4*>(p.h0 + (size_t)b * p.H + chunk * 8);
      reinterpret_cast<uint4*>(sm + g * group_bytes + h_bytes)[k] = v;
    }
  }
  fence_proxy_async_smem();
  tc_fence_before();
  cluster_sync_all();  // barriers and R are there, and every CTA has read the initial h
  tc_fence_after();

  if (working && warp < G) {
    // ------------------------------------------------------------------ MMA issuer of a group
    // (all lanes run the loop with identical values, one elected lane issues: see elect_one.  A warp per group: one warp
    // for all of them left the tensor pipe idle for 200 clk between two groups, and waited for them in one order.)
    if (warp < groups) {
      constexpr uint32_t idesc = umma_idesc_f16(kGateRows, NB);
      const bool leader = elect_one();
      const uint32_t bar_h = bar0 + 32 * warp, d = tmem_base + warp * NB;
      const uint32_t part_bytes = p.B - row0 - warp * NB > NB / 2 ? kBlock : kBlock / 2;
      for (int t = 0; t < p.T; ++t) {
        const uint32_t prev = (uint32_t)(t + 1) & 1u;  // buffer of h_{t-1}
        if (leader && t + 1 < p.T) mbar_expect_tx(bar_h + 8 * (t & 1), p.ctas * part_bytes);
        if (t > 0 && !(mbar_wait_bounded_cl(bar_h + 8 * prev, (uint32_t)((t - 1) >> 1) & 1u, s_abort, p.gerr, 404) &&
                       mbar_wait_bounded(bar_h + 24, (uint32_t)(t - 1) & 1u, s_abort, p.gerr, 403)))
          break;
        tc_fence_after();
        const uint32_t h = plain_lo(base + warp * group_bytes + prev * h_bytes, 128);
        umma_ts_product(leader, d, tmem_base + kColR, h, kBlock / 16, plain_hi(512), idesc, p.H / 16);
        if (leader) umma_commit(bar_h + 16);
      }
    }
  } else if (ROLE == kSecond && working && warp == 5 * G) {
    // ------------------------------------------------------------------ W . x_t of all groups at once, a step or more ahead
    const uint32_t idesc = groups == 2 ? umma_idesc_f16(kGateRows, 2 * NB) : umma_idesc_f16(kGateRows, NB), x_hi = plain_hi(p.H * 16);
    const uint32_t w = plain_lo(base + lay.w, kGateRows * 16);
    const int k_tmem = w_tmem_k(p.H);
    const bool leader = elect_one();
    for (int t = 0; t < p.T; ++t) {
      const int stage = t % kXStages;
      if (!mbar_wait_bounded(bar_xfull + 8 * stage, (uint32_t)(t / kXStages) & 1u, s_abort, p.gerr, 406) ||
          !mbar_wait_bounded(bar_xdrained + 8 * (t & 1), (uint32_t)((t >> 1) + 1) & 1u, s_abort, p.gerr, 411))
        break;
      tc_fence_after();
      const uint32_t d = tmem_base + kColX + (t & 1) * 2 * NB, x = plain_lo(base + lay.x + stage * G * h_bytes, 128);
      umma_ts_product(leader, d, tmem_base + colW, x, 32, x_hi, idesc, k_tmem / 16);
#pragma unroll 4
      for (int k = k_tmem / 16; k < p.H / 16; ++k)
        if (leader) umma_f16_ss_plain(d, w + (k - k_tmem / 16) * 2 * kGateRows, plain_hi(128), x + k * 16, x_hi, idesc);
      if (leader) umma_commit(bar_xempty + 8 * stage);
      if (leader) umma_commit(bar_xready + 8 * (t & 1));
    }
  } else if (ROLE == kSecond && working && warp == 5 * G + 1) {
    // ------------------------------------------------------------------ layer a's steps to shared memory
    if (elect_one()) {
      bool ok = true;
      for (int t = 0; t < p.T && ok; ++t) {
        const int stage = t % kXStages;
        const uint32_t full = bar_xfull + 8 * stage;
        ok = mbar_wait_bounded(bar_xempty + 8 * stage, (uint32_t)(t / kXStages + 1) & 1u, s_abort, p.gerr, 407);
        if (!ok) break;
        mbar_expect_tx(full, (uint32_t)(groups * h_bytes));
        for (int g = 0; g < groups; ++g) {
          const unsigned int target = (unsigned int)p.ctas * (unsigned int)(t + 1);
          const unsigned int* counter = pp->counters + group0 + g;
          if (ld_acquire_gpu(counter) < target) {
            const long long t0 = clock64();
            while (ok && ld_acquire_gpu(counter) < target) {
              if (*s_abort) ok = false;
              else if (clock64() - t0 > AIG_WAIT_CYCLES) {
                *s_abort = 1;
                atomicCAS(p.gerr, 0, 408);
                ok = false;
              } else __nanosleep(40);
            }
          }
          if (!ok) break;
          fence_proxy_async_global();  // written with ordinary stores, read by the bulk copy
          bulk_load(base + lay.x + (stage * G + g) * h_bytes, pp->xs + ((size_t)t * n_groups + group0 + g) * NB * p.H, (uint32_t)h_bytes, full);
        }
      }
    }
    __syncwarp();
  } else if (ROLE == kFirst && working && warp == 5 * G) {
    // ------------------------------------------------------------------ this CTA's part of h_t to the second layer
    // (a warp of its own: the release waits for the stores)
    const uint4* stage = reinterpret_cast<const uint4*>(sm + 2 * h_bytes);
    __half* dst = pp->xs + (size_t)group0 * NB * p.H + (unit0 + lane) * 8;
    bool ok = true;
    for (int t = 0; t < p.T && ok; ++t) {
      for (int g = 0; g < groups && ok; ++g) {
        const uint32_t bar = bar_part + 16 * g;
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(bar, (uint32_t)t & 1u, s_abort, p.gerr, 409));
        if (!ok) break;
        const uint4* src = stage + (g * group_bytes + (t & 1) * kBlock) / 16 + lane;
        const uint4 v0 = src[0], v1 = src[32];
        __syncwarp();
        if (lane == 0) mbar_arrive(bar + 8);
        __half* d = dst + ((size_t)t * n_groups + g) * NB * p.H;
        *reinterpret_cast<uint4*>(d) = v0;
        *reinterpret_cast<uint4*>(d + NB / 2 * p.H) = v1;
      }
      // one release for all groups: it waits for the stores to land, about 1500 clk
      fence_proxy_async_global();
      __syncwarp();
      if (ok && lane < groups) red_release_gpu_add(pp->counters + group0 + lane, 1u);
    }
  } else if (working && warp < 5 * G && (warp - G) >> 2 < groups) {
    // ------------------------------------------------------------------ gates: one thread per gate row
    const int group = (warp - G) >> 2, w4 = (warp - G) & 3, q = warp & 3, tid = w4 * 32 + lane, seq0 = row0 + group * NB;
    const uint32_t sH = base + group * group_bytes, bar_h = bar0 + 32 * group;
    const int n_seq = p.B - seq0;
    const uint32_t part_bytes = n_seq > NB / 2 ? kBlock : kBlock / 2;
    uint8_t* stage = sm + group * group_bytes + 2 * h_bytes;
    const int gate = lane & 3, unit = q * 8 + (lane >> 2);
    // sigmoid(x), or 2*sigmoid(2x) - 1 on the lanes of the g gate
    const float in_scale = gate == 2 ? 2.0f : 1.0f, out_scale = in_scale, out_shift = gate == 2 ? -1.0f : 0.0f;
    const float* gsrc = ROLE == kSecond ? pp->bias + (size_t)gate * p.H + unit0 + unit : p.gx + (size_t)gate * p.H + unit0 + unit;
    float c[NB / 4], gx[NB];
#pragma unroll
    for (int j = 0; j < NB / 4; ++j) {  // this lane's cells: its unit of sequences gate, gate + 4, ...
      const int b = seq0 + 4 * j + gate;
      c[j] = p.c0 && b < p.B ? __half2float(p.c0[(size_t)b * p.H + unit0 + unit]) : 0.f;
    }
    const float bias = ROLE == kSecond ? __ldg(gsrc) : 0.f;
    if (ROLE != kSecond) {
#pragma unroll
      for (int n = 0; n < NB; ++n) gx[n] = seq0 + n < p.B ? __ldg(gsrc + (size_t)(seq0 + n) * p.gx_sB) : 0.f;
    }
    const uint32_t t_addr = tmem_base + group * NB + ((uint32_t)(q * 32) << 16);
    bool ok = true;
    for (int t = 0; t < p.T && ok; ++t) {
      // (what is there early comes before the wait for R . h)
      if (ROLE == kFirst && t > 0) ok = mbar_wait_bounded(bar_part + 16 * group + 8, (uint32_t)(t - 1) & 1u, s_abort, p.gerr, 410);
      if (ROLE == kSecond) ok = mbar_wait_bounded(bar_xready + 8 * (t & 1), (uint32_t)(t >> 1) & 1u, s_abort, p.gerr, 412);
      ok = mbar_wait_bounded(bar_h + 16, (uint32_t)t & 1u, s_abort, p.gerr, 405) && ok;
      tc_fence_after();
      uint32_t r[NB];
      tmem_ld_32x16(t_addr, r);
      if (ROLE == kSecond) tmem_ld_32x16(tmem_base + kColX + ((t & 1) * 2 + group) * NB + ((uint32_t)(q * 32) << 16), reinterpret_cast<uint32_t (&)[NB]>(gx));
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_h + 24);
      if (ROLE == kSecond) {
        if (lane == 0) mbar_arrive(bar_xdrained + 8 * (t & 1));
#pragma unroll
        for (int n = 0; n < NB; ++n) gx[n] += bias;
      }
      __half* st = reinterpret_cast<__half*>(stage + (t & 1) * kBlock);
      auto cells = [&](int j) {  // sequences 4j .. 4j + 3
        float x[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] = fmaf(sigmoid_fast(in_scale * (__uint_as_float(r[4 * j + k]) + gx[4 * j + k])), out_scale, out_shift);
        transpose_quad(x, lane);
        float cn = x[1] * c[j] + x[0] * x[2];
        if (p.clip > 0.f) cn = fminf(p.clip, fmaxf(-p.clip, cn));
        c[j] = __half2float(__float2half(cn));
        const int n = 4 * j + gate;
        st[((n >> 3) * 4 + q) * 64 + (n & 7) * 8 + (lane >> 2)] = __float2half(x[3] * tanh_fast(c[j]));
      };
      if (n_seq > 8) {  // (without branches in between: they interleave)
        cells(0);
        cells(1);
        cells(2);
        cells(3);
      } else {
        cells(0);
        if (n_seq > 4) cells(1);
      }
      fence_proxy_async_smem();
      ok = epilogue_and(group, ok);
      if (!ok) break;
      if (ROLE == kFirst && tid == 0) mbar_arrive(bar_part + 16 * group);
      // (four warps issue: the copies of one warp's lanes go out one after another)
      const int dst = (lane << 2) | w4;
      if (t + 1 < p.T && dst < p.ctas)
        bulk_to_cluster(mapa_shared(sH + (uint32_t)((t & 1) * h_bytes + rank * kBlock), (uint32_t)dst), smem_u32(st), part_bytes,
                        mapa_shared(bar_h + 8 * (t & 1), (uint32_t)dst));
      // under the delivery: this step's h to memory (16 bytes of a sequence per thread), the next step's projection
      if (ROLE != kSecond && t + 1 < p.T) {
        const float* g1 = gsrc + (size_t)(t + 1) * p.gx_sT;
#pragma unroll
        for (int n = 0; n < NB; ++n)
          if (seq0 + n < p.B) gx[n] = __ldg(g1 + (size_t)(seq0 + n) * p.gx_sB);
      }
      if (tid < 4 * NB) {
        const int chunk = tid >> 3 & 3, b = seq0 + (tid >> 5) * 8 + (tid & 7);
        const uint4 v = reinterpret_cast<const uint4*>(st)[tid];
        if (b < p.B) {
          if (ROLE != kFirst) *reinterpret_cast<uint4*>(p.y + (size_t)t * p.y_sT + (size_t)b * p.y_sB + unit0 + chunk * 8) = v;
          if (t == p.T - 1 && p.hT) *reinterpret_cast<uint4*>(p.hT + (size_t)b * p.H + unit0 + chunk * 8) = v;
        }
      }
    }
    if (ok && p.cT)
#pragma unroll
      for (int j = 0; j < NB / 4; ++j) {
        const int b = seq0 + 4 * j + gate;
        if (b < p.B) p.cT[(size_t)b * p.H + unit0 + unit] = __float2half(c[j]);
      }
  }

  if (*s_abort) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // no CTA leaves while another may still write to it
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem_base, tmem_cols);
  }
}

// One layer.  G = groups of 16 sequences per cluster: 1 or 2.
template <int G>
__global__ void __launch_bounds__(lstm_threads(G), 1) lstm_recurrent_kernel(const LstmParams p) {
  uint32_t n_ctarank;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n_ctarank));
  recurrence<G, kAlone>(p, nullptr, (int)(blockIdx.x / n_ctarank));
}

// Two layers: clusters of the first do what lstm_recurrent_kernel does and write each h_t where the bulk copies of the
// second layer's clusters find it as an operand; those run a step or two behind and multiply W . x_t themselves.
template <int GA, int GB>
__global__ void __launch_bounds__(pair_threads(GA, GB), 1) lstm_pair_kernel(const __grid_constant__ LstmPairParams pp) {
  uint32_t n_ctarank;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n_ctarank));
  const int cluster = (int)(blockIdx.x / n_ctarank);
  if (cluster < pp.a_clusters) recurrence<GA, kFirst>(pp.a, &pp, cluster);
  else recurrence<GB, kSecond>(pp.b, &pp, cluster - pp.a_clusters);
  // The last cluster to end (all counting is over then) leaves the counters as it found them, also after a wait that ran out.
  if (cluster_ctarank() == 0 && threadIdx.x == 0) {
    const int n_groups = (pp.a.B + kSeqs - 1) / kSeqs;
    unsigned int done;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(done) : "l"(pp.counters + n_groups) : "memory");
    if (done + 1 == (unsigned int)pp.clusters)
      for (int i = 0; i <= n_groups; ++i) pp.counters[i] = 0u;
  }
}

// Shape of a recurrence launch.
struct LstmLaunch {
  int groups = 1, ctas = 0, cluster = 0;
  size_t smem = 0;
  // two layers side by side: groups per cluster of the first and the second (0: one layer after the other)
  int pair_a = 0, pair_b = 0;
  size_t pair_smem = 0;
};
// (a CTA's shared memory keeps more of them off its SM than TMEM has columns for: one that waits there for another cluster's
// TMEM would make its own cluster wait, too)
size_t recurrent_smem(int H, int groups) {
  const size_t n = (size_t)lstm_smem(H, groups, false).end + 1024, least = (H > 384 ? 116 : 77) * 1024;
  return n < least ? least : n;
}
// (more than half of an SM's: a CTA takes all TMEM columns, so that a second one on its SM could not start)
size_t pair_smem(int H, int ga, int gb) {
  size_t n = lstm_smem(H, ga, false).end;
  if (n < (size_t)lstm_smem(H, gb, true).end) n = lstm_smem(H, gb, true).end;
  return (n < 116 * 1024 ? 116 * 1024 : n) + 1024;
}

int cluster_config(aig_ctx* ctx, const void* kernel, int cluster, int clusters, int threads, size_t smem, bool cooperative, cudaLaunchConfig_t* cfg,
                   cudaLaunchAttribute (&attr)[3]) {
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1] = pdl_attribute(ctx);
  attr[2].id = cudaLaunchAttributeCooperative;
  attr[2].val.cooperative = 1;
  *cfg = cudaLaunchConfig_t{};
  cfg->gridDim = dim3(clusters * cluster);
  cfg->blockDim = dim3(threads);
  cfg->dynamicSmemBytes = smem;
  cfg->stream = ctx->stream;
  cfg->attrs = attr;
  cfg->numAttrs = cooperative ? 3 : 2;
  AIG_CUDA_OK(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  AIG_CUDA_OK(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  return AIG_OK;
}
template <int G>
int recurrent_config(aig_ctx* ctx, const LstmLaunch& l, int batch, cudaLaunchConfig_t* cfg, cudaLaunchAttribute (&attr)[3]) {
  return cluster_config(ctx, (const void*)lstm_recurrent_kernel<G>, l.cluster, ceil_div(batch, G * kSeqs), lstm_threads(G), l.smem, false, cfg, attr);
}
template <int GA, int GB>
int pair_config(aig_ctx* ctx, const LstmLaunch& l, int batch, cudaLaunchConfig_t* cfg, cudaLaunchAttribute (&attr)[3]) {
  return cluster_config(ctx, (const void*)lstm_pair_kernel<GA, GB>, l.cluster, ceil_div(batch, GA * kSeqs) + ceil_div(batch, GB * kSeqs),
                        pair_threads(GA, GB), l.pair_smem, true, cfg, attr);
}

// One group of sequences per cluster, or two where the clusters of one group would not all run at once.
int recurrent_shape(aig_ctx* ctx, int H, int batch, LstmLaunch* l) {
  l->ctas = H / kUnits;
  l->cluster = 1;
  while (l->cluster < l->ctas) l->cluster *= 2;
  l->groups = 1;
  l->smem = recurrent_smem(H, 1);
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[3];
  int rc = recurrent_config<1>(ctx, *l, batch, &cfg, attr), n = 0;
  if (rc != AIG_OK) return rc;
  AIG_CUDA_OK(ctx, cudaOccupancyMaxActiveClusters(&n, lstm_recurrent_kernel<1>, &cfg));
  if (n < 1) return aig_fail(ctx, AIG_ERR_UNSUPPORTED, "lstm: no cluster of %d CTAs fits this device", l->cluster);
  if (ceil_div(batch, kSeqs) > n) {
    l->groups = 2;
    l->smem = recurrent_smem(H, 2);
  }
  return AIG_OK;
}

// The fewest groups per cluster with which the clusters of both layers run at once.
template <int GA, int GB>
int try_pair(aig_ctx* ctx, int H, int batch, LstmLaunch* l) {
  if (l->pair_a) return AIG_OK;
  LstmLaunch t = *l;
  t.pair_a = GA;
  t.pair_b = GB;
  t.pair_smem = pair_smem(H, GA, GB);
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[3];
  int rc = pair_config<GA, GB>(ctx, t, batch, &cfg, attr), n = 0;
  if (rc != AIG_OK) return rc;
  AIG_CUDA_OK(ctx, cudaOccupancyMaxActiveClusters(&n, lstm_pair_kernel<GA, GB>, &cfg));
  if ((int)cfg.gridDim.x <= n * t.cluster) *l = t;
  return AIG_OK;
}
int pair_shape(aig_ctx* ctx, int H, int batch, LstmLaunch* l) {
  int rc = try_pair<1, 1>(ctx, H, batch, l);
  if (rc == AIG_OK) rc = try_pair<2, 2>(ctx, H, batch, l);
  if (rc == AIG_OK) rc = try_pair<3, 2>(ctx, H, batch, l);
  return rc;
}

template <int G>
int launch_recurrent(aig_ctx* ctx, const LstmLaunch& l, const LstmParams& prm) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[3];
  const int rc = recurrent_config<G>(ctx, l, prm.B, &cfg, attr);
  if (rc != AIG_OK) return rc;
  AIG_CUDA_OK(ctx, cudaLaunchKernelEx(&cfg, lstm_recurrent_kernel<G>, prm));
  return AIG_OK;
}
int run_recurrent(aig_ctx* ctx, const LstmLaunch& l, LstmParams prm) {
  prm.ctas = l.ctas;
  prm.gerr = ctx->d_err;
  return l.groups == 1 ? launch_recurrent<1>(ctx, l, prm) : launch_recurrent<2>(ctx, l, prm);
}
template <int GA, int GB>
int launch_pair(aig_ctx* ctx, const LstmLaunch& l, LstmPairParams& pp) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[3];
  const int rc = pair_config<GA, GB>(ctx, l, pp.a.B, &cfg, attr);
  if (rc != AIG_OK) return rc;
  pp.a_clusters = ceil_div(pp.a.B, GA * kSeqs);
  pp.clusters = (int)cfg.gridDim.x / l.cluster;
  AIG_CUDA_OK(ctx, cudaLaunchKernelEx(&cfg, lstm_pair_kernel<GA, GB>, pp));
  return AIG_OK;
}
// sum of a layer's biases, for a second layer (it has no projection to add them)
__global__ void bias_sum_kernel(float* out, const __half* bw, const __half* br, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = __half2float(bw[i]) + (br ? __half2float(br[i]) : 0.f);
}
int run_pair(aig_ctx* ctx, const LstmLaunch& l, LstmPairParams pp) {
  pp.a.ctas = pp.b.ctas = l.ctas;
  pp.a.gerr = pp.b.gerr = ctx->d_err;
  if (l.pair_a == 1) return launch_pair<1, 1>(ctx, l, pp);
  return l.pair_a == 2 ? launch_pair<2, 2>(ctx, l, pp) : launch_pair<3, 2>(ctx, l, pp);
}

}  // namespace

struct aig_lstm_plan {
  aig_ctx* ctx = nullptr;
  int T = 0, L = 0, H = 0, B = 0, in_c = 0;
  float clip = 0.f;
  bool double_bias = true, batch_major = false;
  LstmLaunch shape;
  const __half* blob = nullptr;
  std::vector<size_t> w_off, r_off, bw_off, br_off;
  std::vector<aig_conv_plan*> proj;     // hoisted input projection per layer; none of a pair's second layer
  float* gx = nullptr;                  // [T*B][4H] fp32 scratch
  __half* mid = nullptr;                // outputs that a further layer or pair reads (same layout as y); null: there is none
  __half* xs = nullptr;                 // layers in pairs: the first one's outputs as the second one's operands
  unsigned int* counters = nullptr;     // and how far they are
  float* pair_bias = nullptr;           // per pair the second layer's [4H]
  bool second(int l) const { return shape.pair_a != 0 && (l & 1); }  // (layers 0 and 1, 2 and 3, ...)
};

extern "C" {

size_t aig_lstm_weight_count(int in_c, int hidden, int layers, int double_bias) {
  size_t n = 0;
  for (int l = 0; l < layers; ++l) n += (size_t)4 * hidden * (l == 0 ? in_c : hidden) + (size_t)4 * hidden * hidden;
  n += (size_t)layers * 4 * hidden * (double_bias ? 2 : 1);
  return n;
}

int aig_lstm_plan_create(aig_ctx* ctx, int seq_len, int layers, int hidden, int batch, int in_c, float clip, int double_bias,
                         int batch_major, aig_lstm_plan** out) {
  if (!ctx || !out) return AIG_ERR_INVALID;
  *out = nullptr;
  DeviceGuard g(ctx->device);
  AIG_REQUIRE(ctx, seq_len > 0 && layers > 0 && hidden > 0 && batch > 0 && in_c > 0, "lstm plan: bad extents");
  if (hidden % 64 != 0 || hidden > 512)
    return aig_fail(ctx, AIG_ERR_UNSUPPORTED, "lstm plan: hidden must be a multiple of 64 and at most 512 (got %d)", hidden);
  if (in_c % 16 != 0) return aig_fail(ctx, AIG_ERR_UNSUPPORTED, "lstm plan: in_c must be a multiple of 16 (got %d)", in_c);
  aig_lstm_plan* pl = new aig_lstm_plan();
  pl->ctx = ctx;
  pl->T = seq_len; pl->L = layers; pl->H = hidden; pl->B = batch; pl->in_c = in_c;
  pl->clip = clip; pl->double_bias = double_bias != 0; pl->batch_major = batch_major != 0;
  int rc = recurrent_shape(ctx, hidden, batch, &pl->shape);
  if (rc == AIG_OK && layers > 1) rc = pair_shape(ctx, hidden, batch, &pl->shape);
  if (rc != AIG_OK) {
    delete pl;
    return rc;
  }
  size_t off = 0;
  for (int l = 0; l < layers; ++l) {
    pl->w_off.push_back(off);
    off += (size_t)4 * hidden * (l == 0 ? in_c : hidden);
    pl->r_off.push_back(off);
    off += (size_t)4 * hidden * hidden;
  }
  for (int l = 0; l < layers; ++l) {
    pl->bw_off.push_back(off);
    off += (size_t)4 * hidden;
    pl->br_off.push_back(off);
    if (pl->double_bias) off += (size_t)4 * hidden;
  }
  for (int l = 0; l < layers && rc == AIG_OK; ++l) {
    aig_conv_plan* fp = nullptr;
    if (pl->second(l)) {
      pl->proj.push_back(nullptr);
      continue;
    }
    rc = aig_fc_plan_create(ctx, seq_len * batch, l == 0 ? in_c : hidden, 4 * hidden, AIG_ACT_NONE, 0.f, 0, &fp);
    if (rc == AIG_OK) {
      aig_fc_plan_set_output_f32(fp, 1);
      fc_plan_use_skinny(fp, false);  // a sequence in pieces gives the bits of the whole
      pl->proj.push_back(fp);
    }
  }
  const size_t seq = (size_t)seq_len * batch;
  const bool between = layers > (pl->shape.pair_a ? 2 : 1);
  if (rc == AIG_OK && (cudaMalloc(&pl->gx, seq * 4 * hidden * sizeof(float)) != cudaSuccess ||
                       (between && cudaMalloc(&pl->mid, seq * hidden * sizeof(__half)) != cudaSuccess)))
    rc = aig_fail(ctx, AIG_ERR_CUDA, "lstm plan: device allocation failed");
  const size_t groups = ceil_div(batch, kSeqs), words = (groups + 1) * sizeof(unsigned int);
  if (rc == AIG_OK && pl->shape.pair_a &&
      (cudaMalloc(&pl->xs, groups * kSeqs * seq_len * hidden * sizeof(__half)) != cudaSuccess || cudaMalloc(&pl->counters, words) != cudaSuccess ||
       cudaMalloc(&pl->pair_bias, (size_t)(layers / 2) * 4 * hidden * sizeof(float)) != cudaSuccess ||
       cudaMemsetAsync(pl->counters, 0, words, ctx->stream) != cudaSuccess))
    rc = aig_fail(ctx, AIG_ERR_CUDA, "lstm plan: device allocation failed");
  if (rc != AIG_OK) {
    aig_lstm_plan_destroy(pl);
    return rc;
  }
  *out = pl;
  return AIG_OK;
}

int aig_lstm_plan_pair_groups(const aig_lstm_plan* pl, int* first, int* second) {
  if (!pl || !first || !second) return AIG_ERR_INVALID;
  *first = pl->shape.pair_a;
  *second = pl->shape.pair_b;
  return AIG_OK;
}

int aig_lstm_plan_destroy(aig_lstm_plan* pl) {
  if (!pl) return AIG_OK;
  DeviceGuard g(pl->ctx->device);
  cudaStreamSynchronize(pl->ctx->stream);
  for (aig_conv_plan* fp : pl->proj) aig_conv_plan_destroy(fp);
  cudaFree(pl->gx);
  cudaFree(pl->mid);
  cudaFree(pl->xs);
  cudaFree(pl->counters);
  cudaFree(pl->pair_bias);
  delete pl;
  return AIG_OK;
}

int aig_lstm_plan_set_weights(aig_lstm_plan* pl, const aig_half* blob) {
  if (!pl) return AIG_ERR_INVALID;
  aig_ctx* ctx = pl->ctx;
  DeviceGuard g(ctx->device);
  AIG_REQUIRE(ctx, blob != nullptr && ((uintptr_t)blob & 15) == 0, "lstm set_weights: blob must be non-null and 16-byte aligned");
  pl->blob = (const __half*)blob;
  for (int l = 0; l < pl->L; ++l) {
    if (pl->second(l)) {
      const int n = 4 * pl->H;
      bias_sum_kernel<<<ceil_div(n, 128), 128, 0, ctx->stream>>>(pl->pair_bias + (size_t)(l / 2) * n, (const __half*)blob + pl->bw_off[l],
                                                                 pl->double_bias ? (const __half*)blob + pl->br_off[l] : nullptr, n);
      AIG_LAUNCH_OK(ctx);
      continue;
    }
    int rc = aig_fc_plan_set_weights_out_in(pl->proj[l], blob + pl->w_off[l], blob + pl->bw_off[l]);
    if (rc != AIG_OK) return rc;
    if (pl->double_bias && (rc = aig_fc_plan_add_bias(pl->proj[l], blob + pl->br_off[l])) != AIG_OK) return rc;
  }
  return AIG_OK;
}

// x: [T][B][in] (or [B][T][in] when the plan is batch-major); y: [T][B][H] (or [B][T][H]).
// h_state/c_state: [layers][B][H] fp16 or null; read when use_state != 0, always written when non-null.
int aig_lstm_forward(aig_lstm_plan* pl, const aig_half* x, aig_half* y, aig_half* h_state, aig_half* c_state, int use_state) {
  if (!pl) return AIG_ERR_INVALID;
  aig_ctx* ctx = pl->ctx;
  DeviceGuard g(ctx->device);
  AIG_REQUIRE(ctx, x && y && pl->blob, "lstm forward: null pointer or weights not set");
  AIG_REQUIRE(ctx, ((uintptr_t)x & 15) == 0 && ((uintptr_t)y & 15) == 0, "lstm forward: tensors must be 16-byte aligned");
  AIG_REQUIRE(ctx, (h_state == nullptr) == (c_state == nullptr), "lstm forward: give both state tensors or neither");
  AIG_REQUIRE(ctx, !use_state || h_state, "lstm forward: use_state needs the state tensors");
  const int T = pl->T, B = pl->B, H = pl->H;
  const long long sT = pl->batch_major ? H : (long long)B * H, sB = pl->batch_major ? (long long)T * H : H;
  auto layer = [&](int l) {
    LstmParams prm{};
    prm.T = T; prm.B = B; prm.H = H;
    prm.clip = pl->clip;
    prm.R = pl->blob + pl->r_off[l];
    prm.gx = pl->gx;
    // the projection's rows follow x's memory order
    prm.gx_sT = pl->batch_major ? (long long)4 * H : (long long)B * 4 * H;
    prm.gx_sB = pl->batch_major ? (long long)T * 4 * H : (long long)4 * H;
    // a middle layer may read and write `mid`: its input is fully consumed by the hoisted projection
    // before the recurrence starts overwriting it (a pair's first layer writes `xs` instead)
    prm.y = (l == pl->L - 1) ? (__half*)y : pl->mid;
    prm.y_sT = sT; prm.y_sB = sB;
    prm.h0 = use_state ? (const __half*)h_state + (size_t)l * B * H : nullptr;
    prm.c0 = use_state ? (const __half*)c_state + (size_t)l * B * H : nullptr;
    prm.hT = h_state ? (__half*)h_state + (size_t)l * B * H : nullptr;
    prm.cT = c_state ? (__half*)c_state + (size_t)l * B * H : nullptr;
    return prm;
  };
  const __half* in = (const __half*)x;
  for (int l = 0; l < pl->L;) {
    int rc = aig_conv_forward(pl->proj[l], (const aig_half*)in, nullptr, (aig_half*)pl->gx);
    if (rc != AIG_OK) return rc;
    const LstmParams first = layer(l++);
    in = first.y;
    if (pl->shape.pair_a && l < pl->L) {
      LstmPairParams pp{};
      pp.a = first;
      pp.b = layer(l);
      pp.W = pl->blob + pl->w_off[l];
      pp.bias = pl->pair_bias + (size_t)(l / 2) * 4 * H;
      pp.xs = pl->xs;
      pp.counters = pl->counters;
      in = pp.b.y;
      ++l;
      rc = run_pair(ctx, pl->shape, pp);
    } else {
      rc = run_recurrent(ctx, pl->shape, first);
    }
    if (rc != AIG_OK) return rc;
  }
  return AIG_OK;
}

}  // extern "C"

// =============================================================================================
// Allocation-free single-layer LSTM forward.
//
// For callers that must not allocate device memory once they are running: a frame loop that shares
// the GPU with the game it plays (cudaMalloc/cudaFree synchronise the whole device and stall every
// other stream, and the game may already own nearly all of the memory), or a host application that
// reserves its whole device budget at start-up and forbids later allocations.  Everything the plan
// based entry points keep in a cudaMalloc'ed buffer -- the hoisted input projection -- lives here in one fixed array in
// the library's device image.
//
// The array is part of the module: every GPU that loads the library holds kNoAllocBytes until the
// process exits.  All calls on a device share it, so two calls that overlap on the GPU (different
// streams) race; serialise them.  It keeps the previous call's contents; each call writes what it reads.
namespace {

constexpr size_t kNoAllocProjFloats = (size_t)1 << 19;                       // 2 MiB of fp32 projections
constexpr int kNoAllocMaxBatch = 128;
constexpr int kNoAllocMaxHidden = 512;
constexpr size_t kNoAllocProjBytes = kNoAllocProjFloats * sizeof(float);
constexpr size_t kNoAllocBytes = kNoAllocProjBytes;

// In host code this name is only a handle for the runtime's symbol table, not a device address: the
// device address is fetched once per device with cudaGetSymbolAddress below and that is what kernels get.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

unsigned char* g_noalloc_ptr[64] = {};  // per device, filled by the first call on that device

// gx[row][j] = sum_k x[row][k] * W[j][k] + bW[j] (+ bR[j]); 32x32 output tile per block, fp32 accumulate.
__global__ void noalloc_projection_kernel(const __half* __restrict__ x, const __half* __restrict__ W,
                                          const __half* __restrict__ bW, const __half* __restrict__ bR,
                                          float* __restrict__ gx, int rows, int in_c, int out_c) {
  __shared__ float sx[32][33], sw[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8 threads
  const int row0 = blockIdx.y * 32, col0 = blockIdx.x * 32;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int k0 = 0; k0 < in_c; k0 += 32) {
    for (int i = ty; i < 32; i += 8) {
      const int r = row0 + i, c = col0 + i, k = k0 + tx;
      sx[i][tx] = (r < rows && k < in_c) ? __half2float(x[(size_t)r * in_c + k]) : 0.f;
      sw[i][tx] = (c < out_c && k < in_c) ? __half2float(W[(size_t)c * in_c + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < 32; ++kk) {
      const float wv = sw[tx][kk];
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i] = fmaf(sx[ty + 8 * i][kk], wv, acc[i]);
    }
    __syncthreads();
  }
  const int c = col0 + tx;
  if (c < out_c) {
    const float b = __half2float(bW[c]) + (bR ? __half2float(bR[c]) : 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = row0 + ty + 8 * i;
      if (r < rows) gx[(size_t)r * out_c + c] = acc[i] + b;
    }
  }
}

}  // namespace

extern "C" {

// Single-layer, seq-major LSTM forward with zero initial state: x [T][B][in] -> y [T][B][hidden], the blob
// laid out as aig_lstm_plan_set_weights expects for one layer.  Asynchronous on the context's stream; no
// device or pinned memory is allocated or freed.  The first call on a device resolves the scratch array's
// device address (cudaGetSymbolAddress); make that first call before any stream capture begins.
int aig_lstm_forward_noalloc(aig_ctx* ctx, const aig_half* x, const aig_half* blob, aig_half* y, int seq_len, int batch,
                             int in_c, int hidden, float clip, int double_bias) {
  if (!ctx) return AIG_ERR_INVALID;
  DeviceGuard g(ctx->device);
  AIG_REQUIRE(ctx, x && blob && y && seq_len > 0 && batch > 0 && in_c > 0 && hidden > 0, "lstm noalloc: bad arguments");
  AIG_REQUIRE(ctx, ((uintptr_t)x & 15) == 0 && ((uintptr_t)y & 15) == 0 && ((uintptr_t)blob & 15) == 0,
              "lstm noalloc: tensors must be 16-byte aligned");
  if (hidden % 64 != 0 || hidden > kNoAllocMaxHidden)
    return aig_fail(ctx, AIG_ERR_UNSUPPORTED, "lstm noalloc: hidden must be a multiple of 64 and at most %d (got %d)", kNoAllocMaxHidden, hidden);
  if (batch > kNoAllocMaxBatch)
    return aig_fail(ctx, AIG_ERR_UNSUPPORTED, "lstm noalloc: batch %d exceeds the maximum of %d", batch, kNoAllocMaxBatch);
  if (in_c % 8 != 0) return aig_fail(ctx, AIG_ERR_UNSUPPORTED, "lstm noalloc: in_c must be a multiple of 8 (got %d)", in_c);
  const size_t proj = (size_t)seq_len * batch * 4 * hidden;
  if (proj > kNoAllocProjFloats)
    return aig_fail(ctx, AIG_ERR_UNSUPPORTED,
                    "lstm noalloc: seq_len*batch*4*hidden = %zu exceeds the fixed scratch of %zu floats (%zu bytes)", proj,
                    kNoAllocProjFloats, kNoAllocProjBytes);
  // ---- once per device: resolve the symbol, set the kernel's shared-memory limit
  unsigned char*& base = g_noalloc_ptr[ctx->device & 63];
  if (!base) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) return aig_fail(ctx, AIG_ERR_CUDA, "lstm noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
    base = static_cast<unsigned char*>(p);
  }
  LstmLaunch shape;
  int rc = recurrent_shape(ctx, hidden, batch, &shape);
  if (rc != AIG_OK) return rc;
  float* gx = reinterpret_cast<float*>(base);
  // ---- hoisted input projection into the scratch
  const __half* hb = reinterpret_cast<const __half*>(blob);
  const size_t w_off = 0, r_off = (size_t)4 * hidden * in_c, bw_off = r_off + (size_t)4 * hidden * hidden,
               br_off = bw_off + (size_t)4 * hidden;
  const int rows = seq_len * batch;
  noalloc_projection_kernel<<<dim3(ceil_div(4 * hidden, 32), ceil_div(rows, 32)), 256, 0, ctx->stream>>>(
      (const __half*)x, hb + w_off, hb + bw_off, double_bias ? hb + br_off : nullptr, gx, rows, in_c, 4 * hidden);
  AIG_LAUNCH_OK(ctx);
  // ---- recurrence
  LstmParams prm{};
  prm.T = seq_len; prm.B = batch; prm.H = hidden;
  prm.clip = clip;
  prm.R = hb + r_off;
  prm.gx = gx;
  prm.gx_sT = (long long)batch * 4 * hidden;
  prm.gx_sB = (long long)4 * hidden;
  prm.y = (__half*)y;
  prm.y_sT = (long long)batch * hidden;
  prm.y_sB = hidden;
  return run_recurrent(ctx, shape, prm);
}

}  // extern "C"
