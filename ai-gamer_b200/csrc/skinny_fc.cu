// skinny_fc.cu -- y = x . W^T for few rows of x (at most 64), W K-major as the FC plans keep it.
//
// With few rows the product reads its weights once and does next to nothing with them, so what counts is how many SMs
// stream them and how much each has in flight.  The tiled GEMM gives such a layer N / 64 CTAs that walk K alone: 36864 ->
// 1024 for one frame took 318 us (75 MB at 0.24 TB/s), 64 x 1024 -> 1024 9.9 us.  Here a CTA takes 16 outputs and a share
// of K: eight warps, each a 32-deep block of K in turn, fragments straight from global memory (16 bytes a lane, up to 24
// loads in flight) into mma.sync m16n8k16 -- tensor throughput does not matter at this shape --, the warps' sums through
// shared memory, the shares of a cluster of up to eight CTAs through distributed shared memory, always added in the same
// order.  The two products above take 19 (weights from L2 in part) and 6.2 us.
#include "aig_common.cuh"
#include "skinny_fc.h"

namespace {

constexpr int kThreads = 256, kWarps = 8, kMaxCluster = 8;

__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float ld_cluster(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float round_half(float v) { return __half2float(__float2half(v)); }

// NT = tiles of eight rows of x
template <int NT>
__global__ void __launch_bounds__(kThreads, NT <= 4 ? 2 : 1) skinny_fc_kernel(const SkinnyFc p, int share) {
  constexpr int U = NT <= 1 ? 8 : (NT <= 2 ? 6 : (NT <= 4 ? 4 : 2));  // blocks of K in flight
  __shared__ float red[kWarps / 2][16][NT * 8 + 1];
  __shared__ float sum[16 * NT * 8];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  const int rank = (int)cluster_ctarank(), n0 = blockIdx.y * 16, K = p.in_c;
  const int nkb = (K + 31) >> 5, lo = rank * share, hi = min(nkb, lo + share);  // `share` blocks of K per CTA of the cluster
  griddep_launch_dependents();
  griddep_wait();  // (the weights may be new as well as x)
  const __half* w0 = p.w + (size_t)(n0 + g) * K + q * 8;
  const __half* w1 = w0 + (size_t)8 * K;
  const __half* xr[NT];
  bool on[NT];
  float acc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    on[j] = 8 * j + g < p.rows;
    xr[j] = p.x + (size_t)(on[j] ? 8 * j + g : 0) * K + q * 8;
    acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
  }
  for (int kb0 = lo + warp; kb0 < hi; kb0 += kWarps * U) {
    uint4 a[U][2], b[U][NT];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int kb = kb0 + u * kWarps;
      const bool in = kb < hi && kb * 32 + q * 8 < K;
      a[u][0] = in ? __ldcs(reinterpret_cast<const uint4*>(w0 + kb * 32)) : make_uint4(0, 0, 0, 0);
      a[u][1] = in ? __ldcs(reinterpret_cast<const uint4*>(w1 + kb * 32)) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int j = 0; j < NT; ++j) b[u][j] = in && on[j] ? *reinterpret_cast<const uint4*>(xr[j] + kb * 32) : make_uint4(0, 0, 0, 0);
    }
    // (a lane's 16 bytes of a row and of a column are the two mma steps' k: the order of k is free)
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        mma_16816(acc[j], a[u][0].x, a[u][1].x, a[u][0].y, a[u][1].y, b[u][j].x, b[u][j].y);
        mma_16816(acc[j], a[u][0].z, a[u][1].z, a[u][0].w, a[u][1].w, b[u][j].z, b[u][j].w);
      }
  }
  // the upper four warps' sums, then the lower four's with them
  float(*mine)[NT * 8 + 1] = red[warp & 3];
#pragma unroll
  for (int half = 1; half >= 0; --half) {
    if ((warp >> 2) == half)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float& d = mine[g + 8 * (e >> 1)][8 * j + 2 * q + (e & 1)];
          d = half ? acc[j][e] : d + acc[j][e];
        }
    __syncthreads();
  }
  for (int i = tid; i < 16 * NT * 8; i += kThreads) {  // i = row of x * 16 + output, so that the stores below are in rows
    const int o = i & 15, r = i >> 4;
    sum[i] = (red[0][o][r] + red[1][o][r]) + (red[2][o][r] + red[3][o][r]);
  }
  const int ctas = gridDim.x;  // (one cluster along x)
  if (ctas > 1) cluster_sync_all();
  else __syncthreads();
  // every CTA of the cluster finishes a part of the outputs
  for (int i = rank * kThreads + tid; i < 16 * p.rows; i += ctas * kThreads) {
    const int n = n0 + (i & 15), r = i >> 4;
    if (n >= p.out_c) continue;
    float v = 0.f;
    if (ctas > 1) {
      const uint32_t at = smem_u32(sum + i);
      for (int c = 0; c < ctas; ++c) v += ld_cluster(mapa_shared(at, (uint32_t)c));
    } else {
      v = sum[i];
    }
    if (p.two_step) v = round_half(round_half(v) + p.shift[n]);
    else v = v * p.scale[n] + p.shift[n];
    if (p.tail.gamma) v = round_half(p.tail.gamma[n] * (v - p.tail.mean[n]) * (1.0f / sqrtf(p.tail.var[n] + p.tail.eps)) + p.tail.beta[n]);
    if (p.tail.relu) v = v > 0.f ? v : 0.f;
    if (n < p.tail.n_sigmoid) v = 1.0f / (1.0f + expf(-v));
    if (p.y32) p.y32[(size_t)r * p.out_c + n] = v;
    else p.y[(size_t)r * p.out_c + n] = __float2half(act_apply_fast(v, p.act, p.slope));
  }
  if (ctas > 1) cluster_sync_all();  // no CTA leaves while another reads its sums
}

template <int NT>
cudaError_t launch(aig_ctx* ctx, const SkinnyFc& p, int ctas) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(ctas, (p.out_c + 15) / 16);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ctas;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1] = pdl_attribute(ctx);
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const int nkb = (p.in_c + 31) / 32;
  return cudaLaunchKernelEx(&cfg, skinny_fc_kernel<NT>, p, (nkb + ctas - 1) / ctas);
}

}  // namespace

int skinny_fc_forward(aig_ctx* ctx, const SkinnyFc& p) {
  AIG_REQUIRE(ctx, p.rows >= 1 && p.rows <= kSkinnyRows && p.in_c % 16 == 0 && p.out_c >= 1 && p.out_c <= 16 * 65535, "few-row fc: shape not covered");
  // CTAs along K: as long as a warp keeps two blocks and the launch stays below four CTAs an SM
  const int nkb = (p.in_c + 31) / 32, groups = (p.out_c + 15) / 16;
  int ctas = 1;
  while (ctas < kMaxCluster && nkb >= ctas * 2 * kWarps * 2 && groups * ctas * 2 <= 4 * ctx->sm_count) ctas *= 2;
  const int tiles = (p.rows + 7) / 8;
  cudaError_t e;
  if (tiles <= 1) e = launch<1>(ctx, p, ctas);
  else if (tiles <= 2) e = launch<2>(ctx, p, ctas);
  else if (tiles <= 4) e = launch<4>(ctx, p, ctas);
  else e = launch<8>(ctx, p, ctas);
  AIG_CUDA_OK(ctx, e);
  return AIG_OK;
}
