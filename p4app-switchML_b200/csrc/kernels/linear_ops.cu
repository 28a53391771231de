// What a linear layer needs around its three GEMMs, one launch each.
//
// switchml_cast_weights: fp32 weight and bias -> bf16 for the forward GEMM. Bound by HBM3e (6 bytes per
// element); one tile per block in address order, as in local_pass.cuh.
//
// switchml_column_sums: the bias gradient, sum over the rows of dY [K, M] (bf16), in fp32. Bound by
// reading dY. A cluster of up to eight CTAs shares kSumCols columns along K; the CTAs' partial sums meet in
// the first one's shared memory, added in the order of the ranks: no workspace, no second launch, the same
// bits in every run. 128-byte pieces of a row suffice for HBM3e as long as a CTA has many rows in
// flight (4 loads per thread, 64 rows apart). 8192 x 4096: 15.7 us back to back, where a generic
// reduction took 37 us; 128 or 256 columns per cluster 16 to 37 us, 256 threads 17.5 us.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels/dependent_launch.cuh"
#include "kernels/wgrad_gemm.h"

using switchml::kernels::LaunchOverlapped;
using switchml::kernels::WaitForEarlierKernels;

namespace {

// As in wgrad_gemm.cu: a failed launch does not leave its error for the next caller of cudaGetLastError().
int Launched(cudaError_t e) {
  if (e == cudaSuccess) return 0;
  cudaGetLastError();
  return -4;
}

constexpr int kCastThreads = 256;
constexpr int kCastVecs = 4;  // vectors of 4 elements per thread
constexpr int kCastTile = kCastThreads * kCastVecs * 4;

__device__ __forceinline__ unsigned Pack2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const unsigned*>(&h);
}

__device__ __forceinline__ void CastTile(const float* in, __nv_bfloat16* out, size_t n, size_t tile) {
  const size_t base = tile * kCastTile;
  const bool aligned = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  if (aligned && base + kCastTile <= n) {
    const float4* s = reinterpret_cast<const float4*>(in + base);
    uint2* d = reinterpret_cast<uint2*>(out + base);
    float4 a[kCastVecs];
#pragma unroll
    for (int u = 0; u < kCastVecs; u++) a[u] = s[u * kCastThreads + threadIdx.x];
#pragma unroll
    for (int u = 0; u < kCastVecs; u++) d[u * kCastThreads + threadIdx.x] = make_uint2(Pack2(a[u].x, a[u].y), Pack2(a[u].z, a[u].w));
  } else {
    for (size_t i = base + threadIdx.x; i < n && i < base + kCastTile; i += kCastThreads) out[i] = __float2bfloat16_rn(in[i]);
  }
}

__global__ void __launch_bounds__(kCastThreads)
CastWeightsKernel(const float* w, __nv_bfloat16* w_low, size_t n, unsigned w_tiles, const float* b, __nv_bfloat16* b_low, size_t nb) {
  WaitForEarlierKernels();
  if (blockIdx.x < w_tiles) CastTile(w, w_low, n, blockIdx.x);
  else CastTile(b, b_low, nb, blockIdx.x - w_tiles);
}

constexpr int kSumThreads = 512;
constexpr int kSumCols = 64;              // columns of a cluster: 128 bytes of a row
constexpr int kSumLanes = kSumCols / 8;   // threads per row, 8 columns each
constexpr int kSumRows = kSumThreads / kSumLanes;
constexpr int kSumUnroll = 4;

__global__ void __launch_bounds__(kSumThreads) ColumnSumKernel(const __nv_bfloat16* in, float* out, int K, int M) {
  __shared__ float part[kSumRows][kSumCols + 4];
  __shared__ float total[kSumCols];
  uint32_t rank, ranks;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(ranks));
  const int col0 = static_cast<int>(blockIdx.x / ranks) * kSumCols;
  const int lane = threadIdx.x % kSumLanes, row = threadIdx.x / kSumLanes;
  const int col = col0 + lane * 8;  // M is a multiple of 8: a thread's columns exist all or none
  const int k0 = static_cast<int>(static_cast<long long>(K) * rank / ranks), k1 = static_cast<int>(static_cast<long long>(K) * (rank + 1) / ranks);
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  WaitForEarlierKernels();
  if (col < M) {
    const __nv_bfloat16* p = in + col;
    for (int k = k0 + row; k < k1; k += kSumRows * kSumUnroll) {
      uint4 v[kSumUnroll];
#pragma unroll
      for (int u = 0; u < kSumUnroll; u++) {
        const int r = k + u * kSumRows;
        v[u] = r < k1 ? *reinterpret_cast<const uint4*>(p + static_cast<size_t>(r) * M) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < kSumUnroll; u++) {
        const unsigned w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
          acc[2 * j] += __uint_as_float(w[j] << 16);
          acc[2 * j + 1] += __uint_as_float(w[j] & 0xffff0000u);
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; j++) part[row][lane * 8 + j] = acc[j];
  __syncthreads();
  if (threadIdx.x < kSumCols) {
    float sum = 0.f;
#pragma unroll
    for (int r = 0; r < kSumRows; r++) sum += part[r][threadIdx.x];
    total[threadIdx.x] = sum;
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (rank == 0 && threadIdx.x < kSumCols && col0 + static_cast<int>(threadIdx.x) < M) {
    const uint32_t mine = static_cast<uint32_t>(__cvta_generic_to_shared(&total[threadIdx.x]));
    float v[8];
#pragma unroll
    for (uint32_t r = 0; r < 8; r++) {
      v[r] = 0.f;
      if (r < ranks) {
        uint32_t from;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(from) : "r"(mine), "r"(r));
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[r]) : "r"(from) : "memory");
      }
    }
    float sum = 0.f;
#pragma unroll
    for (int r = 0; r < 8; r++) sum += v[r];
    out[col0 + threadIdx.x] = sum;
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");  // no CTA leaves while it is read
}

}  // namespace

extern "C" int switchml_cast_weights(const float* w, void* w_low, unsigned long long n, const float* b, void* b_low,
                                     unsigned long long nb, void* stream) {
  if (!w || !w_low || n == 0 || (nb && (!b || !b_low))) return -1;
  const unsigned long long w_tiles = (n + kCastTile - 1) / kCastTile, b_tiles = (nb + kCastTile - 1) / kCastTile;
  if (w_tiles + b_tiles > 0x7fffffffull) return -1;
  const cudaError_t e = LaunchOverlapped(CastWeightsKernel, static_cast<unsigned>(w_tiles + b_tiles), kCastThreads, 0, 1,
                                         static_cast<cudaStream_t>(stream), w, static_cast<__nv_bfloat16*>(w_low), n,
                                         static_cast<unsigned>(w_tiles), b, static_cast<__nv_bfloat16*>(b_low), nb);
  return Launched(e);
}

extern "C" int switchml_column_sums(const void* dy, float* out, int K, int M, void* stream) {
  if (!dy || !out || K <= 0 || M <= 0) return -1;
  if ((M % 8) || (reinterpret_cast<uintptr_t>(dy) & 15)) return -2;
  // A CTA gets at least one turn of its unrolled loop (256 rows).
  int ctas = 1;
  while (ctas < 8 && K >= 2 * ctas * kSumRows * kSumUnroll) ctas <<= 1;
  const unsigned blocks = static_cast<unsigned>((M + kSumCols - 1) / kSumCols * ctas);
  const cudaError_t e = LaunchOverlapped(ColumnSumKernel, blocks, kSumThreads, 0, ctas, static_cast<cudaStream_t>(stream),
                                         static_cast<const __nv_bfloat16*>(dy), out, K, M);
  return Launched(e);
}
