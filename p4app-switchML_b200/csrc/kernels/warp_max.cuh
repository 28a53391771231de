// The largest of 32 lanes' magnitudes in one instruction (sm_100a reduces floats across a warp) instead of five
// shuffles and five maxima that wait for one another. With blocks of 256, whose maxima the exact mode takes: one worker,
// 25 MB of bfloat16 7.6 -> 7.0 us, float32 6.7 -> 6.2; two ranks on one GPU, 2^25 elements 131 -> 128.5 us, 2^22 22.8 -> 22.2.
#ifndef SWITCHML_WARP_MAX_CUH_
#define SWITCHML_WARP_MAX_CUH_

namespace switchml {
namespace kernels {
namespace {

// The larger of two magnitudes. kNan: NaN if either is; else a NaN never wins.
template <bool kNan>
__device__ __forceinline__ float Larger(float a, float b) {
  if (!kNan) return fmaxf(a, b);
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// All lanes of a warp: the same over all of them.
template <bool kNan>
__device__ __forceinline__ float WarpLargest(float m) {
  float r;
  if (kNan) asm volatile("redux.sync.max.NaN.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(m));
  else asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(m));
  return r;
}

}  // namespace
}  // namespace kernels
}  // namespace switchml

#endif  // SWITCHML_WARP_MAX_CUH_
