// bf16 conversions and the 16-byte vector accumulators of the plain-sum mode.
#ifndef SWITCHML_VECTOR_SUM_CUH_
#define SWITCHML_VECTOR_SUM_CUH_

#include <cuda_bf16.h>
#include <stdint.h>

#include "kernels/allreduce_kernels.h"

namespace switchml {
namespace kernels {
namespace {

// bf16 pair helpers -----------------------------------------------------------------
__device__ __forceinline__ float2 Bf16x2ToFloat2(unsigned u) {
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}
__device__ __forceinline__ unsigned Float2ToBf16x2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<unsigned*>(&h);
}
__device__ __forceinline__ float Bf16ToFloat(unsigned short u) {
  return __uint_as_float(static_cast<unsigned>(u) << 16);
}
__device__ __forceinline__ unsigned short FloatToBf16(float f) {
  __nv_bfloat16 h = __float2bfloat16_rn(f);
  return *reinterpret_cast<unsigned short*>(&h);
}

// 16-byte vector accumulators of the plain-sum mode.
template <int ELEM> struct VecAcc;
template <> struct VecAcc<ELEM_F32> {
  float4 a;
  __device__ __forceinline__ void Zero() { a = make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ __forceinline__ void Init(uint4 v) { a = make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w)); }
  __device__ __forceinline__ void Add(uint4 v) { a.x += __uint_as_float(v.x); a.y += __uint_as_float(v.y); a.z += __uint_as_float(v.z); a.w += __uint_as_float(v.w); }
  __device__ __forceinline__ uint4 Finish(float s) {
    if (s != 1.0f) { a.x *= s; a.y *= s; a.z *= s; a.w *= s; }
    return make_uint4(__float_as_uint(a.x), __float_as_uint(a.y), __float_as_uint(a.z), __float_as_uint(a.w));
  }
};
template <> struct VecAcc<ELEM_I32> {
  uint4 a;
  __device__ __forceinline__ void Zero() { a = make_uint4(0, 0, 0, 0); }
  __device__ __forceinline__ void Init(uint4 v) { a = v; }
  __device__ __forceinline__ void Add(uint4 v) { a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w; }  // wrapping
  __device__ __forceinline__ uint4 Finish(float) { return a; }
};
template <> struct VecAcc<ELEM_BF16> {
  float a[8];
  __device__ __forceinline__ void Zero() {
#pragma unroll
    for (int j = 0; j < 8; j++) a[j] = 0.f;
  }
  __device__ __forceinline__ void Init(uint4 v) {
    float2 q;
    q = Bf16x2ToFloat2(v.x); a[0] = q.x; a[1] = q.y;
    q = Bf16x2ToFloat2(v.y); a[2] = q.x; a[3] = q.y;
    q = Bf16x2ToFloat2(v.z); a[4] = q.x; a[5] = q.y;
    q = Bf16x2ToFloat2(v.w); a[6] = q.x; a[7] = q.y;
  }
  __device__ __forceinline__ void Add(uint4 v) {
    float2 q;
    q = Bf16x2ToFloat2(v.x); a[0] += q.x; a[1] += q.y;
    q = Bf16x2ToFloat2(v.y); a[2] += q.x; a[3] += q.y;
    q = Bf16x2ToFloat2(v.z); a[4] += q.x; a[5] += q.y;
    q = Bf16x2ToFloat2(v.w); a[6] += q.x; a[7] += q.y;
  }
  __device__ __forceinline__ uint4 Finish(float s) {
    if (s != 1.0f) {
#pragma unroll
      for (int j = 0; j < 8; j++) a[j] *= s;
    }
    return make_uint4(Float2ToBf16x2(a[0], a[1]), Float2ToBf16x2(a[2], a[3]), Float2ToBf16x2(a[4], a[5]),
                      Float2ToBf16x2(a[6], a[7]));
  }
};

}  // namespace
}  // namespace kernels
}  // namespace switchml
#endif  // SWITCHML_VECTOR_SUM_CUH_
