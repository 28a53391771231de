// One worker: nothing to exchange, so a job is a single pass over the tensor. LocalCopyKernel is
// the plain sum out of place, LocalQuantKernel the exact mode's round trip through the block fixed
// point (bit-identical to what the streaming kernels give one worker, and to the CPU oracle).
//
// Both are bound by HBM3e, and both are cut the same way: a block takes one tile of 32 KiB,
// a warp's loads are in flight together, and the grid has as many blocks as there are tiles. Blocks
// then walk the tensor in address order, which the memory likes better than 592 resident blocks
// with strides of megabytes between a thread's vectors. Measured for 1 GiB of float32, read +
// write: copy 350 us -> 307 us (6.1 -> 7.0 TB/s).
#ifndef SWITCHML_LOCAL_PASS_CUH_
#define SWITCHML_LOCAL_PASS_CUH_

#include <cuda_bf16.h>
#include <stdint.h>

#include "kernels/allreduce_kernels.h"
#include "kernels/dependent_launch.cuh"
#include "kernels/warp_max.cuh"
#include "switchml/quant_math.h"

namespace switchml {
namespace kernels {
namespace {

static const int kCopyThreads = 1024;
static const int kCopyUnroll = 2;  // 16-byte vectors per thread: 32 KiB per block
static const int kQuantThreads = 256;
static const int kQuantChunk = 1024;  // elements per warp: a multiple of every block size

// Bytes before the first 16-byte boundary of `out`, at most all of them.
__host__ __device__ __forceinline__ size_t CopyHead(const char* out, size_t bytes) {
  const size_t head = (16 - (reinterpret_cast<uintptr_t>(out) & 15)) & 15;
  return head < bytes ? head : bytes;
}

// kShifted: `in` and `out` lie differently to a 16-byte boundary. The vectors are then those of
// `out`, each put together from the five aligned words of `in` that hold it (a word that holds a
// byte of the input is memory of the input's allocation, aligned as it is); byte by byte, as
// before, 25 MB took 0.5 ms. `in` and `out` do not overlap unless they are equal.
template <bool kShifted>
__global__ void __launch_bounds__(kCopyThreads) LocalCopyKernel(const char* in, char* out, size_t bytes) {
  WaitForEarlierKernels();
  LetNextKernelStart();
  const size_t head = CopyHead(out, bytes);
  const size_t nvec = (bytes - head) / 16;
  const size_t first = static_cast<size_t>(blockIdx.x) * (kCopyThreads * kCopyUnroll) + threadIdx.x;
  const char* s = in + head;
  uint4* d = reinterpret_cast<uint4*>(out + head);
  if (!kShifted) {
    uint4 v[kCopyUnroll];
#pragma unroll
    for (int u = 0; u < kCopyUnroll; u++)
      if (first + u * kCopyThreads < nvec) v[u] = reinterpret_cast<const uint4*>(s)[first + u * kCopyThreads];
#pragma unroll
    for (int u = 0; u < kCopyUnroll; u++)
      if (first + u * kCopyThreads < nvec) d[first + u * kCopyThreads] = v[u];
  } else {
    const unsigned shift = (static_cast<unsigned>(reinterpret_cast<uintptr_t>(s)) & 3) * 8;
    const unsigned* w = reinterpret_cast<const unsigned*>(s - shift / 8);
#pragma unroll
    for (int u = 0; u < kCopyUnroll; u++) {
      const size_t i = first + u * kCopyThreads;
      if (i >= nvec) continue;
      unsigned x[5];
#pragma unroll
      for (int k = 0; k < 4; k++) x[k] = w[i * 4 + k];
      x[4] = shift ? w[i * 4 + 4] : 0;
      d[i] = make_uint4(__funnelshift_r(x[0], x[1], shift), __funnelshift_r(x[1], x[2], shift),
                        __funnelshift_r(x[2], x[3], shift), __funnelshift_r(x[3], x[4], shift));
    }
  }
  if (blockIdx.x == 0) {  // fewer than 16 bytes at either end
    if (threadIdx.x < head) out[threadIdx.x] = in[threadIdx.x];
    const size_t tail = head + nvec * 16 + threadIdx.x;
    if (tail < bytes) out[tail] = in[tail];
  }
}

cudaError_t LaunchLocalCopyImpl(const void* in, void* out, size_t bytes, cudaStream_t stream) {
  const size_t tile = static_cast<size_t>(kCopyThreads) * kCopyUnroll * 16;
  const size_t blocks = (bytes + tile - 1) / tile;
  const char* i = static_cast<const char*>(in);
  char* o = static_cast<char*>(out);
  if (((reinterpret_cast<uintptr_t>(in) ^ reinterpret_cast<uintptr_t>(out)) & 15) == 0)
    return LaunchOverlapped(LocalCopyKernel<false>, static_cast<unsigned>(blocks), kCopyThreads, 0, 1, stream, i, o, bytes);
  return LaunchOverlapped(LocalCopyKernel<true>, static_cast<unsigned>(blocks), kCopyThreads, 0, 1, stream, i, o, bytes);
}

// ---- exact mode ------------------------------------------------------------------------
template <int BYTES> struct RawVec;
template <> struct RawVec<8> { uint2 v; };
template <> struct RawVec<4> { unsigned v; };
template <> struct RawVec<2> { unsigned short v; };

__device__ __forceinline__ unsigned RawWord(const RawVec<8>& r, int i) { return i == 0 ? r.v.x : r.v.y; }
__device__ __forceinline__ unsigned RawWord(const RawVec<4>& r, int) { return r.v; }
__device__ __forceinline__ unsigned RawWord(const RawVec<2>& r, int) { return r.v; }
__device__ __forceinline__ void SetRawWord(RawVec<8>& r, int i, unsigned w) { if (i == 0) r.v.x = w; else r.v.y = w; }
__device__ __forceinline__ void SetRawWord(RawVec<4>& r, int, unsigned w) { r.v = w; }
__device__ __forceinline__ void SetRawWord(RawVec<2>& r, int, unsigned w) { r.v = static_cast<unsigned short>(w); }

// The largest of each quantisation block, in every lane and row that holds some of it: m[u] is what a lane has of row u. A
// block is a power of two of lanes of one row of 2^kLog2Row elements, or of whole rows.
template <int kRows, int kLog2Row, bool kNan>
__device__ __forceinline__ void BlockMaxima(float (&m)[kRows], int log2_block) {
  if (log2_block < kLog2Row) {
    const int lanes = 1 << (log2_block - (kLog2Row - 5));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      if (o < lanes) {  // warp-uniform
#pragma unroll
        for (int u = 0; u < kRows; u++) m[u] = Larger<kNan>(m[u], __shfl_xor_sync(0xffffffffu, m[u], o));
      }
    }
  } else {
    // Fold a block's rows into its first, one reduction per block, and hand the maximum back.
    const int rows = 1 << (log2_block - kLog2Row);
#pragma unroll
    for (int span = 1; span < kRows; span <<= 1) {
      if (span < rows) {
#pragma unroll
        for (int u = 0; u + span < kRows; u += 2 * span) m[u] = Larger<kNan>(m[u], m[u + span]);
      }
    }
#pragma unroll
    for (int u = 0; u < kRows; u++) {
      if ((u & (rows - 1)) == 0) m[u] = WarpLargest<kNan>(m[u]);
    }
#pragma unroll
    for (int span = kRows / 2; span >= 1; span >>= 1) {
      if (span < rows) {
#pragma unroll
        for (int u = 0; u + span < kRows; u += 2 * span) m[u + span] = m[u];
      }
    }
  }
}

template <int ELEM>
__device__ __forceinline__ float LoadElement(const char* p, int i) {
  if (ELEM == ELEM_BF16) return __uint_as_float(static_cast<unsigned>(reinterpret_cast<const unsigned short*>(p)[i]) << 16);
  return reinterpret_cast<const float*>(p)[i];
}
template <int ELEM>
__device__ __forceinline__ void StoreElement(char* p, int i, float x) {
  if (ELEM == ELEM_BF16) reinterpret_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(x);
  else reinterpret_cast<float*>(p)[i] = x;
}

// One chunk of kQuantChunk elements by one warp, in vectors of VB bytes (of VE elements): vector
// u * 32 + lane is lane's u-th, so a row is the 32 * VE elements that a load instruction brings.
// A quantisation block is a power of two of lanes of one row, or of whole rows. kGuard: the chunk
// has only `valid` elements, VB is one element; what is missing counts as zero.
//
// kFast: with one worker the trip x -> int32 -> float rounds x to a multiple of 2^(E-31), E the block's
// exponent. That is (x + C) - C with C = +-2^(E-8): below C the sum's last bit is the grid's, from C on
// x lies on the grid already. Conversions between float and int run at an eighth of the rate of additions,
// two of them per element took 5.9 us of a 25 MB bf16 bucket (kernel 11.6 us -> 9.1 us). Nothing is done and
// false comes back when a value is not finite or so large that the integer saturates; kFast = false takes those.
template <int ELEM, int VB, bool kGuard, bool kFast>
__device__ __forceinline__ bool LocalQuantChunk(const char* in, char* out, int lane, int log2_block, float base,
                                                int valid) {
  constexpr int kEsz = ELEM == ELEM_BF16 ? 2 : 4;
  constexpr int VE = VB / kEsz;
  constexpr int kRows = kQuantChunk / (32 * VE);
  constexpr int kLog2Row = (VE == 4 ? 7 : VE == 2 ? 6 : 5);
  constexpr int kWords = VB >= 4 ? VB / 4 : 1;
  RawVec<VB> x[kRows];
#pragma unroll
  for (int u = 0; u < kRows; u++) {
    if (!kGuard || u * 32 + lane < valid) {
      x[u] = reinterpret_cast<const RawVec<VB>*>(in)[u * 32 + lane];
    } else {
      for (int w = 0; w < kWords; w++) SetRawWord(x[u], w, 0);
    }
  }
  float m[kRows];
#pragma unroll
  for (int u = 0; u < kRows; u++) {
    m[u] = 0.f;
#pragma unroll
    for (int w = 0; w < kWords; w++) {
      const unsigned raw = RawWord(x[u], w);
      if (ELEM == ELEM_F32) {
        m[u] = Larger<kFast>(m[u], fabsf(__uint_as_float(raw)));
      } else {
        m[u] = Larger<kFast>(m[u], fabsf(__uint_as_float(raw << 16)));
        if (VB >= 4) m[u] = Larger<kFast>(m[u], fabsf(__uint_as_float(raw & 0xffff0000u)));
      }
    }
  }
  BlockMaxima<kRows, kLog2Row, kFast>(m, log2_block);
  if (kFast) {
    bool odd = false;
#pragma unroll
    for (int u = 0; u < kRows; u++) odd |= !(m[u] < 0x1p127f);
    if (__any_sync(0xffffffffu, odd)) return false;
  }
#pragma unroll
  for (int u = 0; u < kRows; u++) {
    const int exponent = quant::ClampExponent(quant::LocalExponent(m[u]));
    const float c = __int_as_float((exponent - 8 + 127) << 23);
    // (The scale factor is a power of two here, so that multiplying by its exact reciprocal gives the bits of
    // the division.)
    const float f = quant::ScaleFactorFromBase(exponent, base);
    const float inv = __frcp_rn(f);
    auto trip = [&](float v) {
      if (!kFast) return __int2float_rn(quant::Quantize(v, f)) * inv;
      const float cv = __uint_as_float((__float_as_uint(v) & 0x80000000u) | __float_as_uint(c));
      const float r = __fsub_rn(__fadd_rn(v, cv), cv);
      return fabsf(v) < c ? r : v;
    };
    RawVec<VB> y;
#pragma unroll
    for (int w = 0; w < kWords; w++) {
      const unsigned raw = RawWord(x[u], w);
      if (ELEM == ELEM_F32) {
        SetRawWord(y, w, __float_as_uint(trip(__uint_as_float(raw))));
      } else if (VB >= 4) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(trip(__uint_as_float(raw << 16)), trip(__uint_as_float(raw & 0xffff0000u)));
        SetRawWord(y, w, *reinterpret_cast<const unsigned*>(&h));
      } else {
        const __nv_bfloat16 h = __float2bfloat16_rn(trip(__uint_as_float(raw << 16)));
        SetRawWord(y, w, *reinterpret_cast<const unsigned short*>(&h));
      }
    }
    if (!kGuard || u * 32 + lane < valid) reinterpret_cast<RawVec<VB>*>(out)[u * 32 + lane] = y;
  }
  return true;
}

// The same chunk in whole 16-byte vectors where the first element lies S elements behind a 16-byte boundary, in the input
// and in the output alike (a slice of a flat buffer). Vector v holds the elements v * VE - S to v * VE - S + VE - 1. The first S
// of them belong to the block of the vector before it, of whatever block they are: they count for its
// maximum, and its exponent is theirs, which takes a shuffle each way per row. The neighbours' elements in
// the first vector are left alone, and the chunk's last S elements lie in a vector of the next chunk: both ends go
// element by element. Vectors of one element, which such tensors used to go in, cost their instructions (2^25
// elements in place, blocks of 64: bfloat16 one element off 64.5 us, float32 63.5; of 256: 51 and 50).
//
// kGuard: the chunk has only `valid` elements. False, and nothing done, as in LocalQuantChunk<kFast>.
template <int ELEM, int S, bool kGuard>
__device__ __forceinline__ bool LocalQuantRows(const char* in, char* out, int lane, int log2_block, int valid) {
  constexpr int kEsz = ELEM == ELEM_BF16 ? 2 : 4, VE = 16 / kEsz;
  constexpr int kRows = kQuantChunk / (32 * VE), kLog2Row = VE == 8 ? 8 : 7;
  const uint4* const from = reinterpret_cast<const uint4*>(in - S * kEsz);
  uint4* const to = reinterpret_cast<uint4*>(out - S * kEsz);
  auto element = [&](int e) { return LoadElement<ELEM>(in, e); };
  // Element i of a vector.
  auto get = [](const uint4& v, int i) {
    const unsigned w = ELEM == ELEM_BF16 ? (i < 2 ? v.x : i < 4 ? v.y : i < 6 ? v.z : v.w) : (i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w);
    return __uint_as_float(ELEM == ELEM_F32 ? w : i & 1 ? w & 0xffff0000u : w << 16);
  };
  auto put = [](float x[VE]) {
    if constexpr (ELEM == ELEM_F32) {
      return make_uint4(__float_as_uint(x[0]), __float_as_uint(x[1]), __float_as_uint(x[2]), __float_as_uint(x[3]));
    } else {
      unsigned w[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(x[2 * i], x[2 * i + 1]);
        w[i] = *reinterpret_cast<const unsigned*>(&h);
      }
      return make_uint4(w[0], w[1], w[2], w[3]);
    }
  };
  uint4 x[kRows];
#pragma unroll
  for (int u = 0; u < kRows; u++) {
    const int first = (u * 32 + lane) * VE - S;
    if (!kGuard || first + VE <= valid) {
      x[u] = from[u * 32 + lane];
      if (S > 0 && u == 0 && lane == 0) {  // the chunk before this one's
        float y[VE];
#pragma unroll
        for (int i = 0; i < VE; i++) y[i] = i < S ? 0.f : get(x[u], i);
        x[u] = put(y);
      }
    } else {
      float y[VE];
#pragma unroll
      for (int i = 0; i < VE; i++) y[i] = first + i >= 0 && first + i < valid ? element(first + i) : 0.f;
      x[u] = put(y);
    }
  }
  float end = 0.f;  // lane i: element i of the last S
  const int at_end = kQuantChunk - S + lane;
  if (S > 0 && lane < S && (!kGuard || at_end < valid)) end = element(at_end);
  float m[kRows], low[kRows];
#pragma unroll
  for (int u = 0; u < kRows; u++) {
    m[u] = low[u] = 0.f;
#pragma unroll
    for (int i = 0; i < VE; i++) {
      if (i < S) low[u] = Larger<true>(low[u], fabsf(get(x[u], i)));
      else m[u] = Larger<true>(m[u], fabsf(get(x[u], i)));
    }
  }
  if (S > 0) {
    float end_max = fabsf(end);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) end_max = Larger<true>(end_max, __shfl_xor_sync(0xffffffffu, end_max, o));
#pragma unroll
    for (int u = 0; u < kRows; u++) {
      const float next = u + 1 < kRows ? low[u + 1 < kRows ? u + 1 : u] : end_max;
      m[u] = Larger<true>(m[u], __shfl_sync(0xffffffffu, lane == 0 ? next : low[u], (lane + 1) & 31));
    }
  }
  BlockMaxima<kRows, kLog2Row, true>(m, log2_block);
  bool odd = false;
#pragma unroll
  for (int u = 0; u < kRows; u++) odd |= !(m[u] < 0x1p127f);
  if (__any_sync(0xffffffffu, odd)) return false;
  auto trip = [](float v, float c) {
    const float cv = __uint_as_float((__float_as_uint(v) & 0x80000000u) | __float_as_uint(c));
    const float r = __fsub_rn(__fadd_rn(v, cv), cv);
    return fabsf(v) < c ? r : v;
  };
  float c[kRows];
#pragma unroll
  for (int u = 0; u < kRows; u++) c[u] = __int_as_float((quant::ClampExponent(quant::LocalExponent(m[u])) - 8 + 127) << 23);
#pragma unroll
  for (int u = 0; u < kRows; u++) {
    float before = c[u];
    if (S > 0) before = __shfl_sync(0xffffffffu, lane == 31 && u > 0 ? c[u > 0 ? u - 1 : 0] : c[u], (lane + 31) & 31);
    float y[VE];
#pragma unroll
    for (int i = 0; i < VE; i++) y[i] = trip(get(x[u], i), i < S ? before : c[u]);
    const int first = (u * 32 + lane) * VE - S;
    if ((!kGuard || first + VE <= valid) && !(S > 0 && u == 0 && lane == 0)) {
      to[u * 32 + lane] = put(y);
    } else {
#pragma unroll
      for (int i = 0; i < VE; i++)
        if (first + i >= 0 && (!kGuard || first + i < valid)) StoreElement<ELEM>(out, first + i, y[i]);
    }
  }
  if (S > 0) {
    const float last = __shfl_sync(0xffffffffu, c[kRows - 1], 31);
    if (lane < S && (!kGuard || at_end < valid)) StoreElement<ELEM>(out, at_end, trip(end, last));
  }
  return true;
}

// What the fast way leaves over. Not inlined: its 32 rows would set the kernel's registers.
template <int ELEM>
__device__ __noinline__ void LocalQuantSlow(const char* in, char* out, int lane, int log2_block, float base, int valid) {
  LocalQuantChunk<ELEM, ELEM == ELEM_BF16 ? 2 : 4, true, false>(in, out, lane, log2_block, base, valid);
}

// One chunk per warp; the last warp takes what is left over (fewer than kQuantChunk elements).
// Three blocks per SM (float32, 80 registers) and four (bfloat16, 64) keep 96 and 64 KB in flight. With two and three, the
// slow way inlined, and maxima by shuffles in all of these: 25 MB float32 7.5 us instead of 6.7, bfloat16 8.5 instead of 7.7, 2^27 elements 168 instead of 155
// and 96 instead of 84 (blocks of 256, in place), bfloat16 one element off 133 instead of 98. One block more
// costs registers that the fast way needs (bfloat16 25 MB 10.6). With WarpLargest() instead of shuffles 25 MB take 6.2 and
// 7.0 us, 2^27 elements of bfloat16 78.7 instead of 81.7, one element off 87.5 instead of 91.7.
template <int ELEM, int S>
__global__ void __launch_bounds__(kQuantThreads, ELEM == ELEM_BF16 ? 4 : 3)
LocalQuantRowsKernel(const char* in, char* out, size_t numel, int log2_block, float base) {
  WaitForEarlierKernels();
  LetNextKernelStart();
  constexpr int kEsz = ELEM == ELEM_BF16 ? 2 : 4;
  const int lane = threadIdx.x & 31;
  const size_t off = ((static_cast<size_t>(blockIdx.x) * kQuantThreads + threadIdx.x) >> 5) * kQuantChunk;
  if (off >= numel) return;
  const char* from = in + off * kEsz;
  char* to = out + off * kEsz;
  const int valid = static_cast<int>(numel - off < kQuantChunk ? numel - off : kQuantChunk);
  const bool done = valid == kQuantChunk ? LocalQuantRows<ELEM, S, false>(from, to, lane, log2_block, valid)
                                         : LocalQuantRows<ELEM, S, true>(from, to, lane, log2_block, valid);
  if (!done) LocalQuantSlow<ELEM>(from, to, lane, log2_block, base, valid);
}

// The same where input and output lie differently to a 16-byte boundary, in the widest vectors that both addresses allow.
template <int ELEM, int VB>
__global__ void __launch_bounds__(kQuantThreads)
LocalQuantKernel(const char* in, char* out, size_t numel, int log2_block, float base) {
  WaitForEarlierKernels();
  LetNextKernelStart();
  constexpr int kEsz = ELEM == ELEM_BF16 ? 2 : 4;
  const int lane = threadIdx.x & 31;
  const size_t c = (static_cast<size_t>(blockIdx.x) * kQuantThreads + threadIdx.x) >> 5;
  const size_t off = c * kQuantChunk;
  if (off + kQuantChunk <= numel) {
    const char* from = in + off * kEsz;
    char* to = out + off * kEsz;
    if (!LocalQuantChunk<ELEM, VB, false, true>(from, to, lane, log2_block, base, kQuantChunk))
      LocalQuantChunk<ELEM, kEsz, true, false>(from, to, lane, log2_block, base, kQuantChunk);
  } else if (off < numel) {
    LocalQuantChunk<ELEM, kEsz, true, false>(in + off * kEsz, out + off * kEsz, lane, log2_block, base, static_cast<int>(numel - off));
  }
}

template <int ELEM>
cudaError_t LaunchLocalQuantElem(const void* in, void* out, size_t numel, int log2_block, float base, cudaStream_t stream) {
  constexpr int kEsz = ELEM == ELEM_BF16 ? 2 : 4;
  const uintptr_t a = reinterpret_cast<uintptr_t>(in), b = reinterpret_cast<uintptr_t>(out);
  if ((a | b) % kEsz != 0) return cudaErrorInvalidValue;
  const size_t per_block = static_cast<size_t>(kQuantChunk) * (kQuantThreads / 32);
  const unsigned blocks = static_cast<unsigned>((numel + per_block - 1) / per_block);
  void (*kernel)(const char*, char*, size_t, int, float) = nullptr;
  if (((a ^ b) & 15) == 0) {
    const int shift = static_cast<int>(a & 15) / kEsz;
    if constexpr (ELEM == ELEM_BF16) {
      static constexpr decltype(kernel) kShifted[8] = {LocalQuantRowsKernel<ELEM, 0>, LocalQuantRowsKernel<ELEM, 1>, LocalQuantRowsKernel<ELEM, 2>,
                                                       LocalQuantRowsKernel<ELEM, 3>, LocalQuantRowsKernel<ELEM, 4>, LocalQuantRowsKernel<ELEM, 5>,
                                                       LocalQuantRowsKernel<ELEM, 6>, LocalQuantRowsKernel<ELEM, 7>};
      kernel = kShifted[shift];
    } else {
      static constexpr decltype(kernel) kShifted[4] = {LocalQuantRowsKernel<ELEM, 0>, LocalQuantRowsKernel<ELEM, 1>, LocalQuantRowsKernel<ELEM, 2>,
                                                       LocalQuantRowsKernel<ELEM, 3>};
      kernel = kShifted[shift];
    }
  } else if (((a | b) & 7) == 0) {
    kernel = LocalQuantKernel<ELEM, 8>;
  } else if (((a | b) & 3) == 0) {
    kernel = LocalQuantKernel<ELEM, 4>;
  } else {
    kernel = LocalQuantKernel<ELEM, kEsz>;
  }
  return LaunchOverlapped(kernel, blocks, kQuantThreads, 0, 1, stream, static_cast<const char*>(in), static_cast<char*>(out), numel, log2_block, base);
}

}  // namespace
}  // namespace kernels
}  // namespace switchml
#endif  // SWITCHML_LOCAL_PASS_CUH_
