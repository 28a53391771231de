// What the warps of a CTA of one_gpu_allreduce.cu share, and how they wait for one another and for the other ranks.
//
// Every wait ends: with what it waited for, or when its time is up, or when another one of the CTA has failed. All lanes of
// a warp come out of it together and with the same answer, since what they do next are votes of the whole warp.
//
// csrc/tests/one_gpu_waits_model.cc compiles this file for the host, with a warp of 32 threads.
#ifndef SWITCHML_ONE_GPU_WAITS_CUH_
#define SWITCHML_ONE_GPU_WAITS_CUH_

#include <stdint.h>

#include "kernels/allreduce_kernels.h"
#ifdef __CUDACC__
#include "kernels/bulk_copy.cuh"
#include "kernels/device_sync.cuh"
#endif

namespace switchml {
namespace kernels {
namespace {

#ifdef __CUDACC__
__device__ __forceinline__ unsigned LoadSharedAcquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(BulkSmemAddr(p)) : "memory");
  return v;
}
__device__ __forceinline__ void StoreSharedRelease(unsigned* p, unsigned v) {
  asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(BulkSmemAddr(p)), "r"(v) : "memory");
}
__device__ __forceinline__ bool TryWaitParity(unsigned long long* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done) : "r"(BulkSmemAddr(bar)), "r"(parity) : "memory");
  return done != 0;
}
#endif

constexpr int kNoteLoaded = 8, kNoteReduced = 16;  // (eight and sixteen warps at most)
constexpr int kOneBarriers = 12;
struct OneGpuShared {
  int failed;
  unsigned next[32];  // per warp and role: the first tile that it has not finished
  unsigned seen[3];   // per phase (1 and 2): tiles that all ranks have signalled
  unsigned long long full[kOneBarriers];  // of the stages in shared memory
};

__device__ __forceinline__ bool Failed(OneGpuShared* sh) { return *reinterpret_cast<volatile int*>(&sh->failed) != 0; }
// One lane: the CTA has failed. Its first failure is reported, whichever wait that ended: the waits that follow from it end
// quietly, and none may end the CTA without a status.
__device__ __forceinline__ void Fail(const RankCtx& ctx, OneGpuShared* sh, int channel, int phase) {
  if (atomicExch(&sh->failed, 1) != 0) return;
  ReportStatus(ctx, STATUS_TIMEOUT | (phase << 4) | (channel << 8));
  atomicAdd(ctx.counters + 2, 1ull);
}
constexpr int kInsideCta = 3;  // the phase of a wait that is for the CTA's own warps or copies

// All lanes of a warp: what it wrote so far belongs to the tiles before `next`.
__device__ __forceinline__ void Note(OneGpuShared* sh, int which, int lane, unsigned next) {
  __syncwarp();
  if (lane == 0) StoreSharedRelease(&sh->next[which], next);
}

// All lanes of a warp: until eight neighbouring warps have finished the tiles before `tile`. False after a failure.
__device__ __forceinline__ bool WaitForNotes(const RankCtx& ctx, int channel, OneGpuShared* sh, int which, unsigned tile) {
  const int lane = threadIdx.x & 31;
  unsigned long long start = 0;
  for (unsigned spins = 0;;) {
    if (__all_sync(0xffffffffu, LoadSharedAcquire(&sh->next[which + (lane & 7)]) >= tile)) break;
    if ((++spins & 63) == 0) {
      const unsigned long long now = GlobalTimerNs();
      if (start == 0) start = now;
      // (Twice the time: the wait that holds up the other warps says more than this one.)
      if (__any_sync(0xffffffffu, Failed(sh) || now - start > 2 * ctx.timeout_ns)) {
        if (lane == 0) Fail(ctx, sh, channel, kInsideCta);
        return false;
      }
    }
    __nanosleep(20);
  }
  __syncwarp();
  return true;
}

// Tiles that all ranks are known to have signalled in a phase: the same number in all lanes. (Lanes that kept what each had
// read itself could answer the next call differently, and the votes of two places would then meet.)
struct Seen {
  unsigned tiles = 0;
  // All lanes of a warp: until that are at least `need`. False when the wait ran out or another warp failed.
  __device__ __forceinline__ bool Reach(const RankCtx& ctx, int channel, int phase, unsigned need, OneGpuShared* sh) {
    if (tiles >= need) return true;
    unsigned long long start = 0;
    for (unsigned spins = 0;;) {
      tiles = __reduce_min_sync(0xffffffffu, LoadSharedAcquire(&sh->seen[phase]));
      if (tiles >= need) return true;
      if ((++spins & 63) == 0) {
        const unsigned long long now = GlobalTimerNs();
        if (start == 0) start = now;
        const bool late = now - start > ctx.timeout_ns;
        if (__any_sync(0xffffffffu, late || Failed(sh))) {
          if ((threadIdx.x & 31) == 0) Fail(ctx, sh, channel, phase);
          return false;
        }
      }
      __nanosleep(20);
    }
  }
};

// All lanes of a warp: until the phase of `bar` with this parity is complete. The same answer in every lane.
__device__ __forceinline__ bool WaitForBytes(const RankCtx& ctx, int channel, unsigned long long* bar, uint32_t parity, OneGpuShared* sh) {
  unsigned long long start = 0;
  bool ok = true;
  for (unsigned spins = 0;;) {
    if (TryWaitParity(bar, parity)) break;
    if ((++spins & 255) == 0) {
      const unsigned long long now = GlobalTimerNs();
      if (start == 0) start = now;
      if (Failed(sh) || now - start > ctx.timeout_ns) {
        ok = false;
        break;
      }
    }
  }
  ok = __all_sync(0xffffffffu, ok);
  if (!ok && (threadIdx.x & 31) == 0) Fail(ctx, sh, channel, kInsideCta);
  return ok;
}

}  // namespace
}  // namespace kernels
}  // namespace switchml

#endif  // SWITCHML_ONE_GPU_WAITS_CUH_
