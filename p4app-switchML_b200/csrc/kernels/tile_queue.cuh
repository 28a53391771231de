// Tiles of a persistent GEMM kernel, handed out in the order in which the grid would have launched them.
//
// The grid has one CTA (or cluster) per tile. Those that the GPU starts work on their own block index
// first and then cancel the launch of waiting ones and take over their indices (cluster launch
// control), until none is left. Compared with tile = blockIdx.x + i * gridDim.x the CTAs cannot drift
// apart, so the output is written front to back, and a slow SM takes fewer tiles; compared with a
// counter in global memory there is nothing to reset and nothing that two launches could share.
//
// One thread asks (Run); every consumer (a warp each) follows through Next / Done.
#ifndef SWITCHML_TILE_QUEUE_CUH_
#define SWITCHML_TILE_QUEUE_CUH_

constexpr int kQueueDepth = 2;  // answers that may be outstanding: more would grab tiles that another SM is ready for

struct __align__(16) TileQueue {
  ulonglong2 answer[kQueueDepth];
  uint64_t full[kQueueDepth];
  uint64_t empty[kQueueDepth];

  __device__ __forceinline__ void Init(int consumers) {
    for (int s = 0; s < kQueueDepth; s++) {
      MbarInit(&full[s], 1);
      MbarInit(&empty[s], consumers);
    }
  }
  // Answer number `i` (0, 1, ...): the first block index of the cancelled launch, or -1 at the end (and
  // when the kernel has given up).
  __device__ __forceinline__ int Read(uint32_t i, volatile int* abort) {
    const int s = i % kQueueDepth;
    if (!MbarWait(&full[s], (i / kQueueDepth) & 1, abort)) return -1;
    ulonglong2 a;
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(a.x), "=l"(a.y) : "r"(SmemAddr(&answer[s])) : "memory");
    uint32_t cancelled, x;
    asm volatile(
        "{\n\t.reg .b128 r;\n\t.reg .pred p;\n\t"
        "mov.b128 r, {%2, %3};\n\t"
        "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "mov.u32 %1, 0;\n\t"
        "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, r;\n\t}"
        : "=r"(cancelled), "=r"(x) : "l"(a.x), "l"(a.y) : "memory");
    return cancelled ? static_cast<int>(x) : -1;
  }
  // A consumer has read answer `i`; its slot may be written again (by the async proxy).
  __device__ __forceinline__ void Done(uint32_t i) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    MbarArrive(&empty[i % kQueueDepth]);
  }
};

// Consumer side, called by whole warps: the next tile, or -1.
__device__ __forceinline__ int NextTile(TileQueue& q, uint32_t i, int lane, volatile int* abort) {
  const int tile = q.Read(i, abort);
  __syncwarp();
  if (lane == 0) q.Done(i);
  return tile;
}

// The asking thread. Ends with the first answer that says there is nothing left.
__device__ __forceinline__ void RunTileQueue(TileQueue& q, volatile int* abort) {
  for (uint32_t i = 0;; i++) {
    const int s = i % kQueueDepth;
    if (!MbarWait(&q.empty[s], ((i / kQueueDepth) & 1) ^ 1, abort)) return;
    MbarExpectTx(&q.full[s], 16);
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];"
                 ::"r"(SmemAddr(&q.answer[s])), "r"(SmemAddr(&q.full[s])) : "memory");
    if (q.Read(i, abort) < 0) return;
  }
}

#endif  // SWITCHML_TILE_QUEUE_CUH_
