// The plain GEMM with one CTA per 128 x 256 tile: short reductions (a batch of samples, as in VGG's fully
// connected layers), where dW is much larger than the operands and the time is the time to write it.
// The loads and the MMAs of the next tiles run while a tile is stored:
//   warp 0      TMA producer, a ring of kWideStages stages of 64 K-rows
//   warp 1      MMA issuer, two accumulators in TMEM
//   warp 2      asks for tiles (tile_queue.cuh), allocates TMEM
//   warps 4-7   epilogue: tcgen05.ld 32 columns at a time, swizzled shared memory (kWideBufs buffers), TMA store
//
// kWholeBoxes: the four warps store 128 rows together. Otherwise each stores its 32 rows on its own and waits for nobody,
// which is for short reductions, where the stores are all there is (32 x 4096 x 25088: 67 us = 6.1 TB/s, with the
// barriers 68 to 69). With a long one the main loop's loads have to get past four times as many stores (512 x 8192 x
// 8192: 96.5 us against 90.3 with whole boxes, 2048 x 8192 x 8192: 268 against 259). Eight epilogue warps were
// faster nowhere, and slower at the longer of the short reductions, where their buffers took a stage (256 x 4096 x 4096:
// 21.3 against 18.2 us).
//
// The issuer's loop over a stage is unrolled, with a loop of its own for a last stage that K does not fill: one loop
// with a run-time bound for both cost long reductions a tenth (8192 x 4096 x 1024: 62.5 -> 69.5 us).
constexpr int kWideEpiWarps = 4;
constexpr int kWideThreads = 128 + 32 * kWideEpiWarps;
constexpr int kWideStages = 4;
constexpr int kWideBufs = 2;

struct __align__(1024) WideShared {
  uint8_t stage[kWideStages][kStageBytes];
  uint8_t epi[kWideBufs][kEpiBytes];
  TileQueue queue;
  uint64_t full[kWideStages];
  uint64_t empty[kWideStages];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  volatile int abort;
};

// A barrier of the epilogue's warps that tells all of them whether all of them say yes. One that has given up must not
// leave the others in a barrier without it.
__device__ __forceinline__ bool WideEpilogueAll(bool yes) {
  uint32_t all;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.and.pred q, 1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(all) : "r"(static_cast<uint32_t>(yes)), "n"(kWideEpiWarps * 32) : "memory");
  return all != 0;
}

template <bool kWholeBoxes>
__global__ void __launch_bounds__(kWideThreads, 1)
WgradWideKernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                const __grid_constant__ CUtensorMap map_d, int tiles_n, int K, int* error_flag) {
  extern __shared__ uint8_t smem_raw[];
  WideShared& sh = *reinterpret_cast<WideShared*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k_blocks = (K + kTileK - 1) / kTileK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kWideStages; s++) {
      MbarInit(&sh.full[s], 1);
      MbarInit(&sh.empty[s], 1);
    }
    for (int b = 0; b < 2; b++) {
      MbarInit(&sh.acc_full[b], 1);
      MbarInit(&sh.acc_empty[b], kWideEpiWarps);
    }
    sh.queue.Init(2 + kWideEpiWarps);
    sh.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(SmemAddr(&sh.tmem_base)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = sh.tmem_base;
  WaitForEarlierKernels();

  if (warp == 0) {
    uint32_t it = 0;
    bool ok = true;
    int tile = static_cast<int>(blockIdx.x);
    for (uint32_t t = 0; tile >= 0; tile = NextTile(sh.queue, t++, lane, &sh.abort)) {
      const int m0 = (tile / tiles_n) * kTileM, n0 = (tile % tiles_n) * kTileN;
      if (lane == 0) {
        for (int kb = 0; kb < k_blocks && ok; kb++, it++) {
          const int s = it % kWideStages;
          ok = MbarWait(&sh.empty[s], ((it / kWideStages) & 1) ^ 1, &sh.abort);
          if (!ok) break;
          MbarExpectTx(&sh.full[s], kStageBytes);
          uint8_t* a = sh.stage[s];
          uint8_t* b = a + kABytes;
          // Rows beyond K, and columns beyond M / N, are filled with zeros by the TMA unit.
          for (int j = 0; j < kTileM / kAtomMN; j++)
            TmaLoad2D(a + j * (kTileK * 128), &map_a, m0 + j * kAtomMN, kb * kTileK, &sh.full[s]);
          for (int j = 0; j < kTileN / kAtomMN; j++)
            TmaLoad2D(b + j * (kTileK * 128), &map_b, n0 + j * kAtomMN, kb * kTileK, &sh.full[s]);
        }
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    uint32_t it = 0;
    int tile = static_cast<int>(blockIdx.x);
    for (uint32_t t = 0; tile >= 0; tile = NextTile(sh.queue, t++, lane, &sh.abort)) {
      if (lane == 0) {
        const int acc = t & 1;
        bool ok = MbarWait(&sh.acc_empty[acc], ((t >> 1) & 1) ^ 1, &sh.abort);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tmem_d = tmem_base + acc * kTileN;
        for (int kb = 0; kb < k_blocks && ok; kb++, it++) {
          const int s = it % kWideStages;
          ok = MbarWait(&sh.full[s], (it / kWideStages) & 1, &sh.abort);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a_addr = SmemAddr(sh.stage[s]);
          auto step = [&](int kk) {
            Mma(tmem_d, OperandDesc(a_addr + kk * kMmaK * 128, kTileK * 128),
                OperandDesc(a_addr + kABytes + kk * kMmaK * 128, kTileK * 128), (kb | kk) != 0);
          };
          if (kb < K / kTileK) {
#pragma unroll
            for (int kk = 0; kk < kTileK / kMmaK; kk++) step(kk);
          } else {  // steps that have rows at all
            const int left = (K - kb * kTileK + kMmaK - 1) / kMmaK;
            for (int kk = 0; kk < left; kk++) step(kk);
          }
          MmaCommit(&sh.empty[s]);  // the stage may be refilled once these MMAs have read it
        }
        if (ok) MmaCommit(&sh.acc_full[acc]);
      }
      __syncwarp();
    }
  } else if (warp == 2) {
    if (lane == 0) RunTileQueue(sh.queue, &sh.abort);
    __syncwarp();
  } else if (warp >= 4) {
    const int quarter = warp & 3;  // TMEM lanes 32 * (warp % 4) .. are the warp's own
    const bool issues = threadIdx.x == 128 || (!kWholeBoxes && lane == 0);
    uint32_t stores = 0;
    int tile = static_cast<int>(blockIdx.x);
    for (uint32_t t = 0;; tile = NextTile(sh.queue, t++, lane, &sh.abort)) {
      const int acc = t & 1;
      bool go = tile >= 0 && MbarWait(&sh.acc_full[acc], (t >> 1) & 1, &sh.abort);
      if (kWholeBoxes) go = WideEpilogueAll(go);
      if (!go) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int m0 = (tile / tiles_n) * kTileM, n0 = (tile % tiles_n) * kTileN;
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * kTileN;
      for (int c = 0; c < kTileN / kEpiCols; c++, stores++) {
        uint8_t* box = sh.epi[stores % kWideBufs];
        uint8_t* rows = box + quarter * (32 * 128);
        // The buffer is free once the store that used it last has read it.
        if (issues && stores >= kWideBufs) asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(kWideBufs - 1) : "memory");
        if (kWholeBoxes) {
          NamedBarrier(2, kWideEpiWarps * 32);
          uint32_t v[32];
          TmemLoad32(taddr + c * kEpiCols, v);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          SwizzledRow(v, rows, lane);
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          NamedBarrier(3, kWideEpiWarps * 32);
          if (issues) {
            TmaStore2D(&map_d, box, n0 + c * kEpiCols, m0);  // out-of-range parts are clipped
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        } else {
          __syncwarp();
          StoreBox32(taddr + c * kEpiCols, rows, lane, &map_d, n0 + c * kEpiCols, m0 + quarter * 32);
        }
      }
      // All TMEM reads of this accumulator are done: hand it back to the MMA warp.
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) MbarArrive(&sh.acc_empty[acc]);
    }
    // The stores must have read shared memory; that they have landed is for the end of the grid.
    if (issues) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
  if (threadIdx.x == 0 && sh.abort && error_flag) *reinterpret_cast<volatile int*>(error_flag) = 1;
}
