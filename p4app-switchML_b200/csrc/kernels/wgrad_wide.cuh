// The plain GEMM with one CTA per 128 x 256 tile: short reductions (a batch of samples, as in VGG's fully
// connected layers), where dW is much larger than the operands and the time is the time to write it.
// The loads and the MMAs of the next tiles run while a tile is stored:
//   warp 0       TMA producer, a ring of kWideStages stages of 64 K-rows
//   warp 1       MMA issuer, two accumulators in TMEM
//   warp 2       asks for tiles (tile_queue.cuh), allocates TMEM
//   warps 4-11   epilogue: warp w stores rows 32 * (w % 4) .. of columns 128 * (w / 8) .. on its own:
//                tcgen05.ld, swizzled shared memory (kWideBufs buffers per warp), TMA store. The warps do not
//                wait for one another.
constexpr int kWideThreads = 384;
constexpr int kWideEpiWarps = 8;
constexpr int kBoxBytes = 32 * 128;  // 32 rows of 32 fp32 columns

template <int kWideStages, int kWideBufs>
struct __align__(1024) WideShared {
  uint8_t stage[kWideStages][kStageBytes];
  uint8_t epi[kWideEpiWarps][kWideBufs][kBoxBytes];
  TileQueue queue;
  uint64_t full[kWideStages];
  uint64_t empty[kWideStages];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  volatile int abort;
};

template <int kWideStages, int kWideBufs>
__global__ void __launch_bounds__(kWideThreads, 1)
WgradWideKernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                const __grid_constant__ CUtensorMap map_d, int tiles_n, int K, int* error_flag) {
  extern __shared__ uint8_t smem_raw[];
  using Shared = WideShared<kWideStages, kWideBufs>;
  Shared& sh = *reinterpret_cast<Shared*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
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
          const int left = (K - kb * kTileK + kMmaK - 1) / kMmaK;  // steps that have rows at all
          for (int kk = 0; kk < kTileK / kMmaK && kk < left; kk++)
            Mma(tmem_d, OperandDesc(a_addr + kk * kMmaK * 128, kTileK * 128),
                OperandDesc(a_addr + kABytes + kk * kMmaK * 128, kTileK * 128), (kb | kk) != 0);
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
    const int e = warp - 4, quarter = warp & 3, half = e >> 2;  // TMEM lanes 32 * (warp % 4) .. are the warp's own
    uint32_t stores = 0;
    int tile = static_cast<int>(blockIdx.x);
    for (uint32_t t = 0; tile >= 0; tile = NextTile(sh.queue, t++, lane, &sh.abort)) {
      const int m0 = (tile / tiles_n) * kTileM + quarter * 32, n0 = (tile % tiles_n) * kTileN + half * 128;
      const int acc = t & 1;
      if (!MbarWait(&sh.acc_full[acc], (t >> 1) & 1, &sh.abort)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * kTileN + half * 128;
      for (int c = 0; c < 128 / kEpiCols; c++, stores++) {
        // The buffer is free once the store that used it last has read it.
        if (stores >= kWideBufs) {
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(kWideBufs - 1) : "memory");
          __syncwarp();
        }
        StoreBox32(taddr + c * kEpiCols, sh.epi[e][stores % kWideBufs], lane, &map_d, n0 + c * kEpiCols, m0);
      }
      // All TMEM reads of this accumulator are done: hand it back to the MMA warp.
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) MbarArrive(&sh.acc_empty[acc]);
    }
    // The stores must have read shared memory; that they have landed is for the end of the grid.
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
  if (threadIdx.x == 0 && sh.abort && error_flag) *reinterpret_cast<volatile int*>(error_flag) = 1;
}
