// ---- two CTAs per tile -------------------------------------------------------------------
// Two CTAs of a cluster share one 256 x TN tile: each loads its own 128 rows of A and its own TN / 2
// columns of B, the leader issues tcgen05.mma.cta_group::2 (M256 N=TN K16) which reads B from both
// CTAs' shared memory, and each CTA ends up with its 128 x TN half of the accumulator in its own
// TMEM. Per SM this halves the shared-memory traffic for B, which bounds the one-CTA kernel.
//
// kSplits 1: persistent pairs walk the tiles, the epilogue of a tile overlaps the main loop of the
// next one (two accumulators in TMEM).
//
// kSplits 2 or 4: fewer tiles than pairs. A cluster of that many pairs shares ONE tile along K: each pair
// multiplies its share of the k-blocks and then owns a share of the columns: it reads the other pairs'
// partial sums of them out of their shared memory (the operands' stages, which the MMAs have read by
// then), adds them in the order of the pairs, whoever adds, and stores the result. No workspace, no
// flags in global memory, the same bits in every run. 8192 x 512 x 512 (4 tiles for 74 pairs): 45 -> 18.5 us,
// 8192 x 1024 x 1024: 45 -> 29 us.
//
// A k-block of a 256 x 256 tile takes some 590 cycles, its MMAs 512 and its loads as many (64 bytes per
// cycle is what an SM gets out of L2), whatever the number of stages and of issuing threads; the clock
// under this load is 1.6 to 1.9 GHz.
//
// The epilogue's warps store 32 rows each on their own (StoreBox32) and never wait for one another. While later
// tiles are multiplied four of them do it: eight warps' bursts of stores hold up the main loop's loads (4096 x 8192 x 2048:
// 118 -> 124 us). So do two boxes of a warp in flight, where the main loop is long enough to hide them one by one
// (1024 x 4096 x 4096: 38.1 -> 39.9 us, 2000 x 10000 x 4000: 147 -> 157); up to kShortKBlocks it is not, and a warp has two buffers of
// 4 KiB (559 x 680 x 13744: 24.2 -> 22.7 us, 640 x 8192 x 8192: 105 -> 99). A pair's last tile, which nothing hides, goes
// out by all eight through the stages, every box of a warp in flight.
constexpr int kPairThreads = 384;
constexpr int kPairEpiWarps = 8;
constexpr int kShortKBlocks = 14;  // 900 rows: 900 x 3000 x 3000 24.4 and 24.0 us with one and with two buffers
constexpr uint32_t kPeerBitMask = 0xFEFFFFFFu;  // clears the lowest CTA-rank bit of a shared::cluster address
constexpr int kPairABytes = kTileK * 128 * 2;   // 128 rows of A: 16 KiB

template <int TN>
struct __align__(1024) PairShared {
  static constexpr int kStages = 6;
  static constexpr int kBBytes = kTileK * (TN / 2) * 2;
  static constexpr int kStageBytes = kPairABytes + kBBytes;
  uint8_t stage[kStages][kStageBytes];  // later this CTA's part of the last tile, or its partial sums: 128 rows x TN fp32
  uint8_t epi[4][2][32 * 128];
  uint64_t full[kStages];
  uint64_t empty[kStages];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  volatile int abort;
  static_assert(kStages * kStageBytes >= 128 * TN * 4, "the result must fit");
};

__device__ __forceinline__ void ClusterSync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// TMA load issued by either CTA of the pair; the bytes are counted on the leader's barrier.
__device__ __forceinline__ void TmaLoad2D_2Cta(void* smem_dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(SmemAddr(smem_dst)), "l"(map), "r"(x), "r"(y), "r"(SmemAddr(bar) & kPeerBitMask) : "memory");
}

template <int TN>
__device__ __forceinline__ void Mma2(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t accumulate) {
  constexpr uint32_t kInstr = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                              (static_cast<uint32_t>(TN >> 3) << 17) | (static_cast<uint32_t>(256 >> 4) << 24);
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(kInstr), "r"(accumulate) : "memory");
}

// Arrive, in the CTAs of `mask` (ranks in the cluster), on the barrier at this shared-memory offset once all
// MMAs issued so far are done.
__device__ __forceinline__ void MmaCommit2(uint64_t* bar, uint16_t mask) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(SmemAddr(bar)), "h"(mask) : "memory");
}

// The address of `local` in the shared memory of CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t PeerAddr(uint32_t local, uint32_t rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
  return remote;
}

__device__ __forceinline__ void MbarArriveOn(uint64_t* bar, uint32_t rank) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(PeerAddr(SmemAddr(bar), rank)) : "memory");
}

// A barrier of the epilogue's warps that tells all of them whether any of them says yes.
__device__ __forceinline__ bool EpilogueAny(bool yes) {
  uint32_t any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.or.pred q, 1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(any) : "r"(static_cast<uint32_t>(yes)), "n"(kPairEpiWarps * 32) : "memory");
  return any != 0;
}

// Tile number `t`, in tiles from the top left corner. The shorter side comes first, so that the tiles that are multiplied
// at the same time share strips of both operands: row by row, 3 x 79 tiles read X from memory once for every row
// (2000 x 520 x 20000: 74.2 -> 65.3 us, 6000 x 800 x 16000: 197 -> 183; as many columns as rows: no difference).
struct TilePlace {
  int m, n;
};
__device__ __forceinline__ TilePlace PlaceOf(int t, int tiles_m, int tiles_n) {
  const bool down = tiles_m < tiles_n;
  const int side = down ? tiles_m : tiles_n, q = t / side, r = t - q * side;
  return {down ? r : q, down ? q : r};
}

template <int TN, int kSplits>
__global__ void __launch_bounds__(kPairThreads, 1)
WgradPairKernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                const __grid_constant__ CUtensorMap map_d, int M, int N, int K, int* error_flag) {
  using Shared = PairShared<TN>;
  constexpr int kStages = Shared::kStages;
  constexpr int kGroups = TN / kEpiCols;  // column groups of a tile
  extern __shared__ uint8_t smem_raw[];
  Shared& sh = *reinterpret_cast<Shared*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t cta_rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(cta_rank));
  const uint32_t side = cta_rank & 1, leader_rank = cta_rank & ~1u;  // the pair's leader has the even rank
  const bool leader = side == 0;
  const int tiles_m = (M + 255) / 256, tiles_n = (N + TN - 1) / TN;
  const int num_tiles = tiles_m * tiles_n;
  const int all_k_blocks = (K + kTileK - 1) / kTileK;
  // Split: one tile per cluster, this pair's share of its k-blocks. Otherwise a cluster is one pair.
  constexpr bool kSplit = kSplits > 1;
  const int share = static_cast<int>(cta_rank >> 1);
  const int first_tile = static_cast<int>(blockIdx.x / (2 * kSplits)), stride = static_cast<int>(gridDim.x / (2 * kSplits));
  const int kb0 = all_k_blocks * share / kSplits, kb1 = all_k_blocks * (share + 1) / kSplits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; s++) {
      MbarInit(&sh.full[s], 1);
      MbarInit(&sh.empty[s], 1);
    }
    for (int b = 0; b < 2; b++) {
      MbarInit(&sh.acc_full[b], 1);
      MbarInit(&sh.acc_empty[b], 2 * 4);  // four warps of both CTAs
    }
    sh.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(SmemAddr(&sh.tmem_base)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  ClusterSync();  // both CTAs' barriers exist before anybody signals across the pair
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = sh.tmem_base;
  WaitForEarlierKernels();

  if (warp == 0) {
    if (lane == 0) {
      uint32_t it = 0;
      for (int tile = first_tile; tile < num_tiles && !sh.abort; tile += stride) {
        const TilePlace at = PlaceOf(tile, tiles_m, tiles_n);
        const int m0 = at.m * 256 + static_cast<int>(side) * 128;
        const int n0 = at.n * TN + static_cast<int>(side) * (TN / 2);
        for (int kb = kb0; kb < kb1; kb++, it++) {
          const int s = it % kStages;
          if (!MbarWait(&sh.empty[s], ((it / kStages) & 1) ^ 1, &sh.abort)) break;
          if (leader) MbarExpectTx(&sh.full[s], 2 * Shared::kStageBytes);  // both CTAs' loads
          uint8_t* a = sh.stage[s];
          uint8_t* b = a + kPairABytes;
          for (int j = 0; j < 2; j++) TmaLoad2D_2Cta(a + j * (kTileK * 128), &map_a, m0 + j * kAtomMN, kb * kTileK, &sh.full[s]);
          for (int j = 0; j < TN / 128; j++) TmaLoad2D_2Cta(b + j * (kTileK * 128), &map_b, n0 + j * kAtomMN, kb * kTileK, &sh.full[s]);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && leader) {
      const uint16_t both = static_cast<uint16_t>(3u << cta_rank);
      uint32_t it = 0, local_tile = 0;
      for (int tile = first_tile; tile < num_tiles && !sh.abort; tile += stride, local_tile++) {
        const int acc = local_tile & 1;
        if (!MbarWait(&sh.acc_empty[acc], ((local_tile >> 1) & 1) ^ 1, &sh.abort)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tmem_d = tmem_base + acc * TN;
        bool ok = true;
        for (int kb = kb0; kb < kb1; kb++, it++) {
          const int s = it % kStages;
          ok = MbarWait(&sh.full[s], (it / kStages) & 1, &sh.abort);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a_addr = SmemAddr(sh.stage[s]);
          const uint32_t b_addr = a_addr + kPairABytes;
#pragma unroll
          for (int kk = 0; kk < kTileK / kMmaK; kk++) {
            uint64_t da = OperandDesc(a_addr + kk * kMmaK * 128, kTileK * 128);
            uint64_t db = OperandDesc(b_addr + kk * kMmaK * 128, kTileK * 128);
            Mma2<TN>(tmem_d, da, db, (kb > kb0) | (kk != 0));
          }
          MmaCommit2(&sh.empty[s], both);
        }
        if (!ok) break;
        MmaCommit2(&sh.acc_full[acc], both);
      }
    }
  } else if (warp >= 4) {
    const int e = warp - 4, quarter = warp & 3, half = e >> 2;  // TMEM lanes 32 * (warp % 4) .. are the warp's own
    const uint32_t lanes = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    if (kSplit) {
      // This pair's partial sums into shared memory, box by box as a TMA store would want them.
      if (MbarWait(&sh.acc_full[0], 0, &sh.abort)) {
        LetNextKernelStart();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int g = half * (kGroups / 2); g < (half + 1) * (kGroups / 2); g++) {
          uint32_t v[32];
          TmemLoad32(lanes + g * kEpiCols, v);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          SwizzledRow(v, &sh.stage[0][0] + (g * 4 + quarter) * (32 * 128), lane);
        }
      }
    } else {
      const int last = first_tile + (num_tiles - 1 - first_tile) / stride * stride;
      const int m = static_cast<int>(side) * 128 + quarter * 32;
      const bool two_bufs = all_k_blocks <= kShortKBlocks;
      uint32_t local_tile = 0;
      bool ok = half == 0;
      for (int tile = first_tile; tile < last && ok; tile += stride, local_tile++) {
        const int acc = local_tile & 1;
        ok = MbarWait(&sh.acc_full[acc], (local_tile >> 1) & 1, &sh.abort);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const TilePlace at = PlaceOf(tile, tiles_m, tiles_n);
        for (int g = 0; g < kGroups; g++) {
          // The buffer is free once the store that used it last has read it.
          if (lane == 0) {
            if (two_bufs) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
            else asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          }
          __syncwarp();
          StoreBox32(lanes + acc * TN + g * kEpiCols, sh.epi[e][two_bufs ? g & 1 : 0], lane, &map_d, at.n * TN + g * kEpiCols, at.m * 256 + m);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) MbarArriveOn(&sh.acc_empty[acc], leader_rank);
      }
      // Once the last accumulator is full every load has landed and every MMA has read the stages.
      local_tile = static_cast<uint32_t>((last - first_tile) / stride);
      const int acc = local_tile & 1;
      if (ok) ok = MbarWait(&sh.acc_full[acc], (local_tile >> 1) & 1, &sh.abort);
      if (EpilogueAny(ok)) {
        LetNextKernelStart();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const TilePlace at = PlaceOf(last, tiles_m, tiles_n);
        for (int g = half * (kGroups / 2); g < (half + 1) * (kGroups / 2); g++)
          StoreBox32(lanes + acc * TN + g * kEpiCols, &sh.stage[0][0] + (g * 4 + quarter) * (32 * 128), lane, &map_d,
                     at.n * TN + g * kEpiCols, at.m * 256 + m);
      }
    }
  }
  __syncwarp();
  if (kSplit) {
    ClusterSync();  // every pair's partial sums are in place
    if (warp >= 4 && !sh.abort) {
      const int quarter = warp & 3, half = (warp - 4) >> 2;
      const TilePlace at = PlaceOf(first_tile, tiles_m, tiles_n);
      const int m0 = at.m * 256 + static_cast<int>(side) * 128 + quarter * 32;
      const int n0 = at.n * TN;
      constexpr int mine = kGroups / kSplits;
      for (int i = half; i < mine; i += 2) {
        const int g = share * mine + i;
        // Box by box at the same offset in every CTA, so that a warp reads 512 bytes in a row; row by
        // row, as the accumulator is held, other CTAs' memory gave 6 bytes per ns.
        uint8_t* buf = &sh.stage[0][0] + (g * 4 + quarter) * (32 * 128);  // only this warp reads this pair's own
        const uint32_t box = SmemAddr(buf) + lane * 16;
        float4 x[kSplits][8];  // all loads before the first sum: each takes about a microsecond
#pragma unroll
        for (int p = 0; p < kSplits; p++) {
          const uint32_t from = PeerAddr(box, 2 * p + side);
#pragma unroll
          for (int j = 0; j < 8; j++)
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(x[p][j].x), "=f"(x[p][j].y), "=f"(x[p][j].z), "=f"(x[p][j].w) : "r"(from + j * 512) : "memory");
        }
#pragma unroll
        for (int p = 1; p < kSplits; p++) {
#pragma unroll
          for (int j = 0; j < 8; j++) {
            x[0][j].x += x[p][j].x;
            x[0][j].y += x[p][j].y;
            x[0][j].z += x[p][j].z;
            x[0][j].w += x[p][j].w;
          }
        }
#pragma unroll
        for (int j = 0; j < 8; j++) *reinterpret_cast<float4*>(buf + j * 512 + lane * 16) = x[0][j];
        StoreBuffer(buf, lane, &map_d, n0 + g * kEpiCols, m0);
      }
    }
    __syncwarp();
  }
  // The stores must have read shared memory; that they have landed is for the end of the grid.
  if (warp >= 4 && lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  ClusterSync();  // the peers may still be signalling into, or reading, this CTA's shared memory
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
  if (threadIdx.x == 0 && sh.abort && error_flag) *reinterpret_cast<volatile int*>(error_flag) = 1;
}
