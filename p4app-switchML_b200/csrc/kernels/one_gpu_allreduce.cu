// ALGO_STAGED and ALGO_PUSH for ranks that all live on this GPU and whose tensors all of them can address: slots and
// flags as between GPUs, without the trips that only the fabric asks for.
//
//   loader   brings its tile into the slots: the shards of the other ranks, not its own                  [phase 1]
//   reducer  adds its own shard, read from the tensor, and the others' out of the slots; writes the result into
//            the outputs of ALL ranks                                                                    [phase 2]
// Nothing is copied out of the slots. An element crosses the GPU's L2 3 to 4 times (read; into a slot and out of it
// unless it is the owner's; written), six times in ALGO_STAGED and five in ALGO_PUSH between GPUs. That traffic
// bounds large messages; the others are bound by trips to L2 that follow one another in a tile (700 to 1000 cycles
// each), by the fence in front of a flag (900 cycles on an idle SM, 2000 to 3000 behind its stores) and, in the exact
// mode, by instructions. Hence:
//   - No warp waits for another one of its CTA. Each loads or reduces its own part of every tile at its own pace
//     and notes how far it has come; the signaler warp turns the slowest note of a role into the role's flag, the
//     listener warp asks for the peers' flags and leaves them in shared memory. (With every warp asking for itself,
//     each trip to L2 took 1000 to 2000 cycles: every question invalidates the L1.)
//   - MODE_QUANT: a feeder warp brings tiles into shared memory through the TMA unit, where the loader's warps, a chunk of
//     1024 elements each, take both looks at them. They agree on exponents chunk by chunk, without flags: each rank
//     writes a tagged word per block into everybody's memory kOneAhead tiles before it needs the others', and
//     whoever reads a word of an older tile reads again. A second feeder brings the own shard and the others'
//     contributions to it into shared memory for the reducer's warps.
//   - MODE_SUM: two warps drive the TMA unit, each through a ring of its own and for every second tile, so that the end of
//     one tile's stores is not waited for by the next tile.
//   - The host passes all geometry; with divisions in it a warp's way through a tile was half again as long.
// Kernel times against the streaming kernels, us: 2 ranks x 2^22 push exact 49 -> 22, 8 x 2^20 push exact 67 -> 26, 2 x 2^25
// push exact 252 -> 128, 4 x 2^24 staged exact 276 -> 135, staged sum 174 -> 113, push sum 225 -> 114 (82 us at the
// speed of memory). Tiles of half the size 20 to 60 % slower, twice as many slots up to 15 %, half as many 15 to 20 %.
//
// Flow control (S slots per channel, E = kExpRing exponent slots, A = kOneAhead; "through k": tiles up to k from everybody):
//   * slot k % S is refilled, and the scale factors of tile k - S are overwritten, after phase 2 through k - S;
//   * a warp publishes the exponents of its chunk of tile k + A after it has read everybody's of tile k - 1. Whoever has
//     published that one has read those of tile k - 2 - A before, so the words of tile k + A - E are free if
//     E >= 2 A + 2. Nobody else reads them.
// In place: a result is written to a shard after phase 1 from everybody, that is after every other loader has read it,
// and the owner's input has been read by then, or is read by the thread that overwrites it.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <type_traits>

#include "kernels/allreduce_kernels.h"
#include "kernels/bulk_copy.cuh"
#include "kernels/device_sync.cuh"
#include "kernels/once_per_device.h"
#include "kernels/one_gpu_waits.cuh"
#include "kernels/quant_tile.cuh"
#include "kernels/vector_sum.cuh"
#include "switchml/quant_math.h"

namespace switchml {
namespace kernels {

namespace {

constexpr unsigned kOneQuantTile = 8192;        // elements, largest tile of the exact mode: a chunk per loader warp
constexpr size_t kOneSumTileBytes = 65536;      // largest tile of plain sums
constexpr unsigned kOneChunk = 1024;            // elements of a chunk: whole blocks of every size
constexpr int kOneLoadWarps = 8, kOneAhead = 2;
constexpr int kOneLoadStages = 4, kOneReduceStages = 2;  // exact mode: tiles held by the loader's and by the reducer's warps
constexpr int kOneCopyWarps = 2, kOneCopyStages = 6;
constexpr unsigned kOneCopyBytes = 16384;
constexpr size_t kOneRingBytes = kOneCopyWarps * kOneCopyStages * kOneCopyBytes;
constexpr size_t kOneStageBytes = kOneQuantTile * 4;
static_assert((kOneLoadStages + kOneReduceStages) * kOneStageBytes <= kOneRingBytes, "the tiles must fit");
constexpr unsigned kOneQuantSlots = 8, kOneSumSlots = 4;  // of a channel, at most
static_assert(kExpRing == 8 && kExpRing >= 2 * kOneAhead + 2, "exponent words are still in use when they are published again");

template <int MODE>
struct OneGpuWarps {
  static constexpr int kLoad = MODE == MODE_QUANT ? kOneLoadWarps : kOneCopyWarps;
  static constexpr int kReduce = MODE == MODE_QUANT ? 8 : 16;
  static constexpr int kFeeders = MODE == MODE_QUANT ? 2 : 0;  // bring tiles into shared memory
  static constexpr int kThreads = (kLoad + kReduce + kFeeders + 2) * 32;  // two more talk to the peers
};

static_assert(kOneLoadStages + kOneReduceStages <= kOneBarriers && kOneCopyWarps * kOneCopyStages <= kOneBarriers, "a barrier per stage");

__device__ __forceinline__ void RunOneGpuSignaler(const RankCtx& ctx, OneGpuShared* sh, int channel, Epoch base, unsigned ntiles) {
  const int lane = threadIdx.x & 31, phase = lane < 8 ? 0 : lane < 16 ? 1 : 2, peer = lane & 7;
  Epoch* const flag = phase > 0 && lane < 24 && peer < ctx.nranks ? FlagPtr(ctx.stage_peer[peer], channel, phase, ctx.rank) : nullptr;
  unsigned told = phase == 0 ? ntiles : 0;  // (nothing is told in phase 0)
  for (;;) {
    unsigned v = LoadSharedAcquire(&sh->next[lane]);
    __syncwarp();
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
    const unsigned other = __shfl_xor_sync(0xffffffffu, v, 8);
    if (lane >= 16) v = min(v, other);
    v = min(v, ntiles);
    const bool news = v > told;
    if (__any_sync(0xffffffffu, news)) {
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
      if (news && flag) asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(flag), "l"(base + v) : "memory");
      told = v;
    } else if (Failed(sh)) {
      return;
    } else {
      __nanosleep(20);
    }
    if (__all_sync(0xffffffffu, told >= ntiles)) return;
  }
}

// The listener warp: asks for the flags of all ranks and leaves in shared memory how far each phase has come.
__device__ __forceinline__ void RunOneGpuListener(const RankCtx& ctx, OneGpuShared* sh, int channel, Epoch base, unsigned ntiles, unsigned slots) {
  const int lane = threadIdx.x & 31, phase = lane >> 3, rank = lane & 7;
  const Epoch* const flag = phase > 0 && lane < 24 && rank < ctx.nranks ? FlagPtr(ctx.stage_peer[ctx.rank], channel, phase, rank) : nullptr;
  unsigned seen = 0;
  while (!Failed(sh)) {
    unsigned v = ntiles;
    if (flag) {
      const Epoch e = LoadAcquire(ctx, flag);
      v = e > base ? static_cast<unsigned>(min(e - base, static_cast<Epoch>(ntiles))) : 0;
    }
    __syncwarp();
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (v > seen) {
      seen = v;
      if (rank == 0 && lane < 24) StoreSharedRelease(&sh->seen[phase], v);
    }
    // What the CTA's warps will still ask for: all of phase 1, and room for the last tile.
    if (__all_sync(0xffffffffu, seen >= ntiles || (phase == 2 && seen + slots >= ntiles))) return;
    __nanosleep(20);
  }
}

// On the way out: until the phase of `bar` with this parity is complete, with a limit of its own.
__device__ __forceinline__ void Drain(unsigned long long* bar, uint32_t parity) {
  for (int spins = 0; spins < (1 << 16); spins++)
    if (TryWaitParity(bar, parity)) return;
}

// One lane: a bulk load of `bytes` (a multiple of 16) that completes on `bar`.
__device__ __forceinline__ void BulkLoad(char* smem, const char* from, unsigned bytes, unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(BulkSmemAddr(smem)), "l"(from), "r"(bytes), "r"(BulkSmemAddr(bar)) : "memory");
}
__device__ __forceinline__ void ExpectBytes(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(BulkSmemAddr(bar)), "r"(bytes) : "memory");
}

// Geometry of a launch, the same for all ranks: no CTA divides.
struct OneGpuPlan {
  unsigned size, per;             // elements of a tile and of its shards
  unsigned tail, tail_per;        // ... of the job's last tile
  unsigned tiles, channel_tiles;  // of the job, and of every channel but the last
  unsigned slots;                 // of a channel, a power of two
  size_t slot0, slot_pitch;       // where the slots of channel 0 begin in a staging region, and how far those of the next channel are
  size_t exp0, exp_pitch;         // the same for the exponent words
  unsigned block_words;           // exponent words of a block: a power of two, at least the number of ranks
};

// The tiles of one channel, and where their pieces lie. A shard is whole units, so that no block and no row of 128 lies
// in two.
// kRanks: their number, or 0 for any.
template <int ELEM, int MODE, bool kPush, int kRanks>
struct Tiles {
  static constexpr unsigned kIn = ELEM == ELEM_BF16 ? 2 : 4;       // bytes of an element of the tensors
  static constexpr unsigned kSlot = MODE == MODE_QUANT ? 4 : kIn;  // ... in the slots
  const RankCtx& ctx;
  const JobArgs& job;
  const int channel, n, me;  // n: kRanks where that says it (for the compiler)
  const unsigned size, slots;
  unsigned ntiles;
  unsigned long long first;  // the channel's first element
  const char* in;            // there, in this rank's tensor
  char* mine;                // the channel's slots in this rank's staging region
  size_t slot0;              // where they begin in any rank's region
#ifdef SWITCHML_CHECKED
  const OneGpuPlan& plan;
  OneGpuShared* const sh;
  const char* const ring;
#endif

  __device__ __forceinline__ Tiles(const RankCtx& c, const JobArgs& j, const OneGpuPlan& plan, int ch, OneGpuShared* sh, const char* ring)
      : ctx(c), job(j), channel(ch), n(kRanks ? kRanks : c.nranks), me(c.rank), size(plan.size), slots(plan.slots)
#ifdef SWITCHML_CHECKED
        , plan(plan), sh(sh), ring(ring)
#endif
  {
    const unsigned t0 = static_cast<unsigned>(ch) * plan.channel_tiles;
    ntiles = min(plan.channel_tiles, plan.tiles - t0);
    const bool last = t0 + ntiles == plan.tiles;
    end_len_ = last ? plan.tail : size;
    per_ = plan.per;
    end_per_ = last ? plan.tail_per : per_;
    first = static_cast<unsigned long long>(t0) * size;
    in = static_cast<const char*>(job.in) + first * kIn;
    slot0 = plan.slot0 + ch * plan.slot_pitch;
    mine = ctx.stage_peer[me] + slot0;
  }
  __device__ __forceinline__ unsigned Len(unsigned k) const { return k + 1 < ntiles ? size : end_len_; }
  __device__ __forceinline__ unsigned Per(unsigned k) const { return k + 1 < ntiles ? per_ : end_per_; }
  __device__ __forceinline__ unsigned MostPer() const { return per_; }
  __device__ __forceinline__ const char* In(unsigned k) const { return in + static_cast<size_t>(k) * size * kIn; }
  __device__ __forceinline__ unsigned SlotOff(unsigned k) const { return (k & (slots - 1)) * size * kSlot; }
  // kPush: the bytes of one source's area in a slot, and which of the areas of rank `d` is that of rank `s`.
  __device__ __forceinline__ unsigned AreaBytes() const { return per_ * kSlot; }
  static __device__ __forceinline__ int Area(int s, int d) { return s < d ? s : s - 1; }
  // Where this rank puts element `e` of a tile, which lies in the shard of rank `d` that begins at `begin`, in slot 0.
  __device__ __forceinline__ char* Slot(int d, unsigned begin, unsigned e) const {
    if (!kPush) return mine + static_cast<size_t>(e) * kSlot;
    return ctx.stage_peer[d] + slot0 + Area(me, d) * AreaBytes() + (e - begin) * kSlot;
  }
  // The others' contributions to this rank's shard (which begins at `sb`) in slot 0: rank r's is r * Apart() further
  // (staged; the ranks' staging regions lie side by side), the i-th area's i * Apart() (push).
  __device__ __forceinline__ const char* Others(unsigned sb) const {
    return kPush ? mine : ctx.stage_peer[0] + slot0 + static_cast<size_t>(sb) * kSlot;
  }
  __device__ __forceinline__ size_t Apart() const { return kPush ? AreaBytes() : ctx.stage_bytes; }
  __device__ __forceinline__ char* Out(int p, unsigned long long e) const { return job.user_peer[p] + (job.out_offset + e * kIn); }

  // Whether an access lies in what it is meant for: this channel's part of the tensor, of rank r's slots, exponent words and
  // output; the stages; the scale factors. The checked build (-DSWITCHML_CHECKED) asks for each: one that does not is left out,
  // and the CTA fails with STATUS_BOUNDS. Otherwise always true.
#ifdef SWITCHML_CHECKED
  __device__ __forceinline__ bool Inside(const void* p, size_t bytes, const void* begin, size_t room, unsigned aligned) const {
    const char *a = static_cast<const char*>(p), *b = static_cast<const char*>(begin);
    if (a >= b && bytes <= room && static_cast<size_t>(a - b) <= room - bytes && reinterpret_cast<uintptr_t>(p) % aligned == 0) return true;
    if (atomicExch(&sh->failed, 1) == 0) ReportStatus(ctx, STATUS_BOUNDS | (channel << 8));
    return false;
  }
  __device__ __forceinline__ size_t Bytes() const { return (static_cast<size_t>(ntiles - 1) * size + end_len_) * kIn; }
  __device__ __forceinline__ bool InTensor(const void* p, unsigned bytes, unsigned aligned = 1) const {
    return Inside(p, bytes, in, first * kIn + Bytes() <= job.numel * kIn ? Bytes() : 0, aligned);
  }
  __device__ __forceinline__ bool InSlots(int r, const void* p, unsigned bytes, unsigned aligned = 1) const {
    const size_t room = static_cast<size_t>(slots) * size * kSlot;
    return Inside(p, bytes, ctx.stage_peer[r] + slot0, room <= plan.slot_pitch && slot0 + room <= ctx.stage_bytes ? room : 0, aligned);
  }
  __device__ __forceinline__ bool InWords(int r, const void* p, unsigned bytes) const {
    const size_t begin = plan.exp0 + channel * plan.exp_pitch;
    return Inside(p, bytes, ctx.stage_peer[r] + begin, begin + plan.exp_pitch <= ctx.stage_bytes ? plan.exp_pitch : 0, bytes);
  }
  __device__ __forceinline__ bool InOut(int r, const void* p, unsigned bytes) const {
    const size_t begin = job.out_offset + first * kIn;
    return Inside(p, bytes, job.user_peer[r] + begin, begin + Bytes() <= job.user_bytes ? Bytes() : 0, bytes);
  }
  __device__ __forceinline__ bool InStages(const void* p, unsigned bytes, unsigned aligned = 16) const {
    return Inside(p, bytes, ring, kOneRingBytes, aligned);
  }
  __device__ __forceinline__ bool InStage(int s, const void* p, unsigned bytes) const {
    return Inside(p, bytes, ring + s * kOneStageBytes, kOneStageBytes, bytes);
  }
  __device__ __forceinline__ bool InScales(const float* all, const float* p) const {
    return Inside(p, 4, all, kOneQuantSlots * (kOneQuantTile / 32) * sizeof(float), 4);
  }
#else
  __device__ __forceinline__ bool InTensor(const void*, unsigned, unsigned = 1) const { return true; }
  __device__ __forceinline__ bool InSlots(int, const void*, unsigned, unsigned = 1) const { return true; }
  __device__ __forceinline__ bool InWords(int, const void*, unsigned) const { return true; }
  __device__ __forceinline__ bool InOut(int, const void*, unsigned) const { return true; }
  __device__ __forceinline__ bool InStages(const void*, unsigned, unsigned = 16) const { return true; }
  __device__ __forceinline__ bool InStage(int, const void*, unsigned) const { return true; }
  __device__ __forceinline__ bool InScales(const float*, const float*) const { return true; }
#endif

 private:
  unsigned end_len_, per_, end_per_;
};

// ---- loaders ----------------------------------------------------------------------------
// Exact mode: brings the tiles into the loader warps' stages.
template <int ELEM, bool kPush, int kRanks>
__device__ __forceinline__ void FeedLoader(const Tiles<ELEM, MODE_QUANT, kPush, kRanks>& tiles, int lane, OneGpuShared* sh, char* ring) {
  constexpr unsigned kIn = Tiles<ELEM, MODE_QUANT, kPush, kRanks>::kIn;
  unsigned k = 0;
  if (lane == 0) asm volatile("fence.proxy.async.global;" ::: "memory");  // the input's producers used ordinary stores
  for (; k < tiles.ntiles; k++) {
    if (k >= kOneLoadStages && !WaitForNotes(tiles.ctx, tiles.channel, sh, kNoteLoaded, k + 1 - kOneLoadStages)) break;
    const unsigned s = k % kOneLoadStages, bytes = tiles.Len(k) / kOneChunk * kOneChunk * kIn;
    if (lane == 0) {
      ExpectBytes(&sh->full[s], bytes);
      if (bytes > 0 && tiles.InTensor(tiles.In(k), bytes, 16) && bytes <= kOneStageBytes)
        BulkLoad(ring + s * kOneStageBytes, tiles.In(k), bytes, &sh->full[s]);
    }
  }
  // Nothing may land in this shared memory once the CTA has gone; after a failure nobody else waits for it.
  for (unsigned t = k > kOneLoadStages ? k - kOneLoadStages : 0; t < k; t++) Drain(&sh->full[t % kOneLoadStages], (t / kOneLoadStages) & 1);
}

// Exact mode: brings the own shard and the others' contributions to it into the reducer warps' stages.
template <int ELEM, bool kPush, int kRanks>
__device__ __forceinline__ void FeedReducer(const Tiles<ELEM, MODE_QUANT, kPush, kRanks>& tiles, int lane, OneGpuShared* sh, char* ring) {
  const RankCtx& ctx = tiles.ctx;
  constexpr unsigned kIn = Tiles<ELEM, MODE_QUANT, kPush, kRanks>::kIn;
  const unsigned cap = tiles.MostPer();
  const int i = lane - 1;  // lane 0: the own shard; the others: one contribution each
  const size_t skip = static_cast<size_t>(kPush || i < tiles.me ? i : i + 1) * tiles.Apart();
  const unsigned to = lane == 0 ? 0 : (kIn + 4 * i) * cap;
  Seen loaded;
  unsigned k = 0;
  for (; k < tiles.ntiles; k++) {
    if (!loaded.Reach(ctx, tiles.channel, 1, k + 1, sh)) break;
    if (k >= kOneReduceStages && !WaitForNotes(ctx, tiles.channel, sh, kNoteReduced, k + 1 - kOneReduceStages)) break;
    const unsigned s = k % kOneReduceStages, len = tiles.Len(k), per = tiles.Per(k);
    const unsigned sb = min(per * tiles.me, len), count = (min(sb + per, len) - sb) & ~7u;
    unsigned long long* bar = &sh->full[kOneLoadStages + s];
    if (lane == 0) ExpectBytes(bar, count * (kIn + 4 * (tiles.n - 1)));
    __syncwarp();
    if (lane < tiles.n && count > 0) {
      const char* from = lane == 0 ? tiles.In(k) + static_cast<size_t>(sb) * kIn : tiles.Others(sb) + skip + tiles.SlotOff(k);
      const unsigned bytes = count * (lane == 0 ? kIn : 4);
      char* const stage = ring + (kOneLoadStages + s) * kOneStageBytes + to;
      asm volatile("fence.proxy.async.global;" ::: "memory");  // the slots were filled with ordinary stores
      if (tiles.InStages(stage, bytes) &&
          (lane == 0 ? tiles.InTensor(from, bytes, 16) : tiles.InSlots(kPush ? tiles.me : i < tiles.me ? i : i + 1, from, bytes, 16)))
        BulkLoad(stage, from, bytes, bar);
    }
  }
  for (unsigned t = k > kOneReduceStages ? k - kOneReduceStages : 0; t < k; t++)  // as above
    Drain(&sh->full[kOneLoadStages + t % kOneReduceStages], (t / kOneReduceStages) & 1);
}

template <int ELEM, bool kPush, int kRanks>
__device__ __forceinline__ void QuantLoader(const Tiles<ELEM, MODE_QUANT, kPush, kRanks>& tiles, const OneGpuPlan& plan, int warp, int lane,
                                            Epoch base, OneGpuShared* sh, const char* ring, float* s_sf) {
  const RankCtx& ctx = tiles.ctx;
  constexpr unsigned kIn = Tiles<ELEM, MODE_QUANT, kPush, kRanks>::kIn;
  const int me = tiles.me, n = tiles.n, shift = 31 - __clz(ctx.block_numel);
  const unsigned tile_blocks = tiles.size >> shift, blocks = kOneChunk >> shift, S = tiles.slots;
  // This warp's chunk of a tile, and where it goes (slot 0) if it lies in one shard, which in whole tiles it nearly always
  // does. The own shard is read from the tensor.
  const unsigned c0 = warp * kOneChunk, d0 = min(c0 / tiles.MostPer(), static_cast<unsigned>(n - 1));
  const bool one_shard = (c0 + kOneChunk - 1) / tiles.MostPer() == d0, own = static_cast<int>(d0) == me;
  char* const to0 = tiles.Slot(one_shard ? d0 : me, d0 * tiles.MostPer(), c0 + lane * 4);
  const char* const held = ring + c0 * kIn;
  // A block's exponents: a word of each rank, in all ranks' memory. Words of tile k lie in exponent slot k % kExpRing.
  constexpr int kWords = kRanks ? kRanks : kMaxRanks;
  const size_t exp0 = plan.exp0 + tiles.channel * plan.exp_pitch + warp * blocks * plan.block_words * 4;  // this chunk's in slot 0
  const unsigned exp_bytes = tile_blocks * plan.block_words * 4;
  auto rows = [&](unsigned k, float4 (&x)[8]) {
    if (c0 + kOneChunk <= tiles.Len(k)) {
      const char* smem = held + k % kOneLoadStages * kOneStageBytes;
#pragma unroll
      for (int u = 0; u < 8; u++) {
        x[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (tiles.InStage(k % kOneLoadStages, smem + (u * 32 + lane) * 4 * kIn, 4 * kIn)) x[u] = LoadGroupAsFloat<ELEM>(smem, u * 32 + lane);
      }
    } else {  // the job's end: from the tensor
      const char* in = tiles.In(k);
      const unsigned len = tiles.Len(k);
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const unsigned e = c0 + u * 128 + lane * 4;
        x[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (e < len && !tiles.InTensor(in + e * kIn, min(4u, len - e) * kIn, min(4u, len - e) == 4 ? 4 * kIn : kIn)) continue;
        if (e + 4 <= len) {
          x[u] = LoadGroupAsFloat<ELEM>(in, e / 4);
        } else {
          if (e < len) x[u].x = TileLoadAsFloat(in, e, ELEM);
          if (e + 1 < len) x[u].y = TileLoadAsFloat(in, e + 1, ELEM);
          if (e + 2 < len) x[u].z = TileLoadAsFloat(in, e + 2, ELEM);
        }
      }
    }
  };
  unsigned published = 0;
  auto publish = [&](unsigned k) {
    if (!WaitForBytes(ctx, tiles.channel, &sh->full[k % kOneLoadStages], (k / kOneLoadStages) & 1, sh)) return false;
    if (c0 < tiles.Len(k)) {
      float4 x[8];
      rows(k, x);
      const size_t exp_off = exp0 + (k % kExpRing) * exp_bytes + me * 4;
      const unsigned tag = static_cast<unsigned>(base + k + 1) << 8;
      PublishRows8(ctx.block_numel, lane, x, 0, [&](size_t block, int exponent) {
        for (int p = 0; p < n; p++) {
          char* const to = ctx.stage_peer[p] + exp_off + block * plan.block_words * 4;
          if (tiles.InWords(p, to, 4)) asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(to), "r"(tag | (exponent + 128)) : "memory");
        }
      });
    }
    ++published;
    return true;
  };
  // Lane b has those of the chunk's block b on their way from L2 while the tile before theirs is quantised.
  unsigned word[kWords];
  auto fetch_words = [&](unsigned k) {
    if (static_cast<unsigned>(lane) >= blocks || c0 + (lane << shift) >= tiles.Len(k)) return;
    const char* from = ctx.stage_peer[me] + exp0 + (k % kExpRing) * exp_bytes + lane * plan.block_words * 4;
    if (!tiles.InWords(me, from, kWords == 2 ? 8 : 16)) return;
    if constexpr (kWords == 2) {
      asm volatile("ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%2];" : "=r"(word[0]), "=r"(word[1]) : "l"(from) : "memory");
    } else {
#pragma unroll
      for (int i = 0; i < kWords; i += 4)
        if (i < n)
          asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(word[i]), "=r"(word[i + 1]), "=r"(word[i + 2]), "=r"(word[i + 3]) : "l"(from + i * 4) : "memory");
    }
  };
  // The scale factors of the chunk's blocks, once all ranks' exponents are there. False when the wait ran out.
  auto scale_factors = [&](unsigned k, float* sf) {
    const unsigned tag = static_cast<unsigned>(base + k + 1) & 0xffffffu;
    const bool asks = static_cast<unsigned>(lane) < blocks && c0 + (lane << shift) < tiles.Len(k);
    unsigned long long start = 0;
    for (unsigned spins = 0;; fetch_words(k)) {
      bool there = true;
#pragma unroll
      for (int i = 0; i < kWords; i++)
        if (asks && i < n) there &= (word[i] >> 8) == tag;
      if (__all_sync(0xffffffffu, there)) break;
      if ((++spins & 63) == 0) {
        const unsigned long long now = GlobalTimerNs();
        if (start == 0) start = now;
        const bool late = now - start > ctx.timeout_ns;
        if (__any_sync(0xffffffffu, late || Failed(sh))) {
          if (lane == 0) Fail(ctx, sh, tiles.channel, 0);
          return false;
        }
      }
    }
    if (asks) {
      unsigned m = 0;
#pragma unroll
      for (int i = 0; i < kWords; i++)
        if (i < n) m = max(m, word[i] & 0xff);
      if (tiles.InScales(s_sf, sf + lane)) sf[lane] = quant::ScaleFactorFromBase(static_cast<int>(m) - 128, ctx.quant_base);
    }
    __syncwarp();
    return true;
  };
  Seen reduced;
#pragma unroll
  for (int i = 0; i < kWords; i++) word[i] = 0;
  for (unsigned k = 0; k < tiles.ntiles; k++) {
    while (published < tiles.ntiles && published <= k + kOneAhead)
      if (!publish(published)) return;
    if (k >= S && !reduced.Reach(ctx, tiles.channel, 2, k + 1 - S, sh)) return;
    if (c0 < tiles.Len(k)) {
      float* sf = s_sf + (k & (S - 1)) * tile_blocks + warp * blocks;  // for the reducer, too
      if (!scale_factors(k, sf)) return;
      if (k + 1 < tiles.ntiles) fetch_words(k + 1);
      const bool plain = one_shard && tiles.Len(k) == tiles.size;
      if (!plain || !own) {
        float4 x[8];
        rows(k, x);
        auto quantise = [&](int u, int d, char* to) {
          const float* const scale = sf + ((u * 128 + lane * 4) >> shift);
          if (!tiles.InScales(s_sf, scale) || !tiles.InSlots(kPush ? d : me, to, 16, 16)) return;
          const float f = *scale;
          int4 q;
          q.x = quant::Quantize(x[u].x, f);
          q.y = quant::Quantize(x[u].y, f);
          q.z = quant::Quantize(x[u].z, f);
          q.w = quant::Quantize(x[u].w, f);
          *reinterpret_cast<int4*>(to) = q;
        };
        if (plain) {
          char* to = to0 + tiles.SlotOff(k);
#pragma unroll
          for (int u = 0; u < 8; u++) quantise(u, d0, to + u * 512);
        } else {
          const unsigned per = tiles.Per(k), len = tiles.Len(k);
#pragma unroll
          for (int u = 0; u < 8; u++) {
            const unsigned row = c0 + u * 128, e = row + lane * 4, d = row / per;
            if (static_cast<int>(d) != me && e < len) quantise(u, d, tiles.Slot(d, d * per, e) + tiles.SlotOff(k));
          }
        }
      }
    }
    Note(sh, kNoteLoaded + warp, lane, k + 1);
  }
}

template <int ELEM, bool kPush, int kRanks>
__device__ __forceinline__ void CopyLoader(const Tiles<ELEM, MODE_SUM, kPush, kRanks>& tiles, int warp, int lane, OneGpuShared* sh, char* rings) {
  const RankCtx& ctx = tiles.ctx;
  constexpr unsigned kEsz = Tiles<ELEM, MODE_SUM, kPush, kRanks>::kIn;
  const int n = ctx.nranks, me = ctx.rank, pieces = kPush ? n - 1 : 2;
  char* const ring = rings + static_cast<size_t>(warp) * kOneCopyStages * kOneCopyBytes;
  unsigned long long* const full = sh->full + warp * kOneCopyStages;
  // Piece `i` of a tile, in elements: the shard of the i-th rank after this one (push), or what lies before and behind
  // the own shard (staged).
  auto piece = [&](unsigned k, int i, int* d, unsigned* begin, unsigned* end) {
    const unsigned len = tiles.Len(k), per = tiles.Per(k);
    *d = kPush ? (me + 1 + i < n ? me + 1 + i : me + 1 + i - n) : me;
    const unsigned b = min(per * *d, len), e = min(b + per, len);
    *begin = kPush ? b : i == 0 ? 0 : e;
    *end = kPush ? e : i == 0 ? b : len;
  };
  unsigned load_k = warp, load_off = 0, loads = 0, stores = 0;
  int load_i = 0;
  auto load_next = [&] {  // lane 0: the next copy's load, of whatever tile
    while (load_k < tiles.ntiles) {
      int d;
      unsigned b, e;
      piece(load_k, load_i, &d, &b, &e);
      const unsigned bytes = (e - b) * kEsz & ~15u;
      if (load_i < pieces && load_off < bytes) {
        const unsigned size = min(bytes - load_off, kOneCopyBytes), s = loads % kOneCopyStages;
        const char* const from = tiles.In(load_k) + static_cast<size_t>(b) * kEsz + load_off;
        ExpectBytes(full + s, size);
        if (tiles.InTensor(from, size, 16) && tiles.InStages(ring + s * kOneCopyBytes, size)) BulkLoad(ring + s * kOneCopyBytes, from, size, full + s);
        ++loads;
        load_off += size;
        return;
      }
      load_off = 0;
      if (++load_i >= pieces) {
        load_i = 0;
        load_k += kOneCopyWarps;
      }
    }
  };
  auto run = [&] {
    if (lane == 0) {
      asm volatile("fence.proxy.async.global;" ::: "memory");
#pragma unroll 1
      for (int s = 0; s < kOneCopyStages - 1; s++) load_next();
    }
    Seen reduced;
    for (unsigned k = warp; k < tiles.ntiles; k += kOneCopyWarps) {
      const unsigned S = tiles.slots;
      if (k >= S && !reduced.Reach(ctx, tiles.channel, 2, k + 1 - S, sh)) return;
      const unsigned slot_off = tiles.SlotOff(k);
      for (int i = 0; i < pieces; i++) {
        int d;
        unsigned b, e;
        piece(k, i, &d, &b, &e);
        const unsigned bytes = (e - b) * kEsz & ~15u;
        for (unsigned off = 0; off < bytes; off += kOneCopyBytes) {
          const unsigned s = stores % kOneCopyStages;
          if (!WaitForBytes(ctx, tiles.channel, full + s, (stores / kOneCopyStages) & 1, sh)) return;
          ++stores;
          if (lane == 0) {
            char* const to = tiles.Slot(d, b, b) + slot_off + off;
            const unsigned size = min(bytes - off, kOneCopyBytes);
            if (tiles.InSlots(kPush ? d : me, to, size, 16) && tiles.InStages(ring + s * kOneCopyBytes, size))
              asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                           ::"l"(to), "r"(BulkSmemAddr(ring + s * kOneCopyBytes)), "r"(size) : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");  // the buffer of the store before this one is free
            load_next();
          }
          __syncwarp();
        }
        // Fewer than 16 bytes, at the job's end.
        for (unsigned j = b + bytes / kEsz + lane; j < e; j += 32) {
          char* to = tiles.Slot(d, b, j) + slot_off;
          const char* from = tiles.In(k) + static_cast<size_t>(j) * kEsz;
          if (!tiles.InSlots(kPush ? d : me, to, kEsz, kEsz) || !tiles.InTensor(from, kEsz, kEsz)) continue;
          if (kEsz == 4) *reinterpret_cast<unsigned*>(to) = *reinterpret_cast<const unsigned*>(from);
          else *reinterpret_cast<unsigned short*>(to) = *reinterpret_cast<const unsigned short*>(from);
        }
      }
      if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
      Note(sh, kNoteLoaded + warp, lane, k + kOneCopyWarps);
    }
  };
  run();
  // After a failure: nothing may land in, or be read from, this shared memory once the CTA has gone.
  if (lane == 0) {
    for (; stores < loads; stores++) Drain(full + stores % kOneCopyStages, (stores / kOneCopyStages) & 1);
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  __syncwarp();
}

// ---- reducers ---------------------------------------------------------------------------
// A tile's shard as a reducer sees it.
struct ShardView {
  const char* own;          // in the tensor
  const char* others;       // rank r's contribution is r * apart further (staged), or the a-th area's a * apart (push)
  size_t apart;
  unsigned long long at;    // the shard's first element in the outputs
  const float* sf;          // scale factors of the tile
  const float* scales;      // ... of all slots
  unsigned sb;              // the shard's first element in the tile
  int shift;
};

// U vectors of 16 bytes (v, v + stride, ...) of all ranks, all loads in flight together.
template <int ELEM, bool kPush, int R, int U, typename T>
__device__ __forceinline__ void SumVectors(const T& tiles, const ShardView& s, unsigned v, unsigned stride) {
  constexpr int kMost = R ? R : kMaxRanks;
  const int n = tiles.n, me = tiles.me;
  uint4 x[kMost][U];
#pragma unroll
  for (int i = 0; i < kMost; i++) {
    if (i >= n) continue;
    const char* src = s.others + static_cast<size_t>(kPush ? i - 1 : i) * s.apart;
    if (i == (kPush ? 0 : me)) src = s.own;
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint4* const from = reinterpret_cast<const uint4*>(src) + v + u * stride;
      x[i][u] = make_uint4(0, 0, 0, 0);
      if (i == (kPush ? 0 : me) ? tiles.InTensor(from, 16, 16) : tiles.InSlots(kPush ? me : i, from, 16, 16)) x[i][u] = __ldcg(from);
    }
  }
  // In rank order from zero (staged), or the own shard first (push): the order of the streaming kernels.
  VecAcc<ELEM> acc[U];
#pragma unroll
  for (int u = 0; u < U; u++) {
    if (kPush) acc[u].Init(x[0][u]);
    else acc[u].Zero();
  }
#pragma unroll
  for (int i = kPush ? 1 : 0; i < kMost; i++) {
    if (i >= n) continue;
#pragma unroll
    for (int u = 0; u < U; u++) acc[u].Add(x[i][u]);
  }
#pragma unroll
  for (int u = 0; u < U; u++) x[0][u] = acc[u].Finish(tiles.job.post_scale);
  for (int p = 0; p < n; p++) {
    uint4* out = reinterpret_cast<uint4*>(tiles.Out(p, s.at));
#pragma unroll
    for (int u = 0; u < U; u++)
      if (tiles.InOut(p, out + v + u * stride, 16)) __stcs(out + v + u * stride, x[0][u]);  // leaves L2 to the slots: 4 x 2^24 119 -> 113 us
  }
}

// Exact mode: U groups of four elements of the own shard, out of shared memory: those at `held` + u * stride (own values,
// quantised here), and at `others` + u * stride, `area` bytes further, ... With 2, 4 or 8 ranks the scale factors are powers
// of two: dividing by them is multiplying by their reciprocals.
template <int ELEM, int R, int U, typename T>
__device__ __forceinline__ void QuantGroups(const T& tiles, const ShardView& s, const char* held, const char* others, unsigned area, unsigned g) {
  constexpr unsigned kStride = OneGpuWarps<MODE_QUANT>::kReduce * 32;
  const int n = tiles.n;
  const float post_scale = tiles.job.post_scale;
  float4 y[U];
#pragma unroll
  for (int u = 0; u < U; u++) {
    const float* const scale = s.sf + ((s.sb + (g + u * kStride) * 4) >> s.shift);
    y[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!tiles.InScales(s.scales, scale) || !tiles.InStages(held + (g + u * kStride) * 4 * T::kIn, 4 * T::kIn, 4 * T::kIn) ||
        (n > 1 && !tiles.InStages(others + (n - 2) * area + (g + u * kStride) * 16, 16)))
      continue;
    const float f = *scale;
    const float4 x = LoadGroupAsFloat<ELEM>(held, g + u * kStride);
    auto own = [&](float v) { return static_cast<unsigned>(quant::Quantize(v, f)); };
    uint4 a = make_uint4(own(x.x), own(x.y), own(x.z), own(x.w));  // (sums that wrap: values that saturate)
    const uint4* from = reinterpret_cast<const uint4*>(others) + g + u * kStride;
    for (int i = 0; i < n - 1; i++, from = reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(from) + area)) {
      const uint4 v = *from;
      a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
    }
    const float inv = __uint_as_float(0x7f000000u - __float_as_uint(f));
    auto back = [&](unsigned sum) {
      const int q = static_cast<int>(sum);
      return R ? __int2float_rn(q) * inv : __fdiv_rn(__int2float_rn(q), f);
    };
    y[u] = make_float4(back(a.x), back(a.y), back(a.z), back(a.w));
    if (post_scale != 1.0f) { y[u].x *= post_scale; y[u].y *= post_scale; y[u].z *= post_scale; y[u].w *= post_scale; }
  }
  for (int p = 0; p < n; p++) {
    char* out = tiles.Out(p, s.at);
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (!tiles.InOut(p, out + (g + u * kStride) * 4 * T::kIn, 4 * T::kIn)) continue;
      if (ELEM == ELEM_BF16)
        reinterpret_cast<uint2*>(out)[g + u * kStride] = make_uint2(Float2ToBf16x2(y[u].x, y[u].y), Float2ToBf16x2(y[u].z, y[u].w));
      else
        reinterpret_cast<float4*>(out)[g + u * kStride] = y[u];
    }
  }
}

// One element of the job's ragged end.
template <int ELEM, int MODE, bool kPush, typename T>
__device__ __forceinline__ void ReduceElement(const T& tiles, const ShardView& s, unsigned i) {
  const int n = tiles.n, me = tiles.me;
  for (int j = 0; j < n; j++) {
    const int r = kPush ? (j + me) % n : j;  // (push: the areas of the others, in any order)
    if (r == me ? !tiles.InTensor(s.own + i * T::kIn, T::kIn, T::kIn)
                : !tiles.InSlots(kPush ? me : r, s.others + static_cast<size_t>(kPush ? j - 1 : j) * s.apart + i * T::kSlot, T::kSlot, T::kSlot))
      return;
  }
  unsigned bits;
  if (MODE == MODE_QUANT) {
    if (!tiles.InScales(s.scales, s.sf + ((s.sb + i) >> s.shift))) return;
    const float f = s.sf[(s.sb + i) >> s.shift];
    unsigned a = static_cast<unsigned>(quant::Quantize(TileLoadAsFloat(s.own, i, ELEM), f));
    for (int j = 0; j < n - 1; j++) a += __ldcg(reinterpret_cast<const unsigned*>(s.others + (kPush || j < me ? j : j + 1) * s.apart) + i);
    float y = quant::Dequantize(static_cast<int>(a), f);
    if (tiles.job.post_scale != 1.0f) y *= tiles.job.post_scale;
    bits = __float_as_uint(y);
  } else {
    unsigned a = 0;
    float f = 0.f;
    for (int j = 0; j < n; j++) {
      const char* src = j == (kPush ? 0 : me) ? s.own : s.others + static_cast<size_t>(kPush ? j - 1 : j) * s.apart;
      if (ELEM == ELEM_I32) a += __ldcg(reinterpret_cast<const unsigned*>(src) + i);
      else {
        const float x = ELEM == ELEM_BF16 ? Bf16ToFloat(__ldcg(reinterpret_cast<const unsigned short*>(src) + i)) : __ldcg(reinterpret_cast<const float*>(src) + i);
        f = kPush && j == 0 ? x : f + x;
      }
    }
    if (ELEM != ELEM_I32 && tiles.job.post_scale != 1.0f) f *= tiles.job.post_scale;
    bits = ELEM == ELEM_I32 ? a : __float_as_uint(f);
  }
  for (int p = 0; p < n; p++) {
    char* out = tiles.Out(p, s.at + i);
    if (!tiles.InOut(p, out, T::kIn)) continue;
    if (ELEM == ELEM_BF16) *reinterpret_cast<unsigned short*>(out) = FloatToBf16(__uint_as_float(bits));
    else *reinterpret_cast<unsigned*>(out) = bits;
  }
}

// R: the number of ranks, or 0 for any.
template <int ELEM, int MODE, bool kPush, int R>
__device__ __forceinline__ void Reducer(const Tiles<ELEM, MODE, kPush, R>& tiles, int warp, int lane, OneGpuShared* sh, const char* ring, const float* s_sf) {
  using T = Tiles<ELEM, MODE, kPush, R>;
  constexpr int kWarps = OneGpuWarps<MODE>::kReduce;
  constexpr unsigned kVec = MODE == MODE_QUANT ? 4 : 16 / T::kIn;  // elements that a lane takes at a time
  constexpr int U = R == 0 ? (MODE == MODE_QUANT ? 2 : 1) : 8 / R;  // ... and how often, while more are left
  const RankCtx& ctx = tiles.ctx;
  ShardView s;
  s.shift = 31 - __clz(ctx.block_numel);
  s.apart = tiles.Apart();
  s.scales = s_sf;
  const unsigned tile_blocks = tiles.size >> s.shift;
  Seen loaded;
  for (unsigned k = 0; k < tiles.ntiles; k++) {
    if (MODE == MODE_SUM && !loaded.Reach(ctx, tiles.channel, 1, k + 1, sh)) return;
    const unsigned len = tiles.Len(k), per = tiles.Per(k);
    s.sb = min(per * tiles.me, len);
    const unsigned count = min(s.sb + per, len) - s.sb;
    s.own = tiles.In(k) + static_cast<size_t>(s.sb) * T::kIn;
    s.others = tiles.Others(s.sb) + tiles.SlotOff(k);
    s.at = tiles.first + static_cast<unsigned long long>(k) * tiles.size + s.sb;
    s.sf = s_sf + (k & (tiles.slots - 1)) * tile_blocks;
    unsigned r = warp, nvec;  // rows of 32 vectors
    if constexpr (MODE == MODE_QUANT) {
      nvec = (count & ~7u) / kVec;
      const unsigned stage = k % kOneReduceStages, area = tiles.MostPer() * 4;
      const char* held = ring + (kOneLoadStages + stage) * kOneStageBytes;
      const char* others = held + tiles.MostPer() * T::kIn;
      if (!WaitForBytes(ctx, tiles.channel, &sh->full[kOneLoadStages + stage], (k / kOneReduceStages) & 1, sh)) return;
#pragma unroll 1
      for (; (r + (U - 1) * kWarps) * 32 + 31 < nvec; r += U * kWarps) QuantGroups<ELEM, R, U>(tiles, s, held, others, area, r * 32 + lane);
#pragma unroll 1
      for (; r * 32 < nvec; r += kWarps)
        if (r * 32 + lane < nvec) QuantGroups<ELEM, R, 1>(tiles, s, held, others, area, r * 32 + lane);
    } else {
      nvec = count / kVec;
#pragma unroll 1
      for (; (r + (U - 1) * kWarps) * 32 + 31 < nvec; r += U * kWarps) SumVectors<ELEM, kPush, R, U>(tiles, s, r * 32 + lane, kWarps * 32);
#pragma unroll 1
      for (; r * 32 < nvec; r += kWarps)
        if (r * 32 + lane < nvec) SumVectors<ELEM, kPush, R, 1>(tiles, s, r * 32 + lane, 0);
    }
    if (warp == 0 && nvec * kVec + lane < count) ReduceElement<ELEM, MODE, kPush>(tiles, s, nvec * kVec + lane);
    Note(sh, kNoteReduced + warp, lane, k + 1);
    if (warp == 0 && lane == 0) atomicAdd(ctx.counters, 1ull);
  }
}

template <int ELEM, int MODE, bool kPush, int R>
__global__ void __launch_bounds__(OneGpuWarps<MODE>::kThreads, 1)
AllReduceOneGpuKernel(const __grid_constant__ EmuArgs args, const __grid_constant__ OneGpuPlan plan) {
  extern __shared__ __align__(128) unsigned char s_ring[];
  __shared__ OneGpuShared sh;
  __shared__ float s_sf[MODE == MODE_QUANT ? kOneQuantSlots * kOneQuantTile / 32 : 1];
  __shared__ RankCtx ctx;
  __shared__ JobArgs job;
  constexpr int kLoad = OneGpuWarps<MODE>::kLoad, kReduce = OneGpuWarps<MODE>::kReduce;
  // This rank's arguments as whole words, side by side (see AllReduceEmuKernel).
  static_assert(sizeof(RankCtx) % 4 == 0 && sizeof(JobArgs) % 4 == 0, "copied as words");
  const unsigned* from_ctx = reinterpret_cast<const unsigned*>(&args.ctx[blockIdx.y]);
  const unsigned* from_job = reinterpret_cast<const unsigned*>(&args.job[blockIdx.y]);
  for (unsigned i = threadIdx.x; i < sizeof(RankCtx) / 4; i += blockDim.x) reinterpret_cast<unsigned*>(&ctx)[i] = from_ctx[i];
  for (unsigned i = threadIdx.x; i < sizeof(JobArgs) / 4; i += blockDim.x) reinterpret_cast<unsigned*>(&job)[i] = from_job[i];
  if (threadIdx.x < 32) {
    const int i = threadIdx.x;
    unsigned next = 0xffffffffu;  // no such warp
    if (i < kNoteLoaded) next = 0xffffffffu;
    else if (i < kNoteReduced) next = MODE == MODE_QUANT ? 0 : i - kNoteLoaded < kLoad ? i - kNoteLoaded : next;
    else next = i - kNoteReduced < kReduce ? 0 : next;
    sh.next[i] = next;
    if (i < 3) sh.seen[i] = 0;
    if (i == 0) sh.failed = 0;
    for (int b = i; b < kOneBarriers; b += 32) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(BulkSmemAddr(&sh.full[b])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const int channel = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Epoch base = ctx.epoch_words[channel];
  char* const ring = reinterpret_cast<char*>(s_ring);
  const Tiles<ELEM, MODE, kPush, R> tiles(ctx, job, plan, channel, &sh, ring);
  if (tiles.ntiles > 0) {
    if (warp < kLoad) {
      if constexpr (MODE == MODE_QUANT) QuantLoader<ELEM, kPush, R>(tiles, plan, warp, lane, base, &sh, ring, s_sf);
      else CopyLoader<ELEM, kPush, R>(tiles, warp, lane, &sh, ring);
    } else if (warp < kLoad + kReduce) {
      Reducer<ELEM, MODE, kPush, R>(tiles, warp - kLoad, lane, &sh, ring, s_sf);
    } else if (warp == kLoad + kReduce) {
      RunOneGpuSignaler(ctx, &sh, channel, base, tiles.ntiles);
    } else if (warp == kLoad + kReduce + 1) {
      RunOneGpuListener(ctx, &sh, channel, base, tiles.ntiles, tiles.slots);
    } else if constexpr (MODE == MODE_QUANT) {
      if (warp == kLoad + kReduce + 2) FeedLoader<ELEM, kPush, R>(tiles, lane, &sh, ring);
      else FeedReducer<ELEM, kPush, R>(tiles, lane, &sh, ring);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) ctx.epoch_words[channel] = base + job.epochs;
}

// ---- host side --------------------------------------------------------------------------
// (What QuantLoader loads at a time: 8 bytes with two ranks, else 16.)
unsigned BlockWords(int nranks) { return nranks == 2 ? 2 : nranks <= 4 ? 4 : 8; }
// A channel's exponent words.
size_t ExpBytes(int nranks, int block_numel) { return static_cast<size_t>(kExpRing) * (kOneQuantTile / block_numel) * BlockWords(nranks) * 4; }

// A tile is a multiple of this: whole units on every rank, and whole chunks of the exact mode's loader.
size_t TileUnit(const RankCtx& ctx, int mode) {
  const size_t unit = static_cast<size_t>(ctx.nranks) * (mode == MODE_QUANT && ctx.block_numel > 128 ? ctx.block_numel : 128);
  size_t whole = unit;
  while (mode == MODE_QUANT && whole % kOneChunk) whole += unit;
  return whole;
}

// Elements of the largest tile; 0 if the slots are too small for any.
size_t TileCapacity(const RankCtx& ctx, const JobArgs& job) {
  const size_t in_esz = job.elem_type == ELEM_BF16 ? 2 : 4;
  const size_t by_slot = ctx.slot_bytes / (job.mode == MODE_QUANT ? 4 : in_esz);
  size_t most = job.mode == MODE_QUANT ? kOneQuantTile : kOneSumTileBytes / in_esz;
  if (most > by_slot) most = by_slot;
  const size_t unit = TileUnit(ctx, job.mode);
  return most / unit * unit;
}

template <int ELEM, int MODE, bool kPush, int R>
cudaError_t LaunchRanks(const EmuArgs& emu, int present, const OneGpuPlan& plan, int channels, cudaStream_t stream) {
  void* args[] = {const_cast<EmuArgs*>(&emu), const_cast<OneGpuPlan*>(&plan)};
  const void* kernel = reinterpret_cast<const void*>(AllReduceOneGpuKernel<ELEM, MODE, kPush, R>);
  static std::atomic<unsigned long long> allowed{0};
  int dev = 0;
  cudaGetDevice(&dev);
  const cudaError_t e = OncePerDevice(dev, &allowed, [&] {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kOneRingBytes));
  });
  if (e != cudaSuccess) return e;
  // Cooperative: all CTAs are resident together, which their waiting for one another needs.
  return cudaLaunchCooperativeKernel(kernel, dim3(channels, present), dim3(OneGpuWarps<MODE>::kThreads), args, kOneRingBytes, stream);
}

template <int ELEM, int MODE>
cudaError_t LaunchMode(const EmuArgs& emu, int nranks, int present, const LaunchPlan& launch, cudaStream_t stream) {
  const RankCtx& ctx = emu.ctx[0];
  const JobArgs& job = emu.job[0];
  const unsigned unit = MODE == MODE_QUANT && ctx.block_numel > 128 ? ctx.block_numel : 128;
  OneGpuPlan plan;
  plan.size = static_cast<unsigned>(launch.tile_elems);
  plan.per = plan.size / nranks;
  plan.tiles = static_cast<unsigned>(launch.tiles);
  plan.channel_tiles = launch.epochs;
  plan.tail = static_cast<unsigned>(job.numel - (launch.tiles - 1) * launch.tile_elems);
  plan.tail_per = ((plan.tail + nranks - 1) / nranks + unit - 1) / unit * unit;
  plan.slot0 = ctx.data_offset;
  plan.slot_pitch = ctx.slots_per_channel * ctx.slot_bytes;
  plan.exp0 = ctx.exp_offset;
  plan.block_words = BlockWords(nranks);
  plan.exp_pitch = ExpBytes(nranks, ctx.block_numel);
  const size_t slot = plan.size * static_cast<size_t>(MODE == MODE_QUANT || ELEM != ELEM_BF16 ? 4 : 2);
  plan.slots = 1;
  while (plan.slots < (MODE == MODE_QUANT ? kOneQuantSlots : kOneSumSlots) && 2 * plan.slots * slot <= plan.slot_pitch) plan.slots *= 2;
  // Everything that a CTA indexes lies in its rank's staging region and in its shared memory.
  const size_t channels = launch.channels;
  if (plan.size > (MODE == MODE_QUANT ? kOneQuantTile : kOneSumTileBytes / (ELEM == ELEM_BF16 ? 2 : 4)) || plan.size % (nranks * unit) != 0 ||
      plan.tail == 0 || plan.tail > plan.size || plan.slots * slot > plan.slot_pitch ||
      plan.slot0 + channels * plan.slot_pitch > ctx.stage_bytes ||
      (MODE == MODE_QUANT && (plan.size % kOneChunk != 0 || plan.exp0 + channels * plan.exp_pitch > ctx.stage_bytes)))
    return cudaErrorInvalidValue;
  const bool push = job.algo == ALGO_PUSH;
  const auto start = nranks == 2 ? (push ? LaunchRanks<ELEM, MODE, true, 2> : LaunchRanks<ELEM, MODE, false, 2>)
                   : nranks == 4 ? (push ? LaunchRanks<ELEM, MODE, true, 4> : LaunchRanks<ELEM, MODE, false, 4>)
                   : nranks == 8 ? (push ? LaunchRanks<ELEM, MODE, true, 8> : LaunchRanks<ELEM, MODE, false, 8>)
                                 : (push ? LaunchRanks<ELEM, MODE, true, 0> : LaunchRanks<ELEM, MODE, false, 0>);
  return start(emu, present, plan, launch.channels, stream);
}

}  // namespace

size_t OneGpuExponentBytes(int nranks, int block_numel, int max_channels) { return ExpBytes(nranks, block_numel) * max_channels; }

bool OneGpuFits(const RankCtx& ctx, const JobArgs& job) {
  return (job.algo == ALGO_STAGED || job.algo == ALGO_PUSH) && TileCapacity(ctx, job) > 0;
}

void PlanOneGpu(const RankCtx& ctx, const JobArgs& job, int requested_channels, int max_channels, LaunchPlan* plan) {
  const unsigned long long numel = job.numel ? job.numel : 1;
  const int ch = requested_channels > 0 && requested_channels < max_channels ? requested_channels : max_channels;
  const unsigned long long most = TileCapacity(ctx, job), unit = TileUnit(ctx, job.mode);
  const unsigned long long per_channel = (numel + ch - 1) / ch;
  // As few tiles as it takes, all of the same size.
  const unsigned long long count = (per_channel + most - 1) / most;
  plan->tile_elems = ((per_channel + count - 1) / count + unit - 1) / unit * unit;
  plan->tiles = (numel + plan->tile_elems - 1) / plan->tile_elems;
  const unsigned long long tiles_per_channel = (plan->tiles + ch - 1) / ch;
  plan->elems_per_channel = tiles_per_channel * plan->tile_elems;
  plan->channels = static_cast<int>((numel + plan->elems_per_channel - 1) / plan->elems_per_channel);
  plan->epochs = static_cast<unsigned>(tiles_per_channel);
}

cudaError_t LaunchOneGpuAllReduce(const EmuArgs& args, int nranks, int present, const LaunchPlan& plan, cudaStream_t stream) {
  const JobArgs& job = args.job[0];
  if (job.elem_type == ELEM_I32) return LaunchMode<ELEM_I32, MODE_SUM>(args, nranks, present, plan, stream);
  if (job.mode == MODE_QUANT)
    return (job.elem_type == ELEM_F32 ? LaunchMode<ELEM_F32, MODE_QUANT> : LaunchMode<ELEM_BF16, MODE_QUANT>)(args, nranks, present, plan, stream);
  return (job.elem_type == ELEM_F32 ? LaunchMode<ELEM_F32, MODE_SUM> : LaunchMode<ELEM_BF16, MODE_SUM>)(args, nranks, present, plan, stream);
}

}  // namespace kernels
}  // namespace switchml
