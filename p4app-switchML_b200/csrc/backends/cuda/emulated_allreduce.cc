// EmulatedAllReduce (cuda_backend.h): several ranks of one aggregation played by one
// cooperative kernel on one GPU.
//
// A call used to cost 5 to 25 ms around a kernel of 0.1 to 0.4 ms: cudaGetDeviceProperties
// (2.8 ms), seven to nine cudaMalloc / cudaFree pairs (0.2 to 0.3 ms each, and every free
// waits for the device), clears of the whole staging memory and three blocking copies. Now
// the staging memory of a finished call is kept for the next one, and everything the kernel
// has to know travels as a launch argument. Flags, exponent words and epochs need no clearing
// between calls, for the same reason as between the jobs of a context: epochs only grow.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "backends/cuda/cuda_backend.h"
#include "kernels/allreduce_kernels.h"
#include "switchml/quant_math.h"

namespace switchml {

namespace {

using namespace kernels;

// Staging memory of all ranks of a call, with their epochs, counters and status words.
struct EmuWorkspace {
  int device = -1;
  size_t capacity = 0;              // bytes of `memory`
  char* memory = nullptr;           // [epochs and counters][rank 0's staging region][rank 1's] ...
  int* status = nullptr;            // kMaxRanks words of pinned host memory that the kernel writes
  int* status_dev = nullptr;
  std::string layout;               // geometry that the flags and exponent words in `memory` belong to
  unsigned long long epochs = 0;    // that any channel may have used since they were cleared

  ~EmuWorkspace() {
    int current = -1;
    cudaGetDevice(&current);
    if (device >= 0 && device != current) cudaSetDevice(device);
    if (memory) cudaFree(memory);
    if (status) cudaFreeHost(status);
    if (device >= 0 && device != current) cudaSetDevice(current);
  }
};

constexpr unsigned long long kDirectNumel = 1ull << 18;
constexpr size_t kL2Slots = size_t(44) << 20;  // of 126 MB: inputs and outputs stream through it as well

constexpr size_t kEpochBytes = size_t(kMaxRanks) * kMaxChannels * sizeof(unsigned long long);
constexpr size_t kCounterBytes = size_t(kMaxRanks) * 16 * sizeof(unsigned long long);
constexpr size_t kHeadBytes = (kEpochBytes + kCounterBytes + 4095) / 4096 * 4096;

// Workspaces that no call is using. A call takes one out and puts it back when its kernel has
// ended, so calls of several threads never share one. Bounded: at most kKept, together at
// most kKeptBytes; what does not fit is freed at once, and all are given back when an
// allocation fails or by ReleaseEmulationWorkspaces().
class WorkspacePool {
 public:
  static WorkspacePool& Get() {
    static WorkspacePool* pool = new WorkspacePool;  // never destroyed: the CUDA runtime may be gone by then
    return *pool;
  }
  // The workspace of `layout` if there is one, else the smallest that is large enough.
  std::unique_ptr<EmuWorkspace> Take(int device, size_t bytes, const std::string& layout) {
    std::lock_guard<std::mutex> lk(mu_);
    size_t best = free_.size();
    for (size_t i = 0; i < free_.size(); i++) {
      const EmuWorkspace& w = *free_[i];
      if (w.device != device || w.capacity < bytes) continue;
      if (w.layout == layout) {
        best = i;
        break;
      }
      if (best == free_.size() || w.capacity < free_[best]->capacity) best = i;
    }
    if (best == free_.size()) return nullptr;
    std::unique_ptr<EmuWorkspace> w = std::move(free_[best]);
    free_.erase(free_.begin() + best);
    return w;
  }
  void Put(std::unique_ptr<EmuWorkspace> w) {
    std::vector<std::unique_ptr<EmuWorkspace>> drop;  // freed after the lock is gone
    std::lock_guard<std::mutex> lk(mu_);
    free_.push_back(std::move(w));
    auto kept = [&] {
      size_t sum = 0;
      for (const auto& f : free_) sum += f->capacity;
      return sum;
    };
    while (free_.size() > kKept || (!free_.empty() && kept() > kKeptBytes)) {
      drop.push_back(std::move(free_.front()));  // the one that has been lying here longest
      free_.erase(free_.begin());
    }
  }
  void Clear() {
    std::vector<std::unique_ptr<EmuWorkspace>> drop;
    std::lock_guard<std::mutex> lk(mu_);
    drop.swap(free_);
  }

 private:
  static constexpr size_t kKept = 4;
  static constexpr size_t kKeptBytes = size_t(1) << 29;
  std::mutex mu_;
  std::vector<std::unique_ptr<EmuWorkspace>> free_;
};

std::unique_ptr<EmuWorkspace> NewWorkspace(int device, size_t bytes, cudaError_t* e) {
  std::unique_ptr<EmuWorkspace> w(new EmuWorkspace);
  w->device = device;
  *e = cudaMalloc(reinterpret_cast<void**>(&w->memory), bytes);
  if (*e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    WorkspacePool::Get().Clear();
    *e = cudaMalloc(reinterpret_cast<void**>(&w->memory), bytes);
  }
  if (*e == cudaSuccess)
    *e = cudaHostAlloc(reinterpret_cast<void**>(&w->status), kMaxRanks * sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable);
  if (*e == cudaSuccess) *e = cudaHostGetDevicePointer(reinterpret_cast<void**>(&w->status_dev), w->status, 0);
  w->capacity = bytes;
  if (*e == cudaSuccess) return w;
  cudaGetLastError();
  return nullptr;
}

int SmCount(int device) {
  static int count[64] = {0};
  if (device < 0 || device >= 64) return 0;
  if (count[device] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
    count[device] = n;
  }
  return count[device];
}

}  // namespace

void ReleaseEmulationWorkspaces() { WorkspacePool::Get().Clear(); }

int EmulatedAllReduce(int nranks, void* const* in_ptrs, void* const* out_ptrs,
                      unsigned long long numel, int elem_type, int mode, int algo, int block_numel,
                      size_t slot_bytes, int slots_per_channel, int channels, float post_scale,
                      int repeats, int exponent_lookahead, const EmulationOptions& options, std::string* error) {
  auto fail = [&](const std::string& m, int code) {
    if (error) *error = m;
    return code;
  };
  if (nranks < 1 || nranks > kMaxRanks) return fail("nranks out of range", -1);
  if (options.present < 0 || options.present > nranks) return fail("more ranks come than there are", -1);
  if (block_numel < 1) return fail("block_numel out of range", -1);
  if (algo == ALGO_ZEROCOPY) return fail("zero-copy needs real symmetric memory", -1);
  const bool exact = mode == MODE_QUANT && elem_type != ELEM_I32;
  if (algo != ALGO_ONESHOT) {
    // The streaming kernels and those of one_gpu_allreduce.cu know blocks as a context has them (the words and scale factors
    // of others would lie beyond their arrays); for plain sums a block is nothing but a unit of the geometry. A slot is whole
    // units, or whole blocks where it has no room for one per rank.
    const bool known = block_numel >= 32 && block_numel <= 1024 && (block_numel & (block_numel - 1)) == 0;
    if (exact && !known) return fail("block_numel must be a power of two from 32 to 1024", -1);
    if (!known) block_numel = 128;
    const size_t block = static_cast<size_t>(block_numel > 128 ? block_numel : 128) * 4, unit = nranks * block;
    slot_bytes = slot_bytes >= unit ? slot_bytes / unit * unit : slot_bytes / block * block;
    if (slots_per_channel < 1 || slot_bytes < (exact && elem_type == ELEM_BF16 ? unit : block))
      return fail("no room in the slots for max(block, 128) * 4 bytes, times nranks for bfloat16 in the exact mode", -1);
  }
  if (slot_bytes / 4 / block_numel * slots_per_channel > 8192)
    return fail("slots_per_channel * slot_bytes / (4 * block_numel) exceeds 8192", -1);
  for (int r = 0; r < nranks; r++)
    if (numel > 0 && (!in_ptrs[r] || !out_ptrs[r])) return fail("a rank has no tensor", -1);
  int dev = 0;
  cudaGetDevice(&dev);
  const int sms = SmCount(dev);
  if (sms <= 0) return fail("no CUDA device", -2);
  int esz = elem_type == ELEM_BF16 ? 2 : 4;
  size_t oneshot_bytes = algo == ALGO_ONESHOT ? (numel * esz + 255) / 256 * 256 : 256;
  int max_channels = sms / nranks;  // all virtual ranks share the GPU
  if (max_channels < 1) max_channels = 1;
  if (channels > 0 && channels < max_channels) max_channels = channels;

  // Every rank can address all tensors here, so that results may go straight into the outputs (one_gpu_allreduce.cu), for
  // whole vectors of device memory. Below 2^18 elements per rank, where a message between GPUs takes neither of these
  // algorithms but ALGO_ONESHOT, and in the checked build, the kernels run as they do between GPUs: that is what one
  // looks at there (2 ranks push exact, whole calls: 2^18 elements 36 us with them and 28 straight, 2^22 72 and 46).
  const bool only_direct = options.kernels == EmulationOptions::kOneGpu;
  bool direct = (algo == ALGO_STAGED || algo == ALGO_PUSH) && numel > 0 && options.kernels != EmulationOptions::kStreaming &&
                (only_direct || (numel >= kDirectNumel && !CheckedBuild()));
  uintptr_t bits = 0;
  for (int r = 0; r < nranks; r++) bits |= reinterpret_cast<uintptr_t>(in_ptrs[r]) | reinterpret_cast<uintptr_t>(out_ptrs[r]);
  if (bits & 15) direct = false;
  for (int r = 0; direct && r < nranks; r++) direct = DeviceMemory(in_ptrs[r]) && DeviceMemory(out_ptrs[r]);  // 0.3 us each

  // Plain sums through the slots are bound by memory, and here every rank's slots share one L2: a ring that
  // stays in it spares each tile two trips to HBM (4 ranks x 2^24 float32: 272 us with 155 MB of slots, 200 us
  // with 43 MB; three slots of 64 to 96 KiB, two of 128 KiB and four of 64 KiB come to the same). The
  // exact mode pays too much per tile for smaller ones (256 KiB: 400 us, 128 KiB: 453 us). The caller's geometry is an
  // upper bound there; the results do not depend on it.
  const size_t unit_bytes = static_cast<size_t>(nranks) * (block_numel > 128 ? block_numel : 128) * 4;
  const size_t ring = kL2Slots / (static_cast<size_t>(max_channels) * nranks);  // bytes of a channel's slots
  if (!direct && algo == ALGO_STAGED && mode == MODE_SUM && numel * esz * nranks > kL2Slots && slot_bytes * slots_per_channel > ring) {
    if (slots_per_channel > 3) slots_per_channel = 3;
    const size_t fits = ring / slots_per_channel / unit_bytes * unit_bytes;
    if (fits < slot_bytes) slot_bytes = fits > unit_bytes ? fits : unit_bytes;
  }

  RankCtx proto;
  memset(&proto, 0, sizeof(proto));
  proto.nranks = nranks;
  proto.slot_bytes = slot_bytes;
  proto.slots_per_channel = slots_per_channel;
  proto.one_gpu = 1;
  proto.exp_ring = ExpRingDepth(slots_per_channel);
  proto.exp_lookahead = ExpLookahead(slots_per_channel, exponent_lookahead < 0 ? kDefaultExpLookahead : exponent_lookahead);
  proto.block_numel = block_numel;
  proto.quant_base = quant::QuantBase(nranks);
  proto.oneshot_bytes = oneshot_bytes;
  proto.timeout_ns = options.timeout_ns ? options.timeout_ns : 2000000000ull;  // 2 s: generous for one GPU, still bounded
  JobArgs proto_job;
  memset(&proto_job, 0, sizeof(proto_job));
  proto_job.elem_type = elem_type;
  proto_job.mode = mode;
  proto_job.algo = algo;
  if (direct && !OneGpuFits(proto, proto_job)) direct = false;
  if (only_direct && !direct) return fail("not a call for the kernels of ranks that share a GPU", -1);
  size_t bytes = StagingBytes(slot_bytes, slots_per_channel, block_numel, max_channels,
                                    oneshot_bytes, nranks, &proto.data_offset, &proto.exp_offset,
                                    &proto.oneshot_offset);
  const size_t own_words = direct && mode == MODE_QUANT ? OneGpuExponentBytes(nranks, block_numel, max_channels) : 0;
  if (own_words > 0) {
    proto.exp_offset = bytes;
    bytes += (own_words + 4095) / 4096 * 4096;
  }
  proto.stage_bytes = ReportedStageBytes(bytes);
  if (algo == ALGO_PUSH && PushTileCapacity(proto, elem_type, mode) == 0)
    return fail("ALGO_PUSH needs at least two ranks and slots of about twice nranks * max(block, 128) * 4 bytes", -1);

  // Flags and exponent words of another layout are noise in this one, so they are cleared (with
  // the epochs, which start over) when the layout changes, and only then; or before the epochs outgrow the 24 bits of the tags of
  // one_gpu_allreduce.cu: half a minute of calls back to back (2 ranks x 2^25 exact: 56 epochs in 0.15 ms) to some
  // minutes (calls of one epoch).
  char layout[128];
  snprintf(layout, sizeof(layout), "%d/%d/%zu/%d/%d/%d/%zu", direct, nranks, slot_bytes, slots_per_channel, block_numel, max_channels, bytes);
  const size_t need = kHeadBytes + bytes * nranks;
  cudaError_t e = cudaSuccess;
  std::unique_ptr<EmuWorkspace> ws = WorkspacePool::Get().Take(dev, need, layout);
  if (!ws) ws = NewWorkspace(dev, need, &e);
  if (!ws) return fail(std::string("allocation failed: ") + cudaGetErrorString(e), -3);
  char* const stage0 = ws->memory + kHeadBytes;
  if (ws->layout != layout || ws->epochs > (options.epoch_limit ? options.epoch_limit : 1ull << 23)) {
    ws->layout.clear();
    ws->epochs = 0;
    e = cudaMemsetAsync(ws->memory, 0, kHeadBytes, 0);
    if (e == cudaSuccess) e = cudaMemset2DAsync(stage0, bytes, 0, proto.oneshot_offset, nranks, 0);
    if (e == cudaSuccess && own_words > 0) e = cudaMemset2DAsync(stage0 + proto.exp_offset, bytes, 0, own_words, nranks, 0);
    if (e != cudaSuccess) return fail(std::string("allocation failed: ") + cudaGetErrorString(e), -3);
  }

  // The inputs may still be in the making on any stream.
  e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return fail(std::string("the device reports: ") + cudaGetErrorString(e), -4);

  EmuArgs args;
  memset(&args, 0, sizeof(args));
  LaunchPlan plan;
  for (int it = 0; it < (repeats < 1 ? 1 : repeats); it++) {
    for (int r = 0; r < nranks; r++) {
      RankCtx& c = args.ctx[r];
      c = proto;
      c.rank = r;
      for (int p = 0; p < nranks; p++) c.stage_peer[p] = stage0 + bytes * p;
      c.status = ws->status_dev + r;
      c.epoch_words = reinterpret_cast<unsigned long long*>(ws->memory) + static_cast<size_t>(r) * kMaxChannels;
      c.counters = reinterpret_cast<unsigned long long*>(ws->memory + kEpochBytes) + r * 16;
      JobArgs& j = args.job[r];
      j.in = in_ptrs[r];
      j.out = out_ptrs[r];
      j.numel = numel;
      j.elem_type = elem_type;
      j.mode = mode;
      j.algo = algo;
      j.post_scale = post_scale;
      if (it == 0 && algo != ALGO_ONESHOT) j.bulk_copy = direct || (DeviceMemory(j.in) && DeviceMemory(j.out));
      if (direct) {
        j.out_zero_copy = 1;
        for (int p = 0; p < nranks; p++) j.user_peer[p] = static_cast<char*>(out_ptrs[p]);
        j.user_bytes = ReportedOutputBytes(numel * esz);
      }
      j.oneshot_parity = it & 1;
    }
    if (it == 0) {
      plan = PlanLaunch(args.ctx[0], args.job[0], channels, max_channels);
      for (int r = 0; r < nranks; r++) ws->status[r] = STATUS_OK;
    }
    for (int r = 0; r < nranks; r++) {
      args.job[r].tile_elems = plan.tile_elems;
      args.job[r].epochs = plan.epochs;
    }
    ws->epochs += plan.epochs;
    e = LaunchAllReduceEmulated(args, nranks, options.present ? options.present : nranks, plan, 0);
    if (e != cudaSuccess) break;
  }
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(std::string("emulated launch failed: ") + cudaGetErrorString(e), -4);
  }
  for (int r = 0; r < nranks; r++) {
    const int st = *reinterpret_cast<volatile int*>(ws->status + r);
    if (st != STATUS_OK) return fail("kernel status " + std::to_string(st) + " on rank " + std::to_string(r), st);
  }
  // Only after a call that went well: the ranks' epochs are in step then.
  ws->layout = layout;
  WorkspacePool::Get().Put(std::move(ws));
  return 0;
}

}  // namespace switchml
