// See cuda_backend.h.
#include "backends/cuda/cuda_backend.h"

#include <cuda_runtime.h>
#include <sys/prctl.h>
#if __has_include(<nvtx3/nvToolsExt.h>)
#include <nvtx3/nvToolsExt.h>
#define SML_NVTX 1
#endif

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cctype>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <mutex>
#include <sstream>
#include <thread>
#include <vector>

#include "backends/cuda/fd_channel.h"
#include "backends/cuda/symmetric_memory.h"
#include "kernels/allreduce_kernels.h"
#include "rendezvous/control.h"
#include "switchml/context.h"
#include "switchml/log.h"
#include "switchml/quant_math.h"

namespace switchml {

namespace {

#define SML_CUDA_CHECK(call)                                                        \
  do {                                                                              \
    cudaError_t _e = (call);                                                        \
    SML_CHECK(_e == cudaSuccess) << #call << ": " << cudaGetErrorString(_e);        \
  } while (0)

// Recycles CUDA events; shared with the jobs so that an event outlives the backend if a
// caller still holds the job.
struct EventPool {
  std::mutex mu;
  std::vector<cudaEvent_t> free_list;
  cudaEvent_t Get() {
    {
      std::lock_guard<std::mutex> lk(mu);
      if (!free_list.empty()) {
        cudaEvent_t e = free_list.back();
        free_list.pop_back();
        return e;
      }
    }
    cudaEvent_t e = nullptr;
    cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
    return e;
  }
  void Put(cudaEvent_t e) {
    if (!e) return;
    std::lock_guard<std::mutex> lk(mu);
    free_list.push_back(e);
  }
  ~EventPool() {
    for (cudaEvent_t e : free_list) cudaEventDestroy(e);
  }
};

// Where threads that wait for jobs meet the backend that finishes them. Shared with the jobs: a
// caller may hold one longer than the backend lives.
struct Completions {
  std::mutex mu;                     // held while finished jobs are taken off the queue
  std::function<void()> reap;        // finish every job at the head of the queue whose event has fired; empty once the backend is gone
};

// Looking at events must not disturb a stream capture that goes on elsewhere in the process.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// What tells a stream from every other one of the process's life. Handles do not: that of a destroyed stream may
// come back as another one's, and those of the default streams stand for another stream on every device (or in
// every thread).
struct StreamIdentity {
  unsigned long long id = 0;
  int device = -1;  // current when the stream was looked at; -1: there is no telling
  StreamIdentity() {}
  explicit StreamIdentity(cudaStream_t s) {
    if (cudaStreamGetId(s, &id) != cudaSuccess || cudaGetDevice(&device) != cudaSuccess) {
      cudaGetLastError();
      device = -1;
    }
  }
  bool Is(const StreamIdentity& o) const { return device >= 0 && device == o.device && id == o.id; }
};

struct EventState : public DeviceJobState {
  cudaEvent_t done = nullptr;
  StreamIdentity stream;  // where the job runs
  std::shared_ptr<EventPool> pool;
  std::shared_ptr<Completions> completions;
  ~EventState() override {
    if (pool) pool->Put(done);
  }
  void StreamWait(void* other) override {
    OrderAfter(static_cast<cudaStream_t>(other), StreamIdentity(static_cast<cudaStream_t>(other)));
  }
  // Two work items on the same stream are in order by themselves.
  void OrderAfter(cudaStream_t other, const StreamIdentity& id) {
    if (!stream.Is(id)) cudaStreamWaitEvent(other, done, 0);
  }
  // Whether work on the stream `other` that is enqueued from now on comes after the job without waiting for it.
  bool BehindWithoutWaiting(const StreamIdentity& other) {
    if (stream.Is(other)) return true;
    RelaxedCapture relaxed;
    const cudaError_t e = cudaEventQuery(done);
    if (e != cudaSuccess) cudaGetLastError();
    return e == cudaSuccess;
  }
  void HelpComplete(Job& job, double milliseconds) override {
    const auto start = std::chrono::steady_clock::now();
    RelaxedCapture relaxed;
    for (;;) {
      if (milliseconds < 0) cudaEventSynchronize(done);  // without a limit the driver waits, which answers fastest
      {
        std::lock_guard<std::mutex> lk(completions->mu);
        if (!completions->reap) return;
        completions->reap();
      }
      const JobStatus s = job.GetJobStatus();
      if (s == FINISHED || s == FAILED) return;
      if (milliseconds >= 0) {
        const auto passed = std::chrono::steady_clock::now() - start;
        if (passed > std::chrono::duration<double, std::milli>(milliseconds)) return;
        if (passed > std::chrono::microseconds(100)) std::this_thread::sleep_for(std::chrono::microseconds(10));
      }
      std::this_thread::yield();
    }
  }
};

struct InFlight {
  StreamIdentity stream;  // where the job runs
  std::shared_ptr<Job> job;
  bool via_scheduler = false;
  JobSlice slice;
  cudaEvent_t done = nullptr;
  cudaEvent_t ready = nullptr;
  int status_slot = -1;  // -1: the job's kernel reports no status
  unsigned long long tiles = 0;
  std::string launch_error;
  // Whether input and output are ordinary device memory, once CheckOperands has looked.
  bool checked = false, in_device = true, out_device = true;
};

static const int kStatusSlots = 4096;
// launch = worker: with this many jobs in flight the launcher thread takes over, which may wait for
// room in the stream's queue (about a thousand launches) while the callers go on.
static const size_t kDirectLaunches = 256;
// What a job on the producer's stream may hold up there: read + write at 6 TB/s take 0.4 us (device memory only: over
// PCIe it is 40 us). On that stream and on the library's: 2^12 to 2^18 float32 in exact mode 11.8 and 16 us per job
// behind a kernel of the producer, 13.9 and 14.8 us blocking. The difference stays up to 16 MiB, but by then the
// producer's stream is busy for longer than it saves.
static const uint64_t kBriefBytes = 1 << 20;

// One NVTX range per job for timeline tools; without one the name is not even put together.
struct NvtxRange {
#ifdef SML_NVTX
  NvtxRange(const Job& job, const Tensor& t) {
    static const bool listening = [] {
      const bool on = nvtxRangePushA("switchml") != NVTX_NO_PUSH_POP_TRACKING;
      if (on) nvtxRangePop();
      return on;
    }();
    if (!listening) return;
    char name[96];
    snprintf(name, sizeof(name), "switchml job %llu: %llu x %s", static_cast<unsigned long long>(job.id_),
             static_cast<unsigned long long>(t.numel), DataTypeName(t.data_type));
    nvtxRangePushA(name);
    open = true;
  }
  ~NvtxRange() {
    if (open) nvtxRangePop();
  }
  bool open = false;
#else
  NvtxRange(const Job&, const Tensor&) {}
#endif
};

class CudaBackend : public CudaBackendInterface {
 public:
  CudaBackend(Context& context, Config& config) : CudaBackendInterface(context, config) {}
  ~CudaBackend() override { CleanupWorker(); }

  int NumSchedulerConsumers() const override { return 1; }

  void SetupWorker() override;
  void CleanupWorker() override;
  bool OnSubmit(const std::shared_ptr<Job>& job) override;
  std::string ExtraStatsJson() override;

  void* SymmetricAlloc(size_t bytes) override;
  void SymmetricReset() override;
  bool UsesMultimem() const override { return ctx_.use_multimem != 0; }
  bool SymmetricHeapInfo(void** local, void** peers, void** multicast, size_t* bytes) override {
    if (!heap_.local) return false;
    *local = heap_.local;
    for (int p = 0; p < n_; p++) peers[p] = heap_.peers[p];
    *multicast = heap_.multicast;
    *bytes = heap_.bytes;
    return true;
  }
  int Device() const override { return device_; }
  int RunWaitProbe(double budget_ms) override;

 private:
  void LauncherLoop();
  void CompletionLoop();
  void Reap();
  void FinishInFlight(InFlight& f, cudaError_t e);
  void PushInFlight(InFlight&& f);
  size_t InFlightCount();
  void BindServiceThread(const char* what);
  // Enqueue the kernels of `job` on `stream`; fills `f`. Caller holds launch_mu_.
  // `capturing`: the stream is being captured into a CUDA graph; nothing that belongs to
  // this one submission (events, status slot, buffer parity) may end up in the launch.
  void LaunchJob(const std::shared_ptr<Job>& job, cudaStream_t stream, InFlight* f, bool capturing = false);
  // The same for a single worker, whose job is one pass over the tensor (or none).
  cudaError_t LaunchLocalJob(const Tensor& t, cudaStream_t stream, InFlight* f);
  // Looks at the job's addresses, once: fills `f`, with the error if the GPU cannot reach them.
  void CheckOperands(const Tensor& t, InFlight* f);
  // What follows the kernels (`e`: how their launch went): the job's event and its ordering hooks.
  void FinishLaunch(const std::shared_ptr<Job>& job, cudaStream_t stream, InFlight* f, cudaError_t e, bool capturing);
  cudaEvent_t GetEvent() { return events_->Get(); }
  void PutEvent(cudaEvent_t e) { events_->Put(e); }

  int device_ = 0;
  int rank_ = 0, n_ = 1;
  bool inline_launch_ = false;
  bool set_up_ = false;
  std::unique_ptr<ControlServer> server_;
  ControlClient client_;
  FdChannel fds_;
  std::unique_ptr<SymmetricAllocator> allocator_;
  SymmetricRegion staging_;
  SymmetricRegion heap_;
  size_t heap_used_ = 0;
  kernels::RankCtx ctx_;
  int max_channels_ = 1;
  cudaStream_t comm_stream_ = nullptr;
  StreamIdentity comm_identity_;
  int* dev_status_ = nullptr;
  unsigned long long* dev_counters_ = nullptr;
  unsigned long long* dev_trace_ = nullptr;  // kTraceWords, only with [backend.cuda] trace
  unsigned long long* dev_epochs_ = nullptr;  // per-channel epochs, advanced by the kernels themselves
  int* host_status_ = nullptr;  // pinned ring of status words

  std::mutex launch_mu_;  // serialises launches: one job order on every rank
  // launch = inline: all jobs share the staging slots, the flag pad and the per-channel
  // epochs, so two jobs must never run on the GPU at the same time. A job submitted on a
  // stream other than the previous job's is ordered after that job through its own event.
  std::shared_ptr<EventState> last_job_;
  // launch = worker: jobs handed to the scheduler that the launcher thread has not enqueued yet.
  // While there are none a submitting thread enqueues its job itself.
  int queued_jobs_ = 0;
  unsigned long long epoch_base_ = 0;
  int oneshot_parity_ = 0;
  unsigned long long launched_jobs_ = 0;
  uint64_t oneshot_limit_ = 0;  // messages up to this many bytes take the one-barrier kernel
  unsigned long long kernel_launches_ = 0;  // kernels of this library enqueued so far (under launch_mu_)

  std::shared_ptr<EventPool> events_ = std::make_shared<EventPool>();

  std::thread launcher_, completer_;
  std::mutex q_mu_;
  std::condition_variable q_cv_;
  std::deque<InFlight> inflight_;
  bool stop_completer_ = false;
  bool completer_asleep_ = false;
  std::shared_ptr<Completions> completions_ = std::make_shared<Completions>();
  std::atomic<bool> failed_{false};
};

void CudaBackend::SetupWorker() {
  const GeneralConfig& g = config_.general_;
  const CudaBackendConfig& c = config_.backend_.cuda;
  rank_ = g.rank;
  n_ = g.num_workers;
  SML_CHECK(n_ <= kernels::kMaxRanks)
      << "the cuda backend serves one NVSwitch domain of at most " << kernels::kMaxRanks
      << " GPUs, got num_workers = " << n_;
  inline_launch_ = c.launch == "inline";

  int ndev = 0;
  cudaError_t e = cudaGetDeviceCount(&ndev);
  SML_CHECK(e == cudaSuccess && ndev > 0)
      << "backend = cuda needs a GPU: " << cudaGetErrorString(e);
  device_ = c.device;
  if (device_ < 0) {
    const char* lr = getenv("LOCAL_RANK");
    device_ = (lr && *lr) ? atoi(lr) : static_cast<int>(g.rank);
    device_ %= ndev;
  }
  SML_CHECK(device_ < ndev) << "backend.cuda.device " << device_ << " does not exist";
  SML_CUDA_CHECK(cudaSetDevice(device_));
  cudaDeviceProp prop;
  SML_CUDA_CHECK(cudaGetDeviceProperties(&prop, device_));
  SML_CHECK(prop.major >= 9) << "device " << device_ << " (" << prop.name << ", sm_" << prop.major
                             << prop.minor << ") is too old for this library (built for sm_100a)";

  uint64_t session = static_cast<uint64_t>(
      std::chrono::duration_cast<std::chrono::nanoseconds>(
          std::chrono::system_clock::now().time_since_epoch()).count());
  if (n_ > 1) {
    if (rank_ == 0) {
      server_.reset(new ControlServer());
      SML_CHECK(server_->Start(g.controller_ip_str, g.controller_port, 0))
          << "cannot start the in-process controller on " << g.controller_ip_str << ":"
          << g.controller_port;
    }
    SML_CHECK(client_.Connect(g.controller_ip_str, g.controller_port)) << "controller unreachable";
    SML_CHECK(client_.Broadcast(n_, rank_, 0, &session)) << "session broadcast failed";
    SML_CHECK(fds_.Listen(session, rank_, c.rendezvous_dir)) << "cannot open the fd channel";
    SML_CHECK(client_.Barrier(n_)) << "barrier failed";
  }
  allocator_.reset(new SymmetricAllocator(rank_, n_, device_, &client_, &fds_));

  // Co-residency bound: every CTA of a job must be able to run at the same time.
  max_channels_ = prop.multiProcessorCount;
  if (c.channels > 0 && static_cast<int>(c.channels) < max_channels_) max_channels_ = c.channels;
  if (max_channels_ > kernels::kMaxChannels) max_channels_ = kernels::kMaxChannels;

  memset(&ctx_, 0, sizeof(ctx_));
  ctx_.rank = rank_;
  ctx_.nranks = n_;
  ctx_.slot_bytes = c.slot_bytes;
  ctx_.slots_per_channel = c.slots_per_channel;
  ctx_.sc_fence = c.signal_fence == "sc" ? 1 : 0;
  ctx_.exp_ring = kernels::ExpRingDepth(static_cast<int>(c.slots_per_channel));
  ctx_.exp_lookahead = kernels::ExpLookahead(static_cast<int>(c.slots_per_channel), static_cast<int>(c.exponent_lookahead));
  ctx_.block_numel = static_cast<int>(g.packet_numel);
  ctx_.quant_base = quant::QuantBase(n_);
  // The one-barrier kernel sends every rank's whole message to every rank, n-1 times the
  // traffic of the streaming algorithms: the fewer the ranks, the longer it stays the faster
  // one. The configured limit is the one for eight workers.
  oneshot_limit_ = c.oneshot_max_bytes * 8 / static_cast<uint64_t>(n_ < 2 ? 2 : n_);
  ctx_.oneshot_bytes = (oneshot_limit_ + 255) / 256 * 256;
  ctx_.timeout_ns = static_cast<unsigned long long>(c.wait_timeout_ms * 1e6);
  size_t bytes = kernels::StagingBytes(ctx_.slot_bytes, ctx_.slots_per_channel, ctx_.block_numel,
                                       max_channels_, ctx_.oneshot_bytes, n_, &ctx_.data_offset,
                                       &ctx_.exp_offset, &ctx_.oneshot_offset);
  ctx_.stage_bytes = kernels::ReportedStageBytes(bytes);
  // Two GPUs exchange less data with plain peer loads/stores (N bytes each way) than
  // through the switch (1.5 N); from three GPUs on the in-switch reduction wins.
  bool want_mc = c.transport == "nvls" || (c.transport == "auto" && n_ > 2);
  std::string err;
  SML_CHECK(allocator_->Create(bytes, want_mc, &staging_, &err))
      << "cannot create the symmetric staging region (" << (bytes >> 20) << " MiB): " << err;
  SML_CHECK(!(c.transport == "nvls" && n_ > 1 && !staging_.multicast))
      << "backend.cuda.transport = nvls but NVLink multicast is not available";
  for (int p = 0; p < n_; p++) ctx_.stage_peer[p] = static_cast<char*>(staging_.peers[p]);
  ctx_.stage_mc = static_cast<char*>(staging_.multicast);
  ctx_.use_multimem = staging_.multicast != nullptr;

  if (c.symm_heap_mb > 0) {
    SML_CHECK(allocator_->Create(static_cast<size_t>(c.symm_heap_mb) << 20, ctx_.use_multimem != 0,
                                 &heap_, &err))
        << "cannot create the symmetric heap: " << err;
    if (ctx_.use_multimem && !heap_.multicast) {
      SML_LOG(WARNING) << "symmetric heap has no multicast mapping; zero-copy jobs use peer loads";
    }
  }
  heap_used_ = 0;

  int lo = 0, hi = 0;
  cudaDeviceGetStreamPriorityRange(&lo, &hi);
  SML_CUDA_CHECK(cudaStreamCreateWithPriority(&comm_stream_, cudaStreamNonBlocking, hi));
  comm_identity_ = StreamIdentity(comm_stream_);
  last_job_.reset();
  queued_jobs_ = 0;
  SML_CUDA_CHECK(cudaMalloc(&dev_counters_, 16 * sizeof(unsigned long long)));
  SML_CUDA_CHECK(cudaMemset(dev_counters_, 0, 16 * sizeof(unsigned long long)));
  SML_CUDA_CHECK(cudaMalloc(&dev_epochs_, kernels::kMaxChannels * sizeof(unsigned long long)));
  SML_CUDA_CHECK(cudaMemset(dev_epochs_, 0, kernels::kMaxChannels * sizeof(unsigned long long)));
  // Status words live in pinned host memory that the device can write: a kernel stores
  // its error code there directly, so a job costs no extra copy or memset on the stream.
  SML_CUDA_CHECK(cudaHostAlloc(&host_status_, kStatusSlots * sizeof(int), cudaHostAllocMapped));
  memset(host_status_, 0, kStatusSlots * sizeof(int));
  SML_CUDA_CHECK(cudaHostGetDevicePointer(reinterpret_cast<void**>(&dev_status_), host_status_, 0));
  ctx_.status = dev_status_;
  ctx_.counters = dev_counters_;
  if (c.trace) {
    SML_CUDA_CHECK(cudaMalloc(&dev_trace_, kernels::kTraceWords * sizeof(unsigned long long)));
    SML_CUDA_CHECK(cudaMemset(dev_trace_, 0, kernels::kTraceWords * sizeof(unsigned long long)));
  }
  ctx_.trace = dev_trace_;
  ctx_.epoch_words = dev_epochs_;
  epoch_base_ = 0;
  oneshot_parity_ = 0;
  launched_jobs_ = 0;
  kernel_launches_ = 0;
  failed_ = false;
  SML_CUDA_CHECK(cudaDeviceSynchronize());
  if (n_ > 1) SML_CHECK(client_.Barrier(n_)) << "barrier failed";

  SML_VLOG(0) << "cuda backend ready: rank " << rank_ << "/" << n_ << " on device " << device_
              << " (" << prop.name << "), transport "
              << (n_ == 1 ? "local" : (ctx_.use_multimem ? "nvls (multimem)" : "p2p (peer memory)"))
              << ", staging " << (bytes >> 20) << " MiB, up to " << max_channels_ << " channels, launch "
              << c.launch;
  stop_completer_ = false;
  completer_asleep_ = false;
  completions_->reap = [this] { Reap(); };
  set_up_ = true;
  completer_ = std::thread(&CudaBackend::CompletionLoop, this);
  if (!inline_launch_) launcher_ = std::thread(&CudaBackend::LauncherLoop, this);
}

void CudaBackend::CleanupWorker() {
  if (!set_up_) return;
  set_up_ = false;
  if (launcher_.joinable()) launcher_.join();
  {
    std::lock_guard<std::mutex> lk(q_mu_);
    stop_completer_ = true;
  }
  q_cv_.notify_all();
  if (completer_.joinable()) completer_.join();
  {
    std::lock_guard<std::mutex> lk(completions_->mu);
    completions_->reap = nullptr;
  }
  cudaSetDevice(device_);
  cudaDeviceSynchronize();
  bool peers_alive = !failed_.load();
  if (server_) server_->StopAccepting();
  if (n_ > 1 && peers_alive && !client_.Barrier(n_, 10000)) peers_alive = false;
  if (heap_.local) allocator_->Destroy(&heap_, peers_alive);
  if (staging_.local) allocator_->Destroy(&staging_, peers_alive);
  if (comm_stream_) cudaStreamDestroy(comm_stream_);
  comm_stream_ = nullptr;
  last_job_.reset();
  if (dev_counters_) cudaFree(dev_counters_);
  if (dev_trace_) cudaFree(dev_trace_);
  if (dev_epochs_) cudaFree(dev_epochs_);
  dev_epochs_ = nullptr;
  if (host_status_) cudaFreeHost(host_status_);
  dev_status_ = nullptr;
  dev_counters_ = nullptr;
  dev_trace_ = nullptr;
  host_status_ = nullptr;
  fds_.Close();
  client_.Close();
  if (server_) {
    server_->Stop();
    server_.reset();
  }
}

void* CudaBackend::SymmetricAlloc(size_t bytes) {
  if (!heap_.local) return nullptr;
  size_t need = (bytes + 255) / 256 * 256;
  std::lock_guard<std::mutex> lk(launch_mu_);
  if (heap_used_ + need > heap_.bytes) return nullptr;
  void* p = static_cast<char*>(heap_.local) + heap_used_;
  heap_used_ += need;
  return p;
}

void CudaBackend::SymmetricReset() {
  std::lock_guard<std::mutex> lk(launch_mu_);
  heap_used_ = 0;
}

// nullptr if kernels may dereference `p`, else the reason why not. `device`: whether it is ordinary
// device memory (what kernels::DeviceMemory asks).
static const char* GpuCannotAccess(const void* p, bool* device) {
  if (p == nullptr) return "null pointer";
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    cudaGetLastError();
    return "the address is unknown to CUDA";
  }
  if (at.type == cudaMemoryTypeUnregistered) return "the address is ordinary (pageable) host memory";
  *device = at.type == cudaMemoryTypeDevice;
  return nullptr;
}

// The kernels dereference both pointers on the GPU: refuse anything the GPU cannot be
// trusted to reach (ordinary malloc'ed host memory) instead of launching into a fault.
// Device, managed and pinned (cudaHostAlloc / cudaHostRegister) memory pass.
void CudaBackend::CheckOperands(const Tensor& t, InFlight* f) {
  if (f->checked) return;
  f->checked = true;
  if (t.numel == 0) return;
  const char* why = GpuCannotAccess(t.in_ptr, &f->in_device);
  f->out_device = f->in_device;
  if (!why && t.out_ptr != t.in_ptr) why = GpuCannotAccess(t.out_ptr, &f->out_device);
  if (why) f->launch_error = std::string("backend = cuda needs device, managed or pinned memory: ") + why;
}

void CudaBackend::LaunchJob(const std::shared_ptr<Job>& job, cudaStream_t stream, InFlight* f, bool capturing) {
  const CudaBackendConfig& c = config_.backend_.cuda;
  Tensor t = job->tensor_;
  const Tensor& user = job->tensor_;
  CheckOperands(t, f);
  if (!f->launch_error.empty()) return;
  bool in_device = f->in_device, out_device = f->out_device;
  NvtxRange range(*job, user);
  if (n_ == 1) {
    FinishLaunch(job, stream, f, LaunchLocalJob(t, stream, f), capturing);
    return;
  }
  // uint8: widen into int32 scratch of the stream's memory pool, reduce that in place,
  // narrow into the caller's output. With one worker the sum is the input itself.
  void* widened = nullptr;
  if (t.data_type == UINT8 && t.numel > 0) {
    if (capturing) {
      f->launch_error = "uint8 jobs cannot be captured into a CUDA graph";
      return;
    }
    cudaError_t we = cudaMallocAsync(&widened, t.numel * 4, stream);
    if (we == cudaSuccess) we = kernels::LaunchWidenU8(t.in_ptr, widened, t.numel, stream);
    if (we != cudaSuccess) {
      f->launch_error = std::string("uint8 staging failed: ") + cudaGetErrorString(we);
      cudaGetLastError();
      if (widened) cudaFreeAsync(widened, stream);
      return;
    }
    t.in_ptr = t.out_ptr = widened;
    in_device = out_device = true;
    t.data_type = INT32;
  }
  const bool integer = t.data_type == INT32 || t.data_type == UINT8;
  // A broadcast is a sum to which everybody but the root contributes zeros: clear this
  // rank's buffer in stream order, in front of the kernel; never average.
  const bool broadcast = job->job_type_ == BROADCAST;
  if (broadcast && rank_ != job->extra_job_info_.broadcast_root && t.numel > 0) {
    cudaError_t ce = cudaMemsetAsync(t.in_ptr, 0, t.numel * DataTypeSize(t.data_type), stream);
    if (ce != cudaSuccess) {
      f->launch_error = std::string("broadcast: clearing the buffer failed: ") + cudaGetErrorString(ce);
      cudaGetLastError();
      return;
    }
  }
  kernels::JobArgs a;
  memset(&a, 0, sizeof(a));
  a.in = t.in_ptr;
  a.out = t.out_ptr;
  a.numel = t.numel;
  a.elem_type = t.data_type == FLOAT32 ? kernels::ELEM_F32
              : t.data_type == BFLOAT16 ? kernels::ELEM_BF16 : kernels::ELEM_I32;
  a.mode = (!integer && c.mode == "int32_quant") ? kernels::MODE_QUANT : kernels::MODE_SUM;
  a.post_scale = c.average && !integer && !broadcast ? 1.0f / static_cast<float>(n_) : 1.0f;
  size_t esz = DataTypeSize(t.data_type);
  size_t bytes = t.numel * esz;
  a.bulk_copy = t.numel > 0 && in_device && out_device;

  // Pick the algorithm (identically on every rank: it depends on sizes and on whether the
  // pointers sit in the symmetric heap, which is allocated in lock step).
  auto in_heap = [&](const void* p) {
    return heap_.local && p >= heap_.local &&
           static_cast<const char*>(p) + bytes <= static_cast<const char*>(heap_.local) + heap_.bytes;
  };
  auto heap_usable = [&](const void* p) {
    return in_heap(p) && (reinterpret_cast<uintptr_t>(p) & 15) == 0 && (!ctx_.use_multimem || heap_.multicast);
  };
  const bool out_in_heap = heap_usable(t.out_ptr);
  const bool heap_ok = out_in_heap && heap_usable(t.in_ptr);
  auto describe_heap = [&] {
    for (int p = 0; p < n_; p++) a.user_peer[p] = static_cast<char*>(heap_.peers[p]);
    a.user_mc = static_cast<char*>(heap_.multicast);
    a.user_bytes = heap_.bytes;
    a.in_offset = static_cast<const char*>(t.in_ptr) - static_cast<const char*>(heap_.local);
    a.out_offset = static_cast<const char*>(t.out_ptr) - static_cast<const char*>(heap_.local);
  };
  // Peer-memory transport moves large messages with posted stores only, unless told otherwise.
  const bool push = !ctx_.use_multimem && c.p2p_algo == "push" &&
                    kernels::PushTileCapacity(ctx_, a.elem_type, a.mode) > 0;
  // (Tensors of the symmetric heap are reduced where they lie when the switch can do it;
  // over plain peer memory small ones are quicker through the one-barrier kernel.)
  // Plain sums through the switch leave the one-barrier kernel at a quarter of the configured
  // size already (measured at four GPUs: 4 MiB take 40 us there against 36 us streamed).
  const uint64_t oneshot_limit = (ctx_.use_multimem && a.mode == kernels::MODE_SUM) ? c.oneshot_max_bytes / 4 : oneshot_limit_;
  if (bytes <= oneshot_limit && !(a.mode == kernels::MODE_SUM && heap_ok && ctx_.use_multimem)) {
    a.algo = kernels::ALGO_ONESHOT;
    a.oneshot_parity = oneshot_parity_;
    if (!capturing) oneshot_parity_ ^= 1;
  } else if (push) {
    a.algo = kernels::ALGO_PUSH;
    if (out_in_heap) {  // results go straight into every rank's output
      a.out_zero_copy = 1;
      describe_heap();
    }
  } else if (a.mode == kernels::MODE_SUM && heap_ok) {
    a.algo = kernels::ALGO_ZEROCOPY;
    describe_heap();
  } else {
    a.algo = kernels::ALGO_STAGED;
    if (a.mode == kernels::MODE_QUANT && out_in_heap) {
      a.out_zero_copy = 1;
      describe_heap();
    }
  }
  kernels::LaunchPlan plan = kernels::PlanLaunch(ctx_, a, c.channels, max_channels_);
  a.tile_elems = plan.tile_elems;
  a.epochs = plan.epochs;
  if (capturing && a.algo == kernels::ALGO_ONESHOT) {
    a.trailing_barrier = 1;  // a replayed launch cannot alternate buffers: meet again instead,
    a.oneshot_parity = 2;    // in a buffer set of its own, apart from the alternating pair
    a.epochs = 2;
  }
  epoch_base_ += a.epochs;
  f->tiles = plan.tiles;
  // Replays of a captured launch share one status word that nobody waits on; a timeout in
  // a replay still shows up in the device counters.
  f->status_slot = capturing ? kStatusSlots - 2 : static_cast<int>(launched_jobs_ % (kStatusSlots - 2));

  cudaError_t e = cudaSuccess;
  host_status_[f->status_slot] = kernels::STATUS_OK;  // the ring is far longer than the queue
  kernels::RankCtx job_ctx = ctx_;
  job_ctx.status = dev_status_ + f->status_slot;
  if (t.numel > 0) {
    e = kernels::LaunchAllReduce(job_ctx, a, plan, stream);
    if (e == cudaSuccess) kernel_launches_ += widened ? 3 : 1;
  }
  if (widened) {
    if (e == cudaSuccess) e = kernels::LaunchNarrowI32(widened, user.out_ptr, user.numel, stream);
    cudaFreeAsync(widened, stream);
  }
  SML_VLOG(2) << "job " << job->id_ << ": " << t.numel << " x " << DataTypeName(user.data_type)
              << " algo " << a.algo << " mode " << a.mode << " channels " << plan.channels
              << " epochs " << plan.epochs;
  FinishLaunch(job, stream, f, e, capturing);
}

cudaError_t CudaBackend::LaunchLocalJob(const Tensor& t, cudaStream_t stream, InFlight* f) {
  const size_t bytes = t.numel * DataTypeSize(t.data_type);
  f->tiles = (bytes + ctx_.slot_bytes - 1) / ctx_.slot_bytes;
  if (t.numel == 0) return cudaSuccess;
  const bool integer = t.data_type == INT32 || t.data_type == UINT8;
  cudaError_t e = cudaSuccess;
  if (!integer && config_.backend_.cuda.mode == "int32_quant") {
    // The exact mode rounds every value to its block's grid, also with nobody to add to. (A mean
    // over one worker scales by one.)
    e = kernels::LaunchLocalQuant(t.in_ptr, t.out_ptr, t.numel, t.data_type == BFLOAT16 ? kernels::ELEM_BF16 : kernels::ELEM_F32,
                                  ctx_.block_numel, stream);
  } else if (t.in_ptr != t.out_ptr) {
    e = kernels::LaunchLocalCopy(t.in_ptr, t.out_ptr, bytes, stream);
  } else {
    return cudaSuccess;  // the sum of one term, in place: nothing to do
  }
  if (e == cudaSuccess) kernel_launches_++;
  return e;
}

void CudaBackend::FinishLaunch(const std::shared_ptr<Job>& job, cudaStream_t stream, InFlight* f, cudaError_t e, bool capturing) {
  if (!capturing) launched_jobs_++;  // (its old value was the job's place in the ring of status words)
  f->done = capturing ? nullptr : GetEvent();
  if (e == cudaSuccess && f->done) e = cudaEventRecord(f->done, stream);
  if (e != cudaSuccess) {
    f->launch_error = std::string("kernel launch failed: ") + cudaGetErrorString(e);
    cudaGetLastError();
  }
  if (f->done) {
    auto st = std::make_shared<EventState>();
    st->done = f->done;
    st->stream = f->stream;
    st->pool = events_;
    st->completions = completions_;
    last_job_ = st;
    job->SetDeviceState(st);
  } else {
    job->SetDeviceState(nullptr);  // captured: the work is ordered by the graph itself
  }
}

bool CudaBackend::OnSubmit(const std::shared_ptr<Job>& job) {
  if (job->job_type_ != ALLREDUCE && job->job_type_ != BROADCAST) {
    context_.NotifyJobCompletion(job, false, "only ALLREDUCE and BROADCAST jobs are supported");
    return true;
  }
  if (config_.general_.instant_job_completion) {
    job->SetJobStatus(RUNNING);
    context_.NotifyJobCompletion(job, true);
    return true;
  }
  cudaSetDevice(device_);
  InFlight f;
  f.job = job;
  const cudaStream_t user_stream = static_cast<cudaStream_t>(job->producer_stream_);
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(user_stream, &capture) != cudaSuccess) {
    capture = cudaStreamCaptureStatusNone;
    cudaGetLastError();
  }
  const bool capturing = capture == cudaStreamCaptureStatusActive;
  if (inline_launch_ && InFlightCount() > kStatusSlots / 4) {  // a status word must have been read before its slot comes round again
    std::lock_guard<std::mutex> lk(completions_->mu);
    Reap();
  }
  // launch = worker: a single worker's short pass takes less than handing over from the producer's stream to
  // the backend's and back (two events and the GPU's wait for them), so it may run where its input was made.
  bool brief = false;
  if (!inline_launch_ && !capturing && n_ == 1 && job->tensor_.numel * DataTypeSize(job->tensor_.data_type) <= kBriefBytes) {
    CheckOperands(job->tensor_, &f);
    brief = f.in_device && f.out_device;
  }
  if (!capturing) f.stream = StreamIdentity(user_stream);
  {
    std::lock_guard<std::mutex> lk(launch_mu_);
    cudaStream_t stream = user_stream;
    if (!inline_launch_) {
      const bool queue = capturing || queued_jobs_ > 0 || InFlightCount() >= kDirectLaunches;
      // The producer's stream must not wait for a job before this one: whoever computes there has not asked for that.
      if (queue || !brief || (last_job_ && !last_job_->BehindWithoutWaiting(f.stream))) {
        // Where the producer stream is now: the job comes after it.
        f.ready = GetEvent();
        cudaEventRecord(f.ready, user_stream);
        if (queue) {
          queued_jobs_++;
          job->ready_event_ = f.ready;
          return false;  // goes through the scheduler, so that the caller does not wait for the stream's queue
        }
        // Nobody is ahead of this job: enqueueing it here costs less than waking the launcher thread
        // (a blocking allreduce of 64 Ki elements took 38 us with the hand-over).
        stream = comm_stream_;
        f.stream = comm_identity_;
        cudaStreamWaitEvent(stream, f.ready, 0);
      }
    }
    job->SetJobStatus(QUEUED);
    job->SetJobStatus(RUNNING);
    // Not while capturing: an event recorded outside the capture cannot be waited on inside
    // it. A captured job is ordered by the graph it becomes part of; whoever replays that
    // graph next to other jobs of this context orders the two.
    if (!capturing && last_job_) last_job_->OrderAfter(stream, f.stream);
    LaunchJob(job, stream, &f, capturing);
    if (!capturing) PushInFlight(std::move(f));
  }
  if (capturing) {
    // The kernels now live in the graph under capture and run whenever it is replayed;
    // as far as this submission goes the job is done.
    context_.NotifyJobCompletion(job, f.launch_error.empty(), f.launch_error);
  }
  return true;
}

// [backend.cuda] numa_bind: keep a service thread on the cores next to the GPU (the reference
// pins its RDMA worker threads to the NIC's NUMA node, rdma_worker_thread.cc:77).
void CudaBackend::BindServiceThread(const char* what) {
  if (!config_.backend_.cuda.numa_bind) return;
  char bus[32] = {0};
  if (cudaDeviceGetPCIBusId(bus, sizeof(bus), device_) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  for (char* p = bus; *p; ++p) *p = static_cast<char>(tolower(*p));  // sysfs spells bus ids in lower case
  int node = GetDeviceNuma(bus);
  if (node < 0 || !BindToNumaNode(node)) {
    SML_VLOG(1) << what << " thread: no NUMA binding (device " << bus << ", node " << node << ")";
  } else {
    SML_VLOG(1) << what << " thread bound to NUMA node " << node << " of device " << bus;
  }
}

void CudaBackend::LauncherLoop() {
  cudaSetDevice(device_);
  BindServiceThread("launcher");
  JobSlice js;
  while (context_.GetContextState() == Context::RUNNING && context_.GetJobSlice(0, js)) {
    InFlight f;
    f.job = js.job;
    f.via_scheduler = true;
    f.slice = js;
    f.ready = static_cast<cudaEvent_t>(js.job->ready_event_);
    {
      std::lock_guard<std::mutex> lk(launch_mu_);
      if (f.ready) cudaStreamWaitEvent(comm_stream_, f.ready, 0);
      f.stream = comm_identity_;
      if (last_job_) last_job_->OrderAfter(comm_stream_, f.stream);
      LaunchJob(js.job, comm_stream_, &f);
      PushInFlight(std::move(f));
      queued_jobs_--;
    }
    // The scheduler's barrier (one consumer) lets us take the next job at once: jobs are
    // queued back to back on the stream and complete in order.
  }
}

void CudaBackend::PushInFlight(InFlight&& f) {
  bool wake;
  {
    std::lock_guard<std::mutex> lk(q_mu_);
    inflight_.push_back(std::move(f));
    wake = completer_asleep_;
  }
  if (wake) q_cv_.notify_all();
}

size_t CudaBackend::InFlightCount() {
  std::lock_guard<std::mutex> lk(q_mu_);
  return inflight_.size();
}

// Finishes jobs for those that nobody waits for (a thread that waits for a job does it itself,
// EventState::HelpComplete). It looks at the head of the queue every few microseconds while there
// are jobs, and for a while after the last one: a thread that sits in cudaEventSynchronize holds
// up the launches of the others (9 us per launch instead of 3), and waking one that sleeps costs
// every submission a system call.
void CudaBackend::CompletionLoop() {
  cudaSetDevice(device_);
  BindServiceThread("completion");
  prctl(PR_SET_TIMERSLACK, 1000ul, 0ul, 0ul, 0ul);  // of this thread: sleep 20 us, not 70
  int quiet = 0;  // turns without a job
  for (;;) {
    {
      std::unique_lock<std::mutex> lk(q_mu_);
      if (inflight_.empty() && !stop_completer_ && ++quiet > 100) {
        completer_asleep_ = true;
        q_cv_.wait(lk, [this] { return stop_completer_ || !inflight_.empty(); });
        completer_asleep_ = false;
      }
      if (!inflight_.empty()) quiet = 0;
      else if (stop_completer_) return;  // stop requested and nothing left
    }
    {
      std::unique_lock<std::mutex> lk(completions_->mu, std::try_to_lock);
      if (lk) Reap();
    }
    std::this_thread::sleep_for(std::chrono::microseconds(20));
  }
}

// Caller holds completions_->mu.
void CudaBackend::Reap() {
  RelaxedCapture relaxed;
  for (;;) {
    InFlight* head = nullptr;  // stays where it is: only this function takes jobs off the queue
    {
      std::lock_guard<std::mutex> lk(q_mu_);
      if (inflight_.empty()) return;
      head = &inflight_.front();
    }
    cudaError_t e = cudaSuccess;
    if (head->launch_error.empty()) {
      e = cudaEventQuery(head->done);
      if (e == cudaErrorNotReady) {
        cudaGetLastError();
        return;
      }
    }
    InFlight f = std::move(*head);
    {
      std::lock_guard<std::mutex> lk(q_mu_);
      inflight_.pop_front();
    }
    FinishInFlight(f, e);
  }
}

void CudaBackend::FinishInFlight(InFlight& f, cudaError_t e) {
  Stats& stats = context_.GetStats();
  bool ok = f.launch_error.empty();
  std::string why = f.launch_error;
  if (ok && e != cudaSuccess) {
    ok = false;
    why = std::string("device error: ") + cudaGetErrorString(e);
    failed_ = true;
  } else if (ok && f.status_slot >= 0) {
    int st = *reinterpret_cast<volatile int*>(host_status_ + f.status_slot);
    if (st != kernels::STATUS_OK) {
      ok = false;
      std::ostringstream o;
      if ((st & 0xf) == kernels::STATUS_TIMEOUT) {
        o << "a peer did not arrive within " << config_.backend_.cuda.wait_timeout_ms
          << " ms (channel " << (st >> 8) << ", phase " << ((st >> 4) & 0xf) << ")";
        stats.AddTimeouts(0, 1);
      } else if ((st & 0xf) == kernels::STATUS_BOUNDS) {
        o << "checked build: a tile of channel " << (st >> 8) << " would reach outside its region";
      } else {
        o << "kernel status " << st;
      }
      why = o.str();
      failed_ = true;
    }
  }
  stats.AddTotalPktsSent(0, f.tiles);
  if (ok) stats.AddCorrectPktsReceived(0, f.tiles);
  PutEvent(f.ready);
  // f.done belongs to the job's EventState and returns to the pool with the job.
  if (f.via_scheduler) {
    if (!ok) f.job->failure_reason_ = why;
    context_.NotifyJobSliceCompletion(0, f.slice);
  } else {
    context_.NotifyJobCompletion(f.job, ok, why);
  }
}

std::string CudaBackend::ExtraStatsJson() {
  unsigned long long c[16] = {0};
  if (dev_counters_) {
    cudaSetDevice(device_);
    cudaMemcpy(c, dev_counters_, sizeof(c), cudaMemcpyDeviceToHost);
  }
  std::ostringstream o;
  o << "{\"device\":" << device_ << ",\"multimem\":" << (ctx_.use_multimem ? "true" : "false")
    << ",\"tiles\":" << c[0] << ",\"wait_spins\":" << c[1] << ",\"device_timeouts\":" << c[2]
    << ",\"jobs_launched\":" << launched_jobs_ << ",\"kernel_launches\":" << kernel_launches_
    << ",\"epoch\":" << epoch_base_
    << ",\"channel0_ns\":{\"loader_wait\":" << c[3] << ",\"loader_work\":" << c[4] + c[9] + c[10] + c[11]
    << ",\"loader_scale_factors\":" << c[9] << ",\"loader_payload\":" << c[10] << ",\"loader_exponents_ahead\":" << c[11]
    << ",\"loader_signal\":" << c[4]
    << ",\"reducer_wait\":" << c[5] << ",\"reducer_work\":" << c[6] << ",\"storer_wait\":" << c[7]
    << ",\"storer_work\":" << c[8] << "}";
  if (dev_trace_) {
    // The last job's timeline on channel 0, in ns after the kernel's start: for each role, when its
    // waits for a tile were over and when it had finished the tile (0 = the job had no such tile).
    std::vector<unsigned long long> t(kernels::kTraceWords);
    cudaMemcpy(t.data(), dev_trace_, t.size() * sizeof(t[0]), cudaMemcpyDeviceToHost);
    const unsigned long long t0 = t[6 * kernels::kTraceTiles];
    static const char* names[6] = {"loader_began", "loader_finished", "reducer_began", "reducer_finished",
                                   "storer_began", "storer_finished"};
    o << ",\"channel0_trace_ns\":{";
    for (int row = 0; row < 6; row++) {
      o << (row ? "," : "") << "\"" << names[row] << "\":[";
      for (int k = 0; k < kernels::kTraceTiles; k++) {
        unsigned long long v = t[row * kernels::kTraceTiles + k];
        o << (k ? "," : "") << (v > t0 ? v - t0 : 0);
      }
      o << "]";
    }
    o << "}";
  }
  o << "}";
  return o.str();
}

int CudaBackend::RunWaitProbe(double budget_ms) {
  cudaSetDevice(device_);
  std::lock_guard<std::mutex> lk(launch_mu_);
  kernels::RankCtx probe = ctx_;
  probe.timeout_ns = static_cast<unsigned long long>(budget_ms * 1e6);
  cudaStream_t s = comm_stream_;
  int st = -1;
  int slot = kStatusSlots - 1;
  host_status_[slot] = kernels::STATUS_OK;
  probe.status = dev_status_ + slot;
  cudaError_t e = kernels::LaunchWaitProbe(probe, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e == cudaSuccess) st = *reinterpret_cast<volatile int*>(host_status_ + slot);
  return e == cudaSuccess ? st : -static_cast<int>(e);
}

}  // namespace

Backend* CreateCudaBackend(Context& context, Config& config) {
  return new CudaBackend(context, config);
}

// ---------------------------------------------------------------------------------------

bool KernelsCheckedBuild() { return kernels::CheckedBuild(); }

int ConvertU8OnDevice(bool widen, const void* in, void* out, unsigned long long numel, void* stream,
                      std::string* error) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = widen ? kernels::LaunchWidenU8(in, out, numel, s) : kernels::LaunchNarrowI32(in, out, numel, s);
  if (e != cudaSuccess) {
    if (error) *error = cudaGetErrorString(e);
    cudaGetLastError();
  }
  return static_cast<int>(e);
}

}  // namespace switchml
