// HostPipelinedAllReduce (cuda_backend.h): allreduce of a tensor in pinned host memory, with the
// host→device copy, the reduction and the device→host copy of different chunks at the same time.
//
// PCIe bounds it: n bytes in each direction at once, plus one chunk that is not overlapped, plus
// some 10 us per chunk for starting its copies. The loop is here and not in Python, where
// enqueueing a chunk cost 25 to 30 us. Chunks are reduced where they lie, so nothing is copied
// on the device. 25 MB: 475 + 463 us as one chunk, one copy after the other; 660 us in 4 MiB chunks.
#include <cuda_runtime.h>

#include <memory>
#include <string>
#include <vector>

#include "backends/cuda/cuda_backend.h"
#include "switchml/context.h"

namespace switchml {

namespace {
// An event of the calling thread, for ordering one stream after another (recorded anew for every
// chunk; a wait that was enqueued keeps the record it was made for).
struct ChunkEvent {
  cudaEvent_t e = nullptr;
  ChunkEvent() { cudaEventCreateWithFlags(&e, cudaEventDisableTiming); }
  ~ChunkEvent() {
    if (e) cudaEventDestroy(e);
  }
};

// Nothing may be in flight on the caller's buffers when the call returns, whatever happened: also not when
// AllReduceAsync throws because the context has been stopped.
struct Submitted {
  cudaStream_t in, comm, out;
  std::vector<std::shared_ptr<Job>> jobs;
  bool over = false;
  cudaError_t Finish() {
    if (over) return cudaSuccess;
    over = true;
    cudaError_t e = cudaSuccess;
    for (const cudaStream_t s : {in, comm, out}) {
      const cudaError_t this_one = cudaStreamSynchronize(s);
      if (e == cudaSuccess) e = this_one;
    }
    for (auto& job : jobs) job->WaitToComplete();
    return e;
  }
  ~Submitted() { Finish(); }
};
}  // namespace

int HostPipelinedAllReduce(const void* host_in, void* host_out, void* device, uint64_t numel, DataType type,
                           uint64_t chunk_numel, void* stream_in, void* stream_comm, void* stream_out, std::string* error) {
  Context& ctx = Context::GetInstance();
  const cudaStream_t s_in = static_cast<cudaStream_t>(stream_in), s_out = static_cast<cudaStream_t>(stream_out);
  // One worker's job takes a few microseconds, less than handing over from one stream to another.
  const cudaStream_t s_comm = ctx.GetConfig().general_.num_workers == 1 ? s_out : static_cast<cudaStream_t>(stream_comm);
  const size_t esz = DataTypeSize(type);
  ChunkEvent arrived;
  Submitted submitted{s_in, s_comm, s_out, {}};
  std::vector<std::shared_ptr<Job>>& jobs = submitted.jobs;
  jobs.reserve(numel / chunk_numel + 1);
  cudaError_t e = arrived.e ? cudaSuccess : cudaErrorMemoryAllocation;
  for (uint64_t lo = 0; lo < numel && e == cudaSuccess; lo += chunk_numel) {
    const uint64_t len = numel - lo < chunk_numel ? numel - lo : chunk_numel;
    char* d = static_cast<char*>(device) + lo * esz;
    e = cudaMemcpyAsync(d, static_cast<const char*>(host_in) + lo * esz, len * esz, cudaMemcpyHostToDevice, s_in);
    if (e == cudaSuccess) e = cudaEventRecord(arrived.e, s_in);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s_comm, arrived.e, 0);
    if (e != cudaSuccess) break;
    jobs.push_back(ctx.AllReduceAsync(d, d, len, type, SUM, s_comm));
    if (!jobs.back()->StreamWait(s_out)) break;  // failed: reported below
    e = cudaMemcpyAsync(static_cast<char*>(host_out) + lo * esz, d, len * esz, cudaMemcpyDeviceToHost, s_out);
  }
  const cudaError_t finished = submitted.Finish();
  if (e == cudaSuccess) e = finished;
  for (auto& job : jobs) {
    if (job->GetJobStatus() != FINISHED) {
      *error = job->failure_reason_;
      return -1;
    }
  }
  if (e != cudaSuccess) {
    *error = cudaGetErrorString(e);
    cudaGetLastError();
    return -1;
  }
  return 0;
}

}  // namespace switchml
