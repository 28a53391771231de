// The waits of one_gpu_allreduce.cu (kernels/one_gpu_waits.cuh) on the host: a warp is 32 threads that meet in its votes,
// shared memory is what a case says each lane reads, and time passes when it is asked for. A vote in which lanes of two
// places meet, or which some lanes never come to, is an error (on the GPU nothing would bound that wait).
//
// Prints "ok   <case>" per case; the exit status is the number of failed ones.
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <functional>
#include <mutex>
#include <stdexcept>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

#include "kernels/allreduce_kernels.h"

namespace {

constexpr int kLanes = 32;
thread_local int t_lane = 0;

class Warp {
 public:
  // All lanes: `combine` of their values. `place` tells one vote from another.
  unsigned Meet(int place, unsigned value, const std::function<unsigned(unsigned, unsigned)>& combine) {
    std::unique_lock<std::mutex> lk(mu_);
    if (broken_.empty() && arrived_ > 0 && place != place_) Break("votes of lines " + std::to_string(place_) + " and " + std::to_string(place) + " met");
    if (!broken_.empty()) throw std::runtime_error(broken_);
    place_ = place;
    sum_ = arrived_ == 0 ? value : combine(sum_, value);
    if (++arrived_ == kLanes) {
      arrived_ = 0;
      result_ = sum_;
      generation_++;
      cv_.notify_all();
      return result_;
    }
    const unsigned long long mine = generation_;
    if (!cv_.wait_for(lk, std::chrono::seconds(5), [&] { return generation_ != mine || !broken_.empty(); }))
      Break("lanes never came to the vote of line " + std::to_string(place));
    if (generation_ == mine) throw std::runtime_error(broken_);
    return result_;
  }

 private:
  void Break(const std::string& why) {
    broken_ = why;
    cv_.notify_all();
  }
  std::mutex mu_;
  std::condition_variable cv_;
  int arrived_ = 0, place_ = 0;
  unsigned sum_ = 0, result_ = 0;
  unsigned long long generation_ = 0;
  std::string broken_;
};

Warp* g_warp = nullptr;
std::mutex g_mu;  // of what follows
unsigned long long g_time = 0;
std::vector<int> g_reports;
std::function<unsigned(const unsigned*)> g_load;          // what the calling lane reads
std::function<bool(unsigned long long*)> g_bytes_there;

struct ThreadIdx {
  struct X {
    operator unsigned() const { return static_cast<unsigned>(t_lane); }
  } x;
} threadIdx;

}  // namespace

#define __all_sync(mask, p) (g_warp->Meet(__LINE__, (p) ? 1u : 0u, [](unsigned a, unsigned b) { return a & b; }) != 0)
#define __any_sync(mask, p) (g_warp->Meet(__LINE__, (p) ? 1u : 0u, [](unsigned a, unsigned b) { return a | b; }) != 0)
#define __reduce_min_sync(mask, v) g_warp->Meet(__LINE__, (v), [](unsigned a, unsigned b) { return a < b ? a : b; })
#define __syncwarp() g_warp->Meet(__LINE__, 0u, [](unsigned a, unsigned) { return a; })
#define __nanosleep(ns)
#undef __device__
#undef __forceinline__
#define __device__
#define __forceinline__ inline

namespace switchml {
namespace kernels {
namespace {

typedef unsigned long long Epoch;
inline unsigned long long GlobalTimerNs() {
  std::lock_guard<std::mutex> lk(g_mu);
  return g_time += 1000;
}
inline void ReportStatus(const RankCtx& ctx, int code) {
  std::lock_guard<std::mutex> lk(g_mu);
  *ctx.status = code;
  g_reports.push_back(code);
}
inline void atomicAdd(unsigned long long* p, unsigned long long v) { __atomic_fetch_add(p, v, __ATOMIC_SEQ_CST); }
inline int atomicExch(int* p, int v) { return __atomic_exchange_n(p, v, __ATOMIC_SEQ_CST); }
inline unsigned LoadSharedAcquire(const unsigned* p) { return g_load(p); }
inline void StoreSharedRelease(unsigned* p, unsigned v) { __atomic_store_n(p, v, __ATOMIC_RELEASE); }
inline bool TryWaitParity(unsigned long long* bar, uint32_t) { return g_bytes_there(bar); }

}  // namespace
}  // namespace kernels
}  // namespace switchml

#include "kernels/one_gpu_waits.cuh"

namespace switchml {
namespace kernels {
namespace {

struct Cta {
  RankCtx ctx = {};
  OneGpuShared sh = {};
  int status = STATUS_OK;
  unsigned long long counters[16] = {};
  Cta() {
    ctx.nranks = 2;
    ctx.timeout_ns = 50000;
    ctx.status = &status;
    ctx.counters = counters;
    g_time = 0;
    g_reports.clear();
    g_load = [](const unsigned* p) { return __atomic_load_n(p, __ATOMIC_ACQUIRE); };
    g_bytes_there = [](unsigned long long*) { return false; };
  }
};

int g_failures = 0;
#define EXPECT(cond)                                             \
  if (!(cond)) {                                                 \
    printf("  FAILED line %d: %s\n", __LINE__, #cond);          \
    fails++;                                                     \
  }

// `body` in all lanes of a warp. What broke the warp's votes, or nothing.
std::string RunWarp(const std::function<void()>& body) {
  Warp warp;
  g_warp = &warp;
  std::string why;
  std::mutex mu;
  std::vector<std::thread> lanes;
  for (int l = 0; l < kLanes; l++)
    lanes.emplace_back([&, l] {
      t_lane = l;
      try {
        body();
      } catch (const std::exception& e) {
        std::lock_guard<std::mutex> lk(mu);
        why = e.what();
      }
    });
  for (auto& t : lanes) t.join();
  g_warp = nullptr;
  return why;
}

// A flag that moves on while the lanes read it: what they know afterwards is the same, so that the next call finds all
// of them in the same place.
int LanesThatReadDifferentCounts() {
  int fails = 0;
  Cta cta;
  thread_local int reads;
  g_load = [](const unsigned*) -> unsigned { return reads++ == 0 ? (t_lane < 20 ? 1 : 3) : 3; };
  bool first[kLanes], second[kLanes];
  const std::string why = RunWarp([&] {
    reads = 0;
    Seen seen;
    first[t_lane] = seen.Reach(cta.ctx, 0, 1, 1, &cta.sh);
    second[t_lane] = seen.Reach(cta.ctx, 0, 1, 3, &cta.sh);
    __syncwarp();
  });
  if (!why.empty()) printf("  %s\n", why.c_str());
  EXPECT(why.empty());
  for (int l = 0; l < kLanes; l++) EXPECT(why.empty() && first[l] && second[l]);
  EXPECT(cta.status == STATUS_OK);
  return fails;
}

// Each of the waits runs out: it ends in all lanes, and the CTA has a status, once.
int AWaitThatRunsOutIsReported() {
  int fails = 0;
  for (int wait = 0; wait < 3; wait++) {
    for (bool late : {true, false}) {  // its own time is up, or another warp has failed
      Cta cta;
      cta.sh.failed = !late;
      bool answer[kLanes];
      const std::string why = RunWarp([&] {
        Seen seen;
        answer[t_lane] = wait == 0   ? WaitForNotes(cta.ctx, 5, &cta.sh, kNoteLoaded, 1)
                         : wait == 1 ? seen.Reach(cta.ctx, 5, 2, 1, &cta.sh)
                                     : WaitForBytes(cta.ctx, 5, &cta.sh.full[0], 0, &cta.sh);
        __syncwarp();
      });
      if (!why.empty()) printf("  %s\n", why.c_str());
      EXPECT(why.empty());
      for (int l = 0; l < kLanes; l++) EXPECT(why.empty() && !answer[l]);
      EXPECT(cta.sh.failed == 1);
      const int phase = wait == 1 ? 2 : kInsideCta;
      EXPECT(cta.status == (late ? STATUS_TIMEOUT | (phase << 4) | (5 << 8) : STATUS_OK));
      EXPECT(g_reports.size() == (late ? 1 : 0) && cta.counters[2] == (late ? 1 : 0));
    }
  }
  return fails;
}

void Run(const char* name, int (*test)()) {
  const int fails = test();
  printf("%s %s\n", fails ? "FAIL" : "ok  ", name);
  g_failures += fails != 0;
}

}  // namespace
}  // namespace kernels
}  // namespace switchml

int main() {
  using namespace switchml::kernels;
  Run("lanes_that_read_different_counts", LanesThatReadDifferentCounts);
  Run("a_wait_that_runs_out_is_reported", AWaitThatRunsOutIsReported);
  return g_failures;
}
