// Something that has to be done once on every device before a kernel is launched there.
#ifndef SWITCHML_ONCE_PER_DEVICE_H_
#define SWITCHML_ONCE_PER_DEVICE_H_

#include <atomic>

namespace switchml {
namespace kernels {

// Calls `act` (0 = success) unless it has succeeded before with this device's bit of `done`. What has failed is
// tried again by the next call. Two threads may both call it.
template <typename Act>
auto OncePerDevice(int device, std::atomic<unsigned long long>* done, Act act) -> decltype(act()) {
  const unsigned long long bit = 1ull << (device & 63);
  if (done->load(std::memory_order_acquire) & bit) return static_cast<decltype(act())>(0);
  const auto e = act();
  if (e == 0) done->fetch_or(bit, std::memory_order_release);
  return e;
}

}  // namespace kernels
}  // namespace switchml
#endif  // SWITCHML_ONCE_PER_DEVICE_H_
