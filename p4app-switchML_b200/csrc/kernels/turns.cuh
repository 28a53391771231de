// Loops that keep several loads per thread in flight.
#ifndef SWITCHML_TURNS_CUH_
#define SWITCHML_TURNS_CUH_

#include <stddef.h>

#include <type_traits>

namespace switchml {
namespace kernels {
namespace {

// Walks the elements i, i + n, i + 2n, ... below `count`: whole turns of U of them, then what is left in turns
// of U/2, U/4, ... 1 (log2(U) trips to memory instead of U - 1; predicating one whole turn instead cost
// registers, and a third of the speed of the loop before it); or
// (kHalve = false) one by one: fewer bodies of `f`, hence fewer registers. f(width, i) takes `width` of them.
template <int U, bool kHalve = true, typename F>
__device__ __forceinline__ void Turns(size_t i, size_t count, size_t n, F f) {
  for (; i + (U - 1) * n < count; i += U * n) f(std::integral_constant<int, U>(), i);
  if constexpr (U > 1) {
    if (i < count) Turns<kHalve ? U / 2 : 1, kHalve>(i, count, n, f);
  }
}

}  // namespace
}  // namespace kernels
}  // namespace switchml
#endif  // SWITCHML_TURNS_CUH_
