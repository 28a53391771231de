// Kernels that are launched before the one ahead of them in the stream has ended (programmatic dependent launch).
//
// Ordinarily a kernel's launch begins when its predecessor's last block has left and its stores are
// visible, which back to back costs 2 to 4 us per kernel: blocks to place, barriers, TMEM and tensor maps to set up,
// and the end of a kernel is noticed in steps of 2 us. Launched with LaunchOverlapped, the blocks take the
// SMs' places as these become free, set up, and wait in WaitForEarlierKernels() for the predecessor to be complete
// and its memory to be visible. What the stream promises stays as it was:
//   - a kernel launched this way calls WaitForEarlierKernels() in every thread before it touches global memory, so
//     it cannot end before its predecessor either, and the order holds over any number of them;
//   - a predecessor that knows nothing of this lets the next one start when its last block has left;
//   - an ordinary kernel, copy or event behind one of these waits for its end as ever.
#ifndef SWITCHML_DEPENDENT_LAUNCH_CUH_
#define SWITCHML_DEPENDENT_LAUNCH_CUH_

#include <cuda_runtime.h>

#include <cstring>

namespace switchml {
namespace kernels {

__device__ __forceinline__ void WaitForEarlierKernels() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The next kernel's blocks may be placed once every block of this one has called this or has ended.
__device__ __forceinline__ void LetNextKernelStart() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// `cluster`: CTAs of a cluster.
template <class... Params, class... Args>
cudaError_t LaunchOverlapped(void (*kernel)(Params...), unsigned blocks, unsigned threads, size_t smem, unsigned cluster,
                             cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attrs[2];
  memset(&cfg, 0, sizeof(cfg));
  memset(attrs, 0, sizeof(attrs));
  attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[0].val.programmaticStreamSerializationAllowed = 1;
  attrs[1].id = cudaLaunchAttributeClusterDimension;
  attrs[1].val.clusterDim.x = cluster;
  attrs[1].val.clusterDim.y = attrs[1].val.clusterDim.z = 1;
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attrs;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

}  // namespace kernels
}  // namespace switchml
#endif  // SWITCHML_DEPENDENT_LAUNCH_CUH_
