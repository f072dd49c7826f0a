// Kernels that follow one another on a stream, most of them a few microseconds long.
//
// A kernel launched by Next is a programmatic dependent launch: its blocks start once those of the kernel before it have
// exited, instead of after that grid's memory has been flushed and the launch has gone through the front end.  What it
// does before AwaitPrevious (barriers, tensor memory) overlaps with that; AwaitPrevious returns when the kernel before is
// complete and its writes are seen.  Every kernel that Next launches executes AwaitPrevious before it touches global
// memory, in every thread, and by that waits for all kernels before it: the one before has waited for its own.
// A grid that leaves half of the chip idle also lets the next kernel's blocks start, and set up, at once (they wait in
// AwaitPrevious all the same); a larger one does not, for a kernel that runs under a pending successor gets slower itself.
// Per kernel of a chain on a B200, us, plain / so without an early start: 148 blocks of 256 threads 1.31 / 1.00 replayed
// as a graph, 3.59 / 2.40 launched one by one; a pass over 32 MB 4.55 / 4.14, with an early start 5.71.  A step of an int8
// decoder on 600 rows (120 kernels) 757 / 748, with an early start up to 74 blocks 721, up to 148 blocks 684; but of an f32 decoder on 4096
// rows (157 kernels) 1632 / 1632, 1637 and 1723.
#ifndef SEE_CUDA_LAUNCH_CUH_
#define SEE_CUDA_LAUNCH_CUH_

#include <cuda_runtime.h>

#include <cstddef>
#include <utility>

namespace see::k {

constexpr unsigned kEarlyStartBlocks = 74;
__device__ __forceinline__ void AwaitPrevious() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (gridDim.x * gridDim.y * gridDim.z <= kEarlyStartBlocks) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Next(kernel, grid, block, shared memory, stream)(arguments): kernel<<<grid, block, shared memory, stream>>>(arguments),
// in clusters of `cluster` blocks along x.
template <typename... Params>
struct NextLaunch {
  void (*kernel)(Params...);
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
  unsigned cluster;
  template <typename... Args>
  cudaError_t operator()(Args&&... args) const {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
  }
};
template <typename... Params>
NextLaunch<Params...> Next(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, unsigned cluster = 1) {
  return {kernel, grid, block, smem, stream, cluster};
}

}  // namespace see::k

#endif  // SEE_CUDA_LAUNCH_CUH_
