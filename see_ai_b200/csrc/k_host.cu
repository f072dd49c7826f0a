// Small transfers between the host and a step's stream, as kernels.
//
// A step of a small plan is a few dozen launches of two to five microseconds; a
// copy-engine transfer between them costs its own start-up and the hand-over to
// and from the compute engine (5 to 16 us between a 32 KB upload and the first
// kernel behind it), and two of them at either end of the step were a quarter of
// the feed-forward plan's 121 us.  A kernel that reads or writes pinned host memory
// itself costs one launch.  Scalars travel as kernel parameters.
#include "kernels.h"
#include "launch.cuh"

namespace see::k {

namespace {

__device__ __forceinline__ void CopyBytes(uint8_t* dst, const uint8_t* src, size_t bytes, size_t t, size_t threads) {
  if (((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 15) == 0) {
    const size_t quads = bytes / 16;
    for (size_t i = t; i < quads; i += threads) reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
    for (size_t i = quads * 16 + t; i < bytes; i += threads) dst[i] = src[i];
  } else if (((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 3) == 0) {
    const size_t words = bytes / 4;
    for (size_t i = t; i < words; i += threads) reinterpret_cast<uint32_t*>(dst)[i] = reinterpret_cast<const uint32_t*>(src)[i];
    for (size_t i = words * 4 + t; i < bytes; i += threads) dst[i] = src[i];
  } else {
    for (size_t i = t; i < bytes; i += threads) dst[i] = src[i];
  }
}

__global__ void StageKernel(HostCopy a, HostCopy b) {
  AwaitPrevious();
  const size_t t = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
  const size_t threads = static_cast<size_t>(gridDim.x) * blockDim.x;
  if (a.bytes) CopyBytes(static_cast<uint8_t*>(a.dst), static_cast<const uint8_t*>(a.src), a.bytes, t, threads);
  if (b.bytes) CopyBytes(static_cast<uint8_t*>(b.dst), static_cast<const uint8_t*>(b.src), b.bytes, t, threads);
}

__global__ void PublishKernel(PublishList list, uint32_t* __restrict__ host) {
  AwaitPrevious();
  uint32_t at = 0;
  for (int i = 0; i < list.count; ++i) {
    for (uint32_t w = threadIdx.x; w < list.item[i].words; w += blockDim.x) host[at + w] = list.item[i].src[w];
    at += list.item[i].words;
  }
}

__global__ void SetScalarsKernel(AdamScalars v, AdamScalars* dst) { AwaitPrevious(); *dst = v; }

}  // namespace

void StageFromHost(const HostCopy& a, const HostCopy& b, cudaStream_t s) {
  const size_t quads = (a.bytes + b.bytes) / 16 + 1;
  const size_t blocks = quads < 64 * 256 ? (quads + 255) / 256 : 64;
  Next(StageKernel, static_cast<unsigned>(blocks), 256, 0, s)(a, b);
}

void PublishToHost(const PublishList& list, uint32_t* host, cudaStream_t s) { Next(PublishKernel, 1, 32, 0, s)(list, host); }

void SetScalars(const AdamScalars& v, AdamScalars* dst, cudaStream_t s) { Next(SetScalarsKernel, 1, 1, 0, s)(v, dst); }

}  // namespace see::k
