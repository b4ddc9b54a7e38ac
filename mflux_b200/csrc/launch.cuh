// Launches that overlap the end of the kernel before them in their stream (programmatic dependent launch).
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace mfx {

// A kernel started with launch_overlapped() may begin while its predecessor drains: blocks take the SMs that the
// predecessor's last wave leaves, set up barriers, tensor memory and descriptors, and meet here before their first access
// to memory that another kernel may write or read. Returns once the predecessor has finished and its writes are visible
// (at once where the launch was an ordinary one). Every thread of every such kernel calls it before anything else that
// touches global memory, so a kernel's end still means the end of everything before it in the stream.
// Such a kernel reads global memory by plain or volatile loads, TMA and cp.async, never by the read-only path (__ldg, const
// __restrict__): that path is for memory which nobody writes while the kernel lives, and this one lives while its
// predecessor still writes. The compiler may also move its loads across the wait, the others not (they come behind volatile assembly
// that clobbers memory).
// Without / with it: kernels of a few microseconds one after the other 0.3 to 0.5 us less each (256 x 256 decoded 1.54 /
// 1.13, 333 tokens x 24 heads of attention 10.2 / 9.1), 333 rows of N 9216, K 3072, 4 bits 25.4 / 24.4 us, a step of 380
// launches (8-bit single-stream model, 1613 tokens) 22.21 / 21.82 ms; 24 heads x 4608 tokens of attention 239.5 / 239.1, which
// is noise.
__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// From here on the successor's blocks may be started. They only come to a SM as this kernel's blocks leave it room.
__device__ __forceinline__ void allow_successor() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... Params, typename... Args>
cudaError_t launch_overlapped(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                              Args&&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
  // a failure is the returned value's alone: left pending it would be the next ordinary launch's cudaGetLastError()
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}

}  // namespace mfx
