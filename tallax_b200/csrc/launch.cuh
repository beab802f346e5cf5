// How the kernels are launched: as programmatic dependents of what precedes them on the stream.
//
// A kernel launched this way begins with grid_wait(), or does before it only what needs nothing of its predecessors: the wait
// returns when the predecessor has finished and its writes are visible.  Nothing of a call reads or writes memory before the
// calls before it are complete, which themselves began with the same wait, but the launch's own work, 1 to 2 us between two
// kernels of a stream, is done by then.  A predecessor that knows nothing of this (any other kernel, a copy) is waited for in the
// same way.  A kernel whose successor may start before it has finished (grid_release) is one whose successor waits for it,
// in one CTA at least, before it ends.  The exchange's merge kernel alone reads and writes memory before it waits: the rows as they
// arrive, and its parameters, which nothing may write between the candidate kernel and it (tlx_exchange_merge_and_sample).
//   us a call, queued one after the other, plain launches / these: sampler bf16 [1, 128256] 10.6 / 9.3, [32, 128256] 26.0 / 24.2,
// [256, 128256] 48.4 / 46.2; top-k f32 [8, 32768] 10.3 / 8.5; cumsum f32 [64, 128256] 18.6 / 17.2; gather 4096 of f32 [1024, 262144]
// 78.4 / 76.8; sort bf16 [64, 4097] 10.2 / 7.7.
//   Released at their start, the kernels' successors fill the SMs as these leave room, unevenly: cumsum 21.1 us, sampler of 256
// rows 51.6.
#pragma once
#include "tlx_common.cuh"

namespace tlx {

__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// cluster: CTAs of a thread-block cluster; carveout: the share of an SM's memory that the kernel prefers as shared
// memory, in percent; -1: as set for the kernel.
struct LaunchShape {
  unsigned grid, block;
  size_t smem = 0;
  int cluster = 1;
  int carveout = -1;
  bool plain = false;      // in plain stream order (the kernel's wait is then a no-op)
};

template <typename... Params, typename... Args>
int launch_dependent(void (*kernel)(Params...), const LaunchShape& shape, cudaStream_t st, const char* what, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(shape.grid);
  cfg.blockDim = dim3(shape.block);
  cfg.dynamicSmemBytes = shape.smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[3]{};
  int n = 0;
  if (shape.cluster > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = (unsigned)shape.cluster;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (shape.carveout >= 0) {
    attr[n].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    attr[n++].val.sharedMemCarveout = (unsigned)shape.carveout;
  }
  attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // (the last one: left out where it is not accepted)
  attr[n].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (unsigned)(shape.plain ? n : n + 1);
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
  if (e == cudaErrorNotSupported && !shape.plain) {
    cudaGetLastError();
    cfg.numAttrs = (unsigned)n;
    e = cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return set_error(TLX_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  }
  count_launch();
  return TLX_OK;
}

}  // namespace tlx
