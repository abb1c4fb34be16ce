// hsr_launch.cuh — the kernels of a launch sequence overlap their launches (sm_90 and later:
// programmatic dependent launch).
//
// A sequence is a chain of short kernels, each reading what the one before it wrote; for a small
// draw the gaps between them (drain, launch, first loads: about 3 us each) are much of its time.
// Launched with launch_chained, a kernel's blocks become resident as the blocks of the kernel
// before it exit, and wait at chain_wait until that kernel has completed and its writes are
// visible.  Every block of every kernel of a chain calls chain_wait before it reads or
// writes anything, so no kernel completes before its predecessor and the order of the whole chain
// holds.  The wait orders ordinary loads: a kernel of the chain reads the view descriptors and
// whatever else another kernel of the chain writes by those alone, never by read-only loads (__ldg, or
// what the compiler makes of a const __restrict__ parameter), which are defined only for memory that
// nobody writes while the kernel is resident.  No kernel triggers its successor early (griddepcontrol.launch_dependents): the waiting
// blocks would hold slots that this kernel's work needs (1080p frame: 365 against 356 us).
//
// Whole calls with this, one set-up kernel for copy and memset, and the control block written by
// the raster: 128x128 draw 95 -> 74 us, 1000x600 with shadow 206 -> 185 us, six objects 317 ->
// 290 us, 64 served requests 4,440 -> 4,180 us.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace hsr {

__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class... Params, class... Args>
int launch_chained(void (*kernel)(Params...), int grid, int block, size_t smem, cudaStream_t s, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  // a captured sequence keeps plain edges (the replay is as fast)
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cfg.numAttrs = cudaStreamIsCapturing(s, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone ? 1 : 0;
  return (int)cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace hsr
