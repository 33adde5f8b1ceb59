// launch.cuh -- step kernel launches with programmatic stream serialization.
#pragma once

#include <cuda_runtime.h>

namespace mlbm {

// Launch a step kernel, with programmatic stream serialization when
// `overlap`: it may then begin while the kernel before it in the stream
// finishes, and waits for it at pdl_gate() (pair.cuh).  What a kernel reads
// before its gate must not be written by the kernel launched right before
// it, whose writes are visible only after the gate.
template <typename... KArgs, typename... Args>
void launch_overlapped(bool overlap, void (*kernel)(KArgs...), unsigned grid,
                       unsigned block, size_t smem, cudaStream_t stream,
                       Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = overlap ? 1 : 0;
  // a failed launch is reported by the caller's cudaGetLastError
  (void)cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Launches into a stream that is being captured into a CUDA graph are plain:
// the overlap is used in ordinary stream order only.
inline bool stream_capturing(cudaStream_t stream) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &st) != cudaSuccess) {
    cudaGetLastError();  // a query refused during another capture: be plain
    return true;
  }
  return st != cudaStreamCaptureStatusNone;
}

}  // namespace mlbm
