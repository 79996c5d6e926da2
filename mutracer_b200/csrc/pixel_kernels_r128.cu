// The megakernels at 128 registers (pixel_kernels.cuh).
#include "pixel_kernels.cuh"

namespace mt {

TraceKernel traceKernel512(bool gpuLayout) { return gpuLayout ? k_trace<true, 512> : k_trace<false, 512>; }

BatchKernel batchKernel512(bool gpuLayout) { return gpuLayout ? k_batch<true, 512, 1> : k_batch<false, 512, 1>; }

BatchKernel noallocKernel512(bool gpuLayout) {
  return gpuLayout ? k_batch_noalloc<true, 512, 1> : k_batch_noalloc<false, 512, 1>;
}

BatchKernel shapedBatchKernel(bool gpuLayout) {
  return gpuLayout ? k_batch<true, kShapedThreads, kShapedBlocks> : k_batch<false, kShapedThreads, kShapedBlocks>;
}

BatchKernel shapedNoallocKernel(bool gpuLayout) {
  return gpuLayout ? k_batch_noalloc<true, kShapedThreads, kShapedBlocks>
                   : k_batch_noalloc<false, kShapedThreads, kShapedBlocks>;
}

}  // namespace mt
