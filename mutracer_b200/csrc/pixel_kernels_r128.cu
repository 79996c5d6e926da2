// The megakernels at 128 registers (pixel_kernels.cuh).
#include "pixel_kernels.cuh"

namespace mt {

BatchKernel shapedBatchKernel(bool gpuLayout) {
  return gpuLayout ? k_batch<true, kShapedThreads, kShapedBlocks> : k_batch<false, kShapedThreads, kShapedBlocks>;
}

BatchKernel shapedNoallocKernel(bool gpuLayout) {
  return gpuLayout ? k_batch_noalloc<true, kShapedThreads, kShapedBlocks>
                   : k_batch_noalloc<false, kShapedThreads, kShapedBlocks>;
}

}  // namespace mt
