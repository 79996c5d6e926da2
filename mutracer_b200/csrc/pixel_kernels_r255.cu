// The megakernels at 255 registers (pixel_kernels.cuh).
#include "pixel_kernels.cuh"

namespace mt {

TraceKernel traceKernel256(bool gpuLayout) { return gpuLayout ? k_trace<true, 256> : k_trace<false, 256>; }

BatchKernel batchKernel256(bool gpuLayout) { return gpuLayout ? k_batch<true, 256, 1> : k_batch<false, 256, 1>; }

BatchKernel noallocKernel256(bool gpuLayout) {
  return gpuLayout ? k_batch_noalloc<true, 256, 1> : k_batch_noalloc<false, 256, 1>;
}

}  // namespace mt
