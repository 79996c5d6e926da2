// The megakernels at 255 registers (pixel_kernels.cuh).
#include "pixel_kernels.cuh"

namespace mt {

TraceKernel traceKernel256(bool gpuLayout) { return gpuLayout ? k_trace<true, 256> : k_trace<false, 256>; }

}  // namespace mt
