// The megakernels, as templates over the block they are compiled for.  The
// compiler gives the out-of-line shading code of a source file the registers of
// the smallest budget among the kernels that call it, so each register budget
// has a file of its own:
//   megakernel.cu, batch_noalloc.cu  1,024 threads, 64 registers
//   pixel_kernels_r128.cu            128 registers
#pragma once
#include "batch_table.cuh"

namespace mt {

__device__ __forceinline__ void addCounters(const Counters &cnt, uint32_t paths, mtc_counters *out) {
  if (!out) return;
  unsigned mask = __activemask();
  uint32_t e = __reduce_add_sync(mask, cnt.ext);
  uint32_t s = __reduce_add_sync(mask, cnt.shadow);
  uint32_t p = __reduce_add_sync(mask, paths);
  int leader = __ffs(mask) - 1;
  if ((threadIdx.x & 31) == leader) {
    atomicAdd(&out->extension_rays, (unsigned long long)e);
    atomicAdd(&out->shadow_rays, (unsigned long long)s);
    atomicAdd(&out->path_samples, (unsigned long long)p);
  }
}

// The same, and the launch itself.
__device__ __forceinline__ void flushCounters(const Counters &cnt, uint32_t paths, mtc_counters *out) {
  if (out && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&out->kernel_launches, 1ull);
  addCounters(cnt, paths, out);
}

using BatchKernel = void (*)(const BatchHeader *, uint32_t *, mtc_counters *, uint32_t, uint32_t *);

// Persistent batched kernel over a job table (batch_table.cuh).
template <bool kGpuLayout, uint32_t kThreads, uint32_t kBlocks>
__global__ void __launch_bounds__(kThreads, kBlocks)
    k_batch(const BatchHeader *header, uint32_t *queue, mtc_counters *counters, uint32_t grain, uint32_t *status) {
  Counters cnt;
  uint32_t paths = 0;
  batchWorkLoop<kGpuLayout>(header, queue, grain, status, cnt, paths);
  flushCounters(cnt, paths, counters);
}

// The same over the fixed scratch of batch_noalloc.cu.
template <bool kGpuLayout, uint32_t kThreads, uint32_t kBlocks>
__global__ void __launch_bounds__(kThreads, kBlocks)
    k_batch_noalloc(const BatchHeader *header, uint32_t *queue, mtc_counters *counters, uint32_t grain,
                    uint32_t *status) {
  Counters cnt;
  uint32_t paths = 0;
  batchWorkLoop<kGpuLayout>(header, queue, grain, status, cnt, paths);
  addCounters(cnt, paths, counters);
}

// The kernels for blocks of a size that the host gave (kShapedThreads at most).
BatchKernel shapedBatchKernel(bool gpuLayout);
BatchKernel shapedNoallocKernel(bool gpuLayout);

}  // namespace mt
