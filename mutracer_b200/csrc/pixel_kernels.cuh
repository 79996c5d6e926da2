// The megakernels, as templates over the block they are compiled for.  The
// compiler gives the out-of-line shading code of a source file the registers of
// the smallest budget among the kernels that call it, so each register budget
// has a file of its own:
//   megakernel.cu, batch_noalloc.cu  1,024 threads, 64 registers
//   pixel_kernels_r128.cu            128 registers
//   pixel_kernels_r255.cu            255 registers
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

// The pixels of one image in the order of its 8x4 tiles: the grid's blocks take
// turns at runs of `run` of them, which a block's lanes claim one by one.  Of
// each warp `lanes` lanes ask: a small image is spread over all warps an SM
// holds, a few lanes in each, rather than over full warps of a few.
struct ImageSplit {
  uint32_t run, lanes;
};
struct ImageClaims {
  const JobData &J;
  uint32_t samples;
  uint32_t *cursor;  // shared: the block's next pixel
  ImageSplit split;
  bool exhausted = false;

  MTD void next(bool wants, const JobData *&job, uint32_t &x, uint32_t &y, uint32_t &left) {
    const uint32_t lane = threadIdx.x & 31u, tilesX = (J.width + 7u) / 8u;
    const uint64_t units = uint64_t(tilesX) * ((J.height + 3u) / 4u) * 32u;
    wants = wants && lane < split.lanes;
    unsigned asking = __ballot_sync(0xffffffffu, wants);
    while (asking && !exhausted) {
      uint32_t k = 0;
      if (lane == 0) k = atomicAdd(cursor, uint32_t(__popc(asking)));
      k = __shfl_sync(0xffffffffu, k, 0) + __popc(asking & ((1u << lane) - 1u));
      const uint64_t u = (uint64_t(k / split.run) * gridDim.x + blockIdx.x) * split.run + k % split.run;
      if (wants && u < units) {
        const uint32_t tile = uint32_t(u / 32u), in = uint32_t(u % 32u);
        x = tile % tilesX * 8u + in % 8u;
        y = tile / tilesX * 4u + in / 8u;
        if (x < J.width && y < J.height) {
          job = &J;
          left = samples;
          wants = false;
        }
      }
      // Pixels ascend with the cursor: none is left once one lies past the
      // image.
      exhausted = __any_sync(0xffffffffu, wants && u >= units);
      asking = __ballot_sync(0xffffffffu, wants);
    }
  }
};

// The plain megakernel.  Bound by instruction fetch and by the latency of its
// spilled state; with the 32 warps of an SM's block in step 4 samples of the
// 4M-triangle instanced scene at 960x540 take 29.5 ms (64 free-running warps
// an SM with one thread per pixel: 67.2), 8 of the Cornell box at 512x512 12.8
// (29.6), one of the glass scene at 640x360 20.4 (85.2), one of a 256x256
// Cornell box 0.78 (1.9).  Free-running warps that trace and shade together,
// or that shade once 8, 12 or 20 lanes wait, are slower than one thread per
// pixel: it is the fetches shared by the block that pay.
template <bool kGpuLayout, uint32_t kThreads>
__global__ void __launch_bounds__(kThreads, 1)
    k_trace(const __grid_constant__ JobData J, uint32_t samples, ImageSplit split, mtc_counters *counters) {
  __shared__ uint32_t cursor;
  if (threadIdx.x == 0) cursor = 0;
  __syncthreads();
  Counters cnt;
  uint32_t paths = 0;
  ImageClaims claims{J, samples, &cursor, split};
  tracePixels<kGpuLayout>(claims, cnt, paths);
  flushCounters(cnt, paths, counters);
}

using TraceKernel = void (*)(const JobData, uint32_t, ImageSplit, mtc_counters *);
// The kernels for blocks of up to 512 and 256 threads.
TraceKernel traceKernel512(bool gpuLayout);
TraceKernel traceKernel256(bool gpuLayout);

using BatchKernel = void (*)(const BatchHeader *, uint32_t *, mtc_counters *, uint32_t, uint32_t *);

// Persistent batched kernel over a job table (batch_table.cuh).
template <bool kGpuLayout, uint32_t kThreads, uint32_t kBlocks>
__global__ void __launch_bounds__(kThreads, kBlocks)
    k_batch(const BatchHeader *header, uint32_t *queue, mtc_counters *counters, uint32_t grain, uint32_t *status) {
  Counters cnt;
  uint32_t paths = 0;
  batchWorkLoop<kGpuLayout, kThreads != kShapedThreads>(header, queue, grain, status, cnt, paths);
  flushCounters(cnt, paths, counters);
}

// The same over the fixed scratch of batch_noalloc.cu.
template <bool kGpuLayout, uint32_t kThreads, uint32_t kBlocks>
__global__ void __launch_bounds__(kThreads, kBlocks)
    k_batch_noalloc(const BatchHeader *header, uint32_t *queue, mtc_counters *counters, uint32_t grain,
                    uint32_t *status) {
  Counters cnt;
  uint32_t paths = 0;
  batchWorkLoop<kGpuLayout, kThreads != kShapedThreads>(header, queue, grain, status, cnt, paths);
  addCounters(cnt, paths, counters);
}

// The kernels for blocks of a size that the host gave (kShapedThreads at most).
BatchKernel shapedBatchKernel(bool gpuLayout);
BatchKernel shapedNoallocKernel(bool gpuLayout);
// The kernels for blocks of 512 and of up to 256 threads (BatchGrid).
BatchKernel batchKernel512(bool gpuLayout);
BatchKernel noallocKernel512(bool gpuLayout);
BatchKernel batchKernel256(bool gpuLayout);
BatchKernel noallocKernel256(bool gpuLayout);

}  // namespace mt
