// Job validation, job-table layout and the persistent work loop shared by the
// batched entry points (mtc_batch_prepare / mtc_batch_launch / mtc_trace_batch
// in megakernel.cu and mtc_trace_batch_noalloc in batch_noalloc.cu), so that
// every entry point accepts exactly the same jobs and launch shapes.
#pragma once
#include <cuda_runtime.h>

#include <cstring>

#include "dev_shade.cuh"

namespace mt {

// Header of a batched job table (host table and device copy alike); the
// JobData entries follow at kBatchTableOffset.  The kernels read the job
// count, item total and tile width from it, so a captured launch can be
// replayed after the host table is rewritten with other jobs.
struct BatchHeader {
  uint32_t jobCount, totalItems, tileW, flagsUnion, _pad[60];
};
static_assert(sizeof(BatchHeader) == 256, "batch header size");
constexpr size_t kBatchTableOffset = sizeof(BatchHeader);
// Work items of one table stay below this, so a queue counter that every
// warp advances once past the total cannot wrap.
constexpr uint64_t kBatchMaxItems = 0x7fffffffull;

// Bit set in a batched launch's status word when a warp's work loop ran out
// of iterations before the queue counter passed the item total (cannot
// happen while the counter only grows; reported instead of spinning).
constexpr uint32_t kBatchStatusGuardExhausted = MTC_BATCH_STATUS_GUARD_EXHAUSTED;

// A scene view the kernels can read: every mandatory binding present and
// every vertex-layout field inside the vertex record.
inline bool validScene(const mtc_scene_view *s) {
  return s && s->struct_size == sizeof(mtc_scene_view) && s->bvh && s->instances && s->attributes && s->materials &&
         s->material_count > 0 && s->energy_lut && s->light_sampling &&
         s->vertex_layout.stride >= 4 && s->vertex_layout.normal_offset + (s->vertex_layout.normal_float ? 3u : 1u) <=
                                             s->vertex_layout.stride &&
         (s->vertex_layout.uv_offset == 0 || (s->vertex_layout.uv_offset >= 3 &&
                                              s->vertex_layout.uv_offset + 2 <= s->vertex_layout.stride)) &&
         (s->vertex_layout.uv1_offset == 0 || (s->vertex_layout.uv1_offset >= 3 &&
                                               s->vertex_layout.uv1_offset + 2 <= s->vertex_layout.stride)) &&
         (s->vertex_layout.color_offset == 0 ||
          (s->vertex_layout.color_offset >= 3 &&
           s->vertex_layout.color_offset + (s->vertex_layout.color_float ? 3u : 1u) <= s->vertex_layout.stride));
}

inline bool validUniform(const mtc_trace_uniform *u) {
  if (!u) return false;
  float w = u->output_size[0], h = u->output_size[1];
  return w >= 1.0f && h >= 1.0f && w <= 65536.0f && h <= 65536.0f && u->loop_unroll_guard == 4u;
}

inline bool validOutputs(const mtc_outputs *o) {
  return o && o->color && o->normal && o->albedo && o->shadow_catcher;
}

inline DevScene toDev(const mtc_scene_view *v) {
  DevScene s;
  s.bvh = (const float4 *)v->bvh;
  s.ins = (const float4 *)v->instances;
  s.attr = (const uint32_t *)v->attributes;
  s.mats = (const float4 *)v->materials;
  s.env = (const float4 *)v->env_map;
  s.envDist = (const float2 *)v->env_distribution;
  s.lightData = (const float4 *)v->light_sampling;
  s.lut = (const float *)v->energy_lut;
  s.lights = (const float4 *)v->analytic_lights;
  s.envW = v->env_width;
  s.envH = v->env_height;
  s.vstride = v->vertex_layout.stride;
  s.vnormalOff = v->vertex_layout.normal_offset;
  s.vnormalFloat = v->vertex_layout.normal_float;
  s.flags = v->flags;
  s.insCount = v->instance_count;
  s.matCount = v->material_count;
  s.maps = (const float4 *)v->maps;
  s.mapTexels = (const float4 *)v->map_texels;
  s.mapCount = v->maps && v->map_texels ? v->map_count : 0;
  s.mapTexelCount = v->map_texel_count;
  s.vuvOff = v->vertex_layout.uv_offset;
  s.vcolorOff = v->vertex_layout.color_offset;
  s.vuv1Off = v->vertex_layout.uv1_offset;
  s.triMats = v->triangle_materials;
  s.vcolorFloat = v->vertex_layout.color_float;
  return s;
}

// One job's table entry for warp tiles of tileW x (32 / tileW) pixels.
inline JobData makeJob(const mtc_scene_view *scene, const mtc_camera_uniform *camera,
                       const mtc_trace_uniform *uniform, const mtc_outputs *out, uint32_t samples,
                       uint32_t tileW = 8u) {
  JobData J;
  std::memset(&J, 0, sizeof(J));
  J.s = toDev(scene);
  J.u = *uniform;
  J.cam = *camera;
  J.outColor = (float4 *)out->color;
  J.outNormal = (float4 *)out->normal;
  J.outAlbedo = (float4 *)out->albedo;
  J.outCatcher = (float4 *)out->shadow_catcher;
  J.samples = samples;
  J.width = uint32_t(uniform->output_size[0]);
  J.height = uint32_t(uniform->output_size[1]);
  const uint32_t tileH = 32u / tileW;
  J.tilesX = (J.width + tileW - 1) / tileW;
  J.tilesY = (J.height + tileH - 1) / tileH;
  J.items = samples ? J.tilesX * J.tilesY : 0u;
  return J;
}

// Threads per block the megakernels run with by default: one block fills an SM
// at 64 registers, its 32 warps in step (tracePixels).
constexpr uint32_t kPixelThreads = 1024;

// Blocks of the size a host asks for (32 to 128 threads) run kernels compiled
// for four of 128 threads an SM, at 128 registers.  Smaller blocks share less of
// the code they fetch and gain more from registers than from more warps: 8
// uneven jobs of instanced scenes 176 ms, two samples of a 512x512 Cornell box
// 5.7 ms; eight blocks at 64 registers 186 and 7.1, sixteen at 32 registers 186
// and 7.4 (free-running warps with one thread per pixel: 227 and 8.5).
constexpr uint32_t kShapedThreads = 128, kShapedBlocks = 4;

// Small images: up to 256 pixels an SM go to 8 warps of one block, a few lanes
// each.  Few lanes mean little divergence (61x47 pixels, ms with 8 warps of few
// lanes, 4 of more, full warps in blocks of 1 and of 8: the instanced scene, 4
// samples, 1.71, 1.92, 2.53 and 3.04; glass, 2 samples, 9.1, 10.4, 12.6 and 14.9;
// the Cornell box, 4 samples, 1.11, 1.10, 1.17 and 1.28; with one thread per
// pixel in free-running blocks 4.7, 24.9 and 1.46).  That is a choice for the
// latency of one render: it takes some of every SM, and several at a time hold
// one another up where paths hardly diverge (61x47 Cornell boxes on 1, 2, 4 and
// 8 streams 0.42, 0.65, 1.08 and 1.95 ms, free-running 0.56, 0.59, 0.68 and
// 1.09; the instanced scene 0.72, 0.93, 1.43 and 2.48 against 1.69, 1.69, 1.76
// and 2.21; glass 5.3, 5.5, 9.2 and 15.2 against 14 to 20).  64 or 128 registers
// hardly help those and cost one render 15 to 35 %; a block of one warp for each
// pixel of the smallest images made eight of 24x24 take 1.63 ms, not 1.20.
constexpr uint32_t kSpreadWarps = 8;

struct BatchShape {
  uint32_t blockThreads, tileW, tileH, ctasPerSm, grain;
  bool shaped;  // block size given: kShapedThreads at most
};
// Resolves a (possibly NULL) mtc_batch_config to launch parameters; false for
// out-of-range values.
inline bool batchShape(const mtc_batch_config *c, BatchShape &out) {
  out = BatchShape{kPixelThreads, 8u, 4u, 1u, 1u, false};
  if (!c) return true;
  if (c->struct_size != sizeof(mtc_batch_config)) return false;
  if (c->block_threads) {
    if (c->block_threads > 128u || c->block_threads % 32u) return false;
    out.blockThreads = c->block_threads;
    out.ctasPerSm = kShapedThreads * kShapedBlocks / c->block_threads;
    out.shaped = true;
  }
  if (c->tile_width) {
    if (c->tile_width > 32u || (32u % c->tile_width)) return false;
    out.tileW = c->tile_width;
    out.tileH = 32u / c->tile_width;
  }
  if (c->ctas_per_sm) {
    if (c->ctas_per_sm > 32u) return false;
    out.ctasPerSm = c->ctas_per_sm;
  }
  if (c->items_per_fetch) {
    if (c->items_per_fetch > 16u) return false;
    out.grain = c->items_per_fetch;
  }
  return true;
}

// The grid of a batched launch over `totalItems` work items.  Tables of few
// pixels run like small images: the grid's blocks share them out (TableClaims),
// in blocks of kSpreadWarps at 255 registers.  Full warps of blocks of 1,024, on
// the few SMs whose warps came first, were slower than free-running warps on the
// Cornell box (61x47 pixels, one sample, free-running / in blocks of 1,024 / so:
// 0.65, 0.79, 0.44 ms; of the instanced scene 1.71, 1.77, 0.88; 17x13 pixels,
// three images, 0.57, 0.66, 0.40).  A captured launch may run other tables later:
// it keeps the blocks of 1,024 and spreads over some of their warps (0.56 ms for
// the first of these).  Up to kMediumPixels an SM, 16 warps at 128 registers have
// a lane for every pixel: 333x217 pixels, in blocks of 1,024 / so, Cornell box
// 2.50, 1.87 ms; instanced scene 5.03, 3.99; glass 19.9, 16.3; room 4.69, 4.10.
constexpr uint32_t kMediumPixels = 512;
struct BatchGrid {
  uint32_t blocks, threads;
  bool few;     // blocks of up to 256 threads
  bool medium;  // of 512
};
inline BatchGrid batchGrid(const BatchShape &shape, uint32_t totalItems, uint32_t sms) {
  const uint64_t pixels = uint64_t(totalItems) * 32u, perSm = (pixels + sms - 1u) / sms;
  if (shape.shaped || shape.ctasPerSm != 1u || perSm > kMediumPixels || pixels == 0u)
    return BatchGrid{sms * shape.ctasPerSm, shape.blockThreads, false, false};
  if (perSm > kSpreadWarps * 32u) return BatchGrid{sms, kMediumPixels, false, true};
  return BatchGrid{sms, uint32_t(perSm < kSpreadWarps ? perSm : kSpreadWarps) * 32u, true, false};
}

// Writes the header and `job_count` entries of a job table to host memory
// `base` (kBatchTableOffset + job_count * sizeof(JobData) bytes).
inline mt_status writeBatchTable(const mtc_job_desc *jobs, uint32_t job_count, const BatchShape &shape, void *base,
                                 uint32_t *total_items) {
  char *out = static_cast<char *>(base);
  uint64_t total = 0;
  uint32_t flagsUnion = 0;
  for (uint32_t j = 0; j < job_count; j++) {
    const mtc_job_desc &d = jobs[j];
    if (!validScene(&d.scene) || !validUniform(&d.uniform) || !validOutputs(&d.out))
      return MT_ERROR_INVALID_ARGUMENT;
    JobData J = makeJob(&d.scene, &d.camera, &d.uniform, &d.out, d.samples, shape.tileW);
    J.firstItem = uint32_t(total);
    total += J.items;
    if (total >= kBatchMaxItems) return MT_ERROR_INVALID_ARGUMENT;
    flagsUnion |= d.scene.flags;
    std::memcpy(out + kBatchTableOffset + size_t(j) * sizeof(JobData), &J, sizeof(J));
  }
  BatchHeader h;
  std::memset(&h, 0, sizeof(h));
  h.jobCount = job_count;
  h.totalItems = uint32_t(total);
  h.tileW = shape.tileW;
  h.flagsUnion = flagsUnion;
  std::memcpy(out, &h, sizeof(h));
  if (total_items) *total_items = uint32_t(total);
  return MT_OK;
}

// The pixels of a job table, claimed by the lanes of a persistent grid.
// queue[0] is the next work item; items are warp tiles (tileW x 32/tileW
// pixels) laid out job after job (JobData.firstItem / .items), or, where the
// table has few for the grid (kSpread), slices of them: then some warps of a
// block ask, with as many lanes as a slice has pixels.  A warp takes `grain`
// consecutive items per atomic and hands their pixels to its lanes as they ask.
// A warp is done when the counter passes the item total; its fetch bound only
// guards against a corrupted table, and running out of it sets
// kBatchStatusGuardExhausted in `status` (when given).
struct TableClaims {
  const BatchHeader *header;
  const JobData *jobs;
  uint32_t *queue;
  uint32_t *status;
  uint32_t grain;
  uint32_t slice = 32u;          // pixels of an item, a power of two
  uint64_t cursor = 0, end = 0;  // units (pixels of the items taken) left
  uint32_t fetches = 0;
  bool exhausted = false;

  MTD TableClaims(const BatchHeader *h, uint32_t *q, uint32_t *st, uint32_t g, bool spread)
      : header(h), jobs(reinterpret_cast<const JobData *>(reinterpret_cast<const char *>(h) + kBatchTableOffset)),
        queue(q), status(st), grain(g) {
    const uint64_t perBlock = (uint64_t(h->totalItems) * 32u + gridDim.x - 1u) / gridDim.x;
    if (!spread || perBlock > blockDim.x) return;
    // As many warps of each block as it has work for: the blocks that start first
    // would take all of it.
    const bool few = perBlock <= kSpreadWarps * 32u;
    const uint32_t warps = few ? min(min(kSpreadWarps, blockDim.x / 32u), uint32_t(perBlock))
                               : (uint32_t(perBlock) + 31u) / 32u;
    exhausted = threadIdx.x / 32u >= warps;
    if (!few) return;
    while (slice / 2u * warps >= perBlock && slice > 1u) slice /= 2u;
  }

  MTD void next(bool wants, const JobData *&job, uint32_t &x, uint32_t &y, uint32_t &samples) {
    const uint32_t lane = threadIdx.x & 31u, total = header->totalItems * (32u / slice), tileW = header->tileW;
    wants = wants && lane < slice;
    unsigned asking = __ballot_sync(0xffffffffu, wants);
    while (asking && !exhausted) {
      if (cursor == end) {
        uint32_t first = 0;
        if (lane == 0) first = atomicAdd(queue, grain);
        first = __shfl_sync(0xffffffffu, first, 0);
        if (first >= total || fetches++ > total) {
          if (first < total && status && lane == 0) atomicOr(status, kBatchStatusGuardExhausted);
          exhausted = true;
          break;
        }
        cursor = uint64_t(first) * slice;
        end = uint64_t(min(first + grain, total)) * slice;
      }
      const uint64_t u = cursor + __popc(asking & ((1u << lane) - 1u));
      cursor = min(end, cursor + uint64_t(__popc(asking)));
      if (wants && u < end) {
        const uint32_t item = uint32_t(u / 32u), in = uint32_t(u % 32u);
        // The job owning the item: firstItem ascends.
        uint32_t lo = 0, hi = header->jobCount;
        while (hi - lo > 1u) {
          const uint32_t mid = (lo + hi) / 2u;
          if (jobs[mid].firstItem <= item) lo = mid; else hi = mid;
        }
        const JobData &J = jobs[lo];
        const uint32_t local = item - J.firstItem;
        x = (local % J.tilesX) * tileW + in % tileW;
        y = (local / J.tilesX) * (32u / tileW) + in / tileW;
        if (x < J.width && y < J.height && J.samples) {
          job = &J;
          samples = J.samples;
          wants = false;
        }
      }
      __syncwarp();
      asking = __ballot_sync(0xffffffffu, wants);
    }
  }
};

// The persistent work loop of the batched kernels.
template <bool kGpuLayout, bool kSpread>
__device__ __forceinline__ void batchWorkLoop(const BatchHeader *__restrict__ header, uint32_t *queue, uint32_t grain,
                                              uint32_t *status, Counters &cnt, uint32_t &paths) {
  TableClaims claims(header, queue, status, grain, kSpread);
  tracePixels<kGpuLayout>(claims, cnt, paths);
}

}  // namespace mt
