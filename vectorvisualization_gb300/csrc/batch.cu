// Batched rendering: jobs launched one by one over eight streams or, small ones, in one persistent launch
// (job table, job-major (job, tile) order, CUDA-graph-captured launch sequence); the tile-shape /
// sampler autotuner.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "../../include/vvlic.h"
#include "vvlic_device.cuh"
#include "vvlic_host.hpp"
#include "vvlic_launch.hpp"

using namespace vvlic;

namespace vvlic_batch_order {

__device__ __forceinline__ int job_of(const unsigned* start, int njobs, unsigned g) {
  int lo = 0, hi = njobs - 1;  // largest j with start[j] <= g
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (start[mid] <= g) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Item g of the batch: job j = the job whose tiles contain g, tile g - start[j].  Jobs run in
// submission order and each job's tiles in raster order, so the warps in flight work on one or
// two volumes at a time and share their texels in L1 and L2.  Measured on the 64-volume batch
// (297 views at 512^2): 1065 ms per batch against 1252 ms for a longest-first order over all
// (job, tile) items, which spreads the warps in flight over every volume; the tail this order
// leaves is at most one job's last tiles.
__global__ void batch_order_kernel(const unsigned* start, int njobs, int ntiles, uint2* order) {
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < ntiles; g += gridDim.x * blockDim.x) {
    const int j = job_of(start, njobs, (unsigned)g);
    order[g] = make_uint2((unsigned)j, (unsigned)g - start[j]);
  }
}

}  // namespace vvlic_batch_order

namespace vvlic {

cudaError_t launch_batch_order(const BatchScratch& b, int njobs, int ntiles, cudaStream_t s) {
  using namespace vvlic_batch_order;
  batch_order_kernel<<<std::max(1, std::min((ntiles + 255) / 256, 152 * 8)), 256, 0, s>>>(b.start, njobs, ntiles,
                                                                                          b.order);
  return cudaGetLastError();
}

}  // namespace vvlic

namespace {

vvlic_status grow_device(vvlic_ctx* c, void** p, size_t* cap, size_t bytes, const char* what) {
  if (*cap >= bytes) return VVLIC_OK;
  if (*p) cudaFree(*p);
  *p = nullptr;
  *cap = 0;
  cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaSuccess) return cuda_fail(c, e, what);
  *cap = bytes;
  return VVLIC_OK;
}

void drop_graph(vvlic_ctx* c) {
  if (c->batch_graph) cudaGraphExecDestroy(c->batch_graph);
  c->batch_graph = nullptr;
  std::memset(c->batch_key, 0, sizeof c->batch_key);
}

cudaError_t launch_batch(int storage, const BatchLaunch& b, int sampler, int integ, bool grad, cudaStream_t s) {
  switch (kernel_storage(storage, sampler)) {
    case VVLIC_STORAGE_F32: return launch_batch_f32(b, sampler, integ, grad, s);
    case VVLIC_STORAGE_F16: return launch_batch_f16(b, sampler, integ, grad, s);
    case VVLIC_STORAGE_UNORM8: return launch_batch_u8(b, sampler, integ, grad, s);
    default: return launch_batch_bf16(b, sampler, integ, grad, s);
  }
}

// Validates the jobs, builds their argument blocks into the pinned staging table and the
// per-job tile starts; returns the batch-wide variant and the tile count.
vvlic_status prepare_batch(vvlic_ctx* c, const vvlic_job* jobs, int n, int tw, int sampler_override, cudaStream_t s,
                           int* storage, int* sampler, int* integ, bool* grad, int* ntiles,
                           std::vector<unsigned>& start) {
  if (!jobs || n < 1 || n > 65536) return fail(c, VVLIC_ERR_INVALID_ARGUMENT, "batch: need 1..65536 jobs");
  // the staging table may still be in flight from the previous batch
  if (c->ev_jobs) cudaEventSynchronize(c->ev_jobs);
  const size_t table = (size_t)n * sizeof(RenderArgs);
  if (c->h_jobs_cap < table) {
    if (c->h_jobs) cudaFreeHost(c->h_jobs);
    c->h_jobs = nullptr;
    c->h_jobs_cap = 0;
    cudaError_t e = cudaHostAlloc((void**)&c->h_jobs, table, cudaHostAllocDefault);
    if (e != cudaSuccess) return cuda_fail(c, e, "batch staging allocation");
    c->h_jobs_cap = table;
  }
  start.assign(n + 1, 0);
  double total = 0.0;
  for (int j = 0; j < n; ++j) {
    const vvlic_job& jb = jobs[j];
    auto it = c->vols.find(jb.vol_id);
    if (it == c->vols.end()) return fail(c, VVLIC_ERR_INVALID_ARGUMENT, "batch: job %d: unknown volume %d", j, jb.vol_id);
    if (!jb.d_out || jb.w < 1 || jb.h < 1 || jb.w > 32768 || jb.h > 32768)
      return fail(c, VVLIC_ERR_INVALID_ARGUMENT, "batch: job %d: bad image", j);
    vvlic_params p = jb.params;
    if (sampler_override >= 0) p.sampler = sampler_override;
    if (p.sampler == VVLIC_SAMPLER_BRICK)
      return fail(c, VVLIC_ERR_UNSUPPORTED, "batch: job %d: the BRICK sampler renders single images only", j);
    p.record_tape = 0;
    const vvlic_params& p0 = jobs[0].params;
    const int smp0 = sampler_override >= 0 ? sampler_override : p0.sampler;
    if (it->second.storage != c->vols[jobs[0].vol_id].storage || p.sampler != smp0 || p.integrator != p0.integrator ||
        (p.illum == VVLIC_ILLUM_GRADIENT) != (p0.illum == VVLIC_ILLUM_GRADIENT))
      return fail(c, VVLIC_ERR_INVALID_ARGUMENT,
                  "batch: job %d differs from job 0 in field storage, sampler, integrator or lighting", j);
    if (jb.view.projection != VVLIC_PERSPECTIVE && jb.view.projection != VVLIC_ORTHOGRAPHIC)
      return fail(c, VVLIC_ERR_INVALID_ARGUMENT, "batch: job %d: projection", j);
    JobFilter jf;
    uint8_t tab[1024];
    if (jb.filter_table) {
      if (jb.filter_width < 1 || jb.filter_width > 1024)
        return fail(c, VVLIC_ERR_INVALID_ARGUMENT, "batch: job %d: filter width", j);
      jf.width = centre_filter_table(jb.filter_table, jb.filter_width, tab, &jf.is_box);
      jf.table = tab;
      jf.clamp = jb.filter_clamp;
    }
    vvlic_status st = build_render_args_ex(c, it->second, jb.w, jb.h, s, p, jb.view, jb.filter_table ? &jf : nullptr,
                                           c->h_jobs[j]);
    if (st) return st;
    RenderArgs& a = c->h_jobs[j];
    a.out = jb.d_out;
    a.counters = c->d_counters;
    const int th = 32 / tw;
    const double tiles = (double)((jb.w + tw - 1) / tw) * (double)((jb.h + th - 1) / th);
    start[j] = (unsigned)total;
    total += tiles;
    if (total > 4.0e9) return fail(c, VVLIC_ERR_INVALID_ARGUMENT, "batch: too many tiles");
  }
  start[n] = (unsigned)total;
  *ntiles = (int)total;
  *storage = c->vols[jobs[0].vol_id].storage;
  *sampler = sampler_override >= 0 ? sampler_override : jobs[0].params.sampler;
  *integ = jobs[0].params.integrator;
  *grad = jobs[0].params.illum == VVLIC_ILLUM_GRADIENT;
  return VVLIC_OK;
}

// Jobs of some size are launched one by one, dealt to the caller's stream and seven of the context's so
// that one job's tail runs beside the next ones' starts.  A kernel of its own reads its arguments
// from the constant bank, as operands; the persistent kernel has to hold them in shared memory and loads
// them again and again through the pipe that also serves the noise cells.  24 views of 8 uneven
// volumes, one by one / persistent: 86.5 / 105.6 ms at 512^2 (lit 136 / 223), 26.5 / 37.1 at 256^2, 3.2 /
// 12.7 at 64^2; 320 views at 32^2 14.9 / 21.9 ms, 800 at 16^2 27.6 / 13.6 (launches).  The line lies at a mean
// of a sixteenth of the resident warps in 2x2-ray tiles, 30^2 pixels.  The context's streams have the priority
// of the caller's.
//
// Rays of a few samples leave most lanes of a group idle and frames of them too short for a launch each.
// Batches of them (`samples` a ray, on average) run in the persistent launch up to the size from which
// single frames of such rays take a lane to a ray (head_samples), and there a lane to a ray (lane_per_ray).  All
// opaque, one by one / persistent in groups / a lane to a ray (ms): 320 views at 32^2 1.14 / 0.32 / 0.11, 64 at 64^2
// 0.63 / 0.23 / 0.08, 64 at 128^2 1.08 / 0.69 / 0.20, 24 at 256^2 0.28 / 0.95 / 0.26, 800 at 16^2 - / 0.26 / 0.11.
// Opaque for half of the alphas, where half of the rays go on: 320 at 32^2 1.51 / 0.61 / 0.75, 64 at 128^2 1.15 / 1.27
// / 0.87.
bool job_by_job(const vvlic_ctx* c, const vvlic_job* jobs, int n, double samples) {
  double tiles = 0.0;
  for (int j = 0; j < n; ++j) tiles += (double)((jobs[j].w + 1) / 2) * (double)((jobs[j].h + 1) / 2);
  const double resident = 24.0 * c->num_sms, mean = tiles / n;
  return mean >= resident / 16.0 && !(samples <= 4.0 && mean < 2.0 * resident);
}

// Samples of an average ray of the prepared jobs, taken as two where half of all samples would end it.
double expected_samples(const vvlic_ctx* c, int n) {
  double sum = 0.0;
  for (int j = 0; j < n; ++j) {
    const RenderArgs& a = c->h_jobs[j];
    sum += std::min(a.mean_samples, a.end_share >= 0.5f ? 2.0f : 64.0f);
  }
  return sum / n;
}

vvlic_status launch_jobs(vvlic_ctx* c, int n, int storage, int sampler, int integ, bool grad, cudaStream_t s) {
  constexpr int B = vvlic_ctx::kBatchStreams;
  int priority = 0;
  cudaError_t e = cudaStreamGetPriority(s, &priority);
  if (e != cudaSuccess) return cuda_fail(c, e, "batch stream");
  auto& side = c->batch_streams[priority];  // value-initialised when new
  for (int b = 0; b < B && e == cudaSuccess; ++b) {
    if (!side[b]) e = cudaStreamCreateWithPriority(&side[b], cudaStreamNonBlocking, priority);
    if (e == cudaSuccess && !c->ev_batch_join[b]) e = cudaEventCreateWithFlags(&c->ev_batch_join[b], cudaEventDisableTiming);
  }
  if (e == cudaSuccess && !c->ev_batch_fork) e = cudaEventCreateWithFlags(&c->ev_batch_fork, cudaEventDisableTiming);
  if (e != cudaSuccess) return cuda_fail(c, e, "batch streams");
  const int used = std::min(n - 1, B);
  e = cudaMemsetAsync(c->d_counters, 0, 4 * sizeof(unsigned long long), s);
  if (e == cudaSuccess) e = cudaEventRecord(c->ev0, s);
  if (e == cudaSuccess) e = cudaEventRecord(c->ev_batch_fork, s);
  for (int b = 0; b < used && e == cudaSuccess; ++b) e = cudaStreamWaitEvent(side[b], c->ev_batch_fork, 0);
  for (int j = 0; j < n && e == cudaSuccess; ++j) {
    RenderArgs& a = c->h_jobs[j];
    a.count_steps = 1;
    const int b = j % (used + 1);
    e = launch_raycast(a, storage, sampler, integ, grad, c->num_sms, b == 0 ? s : side[b - 1]);
  }
  // joined even after a failed launch: nothing on the side streams outlives the caller's stream
  for (int b = 0; b < used; ++b) {
    cudaError_t ej = cudaEventRecord(c->ev_batch_join[b], side[b]);
    if (ej == cudaSuccess) ej = cudaStreamWaitEvent(s, c->ev_batch_join[b], 0);
    if (e == cudaSuccess) e = ej;
  }
  if (e == cudaSuccess) e = cudaEventRecord(c->ev1, s);
  if (e != cudaSuccess) return cuda_fail(c, e, "batch launch");
  return VVLIC_OK;
}

vvlic_status batch_render(vvlic_ctx* c, const vvlic_job* jobs, int n, cudaStream_t s, int tw, int sampler_override) {
  int storage, sampler, integ, ntiles;
  bool grad;
  std::vector<unsigned> start;
  // A stream that the caller is capturing is refused before anything is allocated or launched: a layout filled
  // into the caller's graph would count as filled, and the job table would be read at the graph's launch.
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusActive;
  if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone)
    return cuda_fail(c, cudaErrorStreamCaptureUnsupported, "batch on a stream that is being captured");
  if (s == cudaStreamLegacy)  // which the persistent path cannot capture: refused whatever the jobs' sizes
    return cuda_fail(c, cudaErrorStreamCaptureUnsupported, "batch on the legacy default stream");
  vvlic_status st = prepare_batch(c, jobs, n, tw, sampler_override, s, &storage, &sampler, &integ, &grad, &ntiles,
                                  start);
  if (st) return st;
  const double samples = expected_samples(c, n);
  const bool lane_per_ray = samples <= 8.0;
  c->batch_by_job = job_by_job(c, jobs, n, samples);
  if (c->batch_by_job) {
    if ((st = launch_jobs(c, n, storage, sampler, integ, grad, s))) return st;
    c->stats_pending = true;
    c->tape_flag_pending = false;
    c->last_was_batch = true;
    c->tape_valid = false;
    return VVLIC_OK;
  }
  // device buffers; a reallocation invalidates the captured graph
  const void* old_jobs = c->d_jobs;
  const void* old_batch = c->d_batch;
  if ((st = grow_device(c, (void**)&c->d_jobs, &c->d_jobs_cap, (size_t)n * sizeof(RenderArgs), "batch job table")))
    return st;
  const size_t words = batch_scratch(nullptr, n, ntiles).words;
  size_t cap_bytes = c->batch_cap * sizeof(unsigned);
  if ((st = grow_device(c, (void**)&c->d_batch, &cap_bytes, words * sizeof(unsigned), "batch scratch"))) return st;
  c->batch_cap = cap_bytes / sizeof(unsigned);
  if (old_jobs != c->d_jobs || old_batch != c->d_batch) drop_graph(c);
  const BatchScratch bs = batch_scratch(c->d_batch, n, ntiles);
  unsigned* d_start = bs.start;
  // upload the job table and tile starts (outside the graph)
  cudaError_t e = cudaMemcpyAsync(c->d_jobs, c->h_jobs, (size_t)n * sizeof(RenderArgs), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(d_start, start.data(), (n + 1) * sizeof(unsigned), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) {
    if (!c->ev_jobs) e = cudaEventCreateWithFlags(&c->ev_jobs, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventRecord(c->ev_jobs, s);
  }
  if (e != cudaSuccess) return cuda_fail(c, e, "batch upload");
  const uint64_t key[8] = {(uint64_t)n, (uint64_t)ntiles, (uint64_t)storage, (uint64_t)sampler, (uint64_t)integ,
                           (uint64_t)grad, (uint64_t)tw, (uint64_t)lane_per_ray};
  if (!c->batch_graph || std::memcmp(key, c->batch_key, sizeof key) != 0) {
    drop_graph(c);
    // capture: counters reset, order pass, queue reset, the persistent launch
    cudaGraph_t graph = nullptr;
    e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return cuda_fail(c, e, "batch graph capture (a non-default stream is required)");
    cudaError_t ec = cudaMemsetAsync(c->d_counters, 0, 4 * sizeof(unsigned long long), s);
    if (ec == cudaSuccess) ec = launch_batch_order(bs, n, ntiles, s);
    if (ec == cudaSuccess) ec = cudaMemsetAsync(bs.next, 0, sizeof(unsigned), s);
    if (ec == cudaSuccess) {
      BatchLaunch b{c->d_jobs, bs.order, ntiles, bs.next, c->d_tf, c->d_counters, tw, c->num_sms, lane_per_ray};
      ec = launch_batch(storage, b, sampler, integ, grad, s);
    }
    e = cudaStreamEndCapture(s, &graph);
    if (ec != cudaSuccess || e != cudaSuccess) {
      if (graph) cudaGraphDestroy(graph);
      return cuda_fail(c, ec != cudaSuccess ? ec : e, "batch graph capture");
    }
    e = cudaGraphInstantiate(&c->batch_graph, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) {
      c->batch_graph = nullptr;
      return cuda_fail(c, e, "batch graph instantiate");
    }
    std::memcpy(c->batch_key, key, sizeof key);
  }
  e = cudaEventRecord(c->ev0, s);
  if (e == cudaSuccess) e = cudaGraphLaunch(c->batch_graph, s);
  if (e == cudaSuccess) e = cudaEventRecord(c->ev1, s);
  if (e != cudaSuccess) return cuda_fail(c, e, "batch launch");
  c->stats_pending = true;
  c->tape_flag_pending = false;
  c->last_was_batch = true;
  c->tape_valid = false;
  return VVLIC_OK;
}

}  // namespace

extern "C" vvlic_status vvlic_batch_render(vvlic_ctx* c, const vvlic_job* jobs, int32_t n, void* stream) {
  if (!c) return VVLIC_ERR_BAD_HANDLE;
  DeviceGuard g(c->device);
  cudaStream_t s = stream ? (cudaStream_t)stream : c->stream;
  return batch_render(c, jobs, n, s, c->batch_tile_w, c->batch_sampler_override);
}

extern "C" vvlic_status vvlic_batch_autotune(vvlic_ctx* c, const vvlic_job* jobs, int32_t n, void* stream,
                                            int32_t* best_tile_w, int32_t* best_sampler, float* best_ms) {
  if (!c) return VVLIC_ERR_BAD_HANDLE;
  if (!jobs || n < 1) return fail(c, VVLIC_ERR_INVALID_ARGUMENT, "batch_autotune: no jobs");
  DeviceGuard g(c->device);
  cudaStream_t s = stream ? (cudaStream_t)stream : c->stream;
  auto it = c->vols.find(jobs[0].vol_id);
  if (it == c->vols.end()) return fail(c, VVLIC_ERR_INVALID_ARGUMENT, "batch_autotune: unknown volume");
  std::vector<int> samplers = {VVLIC_SAMPLER_HYBRID, VVLIC_SAMPLER_CELL};
  const int tws[4] = {8, 4, 16, 32};
  float best = 1e30f;
  int bt = c->batch_tile_w, bs = jobs[0].params.sampler;
  bool shaped = true;  // launched one by one, the jobs have no tile shape
  for (int smp : samplers) {
    for (int tw : tws) {
      if (!shaped && tw != tws[0]) continue;
      float ms = 0.f;
      for (int rep = 0; rep < 2; ++rep) {  // the first render builds layouts and the graph
        vvlic_status st = batch_render(c, jobs, n, s, tw, smp);
        if (st) return st;
        shaped = !c->batch_by_job;
        cudaError_t e = cudaEventSynchronize(c->ev1);
        if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, c->ev0, c->ev1);
        if (e != cudaSuccess) return cuda_fail(c, e, "batch_autotune");
      }
      if (ms < best) {
        best = ms;
        bt = tw;
        bs = smp;
      }
    }
  }
  if (shaped) c->batch_tile_w = bt;  // otherwise an earlier tuning of small jobs stands
  c->batch_sampler_override = bs;
  drop_graph(c);
  if (best_tile_w) *best_tile_w = bt;
  if (best_sampler) *best_sampler = bs;
  if (best_ms) *best_ms = best;
  return VVLIC_OK;
}
