// Batched wavefront path tracing: many render jobs per launch.
//
// The jobs' sample ranges are concatenated into one work list, which runs in
// one of two ways. Wave mode takes a wave of contiguous work items onto slots
// 0..n-1 and runs the plain render's pipeline on them, each path against its
// job's scene (k_wb_camera, then k_b_trace, k_b_resolve, k_wb_compact, k_b_shade
// per bounce, then k_wb_film). Pooled mode shares one pool of slots among all jobs and
// refills finished slots every iteration of a loop inside a CUDA graph
// while-node:
//
//   k_b_plan     take = min(free slots, work left); reset this iteration's queues
//   k_b_regen    start `take` new camera paths in free slots
//   k_b_trace    closest hit for every live path (each against its job's scene)
//   k_b_shade    one bounce of PathTracing::Li per path (shared shade_one)
//   k_b_trace    shadow rays (any hit) and MIS rays
//   k_b_resolve  direct-light estimate into the path radiance
//   k_b_retire   finished paths' radiance into the job's FP64 film, slot freed
//   k_b_control  flip queues; keep looping while work or live paths remain
//
// Paths of different jobs and depths share every launch. Each path runs the
// plain path's device functions on the same samples; the film's order of
// accumulation differs (FP64 atomics).
#include <cuda_runtime.h>

#include "kernels.h"
#include "shade.cuh"

namespace orion_gb300 {

namespace {

__global__ void k_b_init(BatchView b, int capacity) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < capacity; i += gridDim.x * blockDim.x) b.q_free[i] = i;
}

__global__ void k_b_plan(BatchView b) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  BatchCtl& c = *b.ctl;
  unsigned long long rem = c.total - c.cursor;
  int nfree = c.counters[CNT_FREE];
  int take = (unsigned long long)nfree < rem ? nfree : (int)rem;
  c.take = take;
  c.take_base = c.cursor;
  c.cursor += (unsigned long long)take;
  c.counters[CNT_FREE] = nfree - take;
  c.counters[CNT_NEE] = c.counters[CNT_NEE + 1] = 0;
  c.counters[CNT_RETIRE] = 0;
  c.counters[cnt_rays(RK_EXT, c.cur ^ 1)] = 0;
  for (int k = 1; k < kRayKinds; ++k) c.counters[cnt_rays(k, 0)] = c.counters[cnt_rays(k, 1)] = 0;
  for (int k = 0; k < kRayKinds; ++k) c.counters[CNT_FETCH + k] = 0;
  for (int k = 0; k < kShadeClasses; ++k) c.counters[cnt_cls(k, c.cur)] = 0;
}

__device__ __forceinline__ int job_of_work(const DevJob* jobs, int njobs, unsigned long long work) {
  int lo = 0, hi = njobs - 1;
  while (lo < hi) {  // last job with work_begin <= work
    int mid = (lo + hi + 1) >> 1;
    if ((unsigned long long)jobs[mid].work_begin <= work)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

__global__ void k_b_regen(WaveView w, BatchView b, const uint32_t* sobol) {
  BatchCtl& c = *b.ctl;
  const int take = c.take;
  const int free_after = c.counters[CNT_FREE];
  const int cur = c.cur;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < take; i += gridDim.x * blockDim.x) {
    const int slot = b.q_free[free_after + i];
    const unsigned long long work = c.take_base + (unsigned long long)i;
    const int job = job_of_work(b.jobs, c.njobs, work);
    const DevJob& J = b.jobs[job];
    const long long index = J.first_index + (long long)(work - (unsigned long long)J.work_begin);
    const long long wh = (long long)J.width * J.height;
    const long long pix = index % wh;
    PathSampler smp{sobol, (uint64_t)index, 5u};
    V3 o, d;
    camera_ray(J.scene.cam, smp, (int)(pix % J.width), (int)(pix / J.width), &o, &d);
    // The whole 96-byte record in one go: three full sectors at a scattered slot.
    PathRec r;
    r.o = f4(o, 0.f);
    r.d = f4(d, 0.f);
    r.beta = make_float4(1.f, 1.f, 1.f, 0.f);
    r.L = make_float4(0.f, 0.f, 0.f, __uint_as_float((uint32_t)(unsigned long long)index));
    r.hit = make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
    r.meta = make_int4((int)smp.dim, job, 0, (int)((unsigned long long)index >> 32));
    w.rec[slot] = r;
    queue_append(&c.counters[cnt_rays(RK_EXT, cur)], w.q_ext[cur], slot, true);
  }
}

// Rays of the kinds in `kinds` (trace_kinds). parity: that of the queues to
// trace; pooled mode, whose current parity only the device knows inside a
// graph: kCurrent, or kNext for the rays that this iteration's shading sent out.
constexpr int kCurrent = 2, kNext = 3;

struct BTraceArgs {
  RaySet set[2][kRayKinds];  // [parity][RayKind]
  BatchView b;
  RecI job;
  int kinds, parity;
  int refill_closest, refill_any;
};

template <int SMEM>
__global__ void __launch_bounds__(512, 2) k_b_trace(const __grid_constant__ BTraceArgs a) {
  extern __shared__ int2 stack_smem[];
  BatchCtl& c = *a.b.ctl;
  const int cur = a.parity == kCurrent ? c.cur : a.parity == kNext ? c.cur ^ 1 : a.parity;
  trace_kinds<SMEM, false, kMaxStack>(JobScene{a.b.jobs, a.job}, a.set[cur], a.kinds, c.counters, cur, stack_smem,
                                      a.refill_closest, a.refill_any, &c.error);
}

// Shading of the slots whose extension ray hit a material of class SC (or
// missed, SC_MISS), each against its job's scene.
// Waves (parity 0 or 1): paths are never retired one by one; the queues they go
// to are marked in the slots' qflags bytes (`marks`, for a compaction) or
// appended to. As in plain renders the classes' launches overlap (k_shade). One
// kernel serves both modes so that a path's arithmetic is compiled once.
template <int SC>
__global__ void __launch_bounds__(shade_threads(SC), kShadeThreadsPerSm / shade_threads(SC))
    k_b_shade(WaveView w, BatchView b, const uint32_t* sobol, int parity, int marks) {
  asm volatile("griddepcontrol.launch_dependents;");
  BatchCtl& c = *b.ctl;
  const bool waves = parity != kCurrent;
  const int cur = waves ? parity : c.cur;
  const int n = c.counters[cnt_cls(SC, cur)];
  const int* in_q = w.q_cls + (size_t)SC * w.capacity;
  for (int q0 = blockIdx.x * blockDim.x; q0 < n; q0 += gridDim.x * blockDim.x) {
    const int q = q0 + threadIdx.x;
    __syncthreads();  // the block's warps go through the code together
    if (q >= n) continue;
    const int pid = in_q[q];
    const int4 meta = w.rec[pid].meta;
    const DevJob& J = b.jobs[meta.y];
    const int bounce = meta.z;
    ShadeResult r = shade_one<lobes_of_class(SC), SC == SC_TEXTURED>(
        J.scene, w, sobol, pid, (uint64_t)slot_index(w, pid), meta.x, bounce, J.max_depth, J.rr_depth);
    if (r.alive) w.bounce[pid] = bounce + 1;
    if (marks) {
      w.qflags[pid] = (uint8_t)((r.alive ? kQfExt : 0) | (r.did_nee ? kQfNee : 0) | (r.want_sh ? kQfShadow : 0) |
                                (r.want_mis ? kQfMis : 0) | (r.want_mis_env ? kQfMisEnv : 0));
      continue;
    }
    queue_append(&c.counters[CNT_NEE + (cur ^ 1)], w.q_nee, pid, r.did_nee);
    queue_append(&c.counters[cnt_rays(RK_SHADOW, cur ^ 1)], w.q_sh, pid, r.want_sh);
    queue_append(&c.counters[cnt_rays(RK_MIS, cur ^ 1)], w.q_mis, pid, r.want_mis);
    queue_append(&c.counters[cnt_rays(RK_MIS_ENV, cur ^ 1)], w.q_mis_env, pid, r.want_mis_env);
    queue_append(&c.counters[cnt_rays(RK_EXT, cur ^ 1)], w.q_ext[cur ^ 1], pid, r.alive);
    if (!waves) queue_append(&c.counters[CNT_RETIRE], b.q_retire, pid, !r.alive);
  }
  if (waves) {
    if (blockIdx.x == 0 && threadIdx.x < kRayKinds) c.counters[CNT_FETCH + threadIdx.x] = 0;  // for the next trace
    if (blockIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
  }
}

// parity: that of the paths to resolve, or kNext (pooled mode).
__global__ void k_b_resolve(WaveView w, BatchView b, int parity) {
  const int n = b.ctl->counters[CNT_NEE + (parity == kNext ? b.ctl->cur ^ 1 : parity)];
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    const int pid = w.q_nee[q];
    resolve_one(b.jobs[w.job[pid]].scene, w, pid);
  }
}

__global__ void k_b_retire(WaveView w, BatchView b) {
  BatchCtl& c = *b.ctl;
  const int n = c.counters[CNT_RETIRE];
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    const int pid = b.q_retire[q];
    const float4 l = w.L[pid];
    const int4 meta = w.rec[pid].meta;
    const DevJob& J = b.jobs[meta.y];
    const long long index =
        (long long)(((unsigned long long)(unsigned)meta.w << 32) | (unsigned long long)__float_as_uint(l.w));
    const long long pix = index % ((long long)J.width * J.height);
    atomicAdd(&J.sum[3 * pix], (double)l.x);
    atomicAdd(&J.sum[3 * pix + 1], (double)l.y);
    atomicAdd(&J.sum[3 * pix + 2], (double)l.z);
    if (J.sumsq) {
      atomicAdd(&J.sumsq[3 * pix], (double)l.x * l.x);
      atomicAdd(&J.sumsq[3 * pix + 1], (double)l.y * l.y);
      atomicAdd(&J.sumsq[3 * pix + 2], (double)l.z * l.z);
    }
    if (J.count) atomicAdd(&J.count[pix], 1u);  // null: the caller knows every pixel gets spp samples
    queue_append(&c.counters[CNT_FREE], b.q_free, pid, true);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&c.paths_done, (unsigned long long)n);
}

// ------------------------------------------------------------ wave mode
//
// A batch can also run as waves over its concatenated work list: wave k
// takes work items [base, base + n) onto slots 0..n-1 in order, its paths
// bounce until none is alive (no refills), and the radiance of all n paths
// goes to the jobs' films at the end. A job's work items run pixel after
// pixel in tile order, each pixel's passes in order, so neighbouring slots
// hold neighbouring paths, as in plain waves, whose pipeline (fused trace,
// overlapping shading classes) this is, with a launch that adds the light
// samples once their rays are traced.

// Work item `work`: its job, and the pixel and pass within the job.
struct WorkItem {
  int job, pass;
  long long pixel;  // in tile order
};

__device__ __forceinline__ WorkItem work_item(const DevJob* jobs, int njobs, unsigned long long work) {
  WorkItem it;
  it.job = job_of_work(jobs, njobs, work);
  const DevJob& J = jobs[it.job];
  const long long k = (long long)(work - (unsigned long long)J.work_begin);
  it.pixel = k >> 32 ? k / J.spp : (long long)((uint32_t)k / (uint32_t)J.spp);
  it.pass = (int)(k - it.pixel * J.spp);
  return it;
}

__global__ void k_wb_camera(WaveView w, BatchView b, const uint32_t* sobol, unsigned long long base, int n) {
  BatchCtl& c = *b.ctl;
  if (blockIdx.x == 0 && threadIdx.x < kCounterSlots)
    c.counters[threadIdx.x] = threadIdx.x == cnt_rays(RK_EXT, 0) ? n : 0;
  const int njobs = c.njobs;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const WorkItem it = work_item(b.jobs, njobs, base + (unsigned long long)i);
    const DevJob& J = b.jobs[it.job];
    int px, py;
    tile_pixel(it.pixel, J.width, J.height, &px, &py);
    const long long wh = (long long)J.width * J.height;
    const long long index = J.first_index + it.pass * wh + (long long)py * J.width + px;
    V3 o, d;
    const uint32_t dim = camera_ray_block(J.scene.cam, sobol, (uint64_t)index, px, py, &o, &d);
    PathRec& r = w.rec[i];
    r.o = f4(o, 0.f);
    r.d = f4(d, 0.f);
    r.beta = make_float4(1.f, 1.f, 1.f, 0.f);
    r.L = make_float4(0.f, 0.f, 0.f, __uint_as_float((uint32_t)(unsigned long long)index));
    r.hit = make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
    r.meta = make_int4((int)dim, it.job, 0, (int)((unsigned long long)index >> 32));
  }
}

template <int NQ>
__global__ void __launch_bounds__(kCompactThreads) k_wb_compact(uint8_t* flags, const int* list, const int* count,
                                                                CompactTargets tg) {
  compact_queues<NQ>(flags, list, count, tg);
}

// The wave's radiance into the jobs' films. A block takes 256 slots at a time
// into shared memory; slots of one pixel are neighbours, a run, and a run ends
// in one FP64 atomic per channel (a pixel's samples may go on in the next 256
// slots or another wave). The FP64 unit is its busiest (64% of peak; 2 lanes a clock
// and SM, and a warp holds it as long for one lane as for 32): a run's samples are added in
// pieces of up to kWbPiece slots, one thread per piece and channel, then the
// pieces of a run by one thread, so that the lanes are full whatever the
// samples per pixel. Film stage of a batch, one thread per run / pieces: 33.5M
// paths at 256 spp 3.95 / 1.20 ms, 229M at 64 spp 10.8 / 8.7, 18.9M at 16 spp
// 0.47 / 0.47 (an atomic per path, pass after pass: 1.02, 6.8, 0.56). Pieces of 16:
// 1.35, 8.65, 0.57; loading the next slots early: 1.38, 9.35, 0.51.
// unfinished: -1, or the parity of the extension queue that must be empty.
constexpr int kWbFilmThreads = 256;
constexpr int kWbPiece = 8;
static_assert(kWbPiece > 0 && 32 % kWbPiece == 0, "pieces are cut at multiples within a warp");

__global__ void __launch_bounds__(kWbFilmThreads) k_wb_film(WaveView w, BatchView b, unsigned long long base, int n,
                                                            int unfinished) {
  // A gap after each piece's length, so that threads of different pieces meet in different banks.
  auto at = [](int slot) { return slot + slot / kWbPiece; };
  __shared__ float buf[3][kWbFilmThreads + kWbFilmThreads / kWbPiece + 11];
  __shared__ double piece_sum[3 * kWbFilmThreads], piece_sq[3 * kWbFilmThreads];
  __shared__ int piece_start[kWbFilmThreads + 1];
  __shared__ uint8_t piece_squares[kWbFilmThreads];
  __shared__ int run_piece[kWbFilmThreads + 1];
  __shared__ int warp_counts[kWbFilmThreads / 32];  // pieces, runs << 16
  __shared__ long long run_pix[kWbFilmThreads];
  __shared__ int run_job[kWbFilmThreads];
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  BatchCtl& c = *b.ctl;
  if (blockIdx.x == 0 && t == 0) {
    c.paths_done += (unsigned long long)n;
    if (unfinished >= 0 && c.counters[cnt_rays(RK_EXT, unfinished)] > 0) c.error |= kErrIterationCap;
  }
  const int njobs = c.njobs;
  for (int from = blockIdx.x * kWbFilmThreads; from < n; from += gridDim.x * kWbFilmThreads) {
    const int pid = from + t;
    bool head = false, piece = false;
    WorkItem it{0, 0, 0};
    if (pid < n) {
      it = work_item(b.jobs, njobs, base + (unsigned long long)pid);
      head = t == 0 || it.pass == 0;
      piece = head || t % kWbPiece == 0;
      const float4 l = w.L[pid];
      buf[0][at(t)] = l.x;
      buf[1][at(t)] = l.y;
      buf[2][at(t)] = l.z;
    }
    const unsigned heads = __ballot_sync(0xffffffffu, head), cuts = __ballot_sync(0xffffffffu, piece);
    if (lane == 0) warp_counts[wid] = __popc(cuts) | __popc(heads) << 16;
    __syncthreads();
    int before = 0, all = 0;
#pragma unroll
    for (int k = 0; k < kWbFilmThreads / 32; ++k) {
      if (k < wid) before += warp_counts[k];
      all += warp_counts[k];
    }
    const int pieces = all & 0xffff, runs = all >> 16;
    if (piece) {
      const DevJob& J = b.jobs[it.job];
      const unsigned below = (1u << lane) - 1u;
      const int q = (before & 0xffff) + __popc(cuts & below);
      piece_start[q] = t;
      piece_squares[q] = J.sumsq != nullptr;
      if (head) {
        const int r = (before >> 16) + __popc(heads & below);
        int x, y;
        tile_pixel(it.pixel, J.width, J.height, &x, &y);
        run_piece[r] = q;
        run_job[r] = it.job;
        run_pix[r] = (long long)y * J.width + x;
      }
    }
    if (t == 0) {
      piece_start[pieces] = min(kWbFilmThreads, n - from);
      run_piece[runs] = pieces;
    }
    __syncthreads();
    for (int u = t; u < 3 * pieces; u += kWbFilmThreads) {
      const int q = u / 3;
      const float* v = buf[u - 3 * q];
      const int s1 = piece_start[q + 1];
      double sum = 0, sq = 0;
      if (piece_squares[q]) {
        for (int i = piece_start[q]; i < s1; ++i) {
          const double x = (double)v[at(i)];
          sum += x;
          sq += x * x;
        }
        piece_sq[u] = sq;
      } else {
        for (int i = piece_start[q]; i < s1; ++i) sum += (double)v[at(i)];
      }
      piece_sum[u] = sum;
    }
    __syncthreads();
    for (int u = t; u < 3 * runs; u += kWbFilmThreads) {
      const int r = u / 3, ch = u - 3 * r;
      const DevJob& J = b.jobs[run_job[r]];
      const int q0 = run_piece[r], q1 = run_piece[r + 1];
      double sum = piece_sum[3 * q0 + ch];
      for (int q = q0 + 1; q < q1; ++q) sum += piece_sum[3 * q + ch];
      atomicAdd(&J.sum[3 * run_pix[r] + ch], sum);
      if (J.sumsq) {
        double sq = piece_sq[3 * q0 + ch];
        for (int q = q0 + 1; q < q1; ++q) sq += piece_sq[3 * q + ch];
        atomicAdd(&J.sumsq[3 * run_pix[r] + ch], sq);
      }
      if (J.count && ch == 0) atomicAdd(&J.count[run_pix[r]], (unsigned)(piece_start[q1] - piece_start[q0]));
    }
    __syncthreads();
  }
}

// in_graph: sets the while-node's condition; otherwise leaves the decision in
// ctl->more for a host-driven loop (profiling runs).
__global__ void k_b_control(BatchView b, cudaGraphConditionalHandle cond, int in_graph) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  BatchCtl& c = *b.ctl;
  c.cur ^= 1;
  c.iterations += 1;
  bool more = c.cursor < c.total || c.counters[cnt_rays(RK_EXT, c.cur)] > 0;
  if (more && c.iterations >= c.max_iterations) {
    c.error |= kErrIterationCap;  // bounded loop: report instead of spinning on
    more = false;
  }
  if (in_graph)
    cudaGraphSetConditional(cond, more ? 1u : 0u);
  else
    c.more = more ? 1 : 0;
}

// marks: extension hits mark their slot's shading class in qflags for a
// compaction instead of appending to the class queues.
void b_trace(const LaunchConfig& cfg, const WaveView& bw, const BatchView& b, int kinds, int parity, int grid,
             bool marks, bool camera_rays, cudaStream_t s) {
  BTraceArgs a;
  for (int cur = 0; cur < 2; ++cur) wave_ray_sets(bw, cur, marks, camera_rays, a.set[cur]);
  a.b = b;
  a.job = bw.job;
  a.kinds = kinds;
  a.parity = parity;
  a.refill_closest = cfg.refill_below < 1 ? 1 : (cfg.refill_below > 32 ? 32 : cfg.refill_below);
  a.refill_any = a.refill_closest;  // (the batch loop lost 9-13% of its requests/s at the plain renders' threshold)
  const int block = cfg.trace_block;
  switch (cfg.smem_stack) {
    case 0: k_b_trace<0><<<grid, block, trace_smem_bytes(0, block), s>>>(a); break;
    case 8: k_b_trace<8><<<grid, block, trace_smem_bytes(8, block), s>>>(a); break;
    case 24: k_b_trace<24><<<grid, block, trace_smem_bytes(24, block), s>>>(a); break;
    case 32: k_b_trace<32><<<grid, block, trace_smem_bytes(32, block), s>>>(a); break;
    default: k_b_trace<16><<<grid, block, trace_smem_bytes(16, block), s>>>(a); break;
  }
}

// The wave as the batch's kernels see it: queues and rays are counted in the
// batch's control block.
WaveView batch_view(const WaveView& w, const BatchView& b) {
  WaveView v = w;
  v.counters = b.ctl->counters;
  v.ray_stats = b.ctl->rays;
  v.trace_work = nullptr;
  return v;
}

cudaError_t batch_limit_of(const void* f, int smem_bytes, int* max_block) {
  if (smem_bytes > 0) {
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
    if (e != cudaSuccess) return e;
  }
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, f);
  if (e != cudaSuccess) return e;
  *max_block = *max_block < a.maxThreadsPerBlock ? *max_block : a.maxThreadsPerBlock;
  return cudaSuccess;
}

int grid_cap(int64_t n, int block, int cap) {
  int64_t g = (n + block - 1) / block;
  return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

}  // namespace

cudaError_t configure_batch_kernels(int smem_bytes, KernelLimits* lim) {
  const void* trace[] = {(const void*)k_b_trace<0>, (const void*)k_b_trace<8>, (const void*)k_b_trace<16>,
                         (const void*)k_b_trace<24>, (const void*)k_b_trace<32>};
  const void* shade[] = {(const void*)k_b_shade<SC_DIFFUSE>,    (const void*)k_b_shade<SC_CONDUCTOR>,
                         (const void*)k_b_shade<SC_SPECULAR>,   (const void*)k_b_shade<SC_DIELECTRIC>,
                         (const void*)k_b_shade<SC_PLASTIC>,    (const void*)k_b_shade<SC_GENERAL>,
                         (const void*)k_b_shade<SC_TEXTURED>,
                         (const void*)k_b_shade<SC_MISS>,       (const void*)k_b_resolve,
                         (const void*)k_b_retire};
  for (const void* f : trace) {
    cudaError_t e = batch_limit_of(f, smem_bytes, &lim->max_trace_block);
    if (e != cudaSuccess) return e;
  }
  for (const void* f : shade) {
    cudaError_t e = batch_limit_of(f, 0, &lim->max_shade_block);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

void launch_batch_init(const WaveView& w, const BatchView& b, int capacity, cudaStream_t stream) {
  k_b_init<<<grid_cap(capacity, 256, 4096), 256, 0, stream>>>(b, capacity);
}

namespace {

// One pooled loop iteration's kernels on `stream`, optionally timed per stage.
void enqueue_iteration(const WaveView& w, const BatchView& b, const uint32_t* sobol,
                       const LaunchConfig& cfg, unsigned class_mask, cudaGraphConditionalHandle cond,
                       int in_graph, cudaStream_t stream, StageTimer* timer) {
  const int cap = w.capacity;
  const WaveView bw = batch_view(w, b);
  const int persistent = cfg.num_sms * cfg.blocks_per_sm;
  const int tgrid = grid_cap(cap, cfg.trace_block, persistent);
  const int sgrid = grid_cap(cap, cfg.shade_block, persistent * 2);
  auto begin = [&](int st) {
    if (timer) timer->begin(st, stream);
  };
  auto end = [&]() {
    if (timer) timer->end(stream);
  };
  begin(ST_CAMERA);
  k_b_plan<<<1, 32, 0, stream>>>(b);
  k_b_regen<<<grid_cap(cap, 256, persistent * 4), 256, 0, stream>>>(w, b, sobol);
  end();
  begin(ST_TRACE_EXT);
  b_trace(cfg, bw, b, TK_EXT, kCurrent, tgrid, false, false, stream);
  end();
  begin(ST_SHADE);
  for (int sc = 0; sc < kShadeClasses; ++sc) {
    if (!((class_mask >> sc) & 1u)) continue;
    const ShadeShape shape = shade_shape(sc, cap, cfg);
    switch (sc) {
      case SC_DIFFUSE: k_b_shade<SC_DIFFUSE><<<shape.grid, shape.block, 0, stream>>>(w, b, sobol, kCurrent, 0); break;
      case SC_CONDUCTOR: k_b_shade<SC_CONDUCTOR><<<shape.grid, shape.block, 0, stream>>>(w, b, sobol, kCurrent, 0); break;
      case SC_SPECULAR: k_b_shade<SC_SPECULAR><<<shape.grid, shape.block, 0, stream>>>(w, b, sobol, kCurrent, 0); break;
      case SC_DIELECTRIC: k_b_shade<SC_DIELECTRIC><<<shape.grid, shape.block, 0, stream>>>(w, b, sobol, kCurrent, 0); break;
      case SC_PLASTIC: k_b_shade<SC_PLASTIC><<<shape.grid, shape.block, 0, stream>>>(w, b, sobol, kCurrent, 0); break;
      case SC_GENERAL: k_b_shade<SC_GENERAL><<<shape.grid, shape.block, 0, stream>>>(w, b, sobol, kCurrent, 0); break;
      case SC_TEXTURED: k_b_shade<SC_TEXTURED><<<shape.grid, shape.block, 0, stream>>>(w, b, sobol, kCurrent, 0); break;
      case SC_MISS: k_b_shade<SC_MISS><<<shape.grid, shape.block, 0, stream>>>(w, b, sobol, kCurrent, 0); break;
    }
  }
  end();
  begin(ST_TRACE_SHADOW);
  b_trace(cfg, bw, b, TK_SHADOW, kNext, tgrid, false, false, stream);
  end();
  begin(ST_TRACE_MIS);
  b_trace(cfg, bw, b, TK_MIS | TK_MIS_ENV, kNext, tgrid, false, false, stream);
  end();
  begin(ST_RESOLVE);
  k_b_resolve<<<sgrid, cfg.shade_block, 0, stream>>>(w, b, kNext);
  end();
  begin(ST_FILM);
  k_b_retire<<<sgrid, cfg.shade_block, 0, stream>>>(w, b);
  end();
  begin(ST_OTHER);
  k_b_control<<<1, 32, 0, stream>>>(b, cond, in_graph);
  end();
}

// Shading of one bounce of a batch wave, as launch_shading (kernels.cu).
int launch_wb_shading(const WaveView& bw, const BatchView& b, const uint32_t* sobol, unsigned class_mask, int cur,
                      int append, int n_paths, const LaunchConfig& cfg, cudaStream_t stream) {
  using Kernel = void (*)(WaveView, BatchView, const uint32_t*, int, int);
  static const struct {
    int sc;
    Kernel kernel;
  } kOrder[kShadeClasses] = {{SC_MISS, k_b_shade<SC_MISS>},             {SC_SPECULAR, k_b_shade<SC_SPECULAR>},
                             {SC_DIFFUSE, k_b_shade<SC_DIFFUSE>},       {SC_CONDUCTOR, k_b_shade<SC_CONDUCTOR>},
                             {SC_DIELECTRIC, k_b_shade<SC_DIELECTRIC>}, {SC_PLASTIC, k_b_shade<SC_PLASTIC>},
                             {SC_GENERAL, k_b_shade<SC_GENERAL>},       {SC_TEXTURED, k_b_shade<SC_TEXTURED>}};
  cudaLaunchAttribute early;
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.stream = stream;
  c.attrs = &early;
  int n = 0;
  for (const auto& k : kOrder) {
    if (!((class_mask >> k.sc) & 1u)) continue;
    const ShadeShape shape = shade_shape(k.sc, n_paths, cfg);
    c.blockDim = dim3(shape.block);
    c.gridDim = dim3(shape.grid);
    c.numAttrs = n > 0 ? 1 : 0;
    cudaLaunchKernelEx(&c, k.kernel, bw, b, sobol, cur, append ? 0 : 1);
    ++n;
  }
  return n;
}

}  // namespace

cudaError_t capture_batch_iteration(const WaveView& w, const BatchView& b, const uint32_t* sobol,
                                    const LaunchConfig& cfg, unsigned class_mask, cudaGraphConditionalHandle cond,
                                    cudaStream_t stream, cudaGraph_t body) {
  cudaError_t e = cudaStreamBeginCaptureToGraph(stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) return e;
  enqueue_iteration(w, b, sobol, cfg, class_mask, cond, 1, stream, nullptr);
  cudaGraph_t out = body;
  cudaError_t e2 = cudaStreamEndCapture(stream, &out);
  cudaError_t e3 = cudaGetLastError();
  return e2 != cudaSuccess ? e2 : e3;
}

void launch_batch_iteration(const WaveView& w, const BatchView& b, const uint32_t* sobol, const LaunchConfig& cfg,
                            unsigned class_mask, cudaStream_t stream, StageTimer* timer) {
  enqueue_iteration(w, b, sobol, cfg, class_mask, cudaGraphConditionalHandle{}, 0, stream, timer);
}

namespace {

// launch() on the wave's stream, counted (it returns how many) and timed as `stage`.
template <class F>
void staged(const BatchWave& v, int stage, F&& launch) {
  if (v.timer) v.timer->begin(stage, v.stream);
  const int n = launch();
  if (v.timer) v.timer->end(v.stream);
  if (v.launches) *v.launches += n;
}

}  // namespace

void launch_batch_wave_begin(const BatchWave& v) {
  staged(v, ST_CAMERA, [&] {
    k_wb_camera<<<grid_cap(v.n, 256, v.cfg.num_sms * 32), 256, 0, v.stream>>>(batch_view(v.w, v.b), v.b, v.sobol, v.base, v.n);
    return 1;
  });
}

void launch_batch_wave_bounces(const BatchWave& v, int from, int to, int all) {
  const WaveView bw = batch_view(v.w, v.b);
  const bool append = v.n <= kAppendPaths;
  const int persistent = v.cfg.num_sms * v.cfg.blocks_per_sm;
  const int tgrid = grid_cap(v.n, v.cfg.trace_block, persistent);
  const int sgrid = grid_cap(v.n, v.cfg.shade_block, persistent * 2);
  const int cgrid = grid_cap(v.n, kCompactSpan, v.cfg.num_sms * 8);
  auto trace = [&](int stage, int kinds, int bounce) {
    staged(v, stage, [&] {
      b_trace(v.cfg, bw, v.b, kinds, bounce & 1, tgrid, !append, bounce == 0, v.stream);
      return 1;
    });
  };
  for (int bounce = from; bounce < to; ++bounce) {
    const int cur = bounce & 1;
    if (!v.timer) {
      trace(ST_TRACE_EXT, bounce > 0 ? TK_ALL : TK_EXT, bounce);
    } else {  // timed: kind by kind
      trace(ST_TRACE_EXT, TK_EXT, bounce);
      if (bounce > 0) trace(ST_TRACE_SHADOW, TK_SHADOW, bounce);
      if (bounce > 0) trace(ST_TRACE_MIS, TK_MIS | TK_MIS_ENV, bounce);
    }
    if (bounce > 0)
      staged(v, ST_RESOLVE, [&] {
        k_b_resolve<<<sgrid, v.cfg.shade_block, 0, v.stream>>>(bw, v.b, cur);
        return 1;
      });
    const int* list = bounce == 0 ? nullptr : bw.q_ext[cur];  // the slots traced this bounce
    const int* count = bw.counters + cnt_rays(RK_EXT, cur);
    if (!append)
      staged(v, ST_OTHER, [&] {
        CompactTargets tg{};
        for (int c = 0; c < kShadeClasses; ++c)
          tg.queue[c] = bw.q_cls + (size_t)c * bw.capacity, tg.counter[c] = bw.counters + cnt_cls(c, cur);
        k_wb_compact<kShadeClasses><<<cgrid, kCompactThreads, 0, v.stream>>>(bw.qflags, list, count, tg);
        return 1;
      });
    staged(v, ST_SHADE, [&] {
      return launch_wb_shading(bw, v.b, v.sobol, v.class_mask, cur, append, v.n, v.cfg, v.stream);
    });
    if (!append && bounce + 1 < all)  // no path goes on after the last bounce
      staged(v, ST_OTHER, [&] {
        CompactTargets tg{};
        int* qs[5] = {bw.q_ext[cur ^ 1], bw.q_mis, bw.q_sh, bw.q_mis_env, bw.q_nee};  // as the QueueFlag bits
        for (int k = 0; k < 5; ++k)
          tg.queue[k] = qs[k],
          tg.counter[k] = bw.counters + (k < kRayKinds ? cnt_rays(k, cur ^ 1) : CNT_NEE + (cur ^ 1));
        k_wb_compact<5><<<cgrid, kCompactThreads, 0, v.stream>>>(bw.qflags, list, count, tg);
        return 1;
      });
  }
}

void launch_batch_wave_film(const BatchWave& v, int unfinished) {
  staged(v, ST_FILM, [&] {
    k_wb_film<<<grid_cap(v.n, kWbFilmThreads, v.cfg.num_sms * 8), kWbFilmThreads, 0, v.stream>>>(
        batch_view(v.w, v.b), v.b, v.base, v.n, unfinished < 0 ? -1 : unfinished & 1);
    return 1;
  });
}

// FP64 film sums rounded to FP32 (orion_job.sum32).
__global__ void k_film_to_f32(const double* __restrict__ src, float* __restrict__ dst, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    dst[i] = (float)src[i];
}

void launch_film_to_f32(const double* src, float* dst, long long n, int num_sms, cudaStream_t stream) {
  const long long blocks = std::min<long long>((n + 255) / 256, (long long)num_sms * 8);
  k_film_to_f32<<<(int)std::max<long long>(blocks, 1), 256, 0, stream>>>(src, dst, n);
}

}  // namespace orion_gb300
