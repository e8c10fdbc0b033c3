// Wavefront path tracer kernels for sm_103a.
//
// PathTracing::Li (src/integrator/path.cpp:50-99) is split into stages that
// each run over a device queue of path slots:
//
//   k_camera      Pinhole::generateRay for every path of the wave
//   k_trace       the bounce's extension rays (closest hit), and the previous
//                 bounce's light rays: shadow rays (any hit) and the
//                 BSDF-sampled MIS rays (traced once; the reference traces
//                 that ray twice, once inside Triangle::pdf and once in
//                 estimateDirect)
//   k_shade       emission, BSDF construction, light sampling
//                 (uniformSampleOneLight / estimateDirect,
//                 src/core/integrator.cpp:8-90), BSDF sampling, Russian
//                 roulette; appends shadow / MIS / next-bounce work
//   k_film        per-pixel sums in sample order (RenderTarget::acumulate)
//
// A path's direct-lighting estimate is added to its radiance by its next
// k_shade, before anything else of that bounce, or by k_film if the path
// ended after sampling the light (shade_one, DEFER).
//
// Sample dimensions are consumed in exactly the reference's order, so every
// path sees the same Sobol numbers as the reference path with the same index.
#include <cuda_runtime.h>

#include "kernels.h"
#include "shade.cuh"

namespace orion_gb300 {

namespace {

// The pixel of a wave's local pixel `lp` (WaveArgs).
__device__ __forceinline__ void wave_pixel(const WaveArgs& a, int lp, int* x, int* y) {
  tile_pixel((((int64_t)(lp >> a.chunk_log2) * a.waves + a.wave) << a.chunk_log2) + (lp & ((1 << a.chunk_log2) - 1)),
             a.width, a.height, x, y);
}

__global__ void k_camera(SceneView s, WaveView w, WaveArgs a) {
  if (blockIdx.x == 0 && threadIdx.x < kCounterSlots) w.counters[threadIdx.x] = threadIdx.x == cnt_rays(RK_EXT, 0) ? a.n_paths : 0;
  const int64_t wh = (int64_t)a.width * a.height;
  for (int pid = blockIdx.x * blockDim.x + threadIdx.x; pid < a.n_paths; pid += gridDim.x * blockDim.x) {
    const int lp = pid / a.passes;
    int i, j;
    wave_pixel(a, lp, &i, &j);
    const int64_t index = (a.first_pass + (pid - lp * a.passes)) * wh + (int64_t)j * a.width + i;
    V3 o, d;
    const uint32_t dim = camera_ray_block(s.cam, a.sobol, (uint64_t)index, i, j, &o, &d);
    // Whole 32-byte sectors only (a partly written sector costs L2 a DRAM
    // read): the ray, then the hit and meta sector. The throughput and
    // radiance sector is left out: bounce 0's shading takes 1 and 0 for them
    // (shade_one, FRESH) and writes them.
    PathRec& r = w.rec[pid];
    r.o = f4(o, 0.f);
    r.d = f4(d, 0.f);
    r.hit = make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
    r.meta = make_int4((int)dim, (int)(uint32_t)(uint64_t)index, 0, (int)((uint64_t)index >> 32));
  }
}

// All rays that wait at the start of a bounce (trace_kinds). CAP: traversal
// stack capacity (kTestStackEntries only in the kernels that exercise the
// overflow report).
struct TraceArgs {
  SceneView scene;
  RaySet set[4];  // by TraceKinds bit
  int* counters;
  int* err;
  int kinds;  // the TraceKinds to trace
  int cur;    // parity
  int refill_closest, refill_any;
};

template <int SMEM, bool COUNT = false, int CAP = kMaxStack>
__global__ void __launch_bounds__(512, 2) k_trace(const __grid_constant__ TraceArgs a) {
  extern __shared__ int2 stack_smem[];
  trace_kinds<SMEM, COUNT, CAP>(SingleScene{&a.scene}, a.set, a.kinds, a.counters, a.cur, stack_smem,
                                a.refill_closest, a.refill_any, a.err);
}

// One bounce for every path whose extension ray hit a material of shading
// class SC (or, for SC_MISS, left the scene), with that class's BSDF code only.
// Launch bounds: at most 96 registers (640 threads per SM).
// The queues a path goes to next (next extension ray, shadow ray, MIS rays)
// are recorded as bits of its qflags byte, and k_compact_queues lists them in
// slot order: the next trace then takes rays of neighbouring pixels together
// instead of in the order the shading finished them. Small waves append to the
// queues here (WaveArgs::append).
// The classes' launches do not depend on one another: each lets the next one
// start as soon as its own last blocks run (launch_shading), so the short
// ones overlap; block 0 ends only when the launch before has, which makes the
// end of the last one the end of all.
template <int SC>
__global__ void __launch_bounds__(shade_threads(SC), kShadeThreadsPerSm / shade_threads(SC)) k_shade(SceneView s, WaveView w, WaveArgs a, int bounce, int cur) {
  asm volatile("griddepcontrol.launch_dependents;");
  if (blockIdx.x == 0 && threadIdx.x < kRayKinds) w.counters[CNT_FETCH + threadIdx.x] = 0;  // for the next trace
  const int n = w.counters[cnt_cls(SC, cur)];
  const int* in_q = w.q_cls + (size_t)SC * w.capacity;
  for (int q0 = blockIdx.x * blockDim.x; q0 < n; q0 += gridDim.x * blockDim.x) {
    const int q = q0 + threadIdx.x;
    __syncthreads();  // the block's warps go through the code together
    if (q >= n) continue;
    const int pid = in_q[q];
    const int4 meta = w.rec[pid].meta;
    const uint64_t index = ((uint64_t)(uint32_t)meta.w << 32) | (uint32_t)meta.y;
    ShadeResult r = shade_one<lobes_of_class(SC), SC == SC_TEXTURED, true, true>(
        s, w, a.sobol, pid, index, meta.x, bounce, a.max_depth, a.rr_depth);
    if (a.append) {
      int* next = w.counters + (cur ^ 1);
      queue_append(next + cnt_rays(RK_EXT, 0), w.q_ext[cur ^ 1], pid, r.alive);
      queue_append(next + cnt_rays(RK_MIS, 0), w.q_mis, pid, r.want_mis);
      queue_append(next + cnt_rays(RK_SHADOW, 0), w.q_sh, pid, r.want_sh);
      queue_append(next + cnt_rays(RK_MIS_ENV, 0), w.q_mis_env, pid, r.want_mis_env);
    } else {
      w.qflags[pid] = (uint8_t)((r.alive ? kQfExt : 0) | (r.want_sh ? kQfShadow : 0) |
                                (r.want_mis ? kQfMis : 0) | (r.want_mis_env ? kQfMisEnv : 0));
    }
  }
  if (blockIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Per-pixel accumulation in sample order. A pixel's samples are consecutive
// slots: a block reads whole pixels' samples into shared memory, one thread a
// sample (a path whose last light sample is still pending, since it ended
// right after sampling it, gets it added here), then one thread per pixel and
// channel adds them up in order. Pixels of more samples than threads are read
// in several goes.
constexpr int kFilmThreads = 256;

__global__ void __launch_bounds__(kFilmThreads) k_film(SceneView s, WaveView w, WaveArgs a, FilmView film) {
  // A pixel's samples are padded by one, so that the adding threads meet in different banks.
  __shared__ float buf[3][2 * kFilmThreads];
  const int t = threadIdx.x, P = a.passes;
  const int group = P < kFilmThreads ? kFilmThreads / P : 1;  // pixels of a go
  const int go = P < kFilmThreads ? P : kFilmThreads;         // samples of each
  const int mine = t / go;                                    // this thread's pixel of the group, its sample
  const int n_pixels = a.n_paths / P;
  for (int first = blockIdx.x * group; first < n_pixels; first += gridDim.x * group) {
    const int npx = min(group, n_pixels - first);
    float r = 0.f;  // sums carried from go to go: pixels of several goes only (one pixel, threads 0..2)
    double r64 = 0, rr = 0;
    for (int from = 0; from < P; from += go) {
      const int n = min(go, P - from);
      const int k = t - mine * go;
      if (mine < npx && k < n) {
        const int pid = (first + mine) * P + from + k;
        float4 l = w.L[pid];
        if (w.dim[pid] & kNeePending) {
          const V3 e = xyz(l) + nee_estimate(s, w, pid);
          l.x = e.x;
          l.y = e.y;
          l.z = e.z;
        }
        const int at = mine * (go + 1) + k;
        buf[0][at] = l.x;
        buf[1][at] = l.y;
        buf[2][at] = l.z;
      }
      __syncthreads();
      for (int u = t; u < 3 * npx; u += kFilmThreads) {
        const int px = u / 3, c = u - 3 * px;
        int x, y;
        wave_pixel(a, first + px, &x, &y);
        const int64_t pix = (int64_t)y * a.width + x;
        if (from == 0) {
          r = a.add ? film.sum[3 * pix + c] : 0.f;
          r64 = rr = 0;
        }
        const float* v = buf[c] + px * (go + 1);
        for (int i = 0; i < n; ++i) r += v[i];
        if (film.sum64)
          for (int i = 0; i < n; ++i) {
            r64 += v[i];
            rr += (double)v[i] * v[i];
          }
        if (from + n == P) {
          film.sum[3 * pix + c] = r;
          if (c == 0 && film.count) film.count[pix] = (a.add ? film.count[pix] : 0u) + (uint32_t)P;
          if (film.sum64) {
            film.sum64[3 * pix + c] = (a.add ? film.sum64[3 * pix + c] : 0.0) + r64;
            film.sumsq64[3 * pix + c] = (a.add ? film.sumsq64[3 * pix + c] : 0.0) + rr;
          }
        }
      }
      __syncthreads();
    }
  }
}

template <int NQ>
__global__ void __launch_bounds__(kCompactThreads) k_compact_queues(uint8_t* flags, const int* list, const int* count,
                                                                    CompactTargets tg) {
  compact_queues<NQ>(flags, list, count, tg);
}

__global__ void k_reset_counters(int* counters, int slots, int keep_slot, int keep_value) {
  int i = threadIdx.x;
  if (i < slots) counters[i] = (i == keep_slot) ? keep_value : 0;
}

// ------------------------------------------------------------ test hooks

__global__ void k_sobol(const uint32_t* sobol, int64_t n, const uint64_t* index, const uint32_t* dim, float* out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = sobol_sample(sobol, index[i], dim[i]);
}

// Ray queries (Scene::intersect): closest hit in (tnear, tfar]. Warps take
// their rays from pieces of the list of their own, neighbouring rays together,
// and refill idle lanes from it (no counter to clear); triangles are tested by
// the whole warp. A query of 100,000 rays took 422 us with one ray per thread
// and five device allocations, 181 us so; one ray 216 and 59 us.
constexpr int kQueryStack = 8, kQueryBlock = 128, kQueryRefill = 20;

__global__ void __launch_bounds__(kQueryBlock, 8) k_trace_closest(SceneView s, int64_t n, const float4* rays, float* t,
                                                                  float* u, float* v, int* prim) {
  extern __shared__ int2 stack_smem[];
  constexpr unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  const int64_t warp = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  int64_t next = n * warp / warps;
  const int64_t end = n * (warp + 1) / warps;
  TraversalStack<kQueryStack> st;
  st.smem = stack_smem + threadIdx.x;
  st.stride = blockDim.x;
  st.sp = 0;
  TriScratch* tsc = reinterpret_cast<TriScratch*>(stack_smem + kQueryStack * blockDim.x) + (threadIdx.x >> 5);
  const TraceScene ts = trace_scene(s);
  LaneRay r;
  lane_start(r, make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 1.f, 0.f), kFloatMax, false);
  r.tnear = 0.f;
  int64_t mine = -1;
  while (true) {
    unsigned act = __ballot_sync(kFull, mine >= 0);
    if (next < end && __popc(act) < kQueryRefill) {
      const int64_t k = next + __popc(~act & ((1u << lane) - 1u));
      if (mine < 0 && k < end) {
        const float4 a = __ldcs(rays + 2 * k), b = __ldcs(rays + 2 * k + 1);
        lane_start(r, a, make_float4(a.w, b.x, b.y, 0.f), b.w, false);
        r.tnear = b.z;
        st.sp = 0;
        mine = k;
      }
      next += 32 - __popc(act);
      act = __ballot_sync(kFull, mine >= 0);
    }
    if (act == 0u) break;  // none left in the piece either (next < end would have started some)
    if (mine >= 0) lane_visit<false, kQueryStack, false, kMaxStack, true>(r, ts, st, nullptr);
    warp_triangles<false, false, true, true>(r, ts, tsc, nullptr);
    if (mine >= 0 && lane_pop(r, st)) {
      const bool hit = r.tri >= 0;  // no test by the sign of tmax: hits behind the origin (tnear < 0) count
      t[mine] = hit ? r.tmax : 0.f;
      u[mine] = r.u;
      v[mine] = r.v;
      prim[mine] = hit ? __ldg(s.tri_prim + r.tri) : -1;
      mine = -1;
    }
  }
}

// Any-hit queries: the first hit that a ray's own traversal finds.
template <int SMEM>
__global__ void k_trace_any(SceneView s, int64_t n, const float* rays, float* t, float* u, float* v, int* prim) {
  extern __shared__ int2 stack_smem[];
  TraceScene ts = trace_scene(s);
  TraversalStack<SMEM> st;
  st.smem = stack_smem + threadIdx.x;
  st.stride = blockDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float* r = rays + 8 * i;
    V3 o = V3{r[0], r[1], r[2]}, d = V3{r[3], r[4], r[5]};
    RayHit h = traverse_any(ts, o, d, r[6], r[7], st);
    t[i] = h.tri >= 0 ? h.t : 0.f;
    u[i] = h.u;
    v[i] = h.v;
    prim[i] = h.tri >= 0 ? __ldg(s.tri_prim + h.tri) : -1;
  }
}

// Production-traversal hook: n rays (o, d, tnear = 0, tfar) placed in a
// wave's records as extension rays (closest hit) or shadow rays (occlusion,
// tmax = tfar), so that the renderer's own persistent trace kernels trace them.
__global__ void k_load_rays(WaveView w, int n, const float* rays, int any_hit) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float* r = rays + 8 * (size_t)i;
    if (any_hit) {
      w.sh_o[i] = make_float4(r[0], r[1], r[2], r[7]);
      w.sh_d[i] = make_float4(r[3], r[4], r[5], 0.f);
      w.q_sh[i] = i;
    } else {
      w.ray_o[i] = make_float4(r[0], r[1], r[2], 0.f);
      w.ray_d[i] = make_float4(r[3], r[4], r[5], 0.f);
      w.q_ext[0][i] = i;
    }
  }
}

__global__ void k_store_hits(WaveView w, int n, int any_hit, float* t, float* u, float* v, int* prim) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (any_hit) {
      t[i] = u[i] = v[i] = 0.f;
      prim[i] = w.occluded[i] ? 1 : -1;
    } else {
      const float4 h = w.hit[i];
      const int p = __float_as_int(h.w);
      t[i] = p >= 0 ? h.x : 0.f;
      u[i] = h.y;
      v[i] = h.z;
      prim[i] = p;
    }
  }
}

__global__ void k_camera_rays(SceneView s, const uint32_t* sobol, int64_t n, const int64_t* index, float* rays) {
  const int64_t wh = (int64_t)s.cam.width * s.cam.height;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    int64_t idx = index[q];
    int64_t pix = idx % wh;
    PathSampler smp{sobol, (uint64_t)idx, 5u};
    V3 o, d;
    camera_ray(s.cam, smp, (int)(pix % s.cam.width), (int)(pix / s.cam.width), &o, &d);
    float* r = rays + 6 * q;
    r[0] = o.x;
    r[1] = o.y;
    r[2] = o.z;
    r[3] = d.x;
    r[4] = d.y;
    r[5] = d.z;
  }
}

__global__ void k_bsdf_eval(const DevMaterial* mat, int64_t n, const float* frame, const float* wo, const float* wi,
                            const float* rnd, int type, float* f, float* pdf, float* sf, float* swi, float* spdf,
                            int* stype, int* nbxdf) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float* fr = frame + 12 * i;
    Frame F{ld3(fr), ld3(fr + 3), ld3(fr + 6), ld3(fr + 9)};
    V3 o = ld3(wo + 3 * i), in = ld3(wi + 3 * i);
    V3 fv = bsdf_f(*mat, F, in, o, type);
    f[3 * i] = fv.x;
    f[3 * i + 1] = fv.y;
    f[3 * i + 2] = fv.z;
    pdf[i] = bsdf_pdf(*mat, F, in, o, type);
    V3 w = V3{0, 0, 0};
    float p = 0.f;
    int st = 0;
    V3 s = bsdf_sample_f(*mat, F, o, rnd[2 * i], rnd[2 * i + 1], type, &w, &p, &st);
    sf[3 * i] = s.x;
    sf[3 * i + 1] = s.y;
    sf[3 * i + 2] = s.z;
    swi[3 * i] = w.x;
    swi[3 * i + 1] = w.y;
    swi[3 * i + 2] = w.z;
    spdf[i] = p;
    stype[i] = st;
    nbxdf[i] = bsdf_num_matching(*mat, kNonSpecular);
  }
}

int grid_for(int64_t n, int block, int max_blocks) {
  int64_t g = (n + block - 1) / block;
  if (g > max_blocks) g = max_blocks;
  return (int)(g < 1 ? 1 : g);
}

template <int SMEM, bool COUNT = false, int CAP = kMaxStack>
void launch_trace_kernel(int kinds, const SceneView& s, const WaveView& w, int cur, bool marks, bool camera_rays,
                         const LaunchConfig& cfg, int grid, cudaStream_t stream) {
  TraceArgs a;
  a.scene = s;
  wave_ray_sets(w, cur, marks, camera_rays, a.set);
  a.counters = w.counters;
  a.err = w.error_word;
  a.kinds = kinds;
  a.cur = cur;
  a.refill_closest = cfg.refill_below < 1 ? 1 : (cfg.refill_below > 32 ? 32 : cfg.refill_below);
  a.refill_any = refill_any_hit(a.refill_closest);
  k_trace<SMEM, COUNT, CAP><<<grid, cfg.trace_block, trace_smem_bytes(SMEM, cfg.trace_block), stream>>>(a);
}

// kinds: TraceKinds bits.
void trace_dispatch(int kinds, const SceneView& s, const WaveView& w, int cur, bool marks, bool camera_rays,
                    const LaunchConfig& cfg, int grid, cudaStream_t stream) {
  if (w.trace_work) {  // counting render: the stack's split between shared and local memory is irrelevant
    launch_trace_kernel<0, true>(kinds, s, w, cur, marks, camera_rays, cfg, grid, stream);
    return;
  }
  if (cfg.test_stack_entries) {  // orion_gpu_set_test_limits: kernels with a kTestStackEntries-entry stack
    launch_trace_kernel<0, false, kTestStackEntries>(kinds, s, w, cur, marks, camera_rays, cfg, grid, stream);
    return;
  }
  switch (cfg.smem_stack) {
    case 0: launch_trace_kernel<0>(kinds, s, w, cur, marks, camera_rays, cfg, grid, stream); break;
    case 8: launch_trace_kernel<8>(kinds, s, w, cur, marks, camera_rays, cfg, grid, stream); break;
    case 24: launch_trace_kernel<24>(kinds, s, w, cur, marks, camera_rays, cfg, grid, stream); break;
    case 32: launch_trace_kernel<32>(kinds, s, w, cur, marks, camera_rays, cfg, grid, stream); break;
    default: launch_trace_kernel<16>(kinds, s, w, cur, marks, camera_rays, cfg, grid, stream); break;
  }
}

// Shading of one bounce: a launch per class present, those with the least code
// first (zoo 985x726, 64 spp: 44.7 ms; most code first 48.6 ms; one after the
// other 46.3 ms). All but the first may start before the one before them has ended
// (zoo 333x217, 48 spp, seven classes: 4.85 -> 4.52 ms a render; Cornell 64x64,
// 1 spp 0.66 -> 0.55 ms). One kernel for all classes was slower where it
// matters (zoo 5.35 ms, displaced sphere 60.7 -> 63.1 ms: more spills) and
// contracted other multiply-adds.
int launch_shading(const SceneView& s, const WaveView& w, const WaveArgs& a, int bounce, int cur,
                   const LaunchConfig& cfg, cudaStream_t stream) {
  using Kernel = void (*)(SceneView, WaveView, WaveArgs, int, int);
  static const struct {
    int sc;
    Kernel kernel;
  } kOrder[kShadeClasses] = {{SC_MISS, k_shade<SC_MISS>},             {SC_SPECULAR, k_shade<SC_SPECULAR>},
                             {SC_DIFFUSE, k_shade<SC_DIFFUSE>},       {SC_CONDUCTOR, k_shade<SC_CONDUCTOR>},
                             {SC_DIELECTRIC, k_shade<SC_DIELECTRIC>}, {SC_PLASTIC, k_shade<SC_PLASTIC>},
                             {SC_GENERAL, k_shade<SC_GENERAL>},       {SC_TEXTURED, k_shade<SC_TEXTURED>}};
  cudaLaunchAttribute early;
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.stream = stream;
  c.attrs = &early;
  int n = 0;
  for (const auto& k : kOrder) {
    if (!((a.class_mask >> k.sc) & 1u)) continue;
    const ShadeShape shape = shade_shape(k.sc, a.n_paths, cfg);
    c.blockDim = dim3(shape.block);
    c.gridDim = dim3(shape.grid);
    c.numAttrs = n > 0 ? 1 : 0;
    cudaLaunchKernelEx(&c, k.kernel, s, w, a, bounce, cur);
    ++n;
  }
  return n;
}

}  // namespace

void launch_wave(const SceneView& s, const WaveView& w, const WaveArgs& a, const FilmView& film,
                 const LaunchConfig& cfg, cudaStream_t stream, int* launches, StageTimer* timer,
                 cudaEvent_t film_wait, cudaEvent_t film_done) {
  const int persistent = cfg.num_sms * cfg.blocks_per_sm;
  int nl = 0;
  auto begin = [&](int st) {
    if (timer) timer->begin(st, stream);
  };
  auto end = [&]() {
    if (timer) timer->end(stream);
    ++nl;
  };
  begin(ST_CAMERA);
  k_camera<<<grid_for(a.n_paths, 256, persistent * 4), 256, 0, stream>>>(s, w, a);
  end();
  // The persistent trace grids leave room on each SM for the other stream's
  // shading blocks (6 of 128 threads per SM: 24 of 64 warps; 1012 -> 1023
  // Mpaths/s on the displaced sphere, 2433 -> 2525 on eight spheres, against
  // grids that fill the register file).
  const int tgrid = grid_for(a.n_paths, cfg.trace_block, persistent);
  const int compact_grid = grid_for(a.n_paths, kCompactSpan, cfg.num_sms * 8);
  int cur = 0;
  for (int bounce = 0; bounce <= a.max_depth; ++bounce) {
    // The bounce's extension rays and the previous bounce's light rays. A
    // render that times its stages traces them kind by kind.
    if (!timer) {
      trace_dispatch(bounce > 0 ? TK_ALL : TK_EXT, s, w, cur, !a.append, bounce == 0, cfg, tgrid, stream);
      ++nl;
    } else {
      begin(ST_TRACE_EXT);
      trace_dispatch(TK_EXT, s, w, cur, !a.append, bounce == 0, cfg, tgrid, stream);
      end();
      if (bounce > 0) {
        begin(ST_TRACE_SHADOW);
        trace_dispatch(TK_SHADOW, s, w, cur, !a.append, bounce == 0, cfg, tgrid, stream);
        end();
        begin(ST_TRACE_MIS);
        trace_dispatch(TK_MIS | TK_MIS_ENV, s, w, cur, !a.append, bounce == 0, cfg, tgrid, stream);
        end();
      }
    }
    const int* list = bounce == 0 ? nullptr : w.q_ext[cur];  // the slots traced this bounce
    if (!a.append) {  // the trace marked each finished ray's shading class: list them by class in slot order
      begin(ST_OTHER);
      CompactTargets tg{};
      for (int c = 0; c < kShadeClasses; ++c)
        tg.queue[c] = w.q_cls + (size_t)c * w.capacity, tg.counter[c] = w.counters + cnt_cls(c, cur);
      k_compact_queues<kShadeClasses><<<compact_grid, kCompactThreads, 0, stream>>>(
          w.qflags, list, w.counters + cnt_rays(RK_EXT, cur), tg);
      end();
    }
    begin(ST_SHADE);
    nl += launch_shading(s, w, a, bounce, cur, cfg, stream) - 1;  // end() counts one of them
    end();
    if (!a.append && bounce < a.max_depth) {  // after the last bounce no path goes on and no queue is read
      begin(ST_OTHER);
      CompactTargets tg{};
      int* qs[kRayKinds] = {w.q_ext[cur ^ 1], w.q_mis, w.q_sh, w.q_mis_env};  // as the QueueFlag bits
      for (int k = 0; k < kRayKinds; ++k) tg.queue[k] = qs[k], tg.counter[k] = w.counters + cnt_rays(k, cur ^ 1);
      k_compact_queues<kRayKinds><<<compact_grid, kCompactThreads, 0, stream>>>(
          w.qflags, list, w.counters + cnt_rays(RK_EXT, cur), tg);
      end();
    }
    // No resolve pass: each path's light sample is added to its radiance by
    // its next shading, or by k_film if the path ends here (shade_one, DEFER).
    cur ^= 1;
  }
  if (film_wait) cudaStreamWaitEvent(stream, film_wait, 0);
  begin(ST_FILM);
  k_film<<<grid_for(a.n_paths, kFilmThreads / 2, persistent * 4), kFilmThreads, 0, stream>>>(s, w, a, film);
  end();
  if (film_done) cudaEventRecord(film_done, stream);
  if (launches) *launches += nl;
}

void launch_sobol(const uint32_t* sobol, int64_t n, const uint64_t* index, const uint32_t* dim, float* out,
                  cudaStream_t stream) {
  k_sobol<<<grid_for(n, 256, 4096), 256, 0, stream>>>(sobol, n, index, dim, out);
}

void launch_trace(const SceneView& s, int64_t n, const float* rays, int any_hit, float* t, float* u, float* v,
                  int* prim, const LaunchConfig& cfg, cudaStream_t stream) {
  if (any_hit) {
    const int block = cfg.trace_block;
    const int grid = grid_for(n, block, cfg.num_sms * cfg.blocks_per_sm * 2);
    k_trace_any<16><<<grid, block, (size_t)16 * block * sizeof(int2), stream>>>(s, n, rays, t, u, v, prim);
    return;
  }
  // Pieces of at least two warps' rays, so that there is something to refill with.
  const int grid = grid_for(n, 2 * kQueryBlock, cfg.num_sms * 8);
  k_trace_closest<<<grid, kQueryBlock, trace_smem_bytes(kQueryStack, kQueryBlock), stream>>>(
      s, n, reinterpret_cast<const float4*>(rays), t, u, v, prim);
}

void launch_trace_wave(const SceneView& s, const WaveView& w, int n, const float* rays, int any_hit, float* t,
                       float* u, float* v, int* prim, const LaunchConfig& cfg, cudaStream_t stream) {
  k_reset_counters<<<1, 32, 0, stream>>>(w.counters, kCounterSlots, cnt_rays(any_hit ? RK_SHADOW : RK_EXT, 0), n);
  k_load_rays<<<grid_for(n, 256, 4096), 256, 0, stream>>>(w, n, rays, any_hit);
  const int tgrid = grid_for(n, cfg.trace_block, cfg.num_sms * cfg.blocks_per_sm);
  trace_dispatch(any_hit ? TK_SHADOW : TK_EXT, s, w, 0, true, false, cfg, tgrid, stream);
  k_store_hits<<<grid_for(n, 256, 4096), 256, 0, stream>>>(w, n, any_hit, t, u, v, prim);
}

namespace {

cudaError_t limit_of(const void* f, int smem_bytes, int* max_block) {
  if (smem_bytes > 0) {
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
    if (e != cudaSuccess) return e;
  }
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, f);
  if (e != cudaSuccess) return e;
  *max_block = std::min(*max_block, a.maxThreadsPerBlock);
  return cudaSuccess;
}

}  // namespace

cudaError_t configure_kernels(int smem_bytes, KernelLimits* lim) {
  const void* trace[] = {(const void*)k_trace<0>,        (const void*)k_trace<8>,  (const void*)k_trace<16>,
                         (const void*)k_trace<24>,       (const void*)k_trace<32>, (const void*)k_trace<0, true>,
                         (const void*)k_trace_any<16>};
  const void* shade[] = {(const void*)k_shade<SC_DIFFUSE>, (const void*)k_shade<SC_CONDUCTOR>,
                         (const void*)k_shade<SC_SPECULAR>, (const void*)k_shade<SC_DIELECTRIC>,
                         (const void*)k_shade<SC_PLASTIC>, (const void*)k_shade<SC_GENERAL>, (const void*)k_shade<SC_TEXTURED>,
                         (const void*)k_shade<SC_MISS>};
  for (const void* f : trace) {
    cudaError_t e = limit_of(f, smem_bytes, &lim->max_trace_block);
    if (e != cudaSuccess) return e;
  }
  for (const void* f : shade) {
    cudaError_t e = limit_of(f, 0, &lim->max_shade_block);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

void launch_camera_rays(const SceneView& s, const uint32_t* sobol, int64_t n, const int64_t* index, float* rays,
                        cudaStream_t stream) {
  k_camera_rays<<<grid_for(n, 256, 4096), 256, 0, stream>>>(s, sobol, n, index, rays);
}

void launch_bsdf_eval(const DevMaterial* mat, int64_t n, const float* frame, const float* wo, const float* wi,
                      const float* rnd, int type, float* f, float* pdf, float* sf, float* swi, float* spdf,
                      int* stype, int* nbxdf, cudaStream_t stream) {
  k_bsdf_eval<<<grid_for(n, 128, 4096), 128, 0, stream>>>(mat, n, frame, wo, wi, rnd, type, f, pdf, sf, swi, spdf,
                                                           stype, nbxdf);
}

}  // namespace orion_gb300
