// Host-callable launchers for the wavefront kernels (kernels.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_types.h"

namespace orion_gb300 {

// A resident scene, as the kernels see it.
struct SceneView {
  const float4* nodes;
  const float4* woop;
  const int* tri_prim;
  const uint8_t* tri_class;  // leaf order -> ShadeClass of the triangle's material
  const PrimShade* prims;
  const DevMaterial* mats;
  const DevLight* lights;
  const DevEnvMap* envmaps;  // image environment maps (DevLight::image)
  const DevTexture* textures;      // image textures (DevMaterialSrc::tex)
  const DevMaterialSrc* mat_src;   // builder inputs per material (null when nothing is textured)
  const float* prim_uv;            // texture coordinates, 6 per primitive (null when nothing is textured)
  const float* light_func;
  const float* light_cdf;
  float light_func_int;
  int num_lights;
  int env_idx[8];
  int num_env;
  int num_area_lights;
  float world_radius;
  float world_center[3];  // Bounds3::boundingSphere (distant and environment photons)
  unsigned class_mask;  // shading classes of the scene's triangles (bit ShadeClass), SC_MISS always
  DevCamera cam;
};

// One field of an array of per-path records, seen as an array of its own
// (STRIDE: record size in units of T).
template <class T, int STRIDE>
struct FieldView {
  T* p;
  ORION_HD inline T& operator[](int64_t i) const { return p[i * STRIDE]; }
};

// Per-path state, one 96-byte record (three 32-byte sectors) per path slot,
// so a kernel that reaches a path through a scattered slot index moves whole
// sectors: [o, d] (what a trace reads), [beta, L], [hit, meta].
struct PathRec {
  float4 o;     // ray origin; w unused
  float4 d;     // ray direction; w unused
  float4 beta;  // throughput; w = 1 after a specular bounce
  float4 L;     // radiance so far; w = batched mode: sample index, low 32 bits
  float4 hit;   // t, u, v, primitive (int bits; -1 miss)
  int4 meta;    // Sobol dimension counter; batched mode: job, bounce, sample index high 32 bits
                // (plain waves: y, w hold the sample index)
};
static_assert(sizeof(PathRec) == 96, "PathRec is three sectors");

// Next-event-estimation record of a path, 128 bytes: written whole by the
// shading kernel; the trace reads [sh_o, sh_d] of shadow rays and [mis_o, mis_d]
// of MIS rays, and what adds the sample to the radiance the first two sectors (the
// path's next shading or k_film; in batches k_b_resolve).
struct NeeRec {
  float4 p;      // shading point xyz, light-selection pdf
  float4 beta;   // beta before the bounce, w = flags | light << 8 (int bits)
  float4 ld;     // light-sample contribution rgb, w = BSDF-sample pdf
  float4 f;      // BSDF-sample f * |cos| rgb, w = MIS weight for environment lights
  float4 sh_o;   // shadow ray origin, w = tmax
  float4 sh_d;
  float4 mis_o;
  float4 mis_d;
};
static_assert(sizeof(NeeRec) == 128, "NeeRec is four sectors");

using RecF4 = FieldView<float4, sizeof(PathRec) / sizeof(float4)>;
using RecI = FieldView<int, sizeof(PathRec) / sizeof(int)>;
using NeeF4 = FieldView<float4, sizeof(NeeRec) / sizeof(float4)>;
using F4 = FieldView<float4, 1>;

// Device path state for one wave of `capacity` paths.
struct WaveView {
  PathRec* rec;
  NeeRec* nee;
  RecF4 ray_o, ray_d, beta, L, hit;                          // fields of rec
  RecI dim, job, bounce, index_hi;                           // rec.meta
  NeeF4 nee_p, nee_beta, nee_ld, nee_f, sh_o, sh_d, mis_o, mis_d;  // fields of nee
  float4* mis_hit;   // MIS ray hit: t, u, v, primitive
  int* occluded;
  int* mis_occluded;  // MIS ray towards an environment light: anything hit
  int* q_mis_env;     // MIS rays towards an environment light (occlusion queries)
  int* q_ext[2];     // extension-ray queues (current / next bounce)
  int* q_nee;        // batches: paths that sampled a light this bounce
  int* q_sh;         // shadow rays
  int* q_mis;        // BSDF-sampled rays towards a non-delta light
  int* q_cls;        // extension hits by shading class: kShadeClasses queues of `capacity`
  int* counters;     // kCounterSlots ints
  unsigned long long* ray_stats;  // ext, shadow, mis
  // Null, or (a counting render) 6 counters the trace kernels add to: node
  // visits of the extension, shadow and MIS rays, then their triangle tests.
  unsigned long long* trace_work;
  int* error_word;
  // Plain renders: per slot, the queues its shading appended it to this
  // bounce (kQueueFlag* bits); k_compact_queues turns them into the queues,
  // in slot order, and clears them.
  uint8_t* qflags;
  int capacity;
};

// Bits of WaveView::qflags: the queues a shaded path goes to.
enum QueueFlag { kQfExt = 1, kQfMis = 2, kQfShadow = 4, kQfMisEnv = 8, kQfNee = 16 };

// Bits of a launch's error word (plain renders: WaveView::error_word; batches: BatchCtl::error).
constexpr int kErrIterationCap = 1;    // a batch loop reached its iteration bound
constexpr int kErrTraversalStack = 2;  // a traversal needed more stack entries than its capacity
// Stack capacity of the test-only trace kernels (orion_gpu_set_test_limits).
constexpr int kTestStackEntries = 2;

// Counters of a wave's queues. The queues of rays (one per kind and parity)
// and of shaded classes (one per class and parity) are filled for one bounce
// while the last bounce's counters are still being read, so each has two:
// bounce b's trace reads the ray counters of parity b & 1, counts classes
// under the same parity, and empties the other parity's for the next shading
// and trace to fill.
enum CounterSlot { CNT_RAYS = 0 /* + 2 x kind + parity */, CNT_FETCH = 8 /* + kind */, CNT_NEE = 12 /* + parity */,
                   CNT_RETIRE = 14, CNT_FREE = 15, CNT_CLS = 16 /* + 8 x parity + class */, kCounterSlots = 32 };
ORION_HD constexpr int cnt_rays(int kind, int parity) { return CNT_RAYS + 2 * kind + parity; }
ORION_HD constexpr int cnt_cls(int sc, int parity) { return CNT_CLS + 8 * parity + sc; }
static_assert(kShadeClasses <= 8, "two parities of class counters");

// Ray kinds of one trace launch, by number and as bits.
enum RayKind { RK_EXT = 0, RK_MIS = 1, RK_SHADOW = 2, RK_MIS_ENV = 3, kRayKinds = 4 };
enum TraceKinds { TK_EXT = 1, TK_MIS = 2, TK_SHADOW = 4, TK_MIS_ENV = 8, TK_ALL = 15 };

// ------------------------------------------------------------ batched mode
//
// Many render jobs (scenes, views, resolutions, spp, depths) share one pool
// of path slots (pooled mode; wave mode runs their work list in waves). Each loop iteration refills free slots from the global work
// list (job by job, sample index by sample index), runs one bounce for every
// live path, and retires finished paths into their job's FP64 film.

struct DevJob {
  SceneView scene;
  int width, height;
  int max_depth, rr_depth;
  long long first_index;  // sample index of the job's first path: k0 * W * H
  long long num_paths;    // W * H * spp
  int spp;
  long long work_begin;   // offset of the job in the global work list
  double* sum;            // W*H*3
  double* sumsq;          // W*H*3
  unsigned int* count;    // W*H
};

struct BatchCtl {
  unsigned long long cursor;     // next work item
  unsigned long long total;      // total work items
  unsigned long long take_base;  // first work item taken this iteration
  int take;                      // slots refilled this iteration
  int cur;                       // parity of the current extension queue
  int counters[kCounterSlots];
  int njobs;
  int iterations;
  int max_iterations;
  int error;                     // kErr* bits
  unsigned long long rays[3];    // ext, shadow, mis
  unsigned long long paths_done;
  int more;                      // host-driven loop: 1 while another iteration is needed
};

struct BatchView {
  DevJob* jobs;
  BatchCtl* ctl;
  int* q_retire;
  int* q_free;
};

// One kind of queued rays, as a trace kernel takes them: ray k of `count` is
// that of path slot queue[k], its origin and direction at o / d + slot x
// stride (float4 units).
struct RaySet {
  const int* queue;   // null: ray k is slot k's (a wave's camera rays)
  const int* count;
  int* fetch;         // next ray to take; zero at launch
  const float4* o;    // any hit: w = tmax
  const float4* d;
  float4* hit;        // closest hit: t, u, v, primitive at hit + slot x hit_stride
  int* occluded;      // any hit: 0 or 1 per slot
  int stride, hit_stride;
  // Closest hit, or null: the shading class of what each ray hit goes to its
  // slot's byte here (bit ShadeClass), for a compaction pass, or, without
  // flags, the slot to that class's queue.
  uint8_t* cls_flags;
  int* q_cls;         // kShadeClasses queues, cls_stride ints apart, or null
  int* cls_counters;
  int cls_stride;
  unsigned long long* stat;  // rays traced
  unsigned long long* work;  // counting kernels: node visits at [0], triangle tests at [3]
};

// The rays of a wave of parity `cur`, by RayKind. marks: the shading classes
// go to the slots' flag bytes. camera_rays: the extension rays are those of all
// slots, in order, and no queue lists them.
inline void wave_ray_sets(const WaveView& w, int cur, bool marks, bool camera_rays, RaySet set[kRayKinds]) {
  constexpr int kRec = sizeof(PathRec) / sizeof(float4), kNee = sizeof(NeeRec) / sizeof(float4);
  unsigned long long* work = w.trace_work;
  auto of = [&](int kind, const int* q, const float4* o, const float4* d, int stride, float4* hit, int hit_stride,
                int* occluded, int stat) {
    set[kind] = RaySet{q, w.counters + cnt_rays(kind, cur), w.counters + CNT_FETCH + kind, o, d, hit, occluded,
                       stride, hit_stride, nullptr, nullptr, nullptr, 0, w.ray_stats + stat,
                       work ? work + stat : nullptr};
  };
  of(RK_EXT, camera_rays ? nullptr : w.q_ext[cur], w.ray_o.p, w.ray_d.p, kRec, w.hit.p, kRec, nullptr, 0);
  of(RK_MIS, w.q_mis, w.mis_o.p, w.mis_d.p, kNee, w.mis_hit, 1, nullptr, 2);
  of(RK_SHADOW, w.q_sh, w.sh_o.p, w.sh_d.p, kNee, nullptr, 0, w.occluded, 1);
  of(RK_MIS_ENV, w.q_mis_env, w.mis_o.p, w.mis_d.p, kNee, nullptr, 0, w.mis_occluded, 2);
  set[RK_EXT].cls_flags = marks ? w.qflags : nullptr;
  set[RK_EXT].q_cls = w.q_cls;
  set[RK_EXT].cls_counters = w.counters + cnt_cls(0, cur);
  set[RK_EXT].cls_stride = w.capacity;
}

// Refill threshold of any-hit warps: their rays end early and unevenly, so
// they refill at 4 lanes more (1024x1024 x 64 spp displaced sphere: 804
// Mpaths/s against 798 at the closest-hit threshold of 20, 787 at 16).
inline int refill_any_hit(int refill_closest) { return refill_closest + 4 > 32 ? 32 : refill_closest + 4; }

#ifdef __CUDACC__
// Sample index of a batched path slot (kept in L.w and meta.w).
__device__ __forceinline__ long long slot_index(const WaveView& w, int pid) {
  return (long long)(((unsigned long long)(unsigned)w.index_hi[pid] << 32) |
                     (unsigned long long)__float_as_uint(w.L[pid].w));
}
#endif

// Pixel `pos` of a film in tile order: tiles of 8 x 4 pixels, tile row after
// tile row, row by row within a tile (edge tiles are smaller). Films of more than
// 2^28 pixels a row, where a tile row's pixels pass 32 bits: row by row.
ORION_HD inline void tile_pixel(int64_t pos, int width, int height, int* x, int* y) {
  if (width > 1 << 28) {
    *y = (int)(pos / width);
    *x = (int)(pos - (int64_t)*y * width);
    return;
  }
  const uint32_t band_pixels = 4u * (uint32_t)width;
  const int band = pos >> 32 ? (int)(pos / band_pixels) : (int)((uint32_t)pos / band_pixels), y0 = 4 * band;
  const int left = height - y0, rows = left < 4 ? left : 4, in_band = (int)(pos - (int64_t)band * band_pixels);
  const int tile = in_band / (8 * rows), x0 = 8 * tile, cols = width - x0 < 8 ? width - x0 : 8;
  const int in_tile = in_band - 8 * rows * tile, row = in_tile / cols;
  *x = x0 + in_tile - row * cols;
  *y = y0 + row;
}

// A wave renders `passes` sample passes of some of the film's pixels. Its slots
// hold pixel after pixel, and each pixel's passes in order: slot = local
// pixel x passes + pass, so the rays of a warp leave through one pixel or a few
// neighbouring ones. The render's pixels, in tile order (wave_pixel), are cut
// into chunks of 2^chunk_log2, dealt to its `waves` waves in turn: waves that
// run at once then cost about the same.
struct WaveArgs {
  const uint32_t* sobol;          // Sobol tables (sobol_sample, dmath.cuh)
  int64_t first_pass;  // sample index = (first_pass + pass) x width x height + pixel
  int passes;
  int wave, waves, chunk_log2;
  int add;             // 1: an earlier wave wrote the film for these pixels (other passes)
  int n_paths;         // local pixels x passes
  int width, height;
  int max_depth;
  int rr_depth;
  int append;           // 1: queues are appended to directly (small waves), 0: listed by k_compact_queues
  unsigned class_mask;  // shading classes present in the scene (bit ShadeClass), SC_MISS always
};

// Waves of at most this many paths append to their queues directly: two
// compaction launches fewer a bounce, for queues out of slot order. Medians of
// a render, compacted / appended: Cornell 64x64 x 1 spp (4K paths a wave)
// 0.515 / 0.404 ms; displaced 720p x 1 spp (461K) 1.76 / 1.56; Cornell 512x512 x
// 4 spp (524K) 2.23 / 2.12, zoo the same 2.05 / 2.07; zoo 768x768 x 4 spp (1.2M)
// 3.32 / 3.60; zoo 333x217 x 48 spp (1.7M) 4.11 / 4.72.
constexpr int kAppendPaths = 1 << 19;

struct FilmView {
  float* sum;        // W*H*3
  uint32_t* count;   // W*H
  double* sum64;     // W*H*3 or null
  double* sumsq64;   // W*H*3 or null
};

struct LaunchConfig {
  int num_sms;
  int trace_block;   // threads per block of the trace kernels
  int shade_block;   // threads per block of the shading kernels with little code (shade_shape), resolve and retire
  int blocks_per_sm; // persistent grid size factor
  int smem_stack;    // shared-memory stack entries per thread (0, 8, 16, 24, 32)
  int refill_below;  // a traversal warp refills idle lanes when fewer lanes than this hold a ray (1..32)
  // Test knobs (orion_gpu_set_test_limits), 0 in normal operation:
  int test_stack_entries;   // plain renders trace with kernels whose stack holds kTestStackEntries entries
  int test_batch_iterations;  // batch loops stop (with an error) after this many iterations
};

// Threads of a shading block. Shading waits for instructions about as much as
// for memory, so a block's warps start each path together (a barrier), and the
// classes with the most code run in large blocks: few places in the code at a
// time on an SM. The others keep LaunchConfig::shade_block (at most 128), which
// fits beside another wave's trace blocks. Against 128 threads for all, without
// the barrier: zoo 985x726 x 20 spp 13.7 -> 11.9 ms, zoo 333x217 x 48 spp 4.0 ->
// 3.6, textured 640x359 x 32 spp 4.8 -> 4.5; Cornell, displaced and eight spheres
// unchanged (640 threads: Cornell 1% slower; for all classes: displaced 6%).
constexpr int kShadeThreadsPerSm = 640;
constexpr bool large_code(int sc) {
  return sc == SC_GENERAL || sc == SC_TEXTURED || sc == SC_PLASTIC || sc == SC_DIELECTRIC;
}
constexpr int shade_threads(int sc) { return large_code(sc) ? 320 : 128; }

struct ShadeShape {
  int grid, block;
};
// For up to n paths of class sc: about twice the blocks that run at once.
inline ShadeShape shade_shape(int sc, int64_t n, const LaunchConfig& cfg) {
  const int block = large_code(sc) ? shade_threads(sc) : cfg.shade_block;
  const int64_t most = large_code(sc) ? (int64_t)cfg.num_sms * 2 * (kShadeThreadsPerSm / shade_threads(sc))
                                      : (int64_t)cfg.num_sms * cfg.blocks_per_sm * 2;
  int64_t g = (n + block - 1) / block;
  if (g > most) g = most;
  return ShadeShape{(int)(g < 1 ? 1 : g), block};
}

enum Stage { ST_CAMERA = 0, ST_TRACE_EXT, ST_SHADE, ST_TRACE_SHADOW, ST_TRACE_MIS, ST_RESOLVE, ST_FILM, ST_OTHER,
             kNumStages };

// Optional per-kernel timing: event pairs recorded around every launch.
struct StageTimer {
  cudaEvent_t* events;  // 2 * capacity events
  int* stage;           // capacity
  int capacity;
  int used;
  void begin(int st, cudaStream_t s) {
    if (used < capacity) {
      stage[used] = st;
      cudaEventRecord(events[2 * used], s);
    }
  }
  void end(cudaStream_t s) {
    if (used < capacity) cudaEventRecord(events[2 * used + 1], s);
    ++used;
  }
};

// One full wave: camera rays, then per bounce one trace of all waiting rays (its
// extension rays, the previous bounce's shadow and MIS rays) and the shading, then
// film accumulation. All on `stream`, no host sync.
// The film kernel first waits for `film_wait` (the film write of an earlier
// wave of the same pixels) and then records `film_done`.
void launch_wave(const SceneView& s, const WaveView& w, const WaveArgs& a, const FilmView& film,
                 const LaunchConfig& cfg, cudaStream_t stream, int* launches, StageTimer* timer = nullptr,
                 cudaEvent_t film_wait = nullptr, cudaEvent_t film_done = nullptr);

// Launch limits of the kernel families, and the dynamic shared-memory
// allowance of the traversal kernels (raised to `smem_bytes`, the device's
// opt-in maximum, so any accepted stack depth x block size can launch).
struct KernelLimits {
  int max_trace_block;  // threads per block the traversal kernels can launch with
  int max_shade_block;  // same for the kernels that LaunchConfig::shade_block applies to
};
cudaError_t configure_kernels(int smem_bytes, KernelLimits* lim);
cudaError_t configure_batch_kernels(int smem_bytes, KernelLimits* lim);

// Pooled batches: builds the body of the device-side loop (one iteration)
// into `body` by stream capture on `stream`. The loop keeps running while
// work or live paths remain; `cond` is the graph's while-condition handle.
// Shading kernels are launched for the classes in `class_mask` only.
cudaError_t capture_batch_iteration(const WaveView& w, const BatchView& b, const uint32_t* sobol,
                                    const LaunchConfig& cfg, unsigned class_mask, cudaGraphConditionalHandle cond,
                                    cudaStream_t stream, cudaGraph_t body);
// The same iteration launched directly (a host-driven loop reading ctl->more),
// each stage timed by `timer`: the profiling path of the pooled engine.
void launch_batch_iteration(const WaveView& w, const BatchView& b, const uint32_t* sobol, const LaunchConfig& cfg,
                            unsigned class_mask, cudaStream_t stream, StageTimer* timer);
// Wave mode: the work items [base, base + n) on slots 0..n-1, a plain wave's launches.
// _begin starts the paths. _bounces runs the bounces [from, to); `all` bounces (one more
// than the depth of the deepest job among them) end every path. _film adds the radiance of
// the n paths to their jobs' films; unfinished: -1, or the number of bounces run if paths
// may be left, which are then reported as kErrIterationCap.
struct BatchWave {
  const WaveView& w;
  const BatchView& b;
  const uint32_t* sobol;
  const LaunchConfig& cfg;
  unsigned class_mask;
  unsigned long long base;
  int n;
  cudaStream_t stream;
  int64_t* launches;   // added to
  StageTimer* timer;   // or null
};
void launch_batch_wave_begin(const BatchWave& wave);
void launch_batch_wave_bounces(const BatchWave& wave, int from, int to, int all);
void launch_batch_wave_film(const BatchWave& wave, int unfinished);
// dst[i] = (float)src[i] for i < n.
void launch_film_to_f32(const double* src, float* dst, long long n, int num_sms, cudaStream_t stream);
// Resets the batch control block and the free-slot list for `capacity` slots.
void launch_batch_init(const WaveView& w, const BatchView& b, int capacity, cudaStream_t stream);

// ------------------------------------------------------------------ SPPM
//
// Stochastic progressive photon mapping (src/integrator/sppm.cpp:58-322):
// per iteration a camera pass leaves one visible point per pixel, a hash
// grid over the visible points is built, a photon pass adds photon
// contributions to the visible points near each photon hit, and a per-pixel
// update shrinks the radii and adds the iteration's estimate to the film.

struct SppmGrid {
  float lo[3], hi[3];  // bounds of the visible points' spheres
  int res[3];
  float max_radius;
  int any;             // some pixel has a visible point
};

struct SppmView {
  int width, height, npix;
  int max_depth, iterations, photons;  // photons per iteration
  const uint32_t* sobol;               // Sobol tables (sobol_sample, dmath.cuh)
  // per pixel
  float4* vp_pr;    // visible point p, search radius (kept across iterations)
  float4* vp_wo;    // wo, material index (int bits; -1: no visible point)
  float4* vp_beta;  // beta, texture u
  float4* vp_ns;    // shading normal, texture v
  float4* vp_ng;    // geometric normal
  float4* vp_su;    // shading frame s
  float4* vp_sv;    // shading frame t
  float4* ld;       // direct light sum Ld, photon count N
  float4* tau;      // tau
  float* phi;       // 3 per pixel, photon flux of this iteration
  int* m;           // photons gathered this iteration
  SppmGrid* grid;
  float4* part_lo;  // per block of the bounds pass: lo, max radius
  float4* part_hi;  // hi, any
  // photon hits of this iteration: 3 float4 each (point + hash cell, wi, beta)
  float4* hits;
  int hits_cap;     // photons x (max depth - 1): every hit after a photon's first
  int* hit_count;
  DevMaterial* photon_mats;  // the scene's materials with DevLobe::photon set
  unsigned* photon_next;  // next photon to start (beside hit_count: cleared together)
  int num_sms;
  // hash cell -> photon hits: cell h holds records [cell_start[h], cell_start[h + 1]) of by_cell
  int* cell_start;  // npix + 1 (counts, then their exclusive scan)
  int* cell_fill;   // npix
  int* scan_part;   // per scan block
  float4* by_cell;  // the hits in hash-cell order, 3 float4 each (hits_cap)
  float* film;      // W*H*3 sums of the iterations' estimates
  unsigned* film_count;
  unsigned long long* rays;
};

// Whether the photons [base, base + count) that a warp took from photon_next reach
// the end of an iteration's `photons`. Every warp takes past the end once, at most 32
// photons: the counter is unsigned, so that it holds INT32_MAX photons and that of
// more warps than a launch has.
ORION_HD inline bool photons_dealt(unsigned base, unsigned count, int photons) {
  return base + count >= (unsigned)photons;
}

constexpr int kSppmBoundsBlocks = 1024;  // blocks of the bounds pass (part_lo / part_hi entries)
constexpr int kScanBlock = 1024;         // elements per block of the cell-count scan
constexpr int kScanRaw = 4 * kScanBlock;  // block sums up to which the scan needs no pass over them (k_scan_add)

// Resets per-pixel state (radius r0, no visible point) and the film, and
// fills photon_mats from the scene's materials.
void launch_sppm_init(const SppmView& v, float radius0, const DevMaterial* mats, int num_mats, cudaStream_t stream);
// Camera pass and the grid over the visible points of iteration `iter`.
void launch_sppm_visible_points(const SceneView& s, const SppmView& v, int iter, cudaStream_t stream);
// Exclusive scan of the cell counts (cell_start).
void launch_sppm_scan(const SppmView& v, cudaStream_t stream);
// Photon pass, photon lists by cell, gather at the visible points, pixel
// update and film. No host synchronisation between iterations.
void launch_sppm_photons(const SceneView& s, const SppmView& v, int iter, cudaStream_t stream);

// Averaged FP64 film (W*H*3 sums, W*H counts) -> W*H pixels of bytes B, G,
// R, 255 as saveAsBmp writes them; rows bottom-up when `bottom_up`.
void launch_film_preview(const double* sum, const uint32_t* count, int width, int height, int bottom_up,
                         uint8_t* bgra, cudaStream_t stream);

// Component hooks for the parity tests.
void launch_sobol(const uint32_t* sobol, int64_t n, const uint64_t* index, const uint32_t* dim, float* out,
                  cudaStream_t stream);
void launch_trace(const SceneView& s, int64_t n, const float* rays, int any_hit, float* t, float* u, float* v,
                  int* prim, const LaunchConfig& cfg, cudaStream_t stream);
// The same queries through the renderer's persistent trace kernels: the rays
// become wave `w`'s extension rays (closest hit) or shadow rays (any hit).
void launch_trace_wave(const SceneView& s, const WaveView& w, int n, const float* rays, int any_hit, float* t,
                       float* u, float* v, int* prim, const LaunchConfig& cfg, cudaStream_t stream);
void launch_camera_rays(const SceneView& s, const uint32_t* sobol, int64_t n, const int64_t* index, float* rays,
                        cudaStream_t stream);
void launch_bsdf_eval(const DevMaterial* mat, int64_t n, const float* frame, const float* wo, const float* wi,
                      const float* rnd, int type, float* f, float* pdf, float* sf, float* swi, float* spdf,
                      int* stype, int* nbxdf, cudaStream_t stream);

}  // namespace orion_gb300
