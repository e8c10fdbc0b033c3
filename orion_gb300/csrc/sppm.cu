// Stochastic progressive photon mapping (SPPM::render,
// src/integrator/sppm.cpp:58-322) on the GPU.
//
// One iteration is
//   k_sppm_camera    one lane per pixel: the camera path up to its first
//                    diffuse (or last glossy) hit, direct light at every hit
//                    (uniformSampleOneLight with uniform light choice,
//                    src/core/integrator.cpp:8-27), the visible point kept
//   k_sppm_bounds    bounds of the visible points' spheres, block partials
//   k_sppm_grid      the grid resolution (sppm.cpp:145-160)
//   k_sppm_photons   one lane per photon: Light::sample_Le, then a photon
//                    path with TransportMode::Photon BSDFs and throughput
//                    roulette; every hit after the first that falls inside
//                    the grid is recorded (point, wi, beta) and counted in
//                    its hash cell
//   k_scan_*         exclusive scan: each hash cell's first list entry
//   k_sppm_fill      the photon hits copied into hash-cell order
//   k_sppm_gather    one warp per visible point: for each hash cell its
//                    sphere overlaps, the recorded photons in that cell
//                    within its radius add beta * f(wi, wo) (sppm.cpp:226-247)
//   k_sppm_update    radius / N / tau update and the film (sppm.cpp:272-320)
// The reference walks, per photon hit, the visible points listed in the hit's
// hash cell; here each visible point walks the photon hits listed in the hash
// cells of its own sphere. Both consider a (visible point, photon) pair once
// per cell of the sphere whose hash equals the hash of the photon's cell, so
// the sums have the same terms; only their order differs. A visible point's
// material and frame are loaded once, and no flux atomics are needed.
// The camera and photon kernels hold all of the sampling and BSDF code, and
// with every warp at a place of its own they waited for instructions most of
// the time (12.2 and 10.5 cycles per issue, 10.0 and 4.2 of 32 lanes active,
// 1024x1024 pixels, 1M photons). So all lanes of a block go step by step together
// (trace, shade, shadow rays, ...: block barriers in between), rays are traced by
// whole warps (warp_trace, one copy of each traversal), and warps take new photons
// for those that ended: 2.8 and 6.6 cycles, 14.7 and 9.6 lanes, camera pass 2.01 ->
// 1.16 ms an iteration, photon pass 2.26 -> 1.34 ms, gather 3.84 -> 2.21 ms (see
// there). 512x512, 16 iterations of 262,144 photons: 28.4 -> 18.8 ms.
// Sample indices and dimensions follow the reference: the camera path of
// pixel (i, j) in iteration k uses index k*W*H + j*W + i, photon p uses
// iterations*W*H + k*photons + p, each from dimension 5.
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.h"
#include "shade.cuh"

namespace orion_gb300 {

namespace {

constexpr int kSppmBlock = 256;  // camera paths
constexpr int kPhotonBlock = 512;
constexpr int kSppmStack = 8;  // shared-memory traversal stack entries per thread

__device__ __forceinline__ void count_rays(unsigned long long* ctr, unsigned n) {
  const unsigned mask = __activemask();
  const unsigned total = __reduce_add_sync(mask, n);
  if ((int)(threadIdx.x & 31) == __ffs(mask) - 1) atomicAdd(ctr, (unsigned long long)total);
}

// The lobes of material `mi` at texture coordinates (x, y): the scene's
// record, or built at the hit for a textured material.
__device__ __forceinline__ const DevMaterial* material_at(const SceneView& s, int mi, float x, float y,
                                                          DevMaterial* tm) {
  if (s.mats[mi].shade_class != SC_TEXTURED) return &s.mats[mi];
  textured_material(s, mi, x, y, tm);
  return tm;
}

__device__ __forceinline__ int count_matching(const DevMaterial& m, int t) {
  int n = 0;
  for (int i = 0; i < m.num_lobes; ++i) n += (m.lobes[i].type & t) == m.lobes[i].type ? 1 : 0;
  return n;
}

// What a lane's path needs to trace: the scene's arrays and the block's shared
// memory (warp_trace).
struct Tracer {
  const SceneView& s;
  int2* smem;
  __device__ __forceinline__ RayHit closest(bool on, V3 o, V3 d) const {
    return warp_trace<false, kSppmStack>(s.nodes, s.woop, s.tri_prim, smem, on, o, d, 0.f);
  }
  __device__ __forceinline__ bool occluded(bool on, V3 o, V3 d, float tmax) const {
    return warp_trace<true, kSppmStack>(s.nodes, s.woop, s.tri_prim, smem, on, o, d, tmax).tri >= 0;
  }
};

// uniformSampleOneLight without a light distribution (integrator.cpp:8-27):
// the light chosen uniformly, estimateDirect (integrator.cpp:29-90) with
// its shadow and MIS rays traced here by the whole warp (lanes with nothing to
// shade pass on = false); returns estimateDirect / lightPdf.
__device__ V3 sppm_direct(const SceneView& s, const Tracer& tr, bool on, const DevMaterial& m, const Frame& fr,
                          const Hit& h, V3 rd, PathSampler& smp, unsigned* rays) {
  const int n = s.num_lights;
  if (n == 0) return V3{0, 0, 0};
  int li = 0;
  float a = 0.f, b = 0.f, c = 0.f, d = 0.f;
  if (on) {
    li = min((int)(smp.next() * n), n - 1);
    a = smp.next(), b = smp.next(), c = smp.next(), d = smp.next();  // next2(): .x is the later one
  }
  const float light_pdf = 1.f / n;
  const DevLight& lt = s.lights[li];
  const V3 wo = normalize(-rd);
  V3 Ld = V3{0, 0, 0}, part = V3{0, 0, 0}, o = V3{0, 0, 0}, dir = V3{0, 0, 1};
  bool want = false;
  if (on) {
    const LightSample ls = sample_li(lt, s.prims, s.envmaps, h.p, b, a, s.world_radius);
    if (ls.pdf > 0.f && !is_black(ls.Li)) {
      const V3 f = bsdf_f<kLobeAll>(m, fr, ls.wi, wo, kNonSpecular) * absdot(ls.wi, h.ns);
      const float bpdf = bsdf_pdf<kLobeAll>(m, fr, ls.wi, wo, kNonSpecular);
      if (!is_black(f)) {
        // ShadowTester::unoccluded (light.h:26-29): Intersection::spawnRay to a point.
        o = offset_ray_origin(h.p, h.ng, ls.p_light - h.p);
        dir = ls.p_light - o;
        want = true;
        ++*rays;
        if (is_delta_light(lt.kind))
          part = sdiv(mul(f, ls.Li), ls.pdf);
        else
          part = sdiv(mul(f, ls.Li) * power_heuristic(ls.pdf, bpdf), ls.pdf);
      }
    }
  }
  if (__syncthreads_or(want)) {
    const bool occ = tr.occluded(want, o, dir, 1.f - kShadowEpsilon);
    if (want && !occ) Ld = part;
  }
  bool want_mis = false, env = false;
  V3 fb = V3{0, 0, 0};
  float mis_pdf = 0.f, wgt = 0.f;
  if (on && !is_delta_light(lt.kind)) {
    int stype;
    fb = bsdf_sample_f<kLobeAll>(m, fr, wo, d, c, kNonSpecular, &dir, &mis_pdf, &stype);
    fb = fb * absdot(dir, h.ns);
    if (!is_black(fb) && mis_pdf > 0.f) {
      o = offset_ray_origin(h.p, h.ng, dir);
      env = lt.kind == DL_ENV;
      want_mis = true;
      if (env) {
        const float lpdf = env_pdf_li(lt, s.envmaps, dir);
        if (lpdf != 0.f)
          wgt = power_heuristic(mis_pdf, lpdf);
        else
          want_mis = false;
      }
      *rays += want_mis ? 1u : 0u;
    }
  }
  // Towards an area light the closest hit is needed; rays towards the
  // environment, for which any hit would do, go along.
  if (__syncthreads_or(want_mis)) {
    const RayHit mh = tr.closest(want_mis, o, dir);
    if (want_mis && env) {
      if (mh.tri < 0) Ld = Ld + sdiv(mul(fb, env_le(lt, s.envmaps, dir)) * wgt, mis_pdf);
    } else if (want_mis) {
      const int prim = mh.tri >= 0 ? __ldg(s.tri_prim + mh.tri) : -1;
      if (prim >= 0 && prim == lt.prim) {
        // Triangle::pdf (src/core/triangle.cpp:123-135) on the traced hit.
        const PrimShade& sh = s.prims[prim];
        const V3 ip = point_on(sh, mh.u, mh.v);
        const V3 ing = geometric_normal(sh);
        float lpdf = length_sq(h.p - ip) / (absdot(ing, -dir) * lt.area);
        if (isinf(lpdf)) lpdf = 0.f;
        if (lpdf != 0.f) {
          const float w = power_heuristic(mis_pdf, lpdf);
          const V3 Li = dot(ing, -dir) > 0.f ? ld3(lt.L) : V3{0, 0, 0};
          if (!is_black(Li)) Ld = Ld + sdiv(mul(fb, Li) * w, mis_pdf);
        }
      }
    }
  }
  return sdiv(Ld, light_pdf);
}

// Visible points (sppm.cpp:78-140). A warp follows the paths of 32
// neighbouring pixels (tile order) bounce by bounce, tracing their rays
// together.
__global__ void __launch_bounds__(kSppmBlock, 2) k_sppm_camera(SceneView s, SppmView v, int iter) {
  extern __shared__ int2 stack_smem[];
  const Tracer tr{s, stack_smem};
  const int pos = blockIdx.x * blockDim.x + threadIdx.x;
  const bool mine = pos < v.npix;
  bool on = mine;
  int i, j;
  tile_pixel(mine ? pos : 0, v.width, v.height, &i, &j);
  const int pix = v.width * j + i;
  PathSampler smp{v.sobol, (uint64_t)iter * v.npix + (uint64_t)v.width * j + i, 5u};
  V3 o, d;
  camera_ray(s.cam, smp, i, j, &o, &d);
  V3 beta = V3{1.f, 1.f, 1.f};
  bool specular = false;
  const float4 ld4 = v.ld[pix];
  V3 Ld = xyz(ld4);
  unsigned rays = 0;
  int vp_mat = -1;
  for (int depth = 0; depth < v.max_depth && __syncthreads_or(on); ++depth) {
    const RayHit rh = tr.closest(on, o, d);
    rays += on ? 1u : 0u;
    if (on && rh.tri < 0) {
      for (int e = 0; e < s.num_env; ++e) Ld = Ld + mul(beta, env_le(s.lights[s.env_idx[e]], s.envmaps, d));
      on = false;
    }
    if (!__syncthreads_or(on)) break;
    // Lanes without a hit go along with primitive 0's record (nothing of it is used).
    const int prim = on ? __ldg(s.tri_prim + rh.tri) : 0;
    const PrimShade& sh = s.prims[prim];
    const Hit h = reconstruct(sh, rh.u, rh.v);
    const int mi = sh.material;
    float tu = 0.f, tv = 0.f;
    if (on && s.prim_uv) hit_uv(s.prim_uv + 6 * (size_t)prim, rh.u, rh.v, &tu, &tv);
    DevMaterial tm;
    const DevMaterial& m = *(on ? material_at(s, mi, tu, tv, &tm) : &s.mats[mi]);
    const Frame fr{h.ng, h.ns, h.su, h.sv};
    const V3 wo = -d;
    if (on && (depth == 0 || specular)) {
      const int li = sh.light;
      if (li >= 0 && dot(h.ng, wo) > 0.f) Ld = Ld + mul(beta, ld3(s.lights[li].L));
    }
    const V3 direct = sppm_direct(s, tr, on, m, fr, h, d, smp, &rays);
    if (!on) continue;
    Ld = Ld + mul(beta, direct);
    const bool diffuse = count_matching(m, BXDF_DIFFUSE | BXDF_REFLECTION | BXDF_TRANSMISSION) > 0;
    const bool glossy = count_matching(m, BXDF_GLOSSY | BXDF_REFLECTION | BXDF_TRANSMISSION) > 0;
    if (diffuse || (glossy && depth == v.max_depth - 1)) {
      if (!is_black(beta)) {
        vp_mat = mi;
        v.vp_pr[pix] = f4(h.p, v.vp_pr[pix].w);
        v.vp_wo[pix] = f4(wo, __int_as_float(mi));
        v.vp_beta[pix] = f4(beta, tu);
        v.vp_ns[pix] = f4(h.ns, tv);
        v.vp_ng[pix] = f4(h.ng, 0.f);
        v.vp_su[pix] = f4(h.su, 0.f);
        v.vp_sv[pix] = f4(h.sv, 0.f);
      }
      on = false;
    } else if (depth < v.max_depth - 1) {
      const float a = smp.next(), b = smp.next();
      V3 wi;
      float pdf = 0.f;
      int stype = 0;
      const V3 f = bsdf_sample_f<kLobeAll>(m, fr, wo, b, a, BXDF_ALL, &wi, &pdf, &stype);
      if (pdf == 0.f || is_black(f)) {
        on = false;
      } else {
        specular = (stype & BXDF_SPECULAR) != 0;
        beta = mul(beta, sdiv(f * absdot(wi, h.ns), pdf));
        const float y = spectrum_intensity(beta);
        if (y < 0.25f) {
          const float cont = fminf(1.f, y);
          if (smp.next() > cont)
            on = false;
          else
            beta = sdiv(beta, cont);
        }
        o = offset_ray_origin(h.p, h.ng, wi);
        d = wi;
      }
    }
  }
  if (mine) {
    v.ld[pix] = f4(Ld, ld4.w);
    if (vp_mat < 0) v.vp_wo[pix].w = __int_as_float(-1);
  }
  count_rays(v.rays, rays);
}

__device__ __forceinline__ bool has_vp(const SppmView& v, int pix) { return __float_as_int(v.vp_wo[pix].w) >= 0; }

// Bounds of every visible point's sphere and the largest radius: one
// partial per block.
__global__ void __launch_bounds__(256) k_sppm_bounds(SppmView v) {
  __shared__ float red[8][256];
  float lo[3] = {kFloatMax, kFloatMax, kFloatMax}, hi[3] = {-kFloatMax, -kFloatMax, -kFloatMax}, mr = 0.f, any = 0.f;
  for (int pix = blockIdx.x * blockDim.x + threadIdx.x; pix < v.npix; pix += gridDim.x * blockDim.x) {
    if (!has_vp(v, pix)) continue;
    const float4 pr = v.vp_pr[pix];
    const float p[3] = {pr.x, pr.y, pr.z};
    for (int k = 0; k < 3; ++k) {
      const float a = p[k] - pr.w, b = p[k] + pr.w;  // expand(Bounds3f(p), radius)
      lo[k] = a < lo[k] ? a : lo[k];
      hi[k] = b > hi[k] ? b : hi[k];
    }
    mr = pr.w > mr ? pr.w : mr;
    any = 1.f;
  }
  const int t = threadIdx.x;
  red[0][t] = lo[0], red[1][t] = lo[1], red[2][t] = lo[2];
  red[3][t] = hi[0], red[4][t] = hi[1], red[5][t] = hi[2];
  red[6][t] = mr, red[7][t] = any;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (t < w) {
      for (int k = 0; k < 3; ++k) red[k][t] = fminf(red[k][t], red[k][t + w]);
      for (int k = 3; k < 8; ++k) red[k][t] = fmaxf(red[k][t], red[k][t + w]);
    }
    __syncthreads();
  }
  if (t == 0) {
    v.part_lo[blockIdx.x] = make_float4(red[0][0], red[1][0], red[2][0], red[6][0]);
    v.part_hi[blockIdx.x] = make_float4(red[3][0], red[4][0], red[5][0], red[7][0]);
  }
}

// The grid over the visible points (sppm.cpp:145-160), from the partials.
__global__ void __launch_bounds__(256) k_sppm_grid(SppmView v, int nparts) {
  __shared__ float red[8][256];
  const int t = threadIdx.x;
  float r[8] = {kFloatMax, kFloatMax, kFloatMax, -kFloatMax, -kFloatMax, -kFloatMax, 0.f, 0.f};
  for (int b = t; b < nparts; b += blockDim.x) {
    const float4 l = v.part_lo[b], h = v.part_hi[b];
    r[0] = fminf(r[0], l.x), r[1] = fminf(r[1], l.y), r[2] = fminf(r[2], l.z);
    r[3] = fmaxf(r[3], h.x), r[4] = fmaxf(r[4], h.y), r[5] = fmaxf(r[5], h.z);
    r[6] = fmaxf(r[6], l.w), r[7] = fmaxf(r[7], h.w);
  }
  for (int k = 0; k < 8; ++k) red[k][t] = r[k];
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (t < w) {
      for (int k = 0; k < 3; ++k) red[k][t] = fminf(red[k][t], red[k][t + w]);
      for (int k = 3; k < 8; ++k) red[k][t] = fmaxf(red[k][t], red[k][t + w]);
    }
    __syncthreads();
  }
  if (t == 0) {
    SppmGrid g;
    for (int k = 0; k < 3; ++k) {
      g.lo[k] = red[k][0];
      g.hi[k] = red[k + 3][0];
    }
    g.max_radius = red[6][0];
    g.any = red[7][0] != 0.f;
    g.res[0] = g.res[1] = g.res[2] = 1;
    if (g.any) {
      const float diag[3] = {g.hi[0] - g.lo[0], g.hi[1] - g.lo[1], g.hi[2] - g.lo[2]};
      const float max_diag = fmaxf(diag[0], fmaxf(diag[1], diag[2]));
      const int base = __float2int_rz(max_diag / g.max_radius);
      for (int k = 0; k < 3; ++k) g.res[k] = max(__float2int_rz(__fmul_rn((float)base, diag[k]) / max_diag), 1);
    }
    *v.grid = g;
  }
}

// ToGrid (sppm.cpp:41-51): Bounds3::offset, then the truncated cell, clamped.
__device__ __forceinline__ bool to_grid(const SppmGrid& g, V3 p, int* c) {
  float o[3] = {p.x - g.lo[0], p.y - g.lo[1], p.z - g.lo[2]};
  bool in = true;
  for (int k = 0; k < 3; ++k) {
    if (g.hi[k] > g.lo[k]) o[k] = o[k] / (g.hi[k] - g.lo[k]);
    int ck = __float2int_rz(__fmul_rn((float)g.res[k], o[k]));
    in = in && ck >= 0 && ck < g.res[k];
    c[k] = min(max(ck, 0), g.res[k] - 1);
  }
  return in;
}

// hash (sppm.cpp:53-57), the products modulo 2^32.
__device__ __forceinline__ unsigned cell_hash(int x, int y, int z, int size) {
  return (((unsigned)x * 73856093u) ^ ((unsigned)y * 19349663u) ^ ((unsigned)z * 83492791u)) % (unsigned)size;
}

// Copies the recorded photon hits into hash-cell order (cell_start holds
// each cell's first entry after the scan), so a gather reads a cell's hits
// from consecutive records.
__global__ void __launch_bounds__(256) k_sppm_fill(SppmView v) {
  const unsigned n = (unsigned)min(*v.hit_count, v.hits_cap);  // up to INT32_MAX: i goes past it by a stride
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float4* src = v.hits + 3 * (size_t)i;
    const float4 a = src[0], b = src[1], c = src[2];
    const unsigned h = (unsigned)__float_as_int(a.w);
    float4* dst = v.by_cell + 3 * (size_t)(v.cell_start[h] + atomicAdd(v.cell_fill + h, 1));
    dst[0] = a;
    dst[1] = b;
    dst[2] = c;
  }
}

// Photon flux at each visible point (sppm.cpp:226-247, seen from the visible
// point): the cells its sphere overlaps (sppm.cpp:167-190), the photon hits
// listed under each cell's hash, those within the radius. One warp per
// visible point: the lanes look up the cells (at most 27) at once, then take
// the hits of all cells as one list, and the hits within the radius are
// collected 32 at a time before their BSDF is evaluated, so lanes idle neither
// in short cells nor over the hits outside the sphere (1024x1024 pixels, 1M photons:
// 3.84 -> 2.21 ms against cell after cell, each hit's BSDF where it is found; 2,582M
// -> 1,543M warp instructions, 19.5 -> 30.1 of 32 lanes).
// Every lane runs the same material's BSDF, inline for the diffuse class; the
// lanes' sums are added at the end. The counts of 32 cells are summed in an int:
// where one is above kGatherTogether (films of few pixels, whose few hash cells hold
// many hits and turn up several times in one sphere) the cells go one by one.
constexpr int kGatherWarps = 4;
constexpr int kGatherTogether = 1 << 14;
static_assert(32LL * kGatherTogether <= INT32_MAX, "the counts of a warp's cells are added up in an int");

template <unsigned KM>
__device__ __forceinline__ void gather_photons(const SppmView& v, const DevMaterial& m, const Frame& fr, V3 p, V3 wo,
                                               float rr, const int lo[3], const int hi[3], int* queue, V3* phi_out,
                                               int* count_out) {
  constexpr unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int nx = hi[0] - lo[0] + 1, ny = hi[1] - lo[1] + 1, cells = nx * ny * (hi[2] - lo[2] + 1);
  V3 phi = V3{0, 0, 0};
  int count = 0, queued = 0;
  auto evaluate = [&](int n) {  // the first n queued hits
    if (lane < n) {
      const float4* rec = v.by_cell + 3 * (size_t)queue[lane];
      const float4 wi4 = rec[1], hb = rec[2];
      phi = phi + mul(xyz(hb), bsdf_f<KM>(m, fr, xyz(wi4), wo, BXDF_ALL));
      ++count;
    }
  };
  for (int c0 = 0; c0 < cells;) {
    const int c = c0 + lane;
    int start = 0, in_cell = 0;
    if (c < cells) {
      const int z = c / (nx * ny), y = (c - z * nx * ny) / nx, x = c - (z * ny + y) * nx;
      const unsigned h = cell_hash(lo[0] + x, lo[1] + y, lo[2] + z, v.npix);
      start = v.cell_start[h];
      in_cell = v.cell_start[h + 1] - start;
    }
    const bool alone = __any_sync(kFull, in_cell > kGatherTogether);  // the first cell only
    if (alone && lane > 0) in_cell = 0;
    c0 += alone ? 1 : 32;
    int incl = in_cell;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += y;
    }
    const unsigned total = __shfl_sync(kFull, incl, 31), before = incl - in_cell;
    for (unsigned e0 = 0; e0 < total; e0 += 32) {
      const unsigned e = e0 + lane;
      int cell = 0;  // the last lane whose hits begin at or before e
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const unsigned at = __shfl_sync(kFull, before, cell + step);
        if (at <= e) cell += step;
      }
      const int idx = __shfl_sync(kFull, start, cell) + (int)(e - __shfl_sync(kFull, before, cell));
      const bool in = e < total && !(length_sq(p - xyz(v.by_cell[3 * (size_t)idx])) > rr);
      const unsigned hits = __ballot_sync(kFull, in);
      if (in) queue[queued + __popc(hits & ((1u << lane) - 1u))] = idx;
      queued += __popc(hits);
      __syncwarp();
      if (queued >= 32) {
        evaluate(32);
        queued -= 32;
        const int rest = queue[32 + lane];
        __syncwarp();
        queue[lane] = rest;
        __syncwarp();
      }
    }
  }
  evaluate(queued);
  *phi_out = phi;
  *count_out = count;
}

__global__ void __launch_bounds__(32 * kGatherWarps, 8) k_sppm_gather(SceneView s, SppmView v) {
  __shared__ int queues[kGatherWarps][64];
  const int pos = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (pos >= v.npix) return;  // uniform across the warp
  int px, py;
  tile_pixel(pos, v.width, v.height, &px, &py);
  const int pix = v.width * py + px;
  if (!has_vp(v, pix)) return;
  const SppmGrid g = *v.grid;
  const float4 pr = v.vp_pr[pix], wo4 = v.vp_wo[pix], b4 = v.vp_beta[pix], ns4 = v.vp_ns[pix];
  const V3 p = xyz(pr), wo = xyz(wo4), r = V3{pr.w, pr.w, pr.w};
  const float rr = pr.w * pr.w;
  const int mi = __float_as_int(wo4.w);
  DevMaterial vm;
  const DevMaterial& m = *material_at(s, mi, b4.w, ns4.w, &vm);
  const Frame fr{xyz(v.vp_ng[pix]), xyz(ns4), xyz(v.vp_su[pix]), xyz(v.vp_sv[pix])};
  int lo[3], hi[3];
  to_grid(g, p - r, lo);
  to_grid(g, p + r, hi);
  V3 phi;
  int count;
  if (s.mats[mi].shade_class == SC_DIFFUSE)
    gather_photons<lobes_of_class(SC_DIFFUSE)>(v, m, fr, p, wo, rr, lo, hi, queues[threadIdx.x >> 5], &phi, &count);
  else
    gather_photons<kLobeAll>(v, m, fr, p, wo, rr, lo, hi, queues[threadIdx.x >> 5], &phi, &count);
  for (int off = 16; off > 0; off >>= 1) {
    phi.x += __shfl_xor_sync(0xffffffffu, phi.x, off);
    phi.y += __shfl_xor_sync(0xffffffffu, phi.y, off);
    phi.z += __shfl_xor_sync(0xffffffffu, phi.z, off);
    count += __shfl_xor_sync(0xffffffffu, count, off);
  }
  if (lane == 0) {
    float* ph = v.phi + 3 * (size_t)pix;
    ph[0] = phi.x;
    ph[1] = phi.y;
    ph[2] = phi.z;
    v.m[pix] = count;
  }
}

// Exclusive scan of n ints in place: per-block scans, a scan of the block
// sums, and the block offsets added back.
__global__ void __launch_bounds__(kScanBlock) k_scan_blocks(int* a, int n, int* part) {
  __shared__ int buf[kScanBlock];
  const int t = threadIdx.x, i = blockIdx.x * kScanBlock + t;
  const int x = i < n ? a[i] : 0;
  buf[t] = x;
  __syncthreads();
  for (int off = 1; off < kScanBlock; off <<= 1) {
    const int y = t >= off ? buf[t - off] : 0;
    __syncthreads();
    buf[t] += y;
    __syncthreads();
  }
  if (i < n) a[i] = buf[t] - x;
  if (t == kScanBlock - 1) part[blockIdx.x] = buf[t];
}

__global__ void __launch_bounds__(kScanBlock) k_scan_parts(int* part, int nparts) {
  __shared__ int buf[kScanBlock];
  __shared__ int carry;
  const int t = threadIdx.x;
  if (t == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < nparts; base += kScanBlock) {
    const int i = base + t;
    const int x = i < nparts ? part[i] : 0;
    buf[t] = x;
    __syncthreads();
    for (int off = 1; off < kScanBlock; off <<= 1) {
      const int y = t >= off ? buf[t - off] : 0;
      __syncthreads();
      buf[t] += y;
      __syncthreads();
    }
    if (i < nparts) part[i] = carry + buf[t] - x;
    __syncthreads();
    if (t == kScanBlock - 1) carry += buf[t];
    __syncthreads();
  }
}

// raw: `part` holds the blocks' sums, not their scan: each block adds up those
// before it itself (one launch less, while there are at most kScanRaw).
__global__ void __launch_bounds__(kScanBlock) k_scan_add(int* a, int n, const int* part, int raw) {
  __shared__ int warp_sum[32];
  const int i = blockIdx.x * kScanBlock + threadIdx.x;
  int before = 0;
  if (raw) {
    for (int k = threadIdx.x; k < blockIdx.x; k += kScanBlock) before += part[k];
    before = (int)__reduce_add_sync(0xffffffffu, (unsigned)before);
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = before;
    __syncthreads();
    before = (int)__reduce_add_sync(0xffffffffu, (unsigned)warp_sum[threadIdx.x & 31]);
  } else {
    before = part[blockIdx.x];
  }
  if (i < n) a[i] += before;
}

// Photons (sppm.cpp:197-270). Warps stay in the loop: each turn traces one
// ray of every lane's photon together, and lanes whose photon has ended take
// the next one once fewer than kPhotonRefill still hold one.
constexpr int kPhotonRefill = 24;

__global__ void __launch_bounds__(kPhotonBlock, 2) k_sppm_photons(SceneView s, SppmView v, int iter) {
  extern __shared__ int2 stack_smem[];
  constexpr unsigned kFull = 0xffffffffu;
  const Tracer tr{s, stack_smem};
  const SppmGrid g = *v.grid;
  if (!g.any) return;
  const int lane = threadIdx.x & 31;
  const LightDistrib distrib{s.light_func, s.light_cdf, s.light_func_int, s.num_lights};
  PathSampler smp{v.sobol, 0ull, 5u};
  V3 beta = V3{0, 0, 0}, o = V3{0, 0, 0}, dir = V3{0, 0, 1};
  int depth = 0;
  unsigned rays = 0;
  bool on = false, exhausted = v.max_depth <= 0;
  while (true) {
    const unsigned act = __ballot_sync(kFull, on);
    if (!exhausted && __popc(act) < kPhotonRefill) {
      const unsigned cnt = 32 - __popc(act);
      unsigned base = 0;
      if (lane == 0) base = atomicAdd(v.photon_next, cnt);
      base = __shfl_sync(kFull, base, 0);
      exhausted = photons_dealt(base, cnt, v.photons);
      const unsigned k = base + __popc(~act & ((1u << lane) - 1u));
      if (!on && k < (unsigned)v.photons) {
        smp.index = (uint64_t)v.iterations * v.npix + (uint64_t)iter * v.photons + (uint64_t)k;
        smp.dim = 5u;
        float light_pdf;
        const int ln = sample_discrete(distrib, smp.next(), &light_pdf);
        const float a = smp.next(), b = smp.next(), c = smp.next(), d = smp.next();  // next2(): .x is the later one
        const EmittedRay e = sample_le(s.lights[ln], s.prims, s.envmaps, s.world_center, s.world_radius, b, a, d, c);
        if (!(e.pdf_pos == 0.f || e.pdf_dir == 0.f || is_black(e.Le))) {
          beta = sdiv(absdot(e.n, e.d) * e.Le, light_pdf * e.pdf_pos * e.pdf_dir);
          if (!is_black(beta)) {
            o = e.o, dir = e.d;
            depth = 0;
            on = true;
          }
        }
      }
    }
    if (!__syncthreads_or(on || !exhausted)) break;
    const RayHit rh = tr.closest(on, o, dir);
    __syncthreads();
    if (!on) continue;
    ++rays;
    if (rh.tri < 0) {
      on = false;
      continue;
    }
    const int prim = __ldg(s.tri_prim + rh.tri);
    const PrimShade& sh = s.prims[prim];
    const Hit h = reconstruct(sh, rh.u, rh.v);
    if (depth > 0) {  // recorded for the gather when inside the grid (sppm.cpp:226-229)
      int cell[3];
      const bool in = to_grid(g, h.p, cell);
      const unsigned hc = in ? cell_hash(cell[0], cell[1], cell[2], v.npix) : 0u;
      const unsigned want = __ballot_sync(__activemask(), in);
      if (in) {
        const int leader = __ffs(want) - 1;
        int base = 0;
        if (lane == leader) base = atomicAdd(v.hit_count, __popc(want));
        base = __shfl_sync(want, base, leader);
        const int slot = base + __popc(want & ((1u << lane) - 1u));
        if (slot < v.hits_cap) {
          float4* rec = v.hits + 3 * (size_t)slot;
          rec[0] = f4(h.p, __int_as_float((int)hc));
          rec[1] = f4(-dir, 0.f);
          rec[2] = f4(beta, 0.f);
          atomicAdd(v.cell_start + hc, 1);
        }
      }
    }
    // Intersection::calculateBSDF(TransportMode::Photon)
    const int mi = sh.material;
    float tu = 0.f, tv = 0.f;
    if (s.prim_uv) hit_uv(s.prim_uv + 6 * (size_t)prim, rh.u, rh.v, &tu, &tv);
    DevMaterial tm;
    const DevMaterial* pm = v.photon_mats + mi;
    if (pm->shade_class == SC_TEXTURED) {
      textured_material(s, mi, tu, tv, &tm);
      for (int l = 0; l < tm.num_lobes; ++l) tm.lobes[l].photon = 1;
      pm = &tm;
    }
    const Frame fr{h.ng, h.ns, h.su, h.sv};
    const float u1 = smp.next(), u0 = smp.next();
    V3 wi;
    float pdf = 0.f;
    int stype = 0;
    const V3 f = bsdf_sample_f<kLobeAll>(*pm, fr, -dir, u0, u1, BXDF_ALL, &wi, &pdf, &stype);
    if (is_black(f) || pdf == 0.f) {
      on = false;
      continue;
    }
    const V3 bnew = sdiv(mul(beta, f) * absdot(wi, h.ns), pdf);
    const float q = fmaxf(0.f, 1.f - spectrum_intensity(bnew) / spectrum_intensity(beta));
    if (smp.next() < q) {
      on = false;
      continue;
    }
    beta = sdiv(bnew, 1.f - q);
    o = offset_ray_origin(h.p, h.ng, wi);
    dir = wi;
    on = ++depth < v.max_depth;
  }
  count_rays(v.rays, rays);
}

// Empties hash cell `pix` (there are as many as pixels) and the photon counters.
__device__ __forceinline__ void clear_cells(const SppmView& v, int pix) {
  v.cell_start[pix] = 0;
  v.cell_fill[pix] = 0;
  if (pix == 0) {
    v.cell_start[v.npix] = 0;
    *v.hit_count = 0;
    *v.photon_next = 0u;
  }
}

// Pixel update and film (sppm.cpp:272-320), in the reference's operation
// order without contraction.
__global__ void __launch_bounds__(256) k_sppm_update(SppmView v) {
  const int pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= v.npix) return;
  float4 pr = v.vp_pr[pix];
  float4 ld4 = v.ld[pix];
  float4 tau4 = v.tau[pix];
  const int M = v.m[pix];
  if (M > 0) {
    const float gamma = 2.f / 3.f;
    const float N = ld4.w, r = pr.w;
    const float n_new = __fadd_rn(N, __fmul_rn(gamma, (float)M));
    const float r_new = __fmul_rn(r, __fsqrt_rn(__fdiv_rn(n_new, __fadd_rn(N, (float)M))));
    const float4 b4 = v.vp_beta[pix];
    const float* ph = v.phi + 3 * (size_t)pix;
    const float rr_new = __fmul_rn(r_new, r_new), rr = __fmul_rn(r, r);
    tau4.x = __fdiv_rn(__fmul_rn(__fadd_rn(tau4.x, __fmul_rn(b4.x, ph[0])), rr_new), rr);
    tau4.y = __fdiv_rn(__fmul_rn(__fadd_rn(tau4.y, __fmul_rn(b4.y, ph[1])), rr_new), rr);
    tau4.z = __fdiv_rn(__fmul_rn(__fadd_rn(tau4.z, __fmul_rn(b4.z, ph[2])), rr_new), rr);
    ld4.w = n_new;
    pr.w = r_new;
    v.m[pix] = 0;
    v.phi[3 * (size_t)pix] = v.phi[3 * (size_t)pix + 1] = v.phi[3 * (size_t)pix + 2] = 0.f;
    v.vp_pr[pix] = pr;
    v.ld[pix] = ld4;
    v.tau[pix] = tau4;
  }
  v.vp_wo[pix].w = __int_as_float(-1);  // the visible point is cleared
  const float np = (float)((unsigned long long)v.iterations * (unsigned long long)v.photons);
  const float den = __fmul_rn(__fmul_rn(__fmul_rn(np, kPi), pr.w), pr.w);
  const float fi = (float)v.iterations;
  float* f = v.film + 3 * (size_t)pix;
  f[0] = __fadd_rn(f[0], __fadd_rn(__fdiv_rn(ld4.x, fi), __fdiv_rn(tau4.x, den)));
  f[1] = __fadd_rn(f[1], __fadd_rn(__fdiv_rn(ld4.y, fi), __fdiv_rn(tau4.y, den)));
  f[2] = __fadd_rn(f[2], __fadd_rn(__fdiv_rn(ld4.z, fi), __fdiv_rn(tau4.z, den)));
  v.film_count[pix] += 1u;
  clear_cells(v, pix);  // for the next iteration's photons
}

// Also the materials as photons see them (TransportMode::Photon).
__global__ void k_sppm_init(SppmView v, float radius0, const DevMaterial* mats, int num_mats) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < num_mats; i += gridDim.x * blockDim.x) {
    DevMaterial m = mats[i];
    for (int l = 0; l < kMaxLobes; ++l) m.lobes[l].photon = 1;
    v.photon_mats[i] = m;
  }
  for (int pix = blockIdx.x * blockDim.x + threadIdx.x; pix < v.npix; pix += gridDim.x * blockDim.x) {
    v.vp_pr[pix] = make_float4(0.f, 0.f, 0.f, radius0);
    v.vp_wo[pix] = make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
    v.ld[pix] = make_float4(0.f, 0.f, 0.f, 0.f);
    v.tau[pix] = make_float4(0.f, 0.f, 0.f, 0.f);
    v.phi[3 * (size_t)pix] = v.phi[3 * (size_t)pix + 1] = v.phi[3 * (size_t)pix + 2] = 0.f;
    v.m[pix] = 0;
    v.film[3 * (size_t)pix] = v.film[3 * (size_t)pix + 1] = v.film[3 * (size_t)pix + 2] = 0.f;
    v.film_count[pix] = 0u;
    clear_cells(v, pix);
  }
}

int blocks_for(int64_t n, int block) { return (int)((n + block - 1) / block); }

}  // namespace

void launch_sppm_init(const SppmView& v, float radius0, const DevMaterial* mats, int num_mats, cudaStream_t stream) {
  k_sppm_init<<<std::min(blocks_for(v.npix, 256), 4096), 256, 0, stream>>>(v, radius0, mats, num_mats);
}

// Threads per block for n paths: as few (whole warps) as spread them over all
// SMs four times, at most `most`. Full launches want large blocks (few places
// in the code at a time), small ones many: 512x512 pixels 4.8 ms at 256 threads
// against 5.6 at 64, 128x128 pixels 3.5 against 3.1.
static int sppm_block(int64_t n, int num_sms, int most) {
  const int64_t per_sm = (n + 4LL * num_sms - 1) / (4LL * num_sms);
  return (int)std::min<int64_t>(most, (per_sm + 31) / 32 * 32);
}

void launch_sppm_visible_points(const SceneView& s, const SppmView& v, int iter, cudaStream_t stream) {
  const int block = sppm_block(v.npix, v.num_sms, kSppmBlock);
  k_sppm_camera<<<blocks_for(v.npix, block), block, trace_smem_bytes(kSppmStack, block), stream>>>(s, v, iter);
  const int parts = std::min(blocks_for(v.npix, 256), kSppmBoundsBlocks);
  k_sppm_bounds<<<parts, 256, 0, stream>>>(v);
  k_sppm_grid<<<1, 256, 0, stream>>>(v, parts);
}

void launch_sppm_scan(const SppmView& v, cudaStream_t stream) {
  const int n = v.npix + 1;
  const int nb = blocks_for(n, kScanBlock);
  k_scan_blocks<<<nb, kScanBlock, 0, stream>>>(v.cell_start, n, v.scan_part);
  const bool raw = nb <= kScanRaw;
  if (!raw) k_scan_parts<<<1, kScanBlock, 0, stream>>>(v.scan_part, nb);
  if (nb > 1) k_scan_add<<<nb, kScanBlock, 0, stream>>>(v.cell_start, n, v.scan_part, raw ? 1 : 0);
}

void launch_sppm_photons(const SceneView& s, const SppmView& v, int iter, cudaStream_t stream) {
  if (v.photons > 0) {
    const int block = sppm_block(v.photons, v.num_sms, kPhotonBlock);
    const int grid = std::min(blocks_for(v.photons, block), 1024 / block * v.num_sms);
    k_sppm_photons<<<grid, block, trace_smem_bytes(kSppmStack, block), stream>>>(s, v, iter);
  }
  launch_sppm_scan(v, stream);
  k_sppm_fill<<<std::min(blocks_for(v.hits_cap, 256), 8192), 256, 0, stream>>>(v);
  k_sppm_gather<<<blocks_for(v.npix, kGatherWarps), 32 * kGatherWarps, 0, stream>>>(s, v);
  k_sppm_update<<<blocks_for(v.npix, 256), 256, 0, stream>>>(v);
}

}  // namespace orion_gb300
