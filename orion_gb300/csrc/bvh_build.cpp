// Binned-SAH BVH build on the host, flattened for the GPU.
//
// Replaces the acceleration structure the reference builds inside Embree
// (EmbreeKernel::build, src/core/kernel.cpp:63-110): one static triangle set
// in primID order. Output layout:
//   * 32-byte nodes (BvhNode); the children of an inner node are an
//     adjacent pair, so one 64-byte fetch gives both child boxes;
//   * optionally the first `top_bfs_nodes` slots hold the top levels in
//     breadth-first order (so a kernel can stage them in shared memory),
//     the rest of each subtree follows depth-first for locality;
//   * Woop unit-triangle records (3 x float4 = 48 bytes) in leaf order, and
//     the leaf-order -> primID map.
// Subtrees are built on worker threads.
#include "bvh_build.h"

#include "host_parallel.h"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <condition_variable>
#include <cstring>
#include <deque>
#include <limits>
#include <memory>
#include <mutex>
#include <thread>

namespace orion_gb300 {

void woop_record(const float* p, float out[12]) {
  double v0[3] = {p[0], p[1], p[2]};
  double a[3] = {(double)p[3] - p[0], (double)p[4] - p[1], (double)p[5] - p[2]};  // e1
  double b[3] = {(double)p[6] - p[0], (double)p[7] - p[1], (double)p[8] - p[2]};  // e2
  double c[3] = {a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]};  // n
  auto cross = [](const double* x, const double* y, double* r) {
    r[0] = x[1] * y[2] - x[2] * y[1];
    r[1] = x[2] * y[0] - x[0] * y[2];
    r[2] = x[0] * y[1] - x[1] * y[0];
  };
  double bc[3], ca[3], ab[3];
  cross(b, c, bc);
  cross(c, a, ca);
  cross(a, b, ab);
  double det = a[0] * bc[0] + a[1] * bc[1] + a[2] * bc[2];
  if (!(std::fabs(det) > 0.0) || !std::isfinite(det)) {
    std::memset(out, 0, 12 * sizeof(float));
    return;
  }
  double r0[3], r1[3], r2[3];
  for (int k = 0; k < 3; ++k) {
    r0[k] = bc[k] / det;  // row giving u (along e1)
    r1[k] = ca[k] / det;  // row giving v (along e2)
    r2[k] = ab[k] / det;  // row giving the offset along n
  }
  // Origin-relative form: the fourth components hold v0, and the kernel
  // works with C = o - v0, so t = -(r2.C) / (r2.d), u = r0.C + t r0.d,
  // v = r1.C + t r1.d. Subtracting v0 first keeps t accurate for ray
  // origins close to the triangle's plane (every secondary ray).
  out[0] = (float)r2[0];
  out[1] = (float)r2[1];
  out[2] = (float)r2[2];
  out[3] = (float)v0[0];
  out[4] = (float)r0[0];
  out[5] = (float)r0[1];
  out[6] = (float)r0[2];
  out[7] = (float)v0[1];
  out[8] = (float)r1[0];
  out[9] = (float)r1[1];
  out[10] = (float)r1[2];
  out[11] = (float)v0[2];
}

namespace {

struct TmpNode {
  float lo[3], hi[3];
  int32_t begin = 0, count = 0;  // leaf range in the reference array
  int32_t first = 0, total = 0;  // the subtree's triangles: refs[first, first + total)
  TmpNode* child[2] = {nullptr, nullptr};
  int depth = 0;
};

// Four floats worked on together (the compiler's vector type, SSE or NEON).
// vmin / vmax pick lane by lane exactly what std::min / std::max (box, x) do.
typedef float V4 __attribute__((vector_size(16)));
typedef int32_t I4 __attribute__((vector_size(16)));

inline V4 vmin(V4 box, V4 x) { return x < box ? x : box; }
inline V4 vmax(V4 box, V4 x) { return box < x ? x : box; }
inline V4 splat(float f) { return V4{f, f, f, f}; }

// One triangle's box and id, 32 bytes. The build partitions these records
// themselves (not indices into per-triangle arrays), so every scan of a
// range reads memory in order. The id sits in the fourth lanes as two exact
// small floats, so that no lane ever holds a denormal or a NaN of its own.
struct PrimRef {
  V4 lo, hi;
  void set_id(int32_t id) {
    lo[3] = (float)(id & 0x7fffff);
    hi[3] = (float)(id >> 23);
  }
  int32_t id() const { return (int32_t)lo[3] | ((int32_t)hi[3] << 23); }
  V4 centroids() const { return splat(0.5f) * (lo + hi); }
  float centroid(int k) const { return 0.5f * (lo[k] + hi[k]); }
};

// Boxes of a range of triangles and of their centroids.
struct RangeBox {
  V4 lo = splat(std::numeric_limits<float>::infinity()), hi = -lo;
  V4 clo = lo, chi = hi;
  void add(const PrimRef& r) {
    lo = vmin(lo, r.lo);
    hi = vmax(hi, r.hi);
    const V4 c = r.centroids();
    clo = vmin(clo, c);
    chi = vmax(chi, c);
  }
  void add(const RangeBox& o) {
    lo = vmin(lo, o.lo);
    hi = vmax(hi, o.hi);
    clo = vmin(clo, o.clo);
    chi = vmax(chi, o.chi);
  }
};

// Nodes of one thread, in pieces (a node never moves).
struct Arena {
  static constexpr int kPiece = 1024;
  std::vector<std::unique_ptr<TmpNode[]>> pieces;
  int used = kPiece;
  TmpNode* alloc() {
    if (used == kPiece) {
      pieces.emplace_back(new TmpNode[kPiece]);
      used = 0;
    }
    return &pieces.back()[used++];
  }
};

// A fixed set of threads (the caller's among them) takes subtrees from one
// queue, largest first; whoever splits a large one leaves its right child there
// and goes on with the left. Nobody waits for a subtree: the build is done when
// none is queued or being built.
struct Builder {
  const BvhBuildOptions& opt;
  PrimRef* refs;
  int threads;
  std::vector<Arena> arenas;  // one per thread
  std::atomic<int> max_depth{0};
  std::atomic<int> leaves{0};
  struct Task {
    int begin, end, depth;
    TmpNode** slot;
  };
  std::mutex mu;
  std::condition_variable wake;
  std::deque<Task> queue;
  int unfinished = 0;  // tasks queued or being built
  FirstError error;    // a subtree that failed is given up; the others are built to the end

  Builder(const BvhBuildOptions& o, PrimRef* r, int nthreads) : opt(o), refs(r), threads(nthreads) {}

  TmpNode* run(int count) {
    // As many threads as the triangles can keep busy.
    const int n = std::max(1, std::min(threads, count / kSpawn));
    arenas.resize(n);
    TmpNode* root = nullptr;
    queue.push_back(Task{0, count, 0, &root});
    unfinished = 1;
    std::vector<std::thread> th;
    th.reserve(n);
    for (int t = 1; t < n && start_thread(th, [this, t] { work(arenas[t]); });) ++t;
    work(arenas[0]);
    for (std::thread& x : th) x.join();
    error.rethrow();
    return root;
  }

  void work(Arena& arena) {
    std::unique_lock<std::mutex> g(mu);
    while (true) {
      wake.wait(g, [this] { return !queue.empty() || unfinished == 0; });
      if (queue.empty()) return;
      const Task t = queue.front();
      queue.pop_front();
      g.unlock();
      error.guard([&] { *t.slot = build(t.begin, t.end, t.depth, arena); });
      g.lock();
      if (--unfinished == 0) wake.notify_all();
    }
  }

  static float half_area(const float* a, const float* b) {
    float dx = b[0] - a[0], dy = b[1] - a[1], dz = b[2] - a[2];
    return dx * dy + dy * dz + dz * dx;
  }
  static float half_area(V4 a, V4 b) {
    const V4 d = b - a;
    return d[0] * d[1] + d[1] * d[2] + d[2] * d[0];
  }

  // Ranges above this many primitives are scanned by several threads (the
  // top levels of the tree, which would otherwise run on one thread).
  static constexpr int kParallelScan = 1 << 16;

  // Subtrees of more primitives than this go to the queue (one takes about 0.1
  // ms to build).
  static constexpr int kSpawn = 512;

  int scan_parts(int count) const {
    if (count < kParallelScan) return 1;
    return std::max(1, std::min(threads, count / (kParallelScan / 4)));
  }

  // Boxes over [begin, end), in parallel for large ranges.
  RangeBox boxes(int begin, int end) const {
    const int parts = scan_parts(end - begin);
    RangeBox all;
    if (parts == 1) {
      for (int i = begin; i < end; ++i) all.add(refs[i]);
      return all;
    }
    std::vector<RangeBox> part(parts);
    parallel_parts(begin, end, parts, [&](int s, int e, int t) {
      RangeBox b;
      for (int i = s; i < e; ++i) b.add(refs[i]);
      part[t] = b;
    });
    for (const RangeBox& b : part) all.add(b);
    return all;
  }

  TmpNode* build(int begin, int end, int depth, Arena& arena) {
    TmpNode* n = arena.alloc();
    n->depth = depth;
    const RangeBox box = boxes(begin, end);
    for (int k = 0; k < 3; ++k) n->lo[k] = box.lo[k], n->hi[k] = box.hi[k];
    int count = end - begin;
    n->first = begin;
    n->total = count;
    int cur = max_depth.load();
    while (depth > cur && !max_depth.compare_exchange_weak(cur, depth)) {
    }
    if (count <= 1) return make_leaf(n, begin, count);
    // Remaining depth a balanced split would need from here.
    int need = 0;
    while (((int64_t)opt.max_leaf << need) < count) ++need;
    bool forced_median = depth + need + 1 >= opt.max_depth;
    int mid = -1;
    if (!forced_median) {
      float cost_leaf = (float)count;
      float split_cost;
      mid = sah_split(begin, end, box, &split_cost);
      if (mid < 0 || (count <= opt.max_leaf && cost_leaf <= split_cost)) {
        if (count <= opt.max_leaf) return make_leaf(n, begin, count);
        mid = -1;
      }
    }
    if (mid < 0) mid = median_split(begin, end, box);
    if (end - mid > kSpawn && arenas.size() > 1) {
      {
        std::lock_guard<std::mutex> g(mu);
        queue.push_back(Task{mid, end, depth + 1, &n->child[1]});
        ++unfinished;
      }
      wake.notify_one();
      n->child[0] = build(begin, mid, depth + 1, arena);
    } else {
      n->child[0] = build(begin, mid, depth + 1, arena);
      n->child[1] = build(mid, end, depth + 1, arena);
    }
    return n;
  }

  TmpNode* make_leaf(TmpNode* n, int begin, int count) {
    n->begin = begin;
    n->count = count;
    leaves.fetch_add(1);
    return n;
  }

  int median_split(int begin, int end, const RangeBox& box) {
    int axis = 0;
    for (int k = 1; k < 3; ++k)
      if (box.chi[k] - box.clo[k] > box.chi[axis] - box.clo[axis]) axis = k;
    int mid = begin + (end - begin) / 2;
    std::nth_element(refs + begin, refs + mid, refs + end,
                     [&](const PrimRef& a, const PrimRef& b) { return a.centroid(axis) < b.centroid(axis); });
    return mid;
  }

  struct Bins {
    int cnt[3][64];
    V4 blo[3][64], bhi[3][64];
    void clear(int B) {
      const V4 inf = splat(std::numeric_limits<float>::infinity());
      for (int axis = 0; axis < 3; ++axis)
        for (int b = 0; b < B; ++b) {
          cnt[axis][b] = 0;
          blo[axis][b] = inf;
          bhi[axis][b] = -inf;
        }
    }
  };

  void bin_range(int begin, int end, int B, V4 cl, V4 scale, Bins& bins) const {
    bins.clear(B);
    for (int i = begin; i < end; ++i) {
      const PrimRef& r = refs[i];
      const I4 at = __builtin_convertvector((r.centroids() - cl) * scale, I4);
      for (int axis = 0; axis < 3; ++axis) {
        if (scale[axis] == 0.f) continue;
        const int b = std::min(B - 1, (int)at[axis]);
        bins.cnt[axis][b]++;
        bins.blo[axis][b] = vmin(bins.blo[axis][b], r.lo);
        bins.bhi[axis][b] = vmax(bins.bhi[axis][b], r.hi);
      }
    }
  }

  // Returns the partition point of the best binned SAH split, or -1.
  int sah_split(int begin, int end, const RangeBox& box, float* best_cost_out) {
    const float parent_area = half_area(box.lo, box.hi);
    if (end - begin == 2) {
      // Two primitives part on every axis along which their centres differ,
      // always the same way: the first such axis is the one binning finds.
      for (int axis = 0; axis < 3; ++axis) {
        if (!(box.chi[axis] - box.clo[axis] > 0.f)) continue;
        PrimRef *a = refs + begin, *b = a + 1;
        if (!(a->centroid(axis) < b->centroid(axis))) std::swap(*a, *b);
        const float cost = half_area(a->lo, a->hi) + half_area(b->lo, b->hi);
        *best_cost_out = parent_area > 0.f ? 1.f + cost / parent_area : 1.f;
        return cost < std::numeric_limits<float>::infinity() ? begin + 1 : -1;
      }
      return -1;
    }
    // Small ranges get as many bins as primitives (at least 4): the per-bin
    // clear and sweep would otherwise dominate near the leaves.
    const int B = std::max(2, std::min(std::min(opt.bins, 64), std::max(4, end - begin)));
    int best_axis = -1, best_bin = -1;
    float best_cost = std::numeric_limits<float>::infinity();
    V4 cl = box.clo, scale = splat(0.f);
    cl[3] = 0.f;
    for (int axis = 0; axis < 3; ++axis) {
      // An axis along which the centres lie too close for B / ext is not split.
      const float ext = box.chi[axis] - box.clo[axis], s = B / ext;
      scale[axis] = ext > 0.f && s <= std::numeric_limits<float>::max() ? s : 0.f;
    }
    Bins all;
    const int parts = scan_parts(end - begin);
    if (parts == 1) {
      bin_range(begin, end, B, cl, scale, all);
    } else {  // per-thread bins, merged (counts add, boxes union: independent of timing)
      std::vector<Bins> part(parts);
      parallel_parts(begin, end, parts, [&](int s, int e, int t) { bin_range(s, e, B, cl, scale, part[t]); });
      all.clear(B);
      for (const Bins& pb : part)
        for (int axis = 0; axis < 3; ++axis)
          for (int b = 0; b < B; ++b) {
            all.cnt[axis][b] += pb.cnt[axis][b];
            all.blo[axis][b] = vmin(all.blo[axis][b], pb.blo[axis][b]);
            all.bhi[axis][b] = vmax(all.bhi[axis][b], pb.bhi[axis][b]);
          }
    }
    const V4 inf = splat(std::numeric_limits<float>::infinity());
    for (int axis = 0; axis < 3; ++axis) {
      if (scale[axis] == 0.f) continue;
      const int* cnt = all.cnt[axis];
      float rarea[64];
      int rcnt[64];
      V4 al = inf, ah = -inf;
      int ac = 0;
      for (int b = B - 1; b > 0; --b) {  // an empty bin leaves the sums as they are
        if (cnt[b]) {
          ac += cnt[b];
          al = vmin(al, all.blo[axis][b]);
          ah = vmax(ah, all.bhi[axis][b]);
          rarea[b] = half_area(al, ah);
        } else {
          rarea[b] = ac ? rarea[b + 1] : 0.f;
        }
        rcnt[b] = ac;
      }
      al = inf, ah = -inf;
      ac = 0;
      for (int b = 0; b < B - 1; ++b) {
        if (cnt[b] == 0) continue;  // the split before it again, or no primitive yet
        ac += cnt[b];
        al = vmin(al, all.blo[axis][b]);
        ah = vmax(ah, all.bhi[axis][b]);
        if (rcnt[b + 1] == 0) break;
        float cost = half_area(al, ah) * ac + rarea[b + 1] * rcnt[b + 1];
        if (cost < best_cost) {
          best_cost = cost;
          best_axis = axis;
          best_bin = b;
        }
      }
    }
    if (best_axis < 0) return -1;
    *best_cost_out = parent_area > 0.f ? 1.f + best_cost / parent_area : 1.f;
    float s = scale[best_axis], c0 = cl[best_axis];
    PrimRef* it = std::partition(refs + begin, refs + end, [&](const PrimRef& r) {
      int b = std::min(B - 1, (int)((r.centroid(best_axis) - c0) * s));
      return b <= best_bin;
    });
    int mid = (int)(it - refs);
    if (mid == begin || mid == end) return -1;
    return mid;
  }
};

void write_node(BvhNode* dst, const TmpNode* n) {
  for (int k = 0; k < 3; ++k) {
    constexpr float kMax = std::numeric_limits<float>::max();
    float ext = std::min(n->hi[k] - n->lo[k], kMax);
    float mag = std::max(std::fabs(n->lo[k]), std::fabs(n->hi[k]));
    float pad = ext * 1e-6f + mag * 2e-7f;
    dst->lo[k] = std::max(n->lo[k] - pad, -kMax);
    dst->hi[k] = std::min(n->hi[k] + pad, kMax);
  }
  dst->a = n->count > 0 ? n->begin : 0;
  dst->b = n->count;
}

struct Flattener {
  std::vector<BvhNode>& out;
  explicit Flattener(std::vector<BvhNode>& o) : out(o) {}
  int alloc_pair() {
    int i = (int)out.size();
    out.resize(out.size() + 2);
    return i;
  }
  void dfs(const TmpNode* n, int idx) {
    write_node(&out[idx], n);
    if (n->count > 0) return;
    int c = alloc_pair();
    out[idx].a = c;
    out[idx].b = 0;
    dfs(n->child[0], c);
    dfs(n->child[1], c + 1);
  }
  void run(const TmpNode* root, int top_bfs) {
    out.resize(1);
    if (top_bfs <= 1) {
      dfs(root, 0);
      return;
    }
    // Breadth-first for the first `top_bfs` slots, then depth-first below.
    std::vector<std::pair<const TmpNode*, int>> level{{root, 0}}, frontier;
    write_node(&out[0], root);
    while (!level.empty()) {
      std::vector<std::pair<const TmpNode*, int>> next;
      for (auto& e : level) {
        const TmpNode* n = e.first;
        if (n->count > 0) continue;
        if ((int)out.size() + 2 <= top_bfs) {
          int c = alloc_pair();
          out[e.second].a = c;
          out[e.second].b = 0;
          write_node(&out[c], n->child[0]);
          write_node(&out[c + 1], n->child[1]);
          next.push_back({n->child[0], c});
          next.push_back({n->child[1], c + 1});
        } else {
          frontier.push_back(e);
        }
      }
      level.swap(next);
      if ((int)out.size() + 2 > top_bfs) {
        for (auto& e : level)
          if (e.first->count == 0) frontier.push_back(e);
        break;
      }
    }
    for (auto& e : frontier) dfs(e.first, e.second);
  }
};

// Collapses the binary tree into 8-wide nodes. Each wide node takes the
// children of a binary node and keeps opening its internal child of largest
// surface area until it has 8 children or only leaves; children are placed
// in slots by the direction of their centre from the node's centre (the
// slot order a ray visits depends on its octant); boxes are padded like the
// binary nodes' and quantised outwards.
struct WideCollapser {
  const int32_t* order;            // binary leaf order -> primID
  std::vector<WideNode>& out;
  std::vector<int32_t>& tris;      // wide leaf order -> primID

  static void padded(const TmpNode* n, double lo[3], double hi[3]) {
    BvhNode b;
    write_node(&b, n);
    for (int k = 0; k < 3; ++k) {
      lo[k] = b.lo[k];
      hi[k] = b.hi[k];
    }
  }

  static double area(const TmpNode* n) {
    float dx = n->hi[0] - n->lo[0], dy = n->hi[1] - n->lo[1], dz = n->hi[2] - n->lo[2];
    return (double)dx * dy + (double)dy * dz + (double)dz * dx;
  }

  // A child becomes a leaf slot when its subtree holds at most kWideLeaf triangles.
  static constexpr int kWideLeaf = 3;
  static bool is_leaf(const TmpNode* n) { return n->total <= kWideLeaf; }

  void gather(const TmpNode* n, std::vector<const TmpNode*>& ch) const {
    ch.clear();
    if (is_leaf(n)) {  // a small root: one leaf child
      ch.push_back(n);
      return;
    }
    ch.push_back(n->child[0]);
    ch.push_back(n->child[1]);
    while (ch.size() < 8) {
      int best = -1;
      double best_a = -1.0;
      for (int i = 0; i < (int)ch.size(); ++i)
        if (!is_leaf(ch[i]) && area(ch[i]) > best_a) {
          best_a = area(ch[i]);
          best = i;
        }
      if (best < 0) break;
      const TmpNode* c = ch[best];
      ch[best] = c->child[0];
      ch.push_back(c->child[1]);
    }
    // Slots left over: split leaf-sized subtrees too, for tighter leaf boxes.
    while (ch.size() < 8) {
      int best = -1;
      double best_a = -1.0;
      for (int i = 0; i < (int)ch.size(); ++i)
        if (ch[i]->count == 0 && ch[i]->child[0] && area(ch[i]) > best_a) {
          best_a = area(ch[i]);
          best = i;
        }
      if (best < 0) break;
      const TmpNode* c = ch[best];
      ch[best] = c->child[0];
      ch.push_back(c->child[1]);
    }
  }

  // Slot of each child: greedy matching of child directions to the eight
  // octant directions of the slots.
  static void assign_slots(const std::vector<const TmpNode*>& ch, const double nlo[3], const double nhi[3],
                           int slot_of[8]) {
    const int m = (int)ch.size();
    double score[8][8];
    for (int c = 0; c < m; ++c) {
      double off[3];
      for (int k = 0; k < 3; ++k)
        off[k] = 0.5 * ((double)ch[c]->lo[k] + ch[c]->hi[k]) - 0.5 * (nlo[k] + nhi[k]);
      for (int s = 0; s < 8; ++s) {
        double v = 0.0;
        for (int k = 0; k < 3; ++k) v += ((s >> k) & 1) ? off[k] : -off[k];
        score[c][s] = v;
      }
    }
    bool used_c[8] = {}, used_s[8] = {};
    for (int it = 0; it < m; ++it) {
      int bc = -1, bs = -1;
      double bv = -std::numeric_limits<double>::infinity();
      for (int c = 0; c < m; ++c) {
        if (used_c[c]) continue;
        for (int s = 0; s < 8; ++s)
          if (!used_s[s] && score[c][s] > bv) {
            bv = score[c][s];
            bc = c;
            bs = s;
          }
      }
      used_c[bc] = used_s[bs] = true;
      slot_of[bc] = bs;
    }
  }

  // Builds the wide node of binary node `n` into `w`: its internal children
  // get placeholder slots appended to `nodes` (from w.child_base) and are
  // returned in `kids` in slot order; its leaf triangles are appended to `tris`.
  void fill_node(const TmpNode* n, WideNode& w, std::vector<WideNode>& nodes, std::vector<int32_t>& tris,
                 const TmpNode* kids[8], int* nkids) const {
    std::vector<const TmpNode*> ch;
    ch.reserve(8);
    gather(n, ch);
    const int m = (int)ch.size();
    double clo[8][3], chi[8][3], nlo[3], nhi[3];
    for (int k = 0; k < 3; ++k) {
      nlo[k] = std::numeric_limits<double>::infinity();
      nhi[k] = -std::numeric_limits<double>::infinity();
    }
    for (int c = 0; c < m; ++c) {
      padded(ch[c], clo[c], chi[c]);
      for (int k = 0; k < 3; ++k) {
        nlo[k] = std::min(nlo[k], clo[c][k]);
        nhi[k] = std::max(nhi[k], chi[c][k]);
      }
    }
    int slot_of[8];
    assign_slots(ch, nlo, nhi, slot_of);
    const TmpNode* in_slot[8] = {};
    int child_of_slot[8];
    for (int c = 0; c < m; ++c) {
      in_slot[slot_of[c]] = ch[c];
      child_of_slot[slot_of[c]] = c;
    }
    std::memset(&w, 0, sizeof(w));
    // Empty slots get inverted boxes (lo = 255 > hi = 0 on every axis), which
    // no ray hits whatever its direction.
    std::memset(w.qlo, 0xff, sizeof(w.qlo));
    // Quantisation grid per axis: the smallest power-of-two cell with 255 cells
    // covering the node, at most 2^112 (the traversal scales cells by 2^15).
    double cell[3];
    for (int k = 0; k < 3; ++k) {
      w.p[k] = (float)nlo[k];
      if ((double)w.p[k] > nlo[k]) w.p[k] = std::nextafter(w.p[k], -std::numeric_limits<float>::infinity());
      const double ext = nhi[k] - (double)w.p[k];
      int e = -126;
      if (ext > 0.0) {
        int ex;
        const double m = std::frexp(ext / 255.0, &ex);  // ext / 255 = m * 2^ex, m in [0.5, 1)
        e = std::max(-126, std::min(112, m == 0.5 ? ex - 1 : ex));
      }
      while (e < 112 && std::ldexp(255.0, e) < ext) ++e;  // guards the rounding of ext / 255
      w.e[k] = (uint8_t)(e + 127 + 15);
      cell[k] = std::ldexp(1.0, e);
    }
    // Internal children first (their node slots), then leaf triangles.
    int n_internal = 0;
    for (int s = 0; s < 8; ++s)
      if (in_slot[s] && !is_leaf(in_slot[s])) ++n_internal;
    const int child_base = (int)nodes.size();
    nodes.resize(nodes.size() + n_internal);
    w.child_base = child_base;
    w.tri_base = (int)tris.size();
    for (int s = 0; s < 8; ++s) {
      const TmpNode* c = in_slot[s];
      if (!c) continue;
      const int ci = child_of_slot[s];
      for (int k = 0; k < 3; ++k) {
        double ql = std::floor((clo[ci][k] - w.p[k]) / cell[k]);
        double qh = std::ceil((chi[ci][k] - w.p[k]) / cell[k]);
        ql = std::max(0.0, std::min(255.0, ql));
        qh = std::max(0.0, std::min(255.0, qh));
        while (ql > 0.0 && (double)w.p[k] + ql * cell[k] > clo[ci][k]) ql -= 1.0;
        while (qh < 255.0 && (double)w.p[k] + qh * cell[k] < chi[ci][k]) qh += 1.0;
        w.qlo[k][s] = (uint8_t)ql;
        w.qhi[k][s] = (uint8_t)qh;
      }
      if (!is_leaf(c)) {
        w.imask |= (uint8_t)(1u << s);
        w.meta[s] = 0x80;
      } else {
        const int off = (int)tris.size() - w.tri_base;
        w.meta[s] = (uint8_t)((c->total << 5) | off);
        for (int i = 0; i < c->total; ++i) tris.push_back(order[c->first + i]);
      }
    }
    *nkids = 0;
    for (int s = 0; s < 8; ++s)
      if (in_slot[s] && !is_leaf(in_slot[s])) kids[(*nkids)++] = in_slot[s];
  }

  // The wide subtree of `n` into nodes[idx] and below, depth first.
  void fill(int idx, const TmpNode* n, std::vector<WideNode>& nodes, std::vector<int32_t>& tris) const {
    WideNode w;
    const TmpNode* kids[8];
    int nk;
    fill_node(n, w, nodes, tris, kids, &nk);
    nodes[idx] = w;
    for (int r = 0; r < nk; ++r) fill(w.child_base + r, kids[r], nodes, tris);
  }

  // The top levels breadth first on this thread until there are enough
  // subtrees for every core, then the subtrees in parallel, each into arrays
  // of its own, appended in order with their child and triangle bases shifted.
  void run(const TmpNode* root, int threads) {
    out.assign(1, WideNode{});
    std::vector<std::pair<int, const TmpNode*>> frontier{{0, root}}, next;
    for (int level = 0; level < 6 && !frontier.empty() && (int)frontier.size() < 4 * threads; ++level) {
      next.clear();
      for (auto& f : frontier) {
        WideNode w;
        const TmpNode* kids[8];
        int nk;
        fill_node(f.second, w, out, tris, kids, &nk);
        out[f.first] = w;
        for (int r = 0; r < nk; ++r) next.push_back({w.child_base + r, kids[r]});
      }
      frontier.swap(next);
    }
    struct Task {
      int idx;
      const TmpNode* n;
      WideNode root;
      std::vector<WideNode> nodes;
      std::vector<int32_t> tris;
    };
    std::vector<Task> tasks(frontier.size());
    std::atomic<int> next_task{0};
    auto worker = [&](int, int, int) {
      for (int t; (t = next_task.fetch_add(1)) < (int)tasks.size();) {
        Task& tk = tasks[t];
        tk.idx = frontier[t].first;
        tk.n = frontier[t].second;
        const TmpNode* kids[8];
        int nk;
        fill_node(tk.n, tk.root, tk.nodes, tk.tris, kids, &nk);
        for (int r = 0; r < nk; ++r) fill(tk.root.child_base + r, kids[r], tk.nodes, tk.tris);
      }
    };
    if (!tasks.empty()) parallel_parts(0, threads, std::max(1, std::min(threads, (int)tasks.size())), worker);
    for (Task& tk : tasks) {
      const int node_off = (int)out.size(), tri_off = (int)tris.size();
      for (WideNode& w : tk.nodes) {
        w.child_base += node_off;
        w.tri_base += tri_off;
      }
      tk.root.child_base += node_off;
      tk.root.tri_base += tri_off;
      out[tk.idx] = tk.root;
      out.insert(out.end(), tk.nodes.begin(), tk.nodes.end());
      tris.insert(tris.end(), tk.tris.begin(), tk.tris.end());
    }
  }
};

}  // namespace

void build_bvh(const float* positions, int64_t num_tris, const BvhBuildOptions& opt, BvhBuild* out) {
  const int T = (int)num_tris;
  out->nodes.clear();
  out->woop.assign(12 * (size_t)T, 0.f);
  out->tri_prim.resize(T);
  out->depth = 0;
  out->leaves = 0;
  out->wide.clear();
  if (T == 0 && opt.wide) {
    WideNode empty;
    std::memset(&empty, 0, sizeof(empty));  // no slot in use, inverted boxes: nothing hits
    std::memset(empty.qlo, 0xff, sizeof(empty.qlo));
    for (int k = 0; k < 3; ++k) empty.e[k] = 127 + 15;
    out->wide.push_back(empty);
    return;
  }
  if (T == 0) {
    BvhNode empty;
    std::memset(&empty, 0, sizeof(empty));
    for (int k = 0; k < 3; ++k) {
      empty.lo[k] = 1.f;
      empty.hi[k] = -1.f;  // inverted box: nothing hits
    }
    out->nodes.push_back(empty);
    return;
  }
  int threads = opt.threads > 0 ? opt.threads : (int)std::max(1u, std::thread::hardware_concurrency());
  // Triangles with an infinite or NaN coordinate are never hit (woop_record): they
  // stand at a corner of a triangle that can be, where they widen no box.
  auto finite = [&](int i) {
    const float* p = positions + 9 * (size_t)i;
    return std::all_of(p, p + 9, [](float x) { return std::isfinite(x); });
  };
  int first_finite = 0;
  while (first_finite < T && !finite(first_finite)) ++first_finite;
  float point[9] = {};
  for (int k = 0; k < 9 && first_finite < T; ++k) point[k] = positions[9 * (size_t)first_finite + k % 3];
  std::vector<PrimRef> refs(T);
  parallel_parts(0, T, std::max(1, std::min(threads, T / 4096)), [&](int s, int e, int) {
    for (int i = s; i < e; ++i) {
      const float* p = finite(i) ? positions + 9 * (size_t)i : point;
      PrimRef& r = refs[i];
      for (int k = 0; k < 3; ++k) {
        r.lo[k] = std::min(std::min(p[k], p[3 + k]), p[6 + k]);
        r.hi[k] = std::max(std::max(p[k], p[3 + k]), p[6 + k]);
      }
      r.set_id(i);
    }
  });
  Builder b(opt, refs.data(), threads);
  TmpNode* root = b.run(T);
  out->depth = b.max_depth.load();
  out->leaves = b.leaves.load();
  std::vector<int32_t> order(T);  // binary leaf order -> primID
  for (int i = 0; i < T; ++i) order[i] = refs[i].id();
  // Woop records of triangles in `ids` order, in parallel.
  auto records = [&](const std::vector<int32_t>& ids) {
    parallel_parts(0, T, std::max(1, std::min(threads, T / 4096)), [&](int s, int e, int) {
      for (int i = s; i < e; ++i) {
        out->tri_prim[i] = ids[i];
        woop_record(positions + 9 * (size_t)ids[i], &out->woop[12 * (size_t)i]);
      }
    });
  };
  if (opt.wide) {
    std::vector<int32_t> tris;
    tris.reserve(T);
    WideCollapser wc{order.data(), out->wide, tris};
    wc.run(root, threads);
    records(tris);
    return;
  }
  Flattener fl(out->nodes);
  fl.run(root, opt.top_bfs_nodes);
  records(order);
  // SAH cost of the result (traversal + intersection, relative to the root).
  double root_area = Builder::half_area(out->nodes[0].lo, out->nodes[0].hi);
  double cost = 0.0;
  for (const BvhNode& n : out->nodes) {
    double a = Builder::half_area(n.lo, n.hi) / (root_area > 0 ? root_area : 1.0);
    cost += n.b > 0 ? a * n.b : a;
  }
  out->sah_cost = cost;
}

}  // namespace orion_gb300
