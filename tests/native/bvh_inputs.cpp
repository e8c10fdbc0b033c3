// build_bvh on positions from a file (argv[1]: floats, 9 a triangle), binary and wide, on one thread and
// on eight: every triangle in the tree once, every box around its triangles (those of finite corners).
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "bvh_build.h"

using namespace orion_gb300;

namespace {

std::vector<float> g_pos;

bool finite(int prim) {
  for (int k = 0; k < 9; ++k)
    if (!std::isfinite(g_pos[9 * (size_t)prim + k])) return false;
  return true;
}

// Checks the leaves below node i and adds up their triangles.
bool check(const BvhBuild& b, int i, const float* lo, const float* hi, int* count) {
  const BvhNode& n = b.nodes[i];
  if (n.b == 0) return check(b, n.a, n.lo, n.hi, count) && check(b, n.a + 1, b.nodes[n.a + 1].lo, b.nodes[n.a + 1].hi, count);
  for (int t = n.a; t < n.a + n.b; ++t, ++*count) {
    const int prim = b.tri_prim[t];
    for (int k = 0; finite(prim) && k < 9; ++k) {
      const float x = g_pos[9 * (size_t)prim + k];
      if (!(x >= n.lo[k % 3] && x <= n.hi[k % 3])) return false;
    }
  }
  return true;
}

}  // namespace

int main(int, char** argv) {
  std::FILE* f = std::fopen(argv[1], "rb");
  float x;
  while (f && std::fread(&x, sizeof x, 1, f) == 1) g_pos.push_back(x);
  const int n = (int)(g_pos.size() / 9);
  for (int threads : {1, 8})
    for (bool wide : {false, true}) {
      BvhBuildOptions opt;
      opt.wide = wide;
      opt.max_leaf = wide ? 3 : opt.max_leaf;
      opt.threads = threads;
      BvhBuild b;
      build_bvh(g_pos.data(), n, opt, &b);
      std::vector<char> seen(n, 0);
      for (int p : b.tri_prim)
        if (p < 0 || p >= n || seen[p]++) return std::puts("a triangle is not in the tree once"), 1;
      int count = 0;
      if (!wide && n && !check(b, 0, b.nodes[0].lo, b.nodes[0].hi, &count)) return std::puts("a box too small"), 1;
      if (!wide && count != n) return std::puts("triangles missing"), 1;
    }
  std::puts("ok");
  return 0;
}
