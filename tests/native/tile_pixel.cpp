// tile_pixel: positions [0, width x height) to pixels of the film, each once. Films too large to
// mark every pixel: some positions only, checked for range and against one another.
// argv: width, height.
#include <cstdio>
#include <cstdlib>
#include <set>
#include <vector>

#include "kernels.h"

using namespace orion_gb300;

int main(int, char** argv) {
  const int w = std::atoi(argv[1]), h = std::atoi(argv[2]);
  const int64_t n = (int64_t)w * h;
  auto pixel = [&](int64_t pos, int64_t* out) {
    int x = -1, y = -1;
    tile_pixel(pos, w, h, &x, &y);
    *out = (int64_t)y * w + x;
    return x >= 0 && x < w && y >= 0 && y < h;
  };
  int64_t at;
  if (n <= 1 << 24) {
    std::vector<char> seen(n, 0);
    for (int64_t k = 0; k < n; ++k) {
      if (!pixel(k, &at)) return std::printf("position %lld outside the film\n", (long long)k), 1;
      if (seen[at]++) return std::printf("pixel %lld twice\n", (long long)at), 1;
    }
  } else {
    std::set<int64_t> pos, seen;
    for (int64_t k = 0; k < 4096; ++k)
      for (int64_t p : {k, n - 1 - k, n / 2 + k, (int64_t)w - 2048 + k, ((int64_t)1 << 32) - 2048 + k, n / 4096 * k})
        if (p >= 0 && p < n) pos.insert(p);
    for (int64_t p : pos) {
      if (!pixel(p, &at)) return std::printf("position %lld outside the film\n", (long long)p), 1;
      if (!seen.insert(at).second) return std::printf("pixel %lld twice\n", (long long)at), 1;
    }
  }
  std::puts("ok");
  return 0;
}
