// build_bvh when threads cannot be started (argv[1] = threads: pthread_create fails after the first
// argv[3]) and when memory runs out on one (argv[1] = memory: the caller gets std::bad_alloc).
// argv[2]: triangles.
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <vector>

#include "bvh_build.h"

using namespace orion_gb300;

namespace {
std::atomic<int> g_threads_left{1 << 30};
std::atomic<bool> g_starve{false};
thread_local bool t_main = false;
}  // namespace

// Threads of the C++ runtime come from here while any are left.
extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg) {
  if (g_threads_left-- <= 0) return EAGAIN;
  using Fn = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  return reinterpret_cast<Fn>(dlsym(RTLD_NEXT, "pthread_create"))(t, a, f, arg);
}

void* operator new(size_t n) {
  if (g_starve && !t_main) throw std::bad_alloc();
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void* operator new[](size_t n) { return operator new(n); }
void operator delete(void* p) noexcept { std::free(p); }
void operator delete[](void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }
void operator delete[](void* p, size_t) noexcept { std::free(p); }

int main(int argc, char** argv) {
  t_main = true;
  const int n = std::atoi(argv[2]);
  std::vector<float> pos(9 * (size_t)n);
  unsigned x = 12345u;
  for (int i = 0; i < n; ++i) {
    float c[3];
    for (float& v : c) v = (float)((x = x * 1664525u + 1013904223u) >> 8) / (1 << 24);
    for (int k = 0; k < 9; ++k)
      pos[9 * (size_t)i + k] = c[k % 3] + 0.01f * (float)((x = x * 1664525u + 1013904223u) >> 8) / (1 << 24);
  }
  BvhBuildOptions opt;
  opt.wide = true;
  opt.max_leaf = 3;
  BvhBuild want, got;
  opt.threads = 1;
  build_bvh(pos.data(), n, opt, &want);
  opt.threads = 8;
  if (std::strcmp(argv[1], "memory") == 0) {
    for (int attempt = 0; attempt < 200; ++attempt) {  // (the caller's thread may be quicker than all others)
      try {
        g_starve = true;
        build_bvh(pos.data(), n, opt, &got);
      } catch (const std::bad_alloc&) {
        g_starve = false;
        build_bvh(pos.data(), n, opt, &got);
        std::puts(got.wide.size() == want.wide.size() ? "ok" : "another tree");
        return 0;
      }
    }
    return std::puts("no exception"), 1;
  }
  g_threads_left = std::atoi(argv[3]);
  build_bvh(pos.data(), n, opt, &got);
  const bool same = got.wide.size() == want.wide.size() && got.tri_prim == want.tri_prim && got.woop == want.woop &&
                    got.depth == want.depth && got.leaves == want.leaves;
  std::puts(same ? "ok" : "another tree");
  return 0;
}
