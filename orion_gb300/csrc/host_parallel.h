// Host loops over contiguous pieces on short-lived threads (scene preparation
// and the BVH build).
#pragma once
#include <stdint.h>

#include <algorithm>
#include <thread>
#include <vector>

namespace orion_gb300 {

// f(begin, end, part) over `parts` contiguous pieces of [begin, end); the
// caller's thread takes the last one.
template <class F>
void parallel_parts(int64_t begin, int64_t end, int parts, const F& f) {
  const int64_t n = end - begin;
  std::vector<std::thread> th;
  for (int t = 0; t < parts; ++t) {
    const int64_t b = begin + n * t / parts, e = begin + n * (t + 1) / parts;
    if (t + 1 < parts)
      th.emplace_back([&f, b, e, t] { f(b, e, t); });
    else
      f(b, e, t);
  }
  for (std::thread& x : th) x.join();
}

// Pieces for n items: one per hardware thread, none under `least` items.
inline int parts_for(int64_t n, int64_t least) {
  const int64_t threads = std::max(1u, std::thread::hardware_concurrency());
  return (int)std::max<int64_t>(1, std::min(threads, n / least));
}

}  // namespace orion_gb300
