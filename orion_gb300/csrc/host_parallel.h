// Host loops over contiguous pieces on short-lived threads (scene preparation
// and the BVH build).
#pragma once
#include <stdint.h>

#include <algorithm>
#include <exception>
#include <mutex>
#include <new>
#include <system_error>
#include <thread>
#include <utility>
#include <vector>

namespace orion_gb300 {

// Starts f on a thread of its own, added to `th` (with room for it); false if the
// system gives no more threads.
template <class F>
bool start_thread(std::vector<std::thread>& th, F&& f) {
  try {
    th.emplace_back(std::forward<F>(f));
    return true;
  } catch (const std::system_error&) {
  } catch (const std::bad_alloc&) {
  }
  return false;
}

// The first exception of several threads' work, thrown again once they are joined.
class FirstError {
 public:
  template <class F>
  void guard(F&& f) {
    try {
      f();
    } catch (...) {
      std::lock_guard<std::mutex> g(mu_);
      if (!error_) error_ = std::current_exception();
    }
  }
  void rethrow() const {
    if (error_) std::rethrow_exception(error_);
  }

 private:
  std::mutex mu_;
  std::exception_ptr error_;
};

// f(begin, end, part) over `parts` contiguous pieces of [begin, end); the
// caller's thread takes the last one, and those that get no thread. Throws what
// a piece threw.
template <class F>
void parallel_parts(int64_t begin, int64_t end, int parts, const F& f) {
  const int64_t n = end - begin;
  FirstError error;
  std::vector<std::thread> th;
  th.reserve(parts);
  for (int t = 0; t < parts; ++t) {
    const int64_t b = begin + n * t / parts, e = begin + n * (t + 1) / parts;
    auto piece = [&f, &error, b, e, t] { error.guard([&] { f(b, e, t); }); };
    if (t + 1 == parts || !start_thread(th, piece)) piece();
  }
  for (std::thread& x : th) x.join();
  error.rethrow();
}

// Pieces for n items: one per hardware thread, none under `least` items.
inline int parts_for(int64_t n, int64_t least) {
  const int64_t threads = std::max(1u, std::thread::hardware_concurrency());
  return (int)std::max<int64_t>(1, std::min(threads, n / least));
}

}  // namespace orion_gb300
