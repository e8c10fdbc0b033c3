// plan_waves: each pixel and pass in one wave, every wave within the capacity, the capacity
// within what slots are numbered with. argv: pixels, spp, wave, exact.
#include <cstdio>
#include <cstdlib>

#include "wave_plan.h"

using namespace orion_gb300;

int main(int, char** argv) {
  const int64_t pixels = std::atoll(argv[1]), wave = std::atoll(argv[3]);
  const int spp = std::atoi(argv[2]);
  const bool exact = std::atoi(argv[4]) != 0;
  const WavePlan p = plan_waves(pixels, spp, wave, exact);
  std::printf("%lld groups of %lld waves, %d passes, chunks of 2^%d, capacity %lld\n", (long long)p.groups,
              (long long)p.group_waves, p.passes, p.chunk_log2, (long long)p.capacity());
  if (p.capacity() < 1 || p.capacity() > INT32_MAX) return std::puts("capacity out of range"), 1;
  if (exact && p.capacity() > wave) return std::puts("larger than asked for"), 1;
  if (p.capacity() > wave + wave / 16) return std::puts("over by more than a sixteenth"), 1;
  if (p.passes < 1) return std::puts("no passes"), 1;
  if (spp <= 0 ? p.groups != 0 : (int64_t)(p.groups - 1) * p.passes >= spp || (int64_t)p.groups * p.passes < spp)
    return std::puts("passes left out"), 1;
  int64_t sum = 0;
  for (int64_t k = 0; k < p.group_waves; ++k) {
    const int64_t n = p.pixels_of(k);
    if (n < 1 || n * p.passes > p.capacity()) return std::puts("a wave out of range"), 1;
    sum += n;
  }
  if (sum != pixels) return std::puts("pixels left out"), 1;
  std::puts("ok");
  return 0;
}
