// Warps of k_sppm_photons take photons from SppmView::photon_next until one of their takes
// reaches the end: near the largest photon count every warp must stop, no photon may be taken
// twice and none left. argv[1]: photons; argv[2]: those dealt before the simulated part.
#include <cstdio>
#include <cstdlib>
#include <type_traits>
#include <vector>

#include "kernels.h"

using namespace orion_gb300;

int main(int argc, char** argv) {
  const int photons = std::atoi(argv[1]);
  using Counter = std::remove_pointer<decltype(SppmView::photon_next)>::type;
  Counter next = (Counter)std::atoi(argv[2]);
  const long long left = (long long)photons - (long long)next;
  std::vector<char> done(4864, 0);  // warps of a launch on 152 SMs
  long long taken = 0, expect = (long long)next;
  size_t running = done.size();
  for (long long turn = 0; running && turn < 4 * left + 2 * (long long)done.size(); ++turn) {
    const size_t w = turn % done.size();
    if (done[w]) continue;
    const unsigned cnt = turn % 3 == 0 ? 32 : 9;
    const Counter base = next;
    next += cnt;
    done[w] = photons_dealt(base, cnt, photons);
    running -= done[w] ? 1 : 0;
    for (unsigned i = 0; i < cnt; ++i) {
      const Counter k = base + i;
      if (!(k < (Counter)photons)) continue;
      if ((long long)k != expect++) return std::puts("a photon taken twice or left out"), 1;
      ++taken;
    }
  }
  if (running) return std::printf("%zu warps never stop\n", running), 1;
  if (taken != left) return std::printf("%lld photons of %lld\n", taken, left), 1;
  std::puts("ok");
  return 0;
}
