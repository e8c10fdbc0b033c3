// How a plain render's pixels and passes are cut into waves (WaveArgs).
#pragma once
#include <stdint.h>

#include <algorithm>

namespace orion_gb300 {

// Every wave renders `passes` passes (the last group of passes may have fewer) of some
// chunks of 2^chunk_log2 pixels of the film: wave k of a group takes the chunks k,
// k + group_waves, ... Only a wave smaller than a pixel's samples splits them: then
// several groups of passes follow one another.
struct WavePlan {
  int64_t pixels;
  int64_t groups, group_waves, chunks;
  int passes, chunk_log2;

  // The pixels of wave k of a group; the last chunk may be partial.
  int64_t pixels_of(int64_t k) const {
    const int64_t n = (chunks - k + group_waves - 1) / group_waves;
    const bool has_last = (chunks - 1) % group_waves == k;
    return (n << chunk_log2) - (has_last ? (chunks << chunk_log2) - pixels : 0);
  }
  // Path slots that the largest wave needs.
  int64_t capacity() const {
    return std::min<int64_t>(((chunks + group_waves - 1) / group_waves) << chunk_log2, pixels) * passes;
  }
};

// `wave`: paths per wave (>= 1). exact: no wave is larger. Otherwise there are as few
// waves as `wave` allows, and their last chunk may take one over it, by a sixteenth at
// most; but never past INT32_MAX paths, which slots are numbered with. No samples
// (spp <= 0): no groups.
inline WavePlan plan_waves(int64_t pixels, int spp, int64_t wave, bool exact) {
  WavePlan p;
  p.pixels = pixels;
  p.groups = spp > 0 ? (spp + wave - 1) / wave : 0;
  p.passes = spp > 0 ? (int)((spp + p.groups - 1) / p.groups) : 1;
  const int64_t wave_pixels = std::max<int64_t>(1, wave / p.passes);
  p.chunk_log2 = 8;  // a chunk is at most a sixteenth of a wave's pixels
  while (p.chunk_log2 > 0 && (int64_t)16 << p.chunk_log2 > wave_pixels) --p.chunk_log2;
  p.chunks = (pixels + ((int64_t)1 << p.chunk_log2) - 1) >> p.chunk_log2;
  p.group_waves = std::min<int64_t>(p.chunks, (pixels + wave_pixels - 1) / wave_pixels);
  if (exact || p.capacity() > INT32_MAX) {
    const int64_t wave_chunks = std::max<int64_t>(1, wave_pixels >> p.chunk_log2);
    p.group_waves = (p.chunks + wave_chunks - 1) / wave_chunks;
  }
  return p;
}

}  // namespace orion_gb300
