// pt_wave_size.h -- how many paths a wave may have (host side).
#pragma once
#include <algorithm>
#include <cstdint>

// Shadow-ray list entries: the vertex slot below, the light sample above.
#define PT_LIST_SHIFT 28

namespace pt {

// The largest wave of a job with ln light samples per vertex.  A slot takes
// PT_LIST_SHIFT bits of a list entry, and one 32-bit count covers a bounce's
// closest rays, the list (ln per path) and what the grid's warps claim beyond the
// end (32 each, 0.2 M).
inline int wave_limit(int ln) {
  const int64_t rays = (INT32_MAX - ((int64_t)1 << 20)) / (ln + 1);
  return (int)std::min<int64_t>(rays, ((int64_t)1 << PT_LIST_SHIFT) - 1);
}

// Paths per wave of a render of `total` paths, `npix` per sample: whole samples
// of the film where `cap` holds one.
inline int wave_paths(int64_t npix, int64_t total, int cap, int ln) {
  cap = std::min(cap, wave_limit(ln));
  const int64_t n = npix <= cap ? cap / npix * npix : cap;
  return (int)std::min(n, total);
}

}  // namespace pt
