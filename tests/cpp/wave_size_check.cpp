// Host check of the wave sizes (pt_wave_size.h): for every number of light samples
// and any cap, a wave's slots fit a shadow-list entry and its rays of a bounce a
// 32-bit count, ordinary waves are as large as asked, and they cover the job.
// Prints one line and exits non-zero on a mismatch.
#include "../../pathtracer_gb300/csrc/pt_wave_size.h"

#include <cstdio>
#include <random>

using namespace pt;

int main() {
  std::mt19937_64 gen(5);
  long long bad = 0, tried = 0;
  for (int ln = 1; ln <= 16; ++ln) {
    auto fits = [&](int64_t n) {
      return n < ((int64_t)1 << 28) && n * (ln + 1) + 152 * 16 * 4 * 32 <= INT32_MAX;
    };
    for (int k = 0; k < 20000; ++k) {
      const int64_t npix = 1 + (int64_t)(gen() >> (36 + gen() % 27)), total = npix * (1 + (int64_t)(gen() % 4096));
      const int cap = k % 2 ? INT32_MAX : 1024 + (int)(gen() >> (33 + gen() % 20));
      const int n = wave_paths(npix, total, cap, ln);
      bad += !fits(n) || n < 1 || n > total || n > cap;
      if (n < total) bad += npix <= n && n % npix != 0;
      if (cap <= 1 << 24) bad += n != std::min(total, npix <= cap ? cap / npix * npix : (int64_t)cap);
      ++tried;
    }
  }
  std::printf("%lld wave sizes, %lld wrong\n", tried, bad);
  return bad ? 1 : 0;
}
