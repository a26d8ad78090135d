// Host check of the light sample grid's arithmetic in pt_common.cuh against
// hardware division: div_small for every offset (stratum + k / 2^24 rounded)
// a grid of n <= 16 strata draws, and idiv_small for every pair.  Prints one
// line per check and exits non-zero on a mismatch.
#include "../../pathtracer_gb300/csrc/pt_common.cuh"

#include <cstdio>
#include <cstring>

using namespace pt;

int main() {
  long long bad = 0, count = 0;
  for (int n = 1; n <= 16; ++n) {
    const float r = 1.f / (float)n;
    for (int s = 0; s < n; ++s) {
      // the sums' spacing grows with the stratum: step over equal ones
      const uint32_t step = s < 1 ? 1u : s < 2 ? 2u : s < 4 ? 4u : s < 8 ? 8u : 16u;
      for (uint32_t k = 0; k < (1u << 24); k += step) {
        const float x = (float)s + (float)k * (1.0f / 16777216.0f);
        const float a = div_small(x, (float)n, r), b = x / (float)n;
        bad += std::memcmp(&a, &b, 4) != 0;
        ++count;
      }
      const float x = (float)s + 16777215.0f * (1.0f / 16777216.0f);
      const float a = div_small(x, (float)n, r), b = x / (float)n;
      bad += std::memcmp(&a, &b, 4) != 0;
    }
  }
  printf("div_small: %lld mismatches in %lld quotients\n", bad, count);
  long long bad2 = 0;
  for (int b = 1; b <= 16; ++b)
    for (int a = 0; a < 16; ++a) bad2 += idiv_small(a, 1.f / (float)b) != a / b;
  printf("idiv_small: %lld mismatches\n", bad2);
  return (bad || bad2) ? 1 : 0;
}
