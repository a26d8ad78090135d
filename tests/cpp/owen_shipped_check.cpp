// Host check of the Owen-scrambled dimensions as a render draws them: with the
// tables the library itself makes (make_halton_tables: digit counts, early end)
// and the tables of first digits, every value equals the one that computes every
// digit with the plain permutation_element, and so does the value without the
// tables (pt_sampler_eval's).  Prints one line and exits non-zero on a mismatch.
#include "../../pathtracer_gb300/csrc/pt_common.cuh"

#include <cstdio>
#include <vector>

using namespace pt;

// Every digit, hardware division and permutation_element's own modulo.
static float owen_plain(const HaltonTables &T, int dim, uint32_t index) {
  const int bi = dim % PT_PRIME_COUNT;
  const uint32_t base = (uint32_t)T.prime[bi], hash = (uint32_t)mix_bits(1u + ((uint32_t)dim << 4));
  uint64_t rev = 0;
  uint32_t a = index;
  for (int di = 0; di < T.ndigits[bi]; ++di) {
    const uint32_t dh = (uint32_t)mix_bits(hash ^ (uint32_t)rev ^ ((uint32_t)di << 16));
    rev = rev * base + permutation_element(a % base, base, dh);
    a /= base;
  }
  return clamp_to_float(xdmul(T.inv_base_m[bi], (double)rev));
}

int main() {
  const HaltonTables T = make_halton_tables();
  std::vector<uint32_t> tab(T.owen_at[PT_OWEN_DIMS]);
  for (int dim = 0; dim < PT_OWEN_DIMS; ++dim)
    for (uint32_t r = 0; r < T.owen_pow[dim % PT_PRIME_COUNT]; ++r)
      tab[T.owen_at[dim] + r] = owen_first_digits(T, dim, r);
  long long bad = 0, tried = 0;
  for (int dim = 0; dim < PT_OWEN_DIMS + 36; ++dim) {
    const uint32_t p = T.owen_pow[dim % PT_PRIME_COUNT];
    for (uint64_t k = 0; k < 4000; ++k)
      for (uint32_t i : {(uint32_t)k, ~(uint32_t)k, (uint32_t)splitmix64(k * 257 + dim), (uint32_t)(k * p), (uint32_t)(k * p) - 1u}) {
        const float x = owen_radical_inverse(T, dim, i, tab.data()), y = owen_radical_inverse(T, dim, i);
        const float z = owen_plain(T, dim, i);
        bad += std::memcmp(&x, &z, 4) != 0 || std::memcmp(&y, &z, 4) != 0;
        ++tried;
      }
  }
  std::printf("owen values as shipped: %lld mismatches in %lld\n", bad, tried);
  return bad ? 1 : 0;
}
