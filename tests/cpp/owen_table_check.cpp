// Host check of the tables of first Owen-scrambled digits (pt_common.cuh): the
// radical inverse that starts from a table equals the one that computes every
// digit up to the early end, for every tabulated dimension and the first ones
// beyond, at indices around the multiples of the table's size, the lowest,
// the highest and hashed ones; the divisions by the tables' sizes are exact.
// Prints one line per check and exits non-zero on a mismatch.
#include "../../pathtracer_gb300/csrc/pt_common.cuh"

#include <cstdio>
#include <vector>

using namespace pt;

static HaltonTables tables() {
  static const int primes[PT_PRIME_COUNT] = {2,  3,  5,  7,  11, 13, 17, 19, 23, 29, 31, 37, 41,
                                             43, 47, 53, 59, 61, 67, 71, 73, 79, 83, 89, 97};
  HaltonTables T{};
  for (int b = 0; b < PT_PRIME_COUNT; ++b) {
    const int base = primes[b];
    T.prime[b] = base;
    double m = 1.0;
    int nd = 0;
    while (1.0 - (base - 1) * m < 1.0) {
      ++nd;
      m *= 1.0 / (double)base;
    }
    T.ndigits[b] = nd;
    T.inv_base_m[b] = m;
    div_invariant((uint32_t)base, T.div_magic[b], T.div_shift[b]);
    int check = 0;
    for (uint64_t p = 1; p < (1ull << 38) && check < nd; p *= (uint64_t)base) ++check;
    T.owen_check[b] = check;
    T.owen_tail[b] = 1;
    for (int r = check; r < nd; ++r) T.owen_tail[b] *= (uint64_t)base;
  }
  return T;
}

int main() {
  HaltonTables T = tables();
  const uint32_t n = owen_table_layout(T);
  std::vector<uint32_t> tab(n);
  for (int dim = 0; dim < PT_OWEN_DIMS; ++dim)
    for (uint32_t r = 0; r < T.owen_pow[dim % PT_PRIME_COUNT]; ++r)
      tab[T.owen_at[dim] + r] = owen_first_digits(T, dim, r);
  long long bad = 0, tried = 0, div = 0;
  for (int b = 0; b < PT_PRIME_COUNT; ++b) {
    const uint32_t p = T.owen_pow[b];
    bad += p > PT_OWEN_ENTRIES || p * (uint64_t)T.prime[b] <= PT_OWEN_ENTRIES || T.owen_first[b] > T.owen_check[b];
    for (uint64_t k = 0; k < (1u << 18); ++k)
      for (uint32_t a : {(uint32_t)k, ~(uint32_t)k, (uint32_t)splitmix64(k * 25 + b), (uint32_t)(k * p), (uint32_t)(k * p) - 1u})
        div += div_by(T.owen_pow_magic[b], T.owen_pow_shift[b], a) != a / p;
  }
  for (int dim = 0; dim < PT_OWEN_DIMS + 12; ++dim) {
    const uint32_t p = T.owen_pow[dim % PT_PRIME_COUNT];
    for (uint64_t k = 0; k < 3000; ++k)
      for (uint32_t i : {(uint32_t)k, ~(uint32_t)k, (uint32_t)splitmix64(k * 131 + dim), (uint32_t)(k * p), (uint32_t)(k * p) - 1u}) {
        const float x = owen_radical_inverse(T, dim, i, tab.data()), y = owen_radical_inverse(T, dim, i);
        bad += std::memcmp(&x, &y, 4) != 0;
        ++tried;
      }
  }
  std::printf("owen tables: %lld mismatches in %lld values, %u entries; divisions: %lld mismatches\n", bad, tried, n, div);
  return bad || div ? 1 : 0;
}
