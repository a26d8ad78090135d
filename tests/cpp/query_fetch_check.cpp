// Host check of the ray queries' fetch counters (pt_fetch.h): every query starts
// from 0, whichever of the queries before it were refused at their launch.
// Prints one line and exits non-zero on a mismatch.
#include "../../pathtracer_gb300/csrc/pt_fetch.h"

#include <cstdio>
#include <random>

using namespace pt;

int main() {
  std::mt19937 gen(3);
  int bad = 0, clears = 0, refused = 0, total = 0;
  for (int rate : {0, 2, 3, 10}) {  // 1 launch in `rate` is refused
    int counters[2] = {0, 0};
    QueryFetch F;
    F.counters = counters;
    const int clears_before = clears;
    for (int q = 0; q < 10000; ++q) {
      ++total;
      const FetchPair p = F.begin([&](int *c) {
        c[0] = c[1] = 0;
        ++clears;
      });
      if (rate && gen() % rate == 0) {
        ++refused;
        continue;
      }
      bad += *p.now != 0;  // the kernel: counts in one, clears the other
      *p.now = 1 + (int)(gen() % 1000);
      *p.next = 0;
      F.launched();
    }
    bad += rate == 0 && clears != clears_before;  // none in the usual course
  }
  std::printf("%d queries, %d refused: %d started from a stale counter\n", total, refused, bad);
  return bad ? 1 : 0;
}
