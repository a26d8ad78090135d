// pt_fetch.h -- the fetch counters of the ray queries (host side).
#pragma once

namespace pt {

// Fetch counters of a query: its own (0 at its start) and the next one's.
struct FetchPair {
  int *now, *next;
};

// Two counters in turn: a query's kernel counts in one and clears the other for
// the next query.  That holds only if the kernel runs, so a query that was begun
// and not reported as launched (the launch was refused) leaves them to be
// cleared by the next.
struct QueryFetch {
  int *counters = nullptr;  // two, 0 at first
  int turn = 0;
  bool dirty = false;

  // clear(counters): sets both to 0 before what follows.
  template <class Clear>
  FetchPair begin(Clear clear) {
    if (dirty) clear(counters);
    dirty = true;
    return FetchPair{counters + turn, counters + (turn ^ 1)};
  }
  void launched() {
    turn ^= 1;
    dirty = false;
  }
};

}  // namespace pt
