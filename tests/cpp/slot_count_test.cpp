// Host-only checks of what the engine knows of its mutation count while launches run ahead of the read-backs
// (SlotCount, gf_plan.h): always a bound, and one that follows the counts as they arrive.
#include <cstdio>
#include <deque>

#include "gf_plan.h"

static int failures = 0;
#define CHECK(cond, ...)                                   \
  do {                                                     \
    if (!(cond)) {                                         \
      std::printf("FAIL %s:%d: ", __FILE__, __LINE__);     \
      std::printf(__VA_ARGS__);                            \
      std::printf("\n");                                   \
      ++failures;                                          \
    }                                                      \
  } while (0)

// Windows of `births` that each compact to `living`, the counts arriving `lag` windows later and, as it happens
// while a launch is prepared, after the window was sized and before its births are accounted for.
static void check_bound(long long living, long long births, int lag) {
  gf::SlotCount c;
  c.known(living);
  for (int w = 0; w < 200; ++w) {
    const long long need = c.upper + births;   // what the window is sized for
    CHECK(need >= living + births, "window %d sized for %lld of %lld slots", w, need, living + births);
    if (w >= lag) c.survivors(living);
    c.births(births);
    CHECK(c.upper >= living + births, "window %d: bound %lld of %lld", w, c.upper, living + births);
    c.compaction(gf::PendingCount{});
    CHECK(c.upper <= living + (lag + 1) * births, "window %d, lag %d: the bound has grown to %lld", w, lag, c.upper);
  }
  while (!c.pending.empty()) c.survivors(living);
  CHECK(c.upper == living, "bound %lld of %lld at the end", c.upper, living);
}

int main() {
  for (int lag : {1, 2, 7, 62}) {
    check_bound(1000, 300, lag);
    check_bound(0, 5, lag);
  }
  std::printf(failures ? "FAILED %d\n" : "OK\n", failures);
  return failures ? 1 : 0;
}
