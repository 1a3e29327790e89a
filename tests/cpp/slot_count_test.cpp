// Host-only checks of what the engine knows of its mutation count while launches run ahead of the read-backs
// (SlotCount, gf_plan.h): always a bound, one that follows the counts as they arrive, and the size a window is expected to end with.
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

// What a window is expected to end with: the births of windows that end without a compaction (long cadences are
// cut at 128 generations) are still there, those of windows that compact are not.
static void check_expected() {
  gf::SlotCount c;
  c.known(1000);
  CHECK(c.expected(100) == 1100, "%lld", c.expected(100));
  for (int w = 0; w < 50; ++w) {
    CHECK(c.expected(100) == 1000 + 100 * (w + 1), "window %d without a compaction: %lld", w, c.expected(100));
    c.births(100);
  }
  c.compaction(gf::PendingCount{});
  CHECK(c.expected(100) == 1100, "after the compaction, its count not here: %lld", c.expected(100));
  for (int w = 0; w < 50; ++w) {   // compacting windows ahead of the read-backs
    c.births(100);
    c.compaction(gf::PendingCount{});
  }
  CHECK(c.expected(100) == 1100 && c.upper == 11000, "%lld of %lld", c.expected(100), c.upper);
  c.survivors(1500);
  CHECK(c.expected(100) == 1600, "%lld", c.expected(100));
  c.births(100);
  CHECK(c.expected(100) == 1700, "%lld", c.expected(100));
  c.known(30);
  CHECK(c.expected(5) == 35, "%lld", c.expected(5));
  gf::SlotCount d;
  d.known(10);
  d.births(5);
  d.compaction(gf::PendingCount{});
  d.survivors(3);
  CHECK(d.expected(0) == 3 && d.upper == 3, "%lld of %lld", d.expected(0), d.upper);
}

int main() {
  for (int lag : {1, 2, 7, 62}) {
    check_bound(1000, 300, lag);
    check_bound(0, 5, lag);
  }
  check_expected();
  std::printf(failures ? "FAILED %d\n" : "OK\n", failures);
  return failures ? 1 : 0;
}
