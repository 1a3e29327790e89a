// Host-only checks of which kernel runs a window (gf_plan.h): the kernels that stage a window's generation
// records in shared memory hold at most kMaxWindowGenerations of them.
#include <cstdio>
#include <cstring>
#include <vector>

#include "gf_plan.h"

static int failures = 0;
#define CHECK(cond)                                                  \
  do {                                                               \
    if (!(cond)) {                                                   \
      std::printf("FAIL %s:%d: %s\n", __FILE__, __LINE__, #cond);    \
      ++failures;                                                    \
    }                                                                \
  } while (0)

static gf_replicate rep(int cadence, int generations) {
  gf_replicate r;
  std::memset(&r, 0, sizeof r);
  r.compact_interval = cadence;
  r.num_generations = generations;
  return r;
}

static void check_batches() {
  using gf::WindowForm;
  auto form = [](const std::vector<gf_replicate>& reps, bool pack) {
    return gf::window_form(false, true, pack, 0, gf::longest_window(reps.data(), static_cast<int>(reps.size())));
  };
  for (int cadence : {1, 25, 127, 128}) CHECK(form({rep(cadence, 1000)}, true) == WindowForm::pack);
  for (int cadence : {129, 200, 256, 257, 300, 100000}) CHECK(form({rep(cadence, 1000)}, true) == WindowForm::quads);
  CHECK(form({rep(10, 500), rep(129, 500), rep(25, 500)}, true) == WindowForm::quads);   // one long one is enough
  CHECK(form({rep(300, 128)}, true) == WindowForm::pack);    // a run shorter than its cadence
  CHECK(form({rep(300, 129)}, true) == WindowForm::quads);
  CHECK(form({rep(300, 0)}, true) == WindowForm::pack);
  CHECK(form({rep(25, 1000)}, false) == WindowForm::quads);
}

// The packing rule is the batch's own: it does not move as replicates finish, and needs no resident records.
static void check_packing() {
  auto packs = [](const std::vector<gf_replicate>& reps, long long tiles) {
    return gf::batch_packs(reps.data(), static_cast<int>(reps.size()), tiles);
  };
  CHECK(!packs({rep(25, 100), rep(25, 100)}, 100));
  CHECK(packs({rep(26, 100), rep(26, 100)}, 100));
  CHECK(!packs({rep(10, 100), rep(41, 100)}, 100) && packs({rep(10, 100), rep(42, 100)}, 100));
  CHECK(!packs({rep(10, 100), rep(10, 100)}, 479) && packs({rep(10, 100), rep(10, 100)}, 480));
  CHECK(!packs({rep(10, 100), rep(1000, 0)}, 2));   // a replicate that never runs
  CHECK(packs({rep(30, 100), rep(1, 0)}, 2));
}

static void check_single() {
  using gf::WindowForm;
  const long long line = gf::kSlotWindowSlots;
  CHECK(gf::window_form(true, true, true, line, 128) == WindowForm::slots);
  CHECK(gf::window_form(true, true, true, line + 1, 128) == WindowForm::pack);
  CHECK(gf::window_form(true, true, true, line, 129) == WindowForm::quads);
  CHECK(gf::window_form(true, false, true, 0, 25) == WindowForm::quads);   // another draw schedule
  CHECK(gf::window_form(false, true, true, 0, 25) == WindowForm::pack);    // several replicates
}

int main() {
  check_batches();
  check_packing();
  check_single();
  std::printf(failures ? "FAILED %d\n" : "OK\n", failures);
  return failures ? 1 : 0;
}
