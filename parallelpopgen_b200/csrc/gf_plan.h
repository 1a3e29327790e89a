// Host-only planning logic of the engine, free of CUDA so that it compiles and is tested with a plain
// C++ compiler: the layout of the batched engine's generation records (regions of slabs, resident or
// cycling through a ring of slots), the lock-step finishing schedule of its replicates, which
// generations a multi-population window may hold, and which kernel runs a window.
#pragma once

#include <algorithm>
#include <cstdint>
#include <deque>
#include <vector>

#include "../../include/gofish_b200.h"

namespace gf {

// Generation records of a batch.  Slab j of replicate r is its generations (j * chunk_r,
// (j + 1) * chunk_r] with chunk_r = slab_windows * c_r (c_r its cadence): every replicate advances one
// window per super-step, so all of them enter slab j at super-step j * slab_windows, and no window
// straddles two slabs.  Region j holds slab j of every replicate that runs that long, in replicate
// order.  Resident layout: the regions one after another (region_base); ring layout: region j in slot
// j % ring_slots of slot_records records each.
struct RecordPlan {
  int slab_windows = 1;
  int nregions = 0;
  std::vector<int> chunk;               // [r] generations per slab
  std::vector<long long> region_base;   // [j] first record of region j, resident layout (nregions + 1)
  std::vector<long long> region_jobs;   // [j] slabs in region j
  std::vector<int> region_off;          // [r * nregions + j] offset of replicate r's slab in region j, or -1
  long long total = 0;                  // records of the batch
  long long largest = 0;                // records of the largest region
  int ring_slots = 0;                   // 0: resident; K >= 2: ring of K slots
  long long slot_records = 0;
  long long slots = 0;                  // records the buffers hold

  long long slot_base(int j) const {
    return ring_slots > 0 ? static_cast<long long>(j % ring_slots) * slot_records : region_base[j];
  }
  // Index of replicate r's record of generation g + 1 (g generations done), or -1.
  long long record_index(int r, int g) const {
    const int j = g / chunk[r];
    if (j >= nregions) return -1;
    const int off = region_off[static_cast<size_t>(r) * nregions + j];
    if (off < 0) return -1;
    return slot_base(j) + off + (g - static_cast<long long>(j) * chunk[r]);
  }
};

// Plan the records of `R` replicates for a record budget: resident when the total fits it (and
// record indices stay within int32), else a ring of as many whole regions as fit (at least two).
inline RecordPlan plan_records(const gf_replicate* reps, int R, long long budget, int slab_target) {
  RecordPlan P;
  int cmax = 1;
  for (int r = 0; r < R; ++r) {
    P.total += std::max(reps[r].num_generations, 0);
    cmax = std::max(cmax, reps[r].compact_interval);
  }
  P.slab_windows = std::max(1, (slab_target + cmax - 1) / cmax);
  P.chunk.resize(R);
  for (int r = 0; r < R; ++r) {
    P.chunk[r] = P.slab_windows * std::max(reps[r].compact_interval, 1);
    P.nregions = std::max(P.nregions, (std::max(reps[r].num_generations, 0) + P.chunk[r] - 1) / P.chunk[r]);
  }
  const int nreg = P.nregions;
  P.region_off.assign(static_cast<size_t>(R) * nreg, -1);
  P.region_base.assign(nreg + 1, 0);
  P.region_jobs.assign(nreg, 0);
  long long off = 0;
  for (int j = 0; j < nreg; ++j) {
    P.region_base[j] = off;
    for (int r = 0; r < R; ++r) {
      const int G = reps[r].num_generations;
      const int g0 = j * P.chunk[r];
      if (g0 >= G) continue;
      P.region_off[static_cast<size_t>(r) * nreg + j] = static_cast<int>(off - P.region_base[j]);
      off += std::min(G, g0 + P.chunk[r]) - g0;
      P.region_jobs[j] += 1;
    }
    P.largest = std::max(P.largest, off - P.region_base[j]);
  }
  P.region_base[nreg] = off;
  P.slots = P.total;
  if ((P.total > budget || P.total >= (1ll << 31)) && nreg > 2) {
    const long long K = std::min<long long>(nreg, std::max<long long>(2, budget / std::max<long long>(P.largest, 1)));
    if (K < nreg) {
      P.ring_slots = static_cast<int>(K);
      P.slot_records = P.largest;
      P.slots = K * P.largest;
    }
  }
  return P;
}

// [k]: the replicates whose last window is super-step k (ceil(G / c) windows; none for G = 0).
inline std::vector<std::vector<int>> plan_finish_steps(const gf_replicate* reps, int R) {
  std::vector<std::vector<int>> at;
  for (int r = 0; r < R; ++r) {
    const int G = reps[r].num_generations;
    if (G <= 0) continue;
    const int c = std::max(reps[r].compact_interval, 1);
    const int last = (G + c - 1) / c - 1;
    if (static_cast<int>(at.size()) <= last) at.resize(last + 1);
    at[last].push_back(r);
  }
  return at;
}

// May a multi-population window (2 <= P <= max_pops) hold this generation?  Every population must be
// drifted with Nchrom_e > 0, or not drifted with its rows zero in both state buffers (`live_rows`:
// bit p set when population p's rows may hold a nonzero value).
inline bool mp_window_generation_ok(const gf_generation& g, int P, int live_rows, int max_pops) {
  if (P < 2 || P > max_pops) return false;
  for (int p = 0; p < P; ++p) {
    const gf_population_params& pp = g.pop[p];
    if (pp.drift) {
      if (pp.Nchrom_e <= 0) return false;
    } else if ((live_rows >> p) & 1) {
      return false;
    }
  }
  return true;
}

// A compaction's survivor count on its way to the host: the compaction stores it into h_mail[slot] with the tag
// above it.
struct PendingCount {
  int slot = 0;
  long long added = 0;   // new mutations appended after this compaction
  unsigned tag = 0;
};

// What the host knows of the mutation count while launches are queued ahead of the read-backs.
struct SlotCount {
  long long upper = 0;    // upper bound on the count after everything enqueued
  long long recent = 0;   // the last count read back
  long long open = 0;     // births since the compaction enqueued last: no compaction has thinned them
  std::deque<PendingCount> pending;   // compactions whose survivor counts are not here yet, oldest first

  // The count itself, everything enqueued having run.
  void known(long long M) {
    upper = recent = M;
    open = 0;
  }
  // About how many slots a window with `n` births ends with: the survivors of a compaction differ little from one
  // to the next, while the bound grows by the births of every window enqueued ahead of the read-backs.
  long long expected(long long n) const { return std::min(upper, recent + open) + n; }
  // `n` births enqueued.  They are added to whatever the bound is by then: a count may have arrived since the
  // launch was sized.
  void births(long long n) {
    upper += n;
    open += n;
    for (PendingCount& pc : pending) pc.added += n;
  }
  void compaction(const PendingCount& pc) {
    pending.push_back(pc);
    open = 0;
  }
  // The oldest compaction's count is here: a bound whatever came after (later compactions only lower the count).
  void survivors(long long M) {
    recent = M;
    upper = std::min(upper, M + pending.front().added);
    pending.pop_front();
  }
};

// Generations whose records a block of the single- or multi-population window kernels stages in shared memory.
// The plain engine ends its windows there; a batched replicate's window is its compaction cadence, of any length.
constexpr int kMaxWindowGenerations = 128;

// Generations of the longest window of a batch.
inline int longest_window(const gf_replicate* reps, int R) {
  int n = 0;
  for (int r = 0; r < R; ++r) n = std::max(n, std::min(reps[r].compact_interval, reps[r].num_generations));
  return n;
}

// Whether a batch's windows pack their living slots, decided once: its launches are also captured in graphs.  `tiles`:
// of 1,024 slots, over all segments.  Short windows of small replicates, whose tiles are mostly last ones and share no
// records, do not repay the packing kernel's start.  1,024 replicates, a quad per thread against packing: N0 up to
// 1e4 (some 60 tiles of capacity each) 442 / 508 ms at a cadence of 10, 439 / 456 at 25, 470 / 447 at 35; up to 3e4 (some 140)
// 1.24 / 1.29 s at 20, 1.31 / 1.26 at 30; 128 up to 1e5 (some 350) 2.36 / 1.99 s at 10; spectra of 256 (some 800) 305 / 307 ms at
// 10, 377 / 315 at 25.
inline bool batch_packs(const gf_replicate* reps, int R, long long tiles) {
  constexpr long long kLargeTiles = 240, kPackCadence = 26;
  long long cadences = 0, run = 0;   // of the replicates that run at all
  for (int r = 0; r < R; ++r)
    if (reps[r].num_generations > 0) {
      cadences += reps[r].compact_interval;
      ++run;
    }
  return tiles >= kLargeTiles * R || cadences >= kPackCadence * run;
}

// Expected slots (at the window's end) up to which one replicate's window runs a slot per thread.  Window
// kernels of 25 generations on a B200, a slot per thread against the packing kernel: 23 / 53 us at 12,000
// slots, 27 / 55 at 92,000, 50 / 70 at 368,000, 74 / 80 at 552,000 (N = 1e4, neutral), 92 / 104 at 648,000 (gamma = -10),
// 86 / 86 at 625,000, 98 / 90 at 736,000 and 111 / 94 at 833,000 (neutral, N = 1e4 and 2e5).
#ifndef GF_SLOT_WINDOW_SLOTS
#define GF_SLOT_WINDOW_SLOTS 600000
#endif
constexpr long long kSlotWindowSlots = GF_SLOT_WINDOW_SLOTS;

// The kernel of a single-population window launch: a slot per thread (one small replicate), a quad per thread
// with the living slots packed later (where packing pays), or a quad per thread throughout.  The first two stage
// the window's records, so a launch that holds a longer window takes the third, which reads them from memory.
enum class WindowForm { slots, pack, quads };
inline WindowForm window_form(bool single, bool lane_order, bool pack, long long expected_slots, int longest) {
  if (!lane_order || longest > kMaxWindowGenerations) return WindowForm::quads;
  if (single && expected_slots <= kSlotWindowSlots) return WindowForm::slots;
  return pack ? WindowForm::pack : WindowForm::quads;
}

inline int drifted_populations(const gf_generation& g, int P) {
  int m = 0;
  for (int p = 0; p < P; ++p)
    if (g.pop[p].drift) m |= 1 << p;
  return m;
}

}  // namespace gf
