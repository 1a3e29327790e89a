// Windowed drift: every generation of a compaction window in one launch.
//
// Between two compactions a mutation keeps its slot, and its update in generation g depends only
// on its own frequency, the generation's parameters, the slot index and the mutation count M_g at
// the start of g (which decides the quad / scalar-tail counter layout, go_fish_impl.cuh:97-123).
// M_g = M_start + the host-drawn new-mutation counts of the earlier generations of the window, so
// one thread can carry its quad through all generations in registers: read the row once, drift it
// W times with exactly the per-generation arithmetic (gf_drift.cuh), let slots born inside the
// window start at 1/Nc in their birth generation (add_new_mutations, go_fish_impl.cu:138-145), and
// write the row once with the survival flags of the last generation.  A launch covers any number of
// single-population replicates, each in its own 1024-aligned arena segment with its own window
// length, seeds and parameters: the plain engine uses it with one replicate, the batched engine with
// thousands.  Results are bit-identical to running the per-generation kernel W times.
#include <cuda_runtime.h>

#include <algorithm>

#include "gf_drift.cuh"
#include "gf_internal.h"

namespace gf {

constexpr int kWinThreads = 256;
constexpr int kWinTile = kWinThreads * 4;

__device__ __forceinline__ int list_count(const RepList& L, int nreps) { return L.count ? *L.count : nreps; }
__device__ __forceinline__ int list_rep(const RepList& L, int i) { return L.rep ? L.rep[i] : i; }
__device__ __forceinline__ int list_tile0(const RepList& L, const WinRep* __restrict__ reps, int i) {
  return L.tile0 ? L.tile0[i] : reps[i].tile0;
}

// listed replicate owning launch tile `gt` (the last one whose tile0 <= gt)
__device__ __forceinline__ int find_rep(const RepList& L, const WinRep* __restrict__ reps, int n, int gt) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (list_tile0(L, reps, mid) <= gt) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Shared-memory copy of the listed replicates' first tiles (up to kRepCache of them), so the per-tile
// owner search does not chase global memory.
constexpr int kRepCache = 4096;

__device__ __forceinline__ int find_rep_cached(const int* s_tile0, const RepList& L, const WinRep* __restrict__ reps,
                                               int n, int gt) {
  if (n > kRepCache) return find_rep(L, reps, n, gt);
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (s_tile0[mid] <= gt) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ void load_tile0(int* s_tile0, const RepList& L, const WinRep* __restrict__ reps, int n) {
  if (n <= kRepCache)
    for (int j = threadIdx.x; j < n; j += blockDim.x) s_tile0[j] = list_tile0(L, reps, j);
  __syncthreads();
}

// Tiles of one super-step, assigned on the device: replicate j's births over its window are summed
// from its generation records, and it gets ceil((M_in + births) / 1024) tiles (at least one, at most
// its segment), laid out in replicate order.  One block.
__global__ void __launch_bounds__(1024) batch_tiles_kernel(WinRep* __restrict__ reps, int nreps,
                                                           const int* __restrict__ M_in,
                                                           const WinGen* __restrict__ recs, int* __restrict__ total) {
  __shared__ int s_warp[32];
  __shared__ int s_carry;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (int base = 0; base < nreps; base += 1024) {
    const int j = base + threadIdx.x;
    int need = 0;
    if (j < nreps) {
      WinRep& R = reps[j];
      long long births = 0;
      for (int k = 0; k < R.ngen; ++k) births += recs[R.rec + k].new_count;
      R.births = births;
      const long long end = static_cast<long long>(M_in[R.rep]) + births;
      const long long cap_tiles = R.capacity / kWinTile;
      need = static_cast<int>(max(1ll, min(cap_tiles, (end + kWinTile - 1) / kWinTile)));
    }
    int incl = need;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      int w = s_warp[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xFFFFFFFFu, w, o);
        if (lane >= o) w += y;
      }
      s_warp[lane] = w;
    }
    __syncthreads();
    const int before = s_carry + (warp > 0 ? s_warp[warp - 1] : 0) + incl - need;
    if (j < nreps) {
      reps[j].tile0 = before;
      reps[j].ntiles = need;
    }
    __syncthreads();
    if (threadIdx.x == 0) s_carry += s_warp[31];
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = s_carry;
}

// Tiles of super-step k = *step of a batch with precomputed records, and every replicate's window
// derived on the device: replicate r (cadence c, G generations) runs generations (k c, min(G, (k+1) c)]
// from record slab j = k / slab_windows at its offset in region j; a finished replicate gets no tiles.
// The others get ceil((M_in + births) / 1024) tiles (at least one, at most their segment), in replicate
// order, and are listed (table index, first tile, count) for the window, scan and scatter kernels, which
// then never visit a finished replicate (its state and counts stay as they are).  One block; thread 0
// advances the counter once every thread has read it.
__global__ void __launch_bounds__(1024) batch_step_kernel(WinRep* __restrict__ reps, int R,
                                                          const int* __restrict__ M_in,
                                                          const WinGen* __restrict__ recs, int* __restrict__ total,
                                                          int* __restrict__ step, const BatchStepPlan plan,
                                                          const int* __restrict__ region_off,
                                                          const long long* __restrict__ region_base,
                                                          const StepRep* __restrict__ steprep, int* __restrict__ fault,
                                                          int* __restrict__ list_rep, int* __restrict__ list_tile0,
                                                          int* __restrict__ list_count) {
  __shared__ int s_tiles[32], s_listed[32];
  __shared__ int s_carry_tiles, s_carry_listed;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k = *step;
  const int j = k / plan.slab_windows;
  const bool in_plan = j < plan.nregions;
  const long long slot_base = !in_plan              ? 0
                              : plan.ring_slots > 0 ? static_cast<long long>(j % plan.ring_slots) * plan.slot_records
                                                    : region_base[j];
  if (threadIdx.x == 0) {
    s_carry_tiles = 0;
    s_carry_listed = 0;
  }
  __syncthreads();   // every thread has read *step
  for (int base = 0; base < R; base += 1024) {
    const int r = base + threadIdx.x;
    int need = 0;
    if (r < R) {
      const StepRep sr = steprep[r];
      const long long gen = static_cast<long long>(k) * sr.cadence;
      int ngen = 0, rec = 0;
      long long births = 0;
      if (in_plan && gen < sr.gens) {
        const int off = region_off[static_cast<size_t>(r) * plan.nregions + j];
        if (off < 0) {
          atomicExch(fault, kFaultRecords);
        } else {
          ngen = static_cast<int>(min(static_cast<long long>(sr.cadence), sr.gens - gen));
          rec = static_cast<int>(slot_base + off + (gen - static_cast<long long>(j) * sr.chunk));
          // the window's new-mutation counts, eight independent loads at a time
          for (int g0 = 0; g0 < ngen; g0 += 8) {
            int c[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) c[i] = g0 + i < ngen ? recs[rec + g0 + i].new_count : 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) births += c[i];
          }
          const long long end = static_cast<long long>(M_in[r]) + births;
          const long long cap_tiles = reps[r].capacity / kWinTile;
          need = static_cast<int>(max(1ll, min(cap_tiles, (end + kWinTile - 1) / kWinTile)));
        }
      }
      WinRep& W = reps[r];
      W.rec = rec;
      W.ngen = ngen;
      W.births = births;
      W.compact = need > 0 ? 1 : 0;
      W.ntiles = need;
    }
    // exclusive scans of the tiles and of the listed (unfinished) replicates over the block
    const int listed = need > 0 ? 1 : 0;
    int incl_t = need, incl_l = listed;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int yt = __shfl_up_sync(0xFFFFFFFFu, incl_t, o);
      const int yl = __shfl_up_sync(0xFFFFFFFFu, incl_l, o);
      if (lane >= o) {
        incl_t += yt;
        incl_l += yl;
      }
    }
    if (lane == 31) {
      s_tiles[warp] = incl_t;
      s_listed[warp] = incl_l;
    }
    __syncthreads();
    if (warp == 0) {
      int wt = s_tiles[lane], wl = s_listed[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int yt = __shfl_up_sync(0xFFFFFFFFu, wt, o);
        const int yl = __shfl_up_sync(0xFFFFFFFFu, wl, o);
        if (lane >= o) {
          wt += yt;
          wl += yl;
        }
      }
      s_tiles[lane] = wt;
      s_listed[lane] = wl;
    }
    __syncthreads();
    const int tile0 = s_carry_tiles + (warp > 0 ? s_tiles[warp - 1] : 0) + incl_t - need;
    const int pos = s_carry_listed + (warp > 0 ? s_listed[warp - 1] : 0) + incl_l - listed;
    if (r < R) reps[r].tile0 = tile0;
    if (listed) {
      list_rep[pos] = r;
      list_tile0[pos] = tile0;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      s_carry_tiles += s_tiles[31];
      s_carry_listed += s_listed[31];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    *total = s_carry_tiles;
    *list_count = s_carry_listed;
    *step = k + 1;
  }
}

// DRAW: how a warp schedules its sampler draws (DrawStrategy).  KEYS: a launch of one replicate (the plain
// engine), whose window `one` and Philox round keys `keys` are kernel parameters: no table to read or
// search, and a round's key costs no instruction.
template <int DRAW, bool KEYS>
__global__ void __launch_bounds__(kWinThreads, KEYS ? GF_WINDOW_MIN_BLOCKS_KEYS : GF_WINDOW_MIN_BLOCKS)
    window_kernel(const float* __restrict__ A, float* __restrict__ B, int* __restrict__ id_gp,
                  int* __restrict__ id_tid, unsigned* __restrict__ flags, unsigned* __restrict__ tile_count,
                  const int* __restrict__ M_in, int* __restrict__ M_end, int* __restrict__ M_next,
                  const WinRep* __restrict__ reps, int nreps, const WinGen* __restrict__ recs, int total_tiles,
                  const int* __restrict__ total_dev, unsigned long long* __restrict__ stats,
                  int* __restrict__ fault, const PhiloxKeys keys, int* __restrict__ sched, const RepList list,
                  const WinRep one) {
  __shared__ int s_rep;
  __shared__ int s_tile;
  __shared__ unsigned s_warp[kWinThreads / 32];
  __shared__ int s_tile0[KEYS ? 1 : kRepCache];
  __shared__ WarpDraws s_draws[(DRAW == kDrawWarp || DRAW == kDrawPooledSearch) ? kWinThreads / 32 : 1];
  const int lane = threadIdx.x & 31;
  WarpDraws* wd = &s_draws[(DRAW == kDrawWarp || DRAW == kDrawPooledSearch) ? (threadIdx.x >> 5) : 0];
  const int ntiles_all = total_dev ? *total_dev : total_tiles;
  const int nlist = KEYS ? 1 : list_count(list, nreps);
  if (!KEYS) load_tile0(s_tile0, list, reps, nlist);
  // Tiles are handed out in order by an atomic counter, so a block that drew cheap tiles (slots born
  // late in the window) takes more of them: the launch does not wait on the blocks that a fixed
  // assignment would have given the most expensive tiles.
  for (;;) {
    if (threadIdx.x == 0) {
      const int t = atomicAdd(sched, 1);
      s_tile = t;
      if (!KEYS && t < ntiles_all) s_rep = list_rep(list, find_rep_cached(s_tile0, list, reps, nlist, t));
    }
    __syncthreads();
    const int gt = s_tile;
    if (gt >= ntiles_all) break;   // block-uniform
    const WinRep R = KEYS ? one : reps[s_rep];
    __syncthreads();
    const int t = gt - R.tile0;
    const int q = t * kWinThreads + threadIdx.x;  // quad within the replicate
    const int s0 = 4 * q;
    const int cap = static_cast<int>(R.capacity);
    const int M0 = M_in[R.rep];
    // a tile past the replicate's end-of-window count has nothing to do (tile 0 keeps the bookkeeping)
    if (t > 0 && static_cast<long long>(t) * kWinTile >= M0 + R.births) continue;   // block-uniform
    float* const rowB = B + R.base;
    const float* const rowA = A + R.base;
    int* const gp = id_gp + R.base;
    int* const tid = id_tid + R.base;

    float x[4];
    if (s0 + 3 < M0) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(rowA + s0));
      x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) x[j] = (s0 + j < M0) ? rowA[s0 + j] : 0.f;
    }

    int M = M0;
    int alive = 1;
#pragma unroll 1
    for (int k = 0; k < R.ngen; ++k) {
      const WinGen G = recs[R.rec + k];
      const int N = G.Nc;
      const int g = G.generation;
      alive = G.alive;
      if (N <= 0) {
        // extinction generation: the population's row is cleared
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (s0 + j < M) x[j] = 0.f;
      } else {
        // whole quad: Philox (q + 2, g, 0, 0), lanes x, y, z, w.  Every lane of the warp reaches the
        // draw (N and the loop are uniform over the block), as the warp-pooled strategy requires.
        const bool quad = q < (M >> 2);
        const bool neutral = (G.sel_a == 0.f && G.sel_b == 0.f);
        float xs[4] = {0.f, 0.f, 0.f, 0.f};
        int res[4] = {0, 0, 0, 0};
        unsigned need = 0;
        if (quad) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            xs[j] = neutral ? selected_freq<true>(x[j], 0.f, 0.f, 0.f, 0.f)
                            : selected_freq<false>(x[j], G.sel_a, G.sel_b, G.F, G.h);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            res[j] = (xs[j] == 1.f && N > 6) ? N : 0;
            if (!(xs[j] == 0.f || (xs[j] == 1.f && N > 6))) need |= 1u << j;
          }
        }
        uint4 r = make_uint4(0u, 0u, 0u, 0u);
        if (need) {
          if (KEYS) r = philox4x32_10_keys(make_uint4(static_cast<uint32_t>(q + 2), static_cast<uint32_t>(g), 0u, 0u), keys);
          else r = philox(R.seed1, R.seed2, q + 2, g, 0, 0);
        }
        if (DRAW == kDrawWarp || DRAW == kDrawPooledSearch) {
          draw_quad<DRAW>(xs, r, need, N, lane, wd, res);   // every lane of the warp calls it
        } else if (need) {
          draw_quad<DRAW>(xs, r, need, N, lane, wd, res);
        }
        if (quad) {
          const float Nf = static_cast<float>(N);
#pragma unroll
          for (int j = 0; j < 4; ++j) x[j] = static_cast<float>(clampi(res[j], 0, N)) / Nf;
        } else if (s0 < M) {
          // scalar tail: Philox (slot + 2, g, 0, 0) lane x, variance in double
#pragma unroll 1
          for (int j = 0; j < 4; ++j) {
            const int e = s0 + j;
            if (e >= M) break;
            const float xs1 = neutral ? selected_freq<true>(x[j], 0.f, 0.f, 0.f, 0.f)
                                      : selected_freq<false>(x[j], G.sel_a, G.sel_b, G.F, G.h);
            x[j] = static_cast<float>(clampi(drift_tail(R.seed1, R.seed2, e, g, 0, xs1, N), 0, N)) /
                   static_cast<float>(N);
          }
        }
      }
      // births: slots [M, M + new_count) start at 1/Nc with ID (g, 0, slot - M + 1)
      const int Mn = M + G.new_count;
      if (s0 + 3 >= M && s0 < Mn) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int e = s0 + j;
          if (e >= M && e < Mn && e < cap) {
            x[j] = G.new_freq;
            gp[e] = g;
            tid[e] = e - M + 1;
          }
        }
      }
      M = Mn;
    }
    const int Mw = min(M, cap);
    if (s0 + 3 < Mw) {
      *reinterpret_cast<float4*>(rowB + s0) = make_float4(x[0], x[1], x[2], x[3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (s0 + j < Mw) rowB[s0 + j] = x[j];
    }

    if (R.compact) {
      // flag_segregating_mutations for one population: keep unless lost or fixed (when alive), or
      // if preserved
      unsigned keep = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int e = s0 + j;
        if (e >= Mw) continue;
        // lost or fixed in the (only) population -- or the population is not alive -- removes it
        bool k = alive && !(x[j] <= 0.f || x[j] >= 1.f);
        if (R.check_preserved && e < M0 && tid[e] < 0) k = true;
        if (k) keep |= 1u << j;
      }
      unsigned word = keep << ((lane & 7) * 4);
      word |= __shfl_xor_sync(0xFFFFFFFFu, word, 1);
      word |= __shfl_xor_sync(0xFFFFFFFFu, word, 2);
      word |= __shfl_xor_sync(0xFFFFFFFFu, word, 4);
      if ((lane & 7) == 0) flags[(R.base + s0) >> 5] = word;
      unsigned c = __popc(keep);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
      if (lane == 0) s_warp[threadIdx.x >> 5] = c;
      __syncthreads();
      if (threadIdx.x == 0) {
        unsigned tot = 0;
#pragma unroll
        for (int w = 0; w < kWinThreads / 32; ++w) tot += s_warp[w];
        tile_count[R.base / kWinTile + t] = tot;
      }
      __syncthreads();
    }

    if (t == 0 && threadIdx.x == 0) {
      // window bookkeeping, once per replicate
      unsigned long long mg = 0;
      int m = M0;
      for (int k = 0; k < R.ngen; ++k) {
        mg += static_cast<unsigned long long>(m);
        m += recs[R.rec + k].new_count;
      }
      atomicAdd(stats, mg);
      atomicAdd(stats + 1, static_cast<unsigned long long>(R.ngen));
      if (M > cap) atomicExch(fault, kFaultCapacity);
      M_end[R.rep] = Mw;
      if (M_next && !R.compact) M_next[R.rep] = Mw;
    }
  }
  // every block has drawn past the last tile once it gets here; the last one resets the scheduler
  // for the next launch on this stream
  if (threadIdx.x == 0) {
    __threadfence();   // this block's last draw from sched[0] is ordered before its count in sched[1]
    const int finished = atomicAdd(sched + 1, 1);
    if (finished == static_cast<int>(gridDim.x) - 1) {
      sched[0] = 0;
      sched[1] = 0;
    }
  }
}

// ------------------------------------------------------------------------------------------------
// Small windows: a slot per thread
// ------------------------------------------------------------------------------------------------
// Between compactions a slot depends on nothing but its own frequency and the generations' records, so a
// thread can carry one slot through the window with no barrier.  Every slot then evaluates its quad's
// Philox block alone (four times the work, about 118 thread instructions a draw against 73), but the four
// draws of a quad are no longer one thread's chain: a generation takes the latency of one draw, not of
// four with both sampler branches each.  That is what a state of few mutations waits for: 0.7 us a
// generation against 1.9 at 12,000 slots; see kSlotWindowSlots for where the line lies.
struct __align__(16) SlotGen {   // two 16-byte loads
  int generation, Nc;
  int M;            // mutations at the generation's start
  float Nf;         // Nc
  float sel_a, sel_b, F, h;
};

// Slot e's frequency after the generation (e < G.M): the arithmetic and counters of the generation kernel.
template <bool KEYS>
__device__ __forceinline__ float slot_generation(float x, int e, const SlotGen& G, const PhiloxKeys& keys, int seed1,
                                                 int seed2) {
  const int N = G.Nc, g = G.generation;
  if (N <= 0) return 0.f;   // extinction generation: the population's row is cleared
  const bool neutral = G.sel_a == 0.f && G.sel_b == 0.f;
  const float xs = neutral ? selected_freq<true>(x, 0.f, 0.f, 0.f, 0.f)
                           : selected_freq<false>(x, G.sel_a, G.sel_b, G.F, G.h);
  const float Nf = G.Nf;
  float count = 0.f;
  if (e < (G.M & ~3)) {
    if (xs != 0.f) {
      const int q = e >> 2, j = e & 3;
      uint4 r;
      if (KEYS) r = philox4x32_10_keys(make_uint4(static_cast<uint32_t>(q + 2), static_cast<uint32_t>(g), 0u, 0u), keys);
      else r = philox(seed1, seed2, q + 2, g, 0, 0);
      count = binom_draw_count(j == 0 ? r.x : j == 1 ? r.y : j == 2 ? r.z : r.w, xs, N, Nf);
    }
  } else {   // scalar tail: counter (slot + 2), variance in double
    count = static_cast<float>(clampi(drift_tail(seed1, seed2, e, g, 0, xs, N), 0, N));
  }
  return count / Nf;
}

constexpr int kSlotThreads = 128;   // one SM takes several blocks, and a small state spreads over many SMs
static_assert(kSlotThreads >= kMaxWindowGenerations, "a thread per record");

// The records of a window in shared memory: s_gen, the frequencies of new mutations, and whether a lost slot
// stays lost through every generation (its selected frequency is 0; not so if a coefficient is infinite).
// All threads of the block.
__device__ __forceinline__ void load_slot_generations(SlotGen* s_gen, float* s_new, int* s_scan, int* s_lost_stays,
                                                      const WinGen* __restrict__ recs, int ngen, int M0) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  if (t == 0) *s_lost_stays = 1;
  __syncthreads();
  int births = 0;
  if (t < ngen) {
    const WinGen G = recs[t];
    births = G.new_count;
    s_gen[t] = {G.generation, G.Nc, 0, static_cast<float>(G.Nc), G.sel_a, G.sel_b, G.F, G.h};
    s_new[t] = G.new_freq;
    if (!(G.sel_a == 0.f && G.sel_b == 0.f) && !(selected_freq<false>(0.f, G.sel_a, G.sel_b, G.F, G.h) == 0.f))
      *s_lost_stays = 0;
  }
  int incl = births;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) s_scan[warp] = incl;
  __syncthreads();
  int before = M0 + incl - births;
  for (int w = 0; w < warp; ++w) before += s_scan[w];
  if (t < ngen) s_gen[t].M = before;
  __syncthreads();
}

// One replicate's window, kSlotThreads slots a block; writes the rows, the births' IDs and, before a
// compaction, the flag words.
__global__ void __launch_bounds__(kSlotThreads)
    window_slots_kernel(const float* __restrict__ A, float* __restrict__ B, int* __restrict__ id_gp,
                        int* __restrict__ id_tid, unsigned* __restrict__ flags, const int* __restrict__ M_in,
                        int* __restrict__ M_end, int* __restrict__ M_next, const WinGen* __restrict__ recs,
                        unsigned long long* __restrict__ stats, int* __restrict__ fault, const PhiloxKeys keys,
                        const WinRep R) {
  __shared__ SlotGen s_gen[kMaxWindowGenerations];
  __shared__ float s_new[kMaxWindowGenerations];
  __shared__ int s_scan[kSlotThreads / 32];
  __shared__ int s_lost_stays;
  const int cap = static_cast<int>(R.capacity);
  const int M0 = M_in[R.rep];
  const int Mw = static_cast<int>(min(static_cast<long long>(M0) + R.births, R.capacity));
  const int first = static_cast<int>(blockIdx.x) * kSlotThreads;
  if (first >= Mw && blockIdx.x > 0) return;   // block 0 keeps the books
  load_slot_generations(s_gen, s_new, s_scan, &s_lost_stays, recs + R.rec, R.ngen, M0);
  const bool lost_stays = s_lost_stays != 0;
  const int alive = recs[R.rec + R.ngen - 1].alive;
  for (int s0 = first; s0 < Mw; s0 += static_cast<int>(gridDim.x) * kSlotThreads) {
    const int e = s0 + threadIdx.x;
    bool keep = false;
    if (e < Mw) {
      int k = 0;
      float x;
      if (e < M0) {
        x = A[R.base + e];
      } else {   // born in the last generation k whose births start at or below e
        int hi = R.ngen - 1;
        while (k < hi) {
          const int mid = (k + hi + 1) >> 1;
          if (s_gen[mid].M <= e) k = mid;
          else hi = mid - 1;
        }
        x = s_new[k];
        id_gp[R.base + e] = s_gen[k].generation;
        id_tid[R.base + e] = e - s_gen[k].M + 1;
        ++k;
      }
#pragma unroll 1
      for (; k < R.ngen; ++k) {
        if (lost_stays && __float_as_uint(x) == 0u) break;
        x = slot_generation<true>(x, e, s_gen[k], keys, R.seed1, R.seed2);
      }
      B[R.base + e] = x;
      keep = alive && !(x <= 0.f || x >= 1.f);
      if (R.check_preserved && e < M0 && id_tid[R.base + e] < 0) keep = true;
    }
    if (R.compact) {
      const unsigned word = __ballot_sync(0xFFFFFFFFu, keep);
      if ((threadIdx.x & 31) == 0) flags[(R.base + e) >> 5] = word;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    unsigned long long mg = 0;
    for (int k = 0; k < R.ngen; ++k) mg += static_cast<unsigned long long>(s_gen[k].M);
    atomicAdd(stats, mg);
    atomicAdd(stats + 1, static_cast<unsigned long long>(R.ngen));
    if (static_cast<long long>(M0) + R.births > cap) atomicExch(fault, kFaultCapacity);
    M_end[R.rep] = Mw;
    if (M_next && !R.compact) M_next[R.rep] = Mw;
  }
}

// The compaction of a small window in one launch: a block counts the survivors before its tile from the
// flag words themselves (a few hundred words from L2), then scatters its tile as seg_scatter_kernel does.
__global__ void __launch_bounds__(kWinThreads)
    compact_slots_kernel(const float* __restrict__ src, float* __restrict__ dst, const int* __restrict__ gp_src,
                         const int* __restrict__ tid_src, int* __restrict__ gp_dst, int* __restrict__ tid_dst,
                         const unsigned* __restrict__ flags, const int* __restrict__ M_end, int* __restrict__ M_out,
                         const WinRep R, unsigned long long* mail, unsigned tag) {
  __shared__ int s_sum[kWinThreads / 32];
  const int Mw = M_end[R.rep];
  const int ntiles = max(1, (Mw + kWinTile - 1) / kWinTile), nwords = (Mw + 31) / 32;
  const unsigned* const word0 = flags + (R.base >> 5);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int w0 = tile * (kWinTile / 32);
    int sum = 0;
    for (int w = t; w < w0; w += kWinThreads) sum += __popc(word0[w]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    if (lane == 0) s_sum[warp] = sum;
    __syncthreads();
    int before = 0;
#pragma unroll
    for (int w = 0; w < kWinThreads / 32; ++w) before += s_sum[w];
    __syncthreads();
    // a warp's four words, one after the other: lane l of word w holds slot 32 w + l, and the words of the
    // tile before them are counted by the warp itself
    const unsigned mine = w0 + lane < nwords ? word0[w0 + lane] : 0u;
    int incl = __popc(mine);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += y;
    }
#pragma unroll
    for (int i = 0; i < kWinTile / 32 / (kWinThreads / 32); ++i) {
      const int w = i * (kWinThreads / 32) + warp;
      const unsigned word = __shfl_sync(0xFFFFFFFFu, mine, w);
      const int upto = __shfl_sync(0xFFFFFFFFu, incl, w) - __popc(word);
      if ((word >> lane) & 1u) {
        const long long from = R.base + static_cast<long long>(w0 + w) * 32 + lane;
        const long long to = R.base + before + upto + __popc(word & ((1u << lane) - 1u));
        const int id = tid_src[from];
        dst[to] = src[from];
        gp_dst[to] = gp_src[from];
        tid_dst[to] = R.preserve ? -abs(id) : id;
      }
    }
    if (tile == ntiles - 1 && t == kWinThreads - 1) {   // lane 31 holds the tile's survivors
      M_out[R.rep] = before + incl;
      post_count(mail, tag, before + incl);
    }
  }
}

// ------------------------------------------------------------------------------------------------
// Large windows: a quad per thread while most of its slots live, then the living slots packed
// ------------------------------------------------------------------------------------------------
// A quad per thread shares one Philox block over four draws, but a warp walks all four lane positions, with
// both sampler branches where its lanes differ, as long as one of its 128 slots lives -- and new mutations
// die fast: of a tile of births half the slots are lost after two generations, four fifths after eight.
// Once fewer than kPackPairs of a tile's 256 threads have two living slots or more, the block therefore moves
// the frequencies to shared memory and hands out the living slots one per thread, densely (each evaluating
// its quad's Philox block alone), repacking every few generations.  A slot's counters depend on its position
// only, so who computes it does not matter.  Lost slots cost nothing from then on.
//
// Issue-bound (79 % of issue slots, 23 of 32 lanes).  Windows of 25 generations on a B200, against a quad per
// thread throughout (window_kernel): N = 2e5, L = 2.5e8, neutral 354 -> 293 us, gamma = -10 357 -> 293; N = 1e4 with 4
// million slots 201 -> 157; the batched windows of 256 replicates (N0 in [1e3, 1e4]) 400 -> 310 ms in all.
// A third of that is the shorter draw (binom_draw_count) and generation loop: 20 % fewer warp instructions.
//
// kPackPairs: 100 and 190 measured 1 % slower (the neutral half below).  The threads are counted after two
// generations of a full tile of births and then after each, after four of a tile the window began with and
// then after every fifth (one barrier: counting the slots themselves every third generation cost 8 % of the
// instructions); the first packed stage lasts three generations, each later one a generation longer (2 or 4
// at first: the same within 1 %).
constexpr int kPackPairs = 150;

// A whole quad's generation: Philox (q + 2, g, 0, 0), lanes x, y, z, w.
template <bool KEYS>
__device__ __forceinline__ void quad_generation(float (&x)[4], int q, const SlotGen& G, const PhiloxKeys& keys,
                                                int seed1, int seed2) {
  const int N = G.Nc, g = G.generation;
  if (N <= 0) {   // extinction generation: the population's row is cleared
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = 0.f;
    return;
  }
  if (!(G.sel_a == 0.f && G.sel_b == 0.f)) {
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = selected_freq<false>(x[j], G.sel_a, G.sel_b, G.F, G.h);
  }
  const float Nf = G.Nf;
  if (x[0] != 0.f || x[1] != 0.f || x[2] != 0.f || x[3] != 0.f) {
    uint4 r;
    if (KEYS) r = philox4x32_10_keys(make_uint4(static_cast<uint32_t>(q + 2), static_cast<uint32_t>(g), 0u, 0u), keys);
    else r = philox(seed1, seed2, q + 2, g, 0, 0);
    const uint32_t bits[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (x[j] != 0.f) x[j] = binom_draw_count(bits[j], x[j], N, Nf) / Nf;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (x[j] == 0.f) x[j] = 0.f;   // a negative zero of the caller's becomes a positive one, as a draw gives
}

// Exclusive position of this thread's `c` items in the block's order of (round, thread), and their total.
// s_part: [kWinThreads / 32] words.  Ends with the block past a barrier; s_part is free again after the next one.
__device__ __forceinline__ int pack_position(int c, int* s_part, int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) s_part[warp] = incl;
  __syncthreads();
  int before = 0;
  total = 0;
#pragma unroll
  for (int w = 0; w < kWinThreads / 32; ++w) {
    const int v = s_part[w];
    before += w < warp ? v : 0;
    total += v;
  }
  return before + incl - c;
}

template <bool KEYS>
__global__ void __launch_bounds__(kWinThreads, KEYS ? GF_WINDOW_MIN_BLOCKS_KEYS : GF_WINDOW_MIN_BLOCKS)
    window_pack_kernel(const float* __restrict__ A, float* __restrict__ B, int* __restrict__ id_gp,
                       int* __restrict__ id_tid, unsigned* __restrict__ flags, unsigned* __restrict__ tile_count,
                       const int* __restrict__ M_in, int* __restrict__ M_end, int* __restrict__ M_next,
                       const WinRep* __restrict__ reps, int nreps, const WinGen* __restrict__ recs, int total_tiles,
                       const int* __restrict__ total_dev, unsigned long long* __restrict__ stats,
                       int* __restrict__ fault, const PhiloxKeys keys, int* __restrict__ sched, const RepList list,
                       const WinRep one) {
  __shared__ int s_rep;
  __shared__ int s_tile;
  __shared__ int s_part[2][kWinThreads / 32];
  __shared__ int s_tile0[KEYS ? 1 : kRepCache];
  __shared__ SlotGen s_gen[kMaxWindowGenerations];
  __shared__ float s_new[kMaxWindowGenerations];
  __shared__ int s_scan[kWinThreads / 32];
  __shared__ int s_lost_stays;
  __shared__ float4 s_x[kWinThreads];
  __shared__ unsigned short s_list[2][kWinTile];
  const int lane = threadIdx.x & 31;
  const int ntiles_all = total_dev ? *total_dev : total_tiles;
  const int nlist = KEYS ? 1 : list_count(list, nreps);
  if (!KEYS) load_tile0(s_tile0, list, reps, nlist);
  int loaded = -1;   // the replicate whose records s_gen holds
  // tiles are handed out in order by an atomic counter, as in window_kernel
  for (;;) {
    if (threadIdx.x == 0) {
      const int t = atomicAdd(sched, 1);
      s_tile = t;
      s_rep = KEYS ? 0 : t < ntiles_all ? list_rep(list, find_rep_cached(s_tile0, list, reps, nlist, t)) : -1;
    }
    __syncthreads();
    const int gt = s_tile, rep = s_rep;
    if (gt >= ntiles_all) break;   // block-uniform
    const WinRep R = KEYS ? one : reps[rep];
    __syncthreads();
    const int t = gt - R.tile0;
    const int q = t * kWinThreads + threadIdx.x;  // quad within the replicate
    const int s0 = 4 * q;
    const int cap = static_cast<int>(R.capacity);
    const int M0 = M_in[R.rep];
    const long long end = M0 + R.births;
    // a tile past the replicate's end-of-window count has nothing to do (tile 0 keeps the bookkeeping)
    if (t > 0 && static_cast<long long>(t) * kWinTile >= end) continue;   // block-uniform
    if (rep != loaded) {
      load_slot_generations(s_gen, s_new, s_scan, &s_lost_stays, recs + R.rec, R.ngen, M0);
      loaded = rep;
    }
    float* const rowB = B + R.base;
    const float* const rowA = A + R.base;
    int* const gp = id_gp + R.base;
    int* const tid = id_tid + R.base;

    float x[4];
    if (s0 + 3 < M0) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(rowA + s0));
      x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) x[j] = (s0 + j < M0) ? rowA[s0 + j] : 0.f;
    }

    // a tile of births starts with the generation that appends its first one
    const int tile_first = t * kWinTile;
    int k = 0;
    if (tile_first >= M0) {
      int hi = R.ngen - 1;
      while (k < hi) {
        const int mid = (k + hi + 1) >> 1;
        if (s_gen[mid].M <= tile_first) k = mid;
        else hi = mid - 1;
      }
    }
    // ---- until every slot of the tile is born: whole quads, the scalar tail and births ----
#pragma unroll 1
    for (; k < R.ngen && s_gen[k].M < tile_first + kWinTile; ++k) {
      const SlotGen& G = s_gen[k];
      const int M = G.M;
      if (s0 + 3 < (M & ~3)) {
        quad_generation<KEYS>(x, q, G, keys, R.seed1, R.seed2);
      } else if (s0 < M) {
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {
          if (s0 + j >= M) break;
          const float v = slot_generation<KEYS>(j == 0 ? x[0] : j == 1 ? x[1] : j == 2 ? x[2] : x[3], s0 + j, G, keys,
                                                R.seed1, R.seed2);
          x[0] = j == 0 ? v : x[0];
          x[1] = j == 1 ? v : x[1];
          x[2] = j == 2 ? v : x[2];
          x[3] = j == 3 ? v : x[3];
        }
      }
      // births: slots [M, M + new_count) start at 1/Nc with ID (g, 0, slot - M + 1)
      const int Mn = k + 1 < R.ngen ? s_gen[k + 1].M : static_cast<int>(end);
      if (s0 + 3 >= M && s0 < Mn) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int e = s0 + j;
          if (e >= M && e < Mn && e < cap) {
            x[j] = s_new[k];
            gp[e] = G.generation;
            tid[e] = e - M + 1;
          }
        }
      }
    }
    // ---- a full tile: whole quads only, and now and then a count of the threads with two living slots ----
    bool packed = false;
    int check = tile_first >= M0 ? 2 : 4;
#pragma unroll 1
    while (k < R.ngen) {
      quad_generation<KEYS>(x, q, s_gen[k], keys, R.seed1, R.seed2);
      ++k;
      if (--check > 0) continue;
      check = tile_first >= M0 ? 1 : 5;
      if (k + 2 > R.ngen || !s_lost_stays) continue;
      int c = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) c += __float_as_uint(x[j]) != 0u ? 1 : 0;
      if (__syncthreads_count(c >= 2) <= kPackPairs) {
        packed = true;
        break;
      }
    }
    if (packed) {   // block-uniform
      int living;
      {
        s_x[threadIdx.x] = make_float4(x[0], x[1], x[2], x[3]);
        int c = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) c += __float_as_uint(x[j]) != 0u ? 1 : 0;
        int living_at = pack_position(c, s_part[0], living);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (__float_as_uint(x[j]) != 0u) s_list[0][living_at++] = static_cast<unsigned short>(4 * threadIdx.x + j);
        __syncthreads();
      }
      float* const s_xs = reinterpret_cast<float*>(s_x);
      int cur = 0, stage = 3;
      while (living > 0) {
        const int k1 = min(R.ngen, k + stage);
        int stays = 0;   // of this thread's slots, at positions t, t + 256, ...: how many still live
#pragma unroll 1
        for (int at = threadIdx.x; at < living; at += kWinThreads) {
          const int local = s_list[cur][at];
          float v = s_xs[local];
#pragma unroll 1
          for (int kk = k; kk < k1; ++kk) {
            v = slot_generation<KEYS>(v, tile_first + local, s_gen[kk], keys, R.seed1, R.seed2);
            if (__float_as_uint(v) == 0u) break;
          }
          s_xs[local] = v;
          stays += __float_as_uint(v) != 0u ? 1 : 0;
        }
        k = k1;
        if (k >= R.ngen) break;   // block-uniform
        const int had = living;
        int to = pack_position(stays, s_part[cur ^ 1], living);
#pragma unroll 1
        for (int at = threadIdx.x; at < had; at += kWinThreads) {
          const int local = s_list[cur][at];
          if (__float_as_uint(s_xs[local]) != 0u) s_list[cur ^ 1][to++] = static_cast<unsigned short>(local);
        }
        __syncthreads();
        cur ^= 1;
        stage += 1;
      }
      __syncthreads();
      const float4 v = s_x[threadIdx.x];
      x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
    }
    const int Mw = static_cast<int>(min(end, static_cast<long long>(cap)));
    if (s0 + 3 < Mw) {
      *reinterpret_cast<float4*>(rowB + s0) = make_float4(x[0], x[1], x[2], x[3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (s0 + j < Mw) rowB[s0 + j] = x[j];
    }

    if (R.compact) {
      // flag_segregating_mutations for one population: keep unless lost or fixed (when alive), or
      // if preserved
      const int alive = R.ngen > 0 ? recs[R.rec + R.ngen - 1].alive : 1;
      unsigned keep = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int e = s0 + j;
        if (e >= Mw) continue;
        // lost or fixed in the (only) population -- or the population is not alive -- removes it
        bool kp = alive && !(x[j] <= 0.f || x[j] >= 1.f);
        if (R.check_preserved && e < M0 && tid[e] < 0) kp = true;
        if (kp) keep |= 1u << j;
      }
      unsigned word = keep << ((lane & 7) * 4);
      word |= __shfl_xor_sync(0xFFFFFFFFu, word, 1);
      word |= __shfl_xor_sync(0xFFFFFFFFu, word, 2);
      word |= __shfl_xor_sync(0xFFFFFFFFu, word, 4);
      if ((lane & 7) == 0) flags[(R.base + s0) >> 5] = word;
      const int c = __reduce_add_sync(0xFFFFFFFFu, __popc(keep));
      if (lane == 0) s_scan[threadIdx.x >> 5] = c;
      __syncthreads();
      if (threadIdx.x == 0) {
        unsigned tot = 0;
#pragma unroll
        for (int w = 0; w < kWinThreads / 32; ++w) tot += s_scan[w];
        tile_count[R.base / kWinTile + t] = tot;
      }
      __syncthreads();
    }

    if (t == 0 && threadIdx.x == 0) {
      // window bookkeeping, once per replicate
      unsigned long long mg = 0;
      for (int kk = 0; kk < R.ngen; ++kk) mg += static_cast<unsigned long long>(s_gen[kk].M);
      atomicAdd(stats, mg);
      atomicAdd(stats + 1, static_cast<unsigned long long>(R.ngen));
      if (end > cap) atomicExch(fault, kFaultCapacity);
      M_end[R.rep] = Mw;
      if (M_next && !R.compact) M_next[R.rep] = Mw;
    }
  }
  // the launch's last block sets the scheduler back to zero, as in window_kernel
  if (threadIdx.x == 0) {
    __threadfence();
    const int finished = atomicAdd(sched + 1, 1);
    if (finished == static_cast<int>(gridDim.x) - 1) {
      sched[0] = 0;
      sched[1] = 0;
    }
  }
}

// One block per replicate: exclusive scan of its tile survivor counts, compacted count.  Each thread
// takes kSegScanItems consecutive tiles, so one pass covers 8,192 tiles (8.4 M slots).  SINGLE: one
// replicate, `one`, whose count also goes to the host.
constexpr int kSegScanThreads = 1024;
constexpr int kSegScanItems = 8;
template <bool SINGLE>
__global__ void __launch_bounds__(kSegScanThreads)
    seg_scan_kernel(const unsigned* __restrict__ tile_count, unsigned* __restrict__ tile_offset,
                    const WinRep* __restrict__ reps, const int* __restrict__ M_end, int* __restrict__ M_out,
                    const RepList list, const WinRep one, unsigned long long* mail, unsigned tag) {
  if (!SINGLE && list.count && static_cast<int>(blockIdx.x) >= *list.count) return;
  const WinRep R = SINGLE ? one : reps[list_rep(list, blockIdx.x)];
  if (!R.compact) return;
  __shared__ unsigned s_warp[kSegScanThreads / 32];
  __shared__ unsigned s_carry;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = (M_end[R.rep] + kWinTile - 1) / kWinTile;
  const long long t0 = R.base / kWinTile;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (int base = 0; base < n; base += kSegScanThreads * kSegScanItems) {
    const int first = base + threadIdx.x * kSegScanItems;
    unsigned v[kSegScanItems];
    unsigned sum = 0;
#pragma unroll
    for (int k = 0; k < kSegScanItems; ++k) {
      v[k] = first + k < n ? tile_count[t0 + first + k] : 0u;
      sum += v[k];
    }
    unsigned incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      const unsigned wv = s_warp[lane];
      unsigned wi = wv;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xFFFFFFFFu, wi, o);
        if (lane >= o) wi += y;
      }
      s_warp[lane] = wi - wv;
    }
    __syncthreads();
    unsigned run = s_carry + s_warp[warp] + incl - sum;
#pragma unroll
    for (int k = 0; k < kSegScanItems; ++k) {
      if (first + k < n) tile_offset[t0 + first + k] = run;
      run += v[k];
    }
    __syncthreads();
    if (threadIdx.x == kSegScanThreads - 1) s_carry = run;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    M_out[R.rep] = static_cast<int>(s_carry);
    if (SINGLE) post_count(mail, tag, static_cast<int>(s_carry));
  }
}

// Stable scatter of every compacting replicate's survivors (scatter_arrays, go_fish_impl.cu:147-189),
// staged through shared memory into one contiguous run per tile.  FUSED stages the frequency and
// both ID words of a tile together (one barrier, the three loads in flight at once, 12 KB of staging)
// -- faster for one large replicate, passed by value as `one`; otherwise the arrays go one after the other through one 4 KB
// buffer, which keeps more blocks resident for the many small tiles of a batch.
template <bool FUSED>
__global__ void __launch_bounds__(kWinThreads)
    seg_scatter_kernel(const float* __restrict__ src, float* __restrict__ dst, const int* __restrict__ gp_src,
                       const int* __restrict__ tid_src, int* __restrict__ gp_dst, int* __restrict__ tid_dst,
                       const unsigned* __restrict__ flags, const unsigned* __restrict__ tile_offset,
                       const WinRep* __restrict__ reps, int nreps, const int* __restrict__ M_end, int total_tiles,
                       const int* __restrict__ total_dev, const RepList list, const WinRep one) {
  __shared__ int s_rep;
  __shared__ int s_tile0[FUSED ? 1 : kRepCache];
  const int ntiles_all = total_dev ? *total_dev : total_tiles;
  const int nlist = FUSED ? 1 : list_count(list, nreps);
  if (!FUSED) load_tile0(s_tile0, list, reps, nlist);
  __shared__ unsigned s_words[32];
  __shared__ unsigned s_prefix[32];
  __shared__ float s_stage[FUSED ? 3 * kWinTile : kWinTile];
  const int t = threadIdx.x;
  for (int gt = blockIdx.x; gt < ntiles_all; gt += gridDim.x) {
    if (!FUSED) {
      if (t == 0) s_rep = list_rep(list, find_rep_cached(s_tile0, list, reps, nlist, gt));
      __syncthreads();
    }
    const WinRep R = FUSED ? one : reps[s_rep];
    if (!FUSED) __syncthreads();
    const int tile = gt - R.tile0;
    const int ntiles = (M_end[R.rep] + kWinTile - 1) / kWinTile;
    if (!R.compact || tile >= ntiles) continue;  // block-uniform
    const long long atile = R.base / kWinTile + tile;
    if (t < 32) {
      const unsigned w = flags[atile * 32 + t];
      s_words[t] = w;
      const unsigned c = __popc(w);
      unsigned incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (t >= o) incl += y;
      }
      s_prefix[t] = incl - c;
    }
    __syncthreads();
    const int w = t >> 3, sh = (t & 7) * 4;
    const unsigned word = s_words[w];
    const unsigned nib = (word >> sh) & 0xFu;
    const int local = static_cast<int>(s_prefix[w] + __popc(word & ((1u << sh) - 1u)));
    const int count = static_cast<int>(s_prefix[31] + __popc(s_words[31]));
    const long long out0 = R.base + tile_offset[atile];
    const long long in0 = R.base + static_cast<long long>(tile) * kWinTile + 4 * t;
    if constexpr (FUSED) {
      int* s_gstage = reinterpret_cast<int*>(s_stage + kWinTile);
      int* s_tstage = s_gstage + kWinTile;
      if (nib) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(src + in0));
        const int4 g = __ldg(reinterpret_cast<const int4*>(gp_src + in0));
        const int4 d = __ldg(reinterpret_cast<const int4*>(tid_src + in0));
        const bool mark = R.preserve != 0;
        const float vv[4] = {v.x, v.y, v.z, v.w};
        const int gg[4] = {g.x, g.y, g.z, g.w};
        const int dd[4] = {d.x, d.y, d.z, d.w};
        int k = local;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (!((nib >> j) & 1u)) continue;
          s_stage[k] = vv[j];
          s_gstage[k] = gg[j];
          s_tstage[k++] = mark ? -abs(dd[j]) : dd[j];
        }
      }
      __syncthreads();
      for (int k = t; k < count; k += kWinThreads) {
        dst[out0 + k] = s_stage[k];
        gp_dst[out0 + k] = s_gstage[k];
        tid_dst[out0 + k] = s_tstage[k];
      }
      __syncthreads();
      continue;
    }
    if (nib) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(src + in0));
      int k = local;
      if (nib & 1u) s_stage[k++] = v.x;
      if (nib & 2u) s_stage[k++] = v.y;
      if (nib & 4u) s_stage[k++] = v.z;
      if (nib & 8u) s_stage[k++] = v.w;
    }
    __syncthreads();
    for (int k = t; k < count; k += kWinThreads) dst[out0 + k] = s_stage[k];
    __syncthreads();
    int* s_istage = reinterpret_cast<int*>(s_stage);
    for (int arr = 0; arr < 2; ++arr) {
      const int* s = arr ? tid_src : gp_src;
      int* d = arr ? tid_dst : gp_dst;
      if (nib) {
        const int4 v = __ldg(reinterpret_cast<const int4*>(s + in0));
        int k = local;
        const bool mark = arr && R.preserve;
        if (nib & 1u) s_istage[k++] = mark ? -abs(v.x) : v.x;
        if (nib & 2u) s_istage[k++] = mark ? -abs(v.y) : v.y;
        if (nib & 4u) s_istage[k++] = mark ? -abs(v.z) : v.z;
        if (nib & 8u) s_istage[k++] = mark ? -abs(v.w) : v.w;
      }
      __syncthreads();
      for (int k = t; k < count; k += kWinThreads) d[out0 + k] = s_istage[k];
      __syncthreads();
    }
  }
}

// Tile assignment of a batched super-step (batch_tiles_kernel), on the engine stream.
void assign_batch_tiles(Engine* e, WinRep* d_reps, int nreps, const int* M_in, const WinGen* recs,
                        int* total_out) {
  batch_tiles_kernel<<<1, 1024, 0, e->stream>>>(d_reps, nreps, M_in, recs, total_out);
  e->kernel_launches += 1;
}

void batch_step_tiles(Engine* e, WinRep* d_table, int R, const int* M_in, const WinGen* recs, int* total_out,
                      int* d_step, const BatchStepPlan& plan, const int* region_off, const long long* region_base,
                      const StepRep* steprep, int* fault, int* list_rep, int* list_tile0, int* list_count) {
  batch_step_kernel<<<1, 1024, 0, e->stream>>>(d_table, R, M_in, recs, total_out, d_step, plan, region_off,
                                               region_base, steprep, fault, list_rep, list_tile0, list_count);
  e->kernel_launches += 1;
}

template <bool KEYS, typename Kernel>
static void launch_window_tiles(Engine* e, const WindowLaunch& w, Kernel kernel, int occupancy) {
  const int per_sm = e->blocks_per_sm > 0 ? std::min(e->blocks_per_sm, occupancy) : occupancy;
  const int blocks = std::max(1, std::min(w.total_tiles, e->num_sms * per_sm));
  const PhiloxKeys keys = philox_round_keys(w.one.seed1, w.one.seed2);
  kernel<<<blocks, kWinThreads, 0, e->stream>>>(w.A, w.B, w.id_gp_cur, w.id_tid_cur, w.flags, w.tile_count, w.M_in,
                                                w.M_end, w.M_next, w.reps, w.nreps, w.recs, w.total_tiles,
                                                w.total_tiles_dev, w.stats, w.fault, keys, w.sched, w.list, w.one);
}

// Resident blocks per SM of a kernel (the same on every B200).
template <typename Kernel>
static int resident_blocks(Kernel kernel) {
  int o = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, kernel, kWinThreads, 0) != cudaSuccess || o < 1) {
    cudaGetLastError();
    o = 1;
  }
  return o;
}

// One large or several replicates: window_pack_kernel (lane order only) or window_kernel.
template <int DRAW, bool KEYS>
static void launch_window_kernel(Engine* e, const WindowLaunch& w, WindowForm form) {
  if (DRAW == kDrawLanes && form == WindowForm::pack) {
    static const int occupancy = resident_blocks(window_pack_kernel<KEYS>);   // thread-safe, once
    launch_window_tiles<KEYS>(e, w, window_pack_kernel<KEYS>, occupancy);
  } else {
    static const int occupancy = resident_blocks(window_kernel<DRAW, KEYS>);
    launch_window_tiles<KEYS>(e, w, window_kernel<DRAW, KEYS>, occupancy);
  }
}

// Launch a window over w.nreps replicates (one passed by value) and, for the replicates that compact, the
// segmented scan and scatter into `compact_dst` (the other state buffer).
gf_status window_run(Engine* e, const WindowLaunch& w, float* compact_dst, cudaEvent_t after_window,
                     cudaEvent_t before_compaction) {
  const bool single = w.reps == nullptr;
  const WindowForm form = window_form(single, e->draw_strategy == kDrawLanes, w.pack, w.expected_slots, w.longest);
  const bool slots = form == WindowForm::slots;
  if (slots) {
    const long long blocks = (w.one.ntiles * static_cast<long long>(kWinTile) + kSlotThreads - 1) / kSlotThreads;
    window_slots_kernel<<<static_cast<int>(std::max(1ll, std::min(blocks, 16ll * e->num_sms))), kSlotThreads, 0,
                          e->stream>>>(w.A, w.B, w.id_gp_cur, w.id_tid_cur, w.flags, w.M_in, w.M_end, w.M_next, w.recs,
                                       w.stats, w.fault, philox_round_keys(w.one.seed1, w.one.seed2), w.one);
  } else {
    switch (e->draw_strategy) {
      case kDrawWarp:
        if (single) launch_window_kernel<kDrawWarp, true>(e, w, form);
        else launch_window_kernel<kDrawWarp, false>(e, w, form);
        break;
      case kDrawGrouped:
        if (single) launch_window_kernel<kDrawGrouped, true>(e, w, form);
        else launch_window_kernel<kDrawGrouped, false>(e, w, form);
        break;
      case kDrawNormalAll:
        if (single) launch_window_kernel<kDrawNormalAll, true>(e, w, form);
        else launch_window_kernel<kDrawNormalAll, false>(e, w, form);
        break;
      case kDrawPooledSearch:
        if (single) launch_window_kernel<kDrawPooledSearch, true>(e, w, form);
        else launch_window_kernel<kDrawPooledSearch, false>(e, w, form);
        break;
      default:
        if (single) launch_window_kernel<kDrawLanes, true>(e, w, form);
        else launch_window_kernel<kDrawLanes, false>(e, w, form);
        break;
    }
  }
  GF_CUDA(e, cudaGetLastError());
  e->kernel_launches += 1;
  if (after_window) GF_CUDA(e, cudaEventRecord(after_window, e->stream));
  if (before_compaction) GF_CUDA(e, cudaEventRecord(before_compaction, e->stream));
  if (!w.any_compact) return GF_OK;
  const int sblocks = std::max(1, std::min(w.total_tiles, e->num_sms * 8));
  if (slots) {
    compact_slots_kernel<<<sblocks, kWinThreads, 0, e->stream>>>(w.B, compact_dst, w.id_gp_cur, w.id_tid_cur,
                                                                 w.id_gp_next, w.id_tid_next, w.flags, w.M_end, w.M_out,
                                                                 w.one, w.mail, w.mail_tag);
    GF_CUDA(e, cudaGetLastError());
    e->kernel_launches += 1;
    return GF_OK;
  }
  auto scan = single ? seg_scan_kernel<true> : seg_scan_kernel<false>;
  scan<<<w.nreps, kSegScanThreads, 0, e->stream>>>(w.tile_count, w.tile_offset, w.reps, w.M_end, w.M_out, w.list, w.one,
                                                   w.mail, w.mail_tag);
  GF_CUDA(e, cudaGetLastError());
  auto scatter = single ? seg_scatter_kernel<true> : seg_scatter_kernel<false>;
  scatter<<<sblocks, kWinThreads, 0, e->stream>>>(w.B, compact_dst, w.id_gp_cur, w.id_tid_cur, w.id_gp_next,
                                                  w.id_tid_next, w.flags, w.tile_offset, w.reps, w.nreps, w.M_end,
                                                  w.total_tiles, w.total_tiles_dev, w.list, w.one);
  GF_CUDA(e, cudaGetLastError());
  e->kernel_launches += 2;
  return GF_OK;
}

}  // namespace gf
