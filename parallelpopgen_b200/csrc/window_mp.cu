// Windowed drift for 2 to 8 populations: every generation of a compaction window in one launch.
//
// Migration mixes the frequencies of one mutation across populations and nothing else, so a thread
// can carry the P rows of one slot through all generations of a window, as the single-population
// window kernels (window.cu) do for one row.  Each generation repeats the per-generation kernel's
// arithmetic for every drifted population in order (migration_selection_drift,
// go_fish_impl.cuh:93-124): the migration sum over the rows as they stood at the start of the
// generation, selection, the draw with counter (q + 2, g, p, 0) for whole quads and (slot + 2, g, p, 0)
// for the scalar tail, float(j) / Nc.  Births are appended after the drift (add_new_mutations,
// go_fish_impl.cu:138-145: row p = 1/Nc of the population that drew them, other rows 0, in population
// order), and only the last generation writes the rows and the compaction flags
// (flag_segregating_mutations, go_fish_impl.cuh:137-176).
//
// The per-generation kernel leaves the rows of populations that it does not drift untouched; the engine
// forms a window only while every such row is zero in both state buffers (a population that has not
// been founded yet), so writing those rows back unchanged is the same as not writing them.
#include <cuda_runtime.h>

#include <algorithm>

#include "gf_drift.cuh"
#include "gf_internal.h"

namespace gf {

// A slot per thread, and the four lanes of a quad share its Philox blocks: lane p computes population p's and
// a 4 x 4 transposition hands every lane its word of each (a block and 16 instructions instead of P blocks).
// New mutations die fast and a block's other warps do not: once the living slots of a tile are few enough the
// block packs them, one per thread, each then evaluating its blocks alone, and packs again every few
// generations (window_pack_kernel does the same for one population).
//
// Issue-bound (76 % of issue slots, 24 of 32 lanes).  Windows of 25 generations on a B200, against a quad per
// thread with the rows of its four slots in registers (four blocks an SM, lost slots carried along): three
// populations, N = 50,000, L = 1e8 (35 generations, 1.6 M slots at the end) 462 -> 370 us; two, N = 100,000 285 -> 265;
// four, N = 30,000 391 -> 282; three of N = 2,000 to 20,000 (4,000 to 130,000 slots) 137 -> 50 to 61.  Five to
// eight populations, which had a launch per generation: 25 generations of six, N = 2,000 532 -> 87 us, N = 30,000,
// L = 5e7 776 -> 398; of eight 637 -> 111, N = 30,000, L = 4e7 982 -> 604.  Packing at half
// the tile instead of three quarters: the same within 1 %.
// Resident blocks: 5 (48 registers), 4 from four populations on, whose rows would spill.  6 is 10 % slower for three.
constexpr int mp_min_blocks(int P, bool small) { return small ? (P <= 4 ? 8 : 6) : P <= 3 ? 5 : P <= 4 ? 4 : 3; }

// Slots of a thread, threads of a block: large states hand out half compaction tiles (512 slots; a whole one is
// too coarse for the few hundred that carry the old mutations) and pack them; small ones spread over many SMs.
template <bool SMALL>
struct MpShape {
  static constexpr int kSlots = SMALL ? 1 : 2;
  static constexpr int kThreads = SMALL ? 128 : 256;
  static constexpr int kTile = kSlots * kThreads;
};
static_assert(2 * MpShape<false>::kTile == kTileSlots, "a window tile is half a compaction tile");
static_assert(MpShape<true>::kThreads >= kMaxWindowGenerations, "a thread per record");

template <int P>
struct MpLimit {
  static constexpr int kGens = mp_max_window(P);
};

// The fields of one generation record the drift reads.
template <int P>
struct __align__(16) MpGen {
  int generation;
  int M;           // mutations at the generation's start
  int neutral;     // every drifted population has s(x) == 0 (the per-generation kernel's NEUTRAL case)
  int drift_mask;
  struct Pop {
    int Nc;
    float Nf;      // Nc
    float sel_a, sel_b, F, h;
  } pop[P];
  float mig[P * P];  // [from * P + to]
};

// Drift of one population's slot in a whole quad: `bits` is its word of the quad's Philox block.  The count of
// binom_draw_count, with a shorter way out for the tiny means that migrants give: the Poisson search returns 0
// if u <= exp(-mean), and exp(-mean) > 0.9999 - mean whatever the rounding.
__device__ __forceinline__ float mp_draw(uint32_t bits, float x, int N, float Nf) {
  const float mean = x * N;
  if (Nf >= kBinomNBoundary && u01(bits) <= 0.9999f - mean) return 0.f;
  return binom_draw_count(bits, x, N, Nf);
}

// After this, lane j of each four lanes holds word j of the blocks of the four.
__device__ __forceinline__ void transpose_quad(uint32_t (&r)[4], int lane) {
  const bool b0 = lane & 1, b1 = lane & 2;
#pragma unroll
  for (int i = 0; i < 4; i += 2) {
    const uint32_t got = __shfl_xor_sync(0xFFFFFFFFu, b0 ? r[i] : r[i + 1], 1);
    if (b0) r[i] = got;
    else r[i + 1] = got;
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint32_t got = __shfl_xor_sync(0xFFFFFFFFu, b1 ? r[i] : r[i + 2], 2);
    if (b1) r[i] = got;
    else r[i + 2] = got;
  }
}

template <int P>
__device__ __forceinline__ bool mp_living(const float (&x)[P]) {
  unsigned any = 0;
#pragma unroll
  for (int p = 0; p < P; ++p) any |= __float_as_uint(x[p]);
  return any != 0;
}

template <int P>
__device__ __forceinline__ float mp_migrated(const float (&x)[P], const MpGen<P>& G, int p) {
  float xm = 0.f;
#pragma unroll
  for (int kk = 0; kk < P; ++kk) xm += G.mig[kk * P + p] * x[kk];
  return xm;
}

// Slot e of a whole quad through generation G.  QUAD: the warp's lanes hold consecutive slots and all call this,
// `live` or not (a slot that is not keeps its rows).
template <int P, bool QUAD>
__device__ __forceinline__ void mp_generation(float (&x)[P], bool live, int e, const MpGen<P>& G, const PhiloxKeys& keys,
                                              int lane) {
  const uint32_t q2 = static_cast<uint32_t>((e >> 2) + 2), g = static_cast<uint32_t>(G.generation);
  uint32_t bits[(P + 3) / 4][4];
  if (QUAD) {
#pragma unroll
    for (int b = 0; b < (P + 3) / 4; ++b) {   // four populations at a time
      const uint4 r = philox4x32_10_keys(make_uint4(q2, g, static_cast<uint32_t>(4 * b + (lane & 3)), 0u), keys);
      bits[b][0] = r.x;
      bits[b][1] = r.y;
      bits[b][2] = r.z;
      bits[b][3] = r.w;
      transpose_quad(bits[b], lane);
    }
  }
  if (!live) return;
  float xm[P];
#pragma unroll
  for (int p = 0; p < P; ++p) xm[p] = mp_migrated<P>(x, G, p);
#pragma unroll
  for (int p = 0; p < P; ++p) {
    if (!((G.drift_mask >> p) & 1)) continue;
    const auto& pop = G.pop[p];
    const int N = pop.Nc;
    float count = 0.f;
    if (N > 0) {  // N == 0: extinction generation, the population's row is cleared
      float xs = xm[p];
      if (!G.neutral) xs = selected_freq<false>(xs, pop.sel_a, pop.sel_b, pop.F, pop.h);
      if (xs != 0.f) {
        uint32_t b;
        if (QUAD) {
          b = bits[p / 4][p % 4];
        } else {
          const uint4 r = philox4x32_10_keys(make_uint4(q2, g, static_cast<uint32_t>(p), 0u), keys);
          b = (e & 2) ? ((e & 1) ? r.w : r.z) : ((e & 1) ? r.y : r.x);
        }
        count = mp_draw(b, xs, N, pop.Nf);
      }
    }
    x[p] = N > 0 ? count / pop.Nf : 0.f;
  }
}

// The same for a slot of the scalar tail: counter (slot + 2), variance in double.
template <int P>
__device__ __noinline__ void mp_tail(float* x, int e, const MpGen<P>& G, int seed1, int seed2) {
  float xo[P];
#pragma unroll
  for (int p = 0; p < P; ++p) xo[p] = x[p];
#pragma unroll 1
  for (int p = 0; p < P; ++p) {
    if (!((G.drift_mask >> p) & 1)) continue;
    const auto& pop = G.pop[p];
    const float xm = mp_migrated<P>(xo, G, p);
    float o = 0.f;
    if (pop.Nc > 0) {
      const float xs = G.neutral ? selected_freq<true>(xm, 0.f, 0.f, 0.f, 0.f)
                                 : selected_freq<false>(xm, pop.sel_a, pop.sel_b, pop.F, pop.h);
      o = static_cast<float>(clampi(drift_tail(seed1, seed2, e, G.generation, p, xs, pop.Nc), 0, pop.Nc)) / pop.Nf;
    }
    x[p] = o;
  }
}

// The window's records, and whether a mutation lost everywhere stays lost through every generation (not so where
// a selected frequency of 0 is not 0, or a migration factor is not finite).  All threads of the block.
template <int P, int THREADS>
__device__ __forceinline__ void load_mp_generations(MpGen<P>* s_gen, int* s_scan, int* s_lost_stays,
                                                    const GenArgs* __restrict__ table, int ngen, int M0) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  if (t == 0) *s_lost_stays = 1;
  __syncthreads();
  int births = 0;
  if (t < ngen) {
    const GenArgs& a = table[t];
    MpGen<P>& G = s_gen[t];
    births = a.new_offset[P];
    G.generation = a.generation;
    G.drift_mask = a.drift_mask;
    int neutral = 1;
    bool stays = true;
#pragma unroll
    for (int p = 0; p < P; ++p) {
      G.pop[p] = {a.Nc[p], static_cast<float>(a.Nc[p]), a.sel_a[p], a.sel_b[p], a.F[p], a.h[p]};
      if (((a.drift_mask >> p) & 1) && (a.sel_a[p] != 0.f || a.sel_b[p] != 0.f)) {
        neutral = 0;
      }
    }
    G.neutral = neutral;
#pragma unroll
    for (int p = 0; p < P; ++p)
      if (!neutral && !(selected_freq<false>(0.f, a.sel_a[p], a.sel_b[p], a.F[p], a.h[p]) == 0.f)) stays = false;
#pragma unroll
    for (int i = 0; i < P * P; ++i) {
      G.mig[i] = a.mig[i];
      if (!isfinite(a.mig[i])) stays = false;
    }
    if (!stays) *s_lost_stays = 0;
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

// Exclusive position of this thread's `c` items in the block's order of threads, and their total.  Ends past a
// barrier; s_part is free again after the next one.
template <int THREADS>
__device__ __forceinline__ int mp_position(int c, int* s_part, int& total) {
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
  for (int w = 0; w < THREADS / 32; ++w) {
    const int v = s_part[w];
    before += w < warp ? v : 0;
    total += v;
  }
  return before + incl - c;
}

template <int P, bool SMALL>
__global__ void __launch_bounds__(MpShape<SMALL>::kThreads, mp_min_blocks(P, SMALL))
    window_mp_kernel(const float* __restrict__ A, float* __restrict__ B, long long stride, int* __restrict__ id_gp,
                     int* __restrict__ id_tid, unsigned* __restrict__ flags, unsigned* __restrict__ tile_count,
                     int* __restrict__ d_count, int slot_in, int slot_out, long long capacity,
                     const GenArgs* __restrict__ table, int ngen, long long births, int compact, int check_preserved,
                     int seed1, int seed2, unsigned long long* __restrict__ stats, const PhiloxKeys keys) {
  constexpr int kThreads = MpShape<SMALL>::kThreads, kSlots = MpShape<SMALL>::kSlots, kTile = MpShape<SMALL>::kTile;
  __shared__ MpGen<P> s_gen[MpLimit<P>::kGens];
  __shared__ float s_x[SMALL ? 1 : P][SMALL ? 1 : kTile];
  __shared__ unsigned short s_list[2][SMALL ? 1 : kTile];
  __shared__ int s_part[2][kThreads / 32];
  __shared__ int s_scan[kThreads / 32];
  __shared__ int s_lost_stays;
  __shared__ int s_tile;
  int* const sched = d_count + kSchedWord;   // tile scheduler: next tile, blocks finished
  const int lane = threadIdx.x & 31;
  const int M0 = d_count[slot_in];
  const long long end = static_cast<long long>(M0) + births;  // slots at the window end
  const int cap = static_cast<int>(capacity);
  const int Mw = static_cast<int>(min(end, capacity));
  const int ntiles = SMALL ? (Mw + kTile - 1) / kTile : 2 * ((Mw + kTileSlots - 1) / kTileSlots);
  if (SMALL && static_cast<int>(blockIdx.x) >= ntiles && blockIdx.x > 0) return;   // block 0 keeps the books
  load_mp_generations<P, kThreads>(s_gen, s_scan, &s_lost_stays, table, ngen, M0);
  const bool lost_stays = s_lost_stays != 0;
  const int alive = table[ngen - 1].alive_mask;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    d_count[slot_out] = Mw;
    d_count[3] = Mw;
    if (end > capacity) atomicExch(d_count + 2, kFaultCapacity);  // births past the rows are not written
    unsigned long long mg = 0;
    for (int k = 0; k < ngen; ++k) mg += static_cast<unsigned long long>(s_gen[k].M);
    stats[0] += mg;
    stats[1] += static_cast<unsigned long long>(ngen);
  }

  // tiles of a large state are handed out in order by an atomic counter (cheap tiles of late-born slots balance out)
  for (int t = blockIdx.x;; t += gridDim.x) {
    if (!SMALL) {
      if (threadIdx.x == 0) s_tile = atomicAdd(sched, 1);
      __syncthreads();
      t = s_tile;
      __syncthreads();
    }
    if (t >= ntiles) break;   // block-uniform
    const int tile_first = t * kTile;
    // a tile of births starts with the generation that appends its first one
    int k = 0;
    if (tile_first >= M0) {
      int hi = ngen - 1;
      while (k < hi) {
        const int mid = (k + hi + 1) >> 1;
        if (s_gen[mid].M <= tile_first) k = mid;
        else hi = mid - 1;
      }
    }
    // ---- consecutive slots, until few of them live ----
    float x[P];
    bool packed = false, first = true;
    int stage = SMALL ? ngen : tile_first >= M0 ? 3 : 5, living = 0;
#pragma unroll 1
    while (k < ngen) {
      const int k1 = min(ngen, k + stage);
      unsigned here = 0;   // bit i: this thread's slot i lives
#pragma unroll 1
      for (int i = 0; i < kSlots; ++i) {
        const int local = i * kThreads + threadIdx.x, e = tile_first + local;
#pragma unroll
        for (int p = 0; p < P; ++p) x[p] = first ? (e < M0 ? A[p * stride + e] : 0.f) : s_x[SMALL ? 0 : p][SMALL ? 0 : local];
#pragma unroll 1
        for (int kk = k; kk < k1; ++kk) {
          const MpGen<P>& G = s_gen[kk];
          const int M = G.M;
          const bool live = e < M && (!lost_stays || mp_living<P>(x));
          if (__any_sync(0xFFFFFFFFu, live)) {
            mp_generation<P, true>(x, live && e < (M & ~3), e, G, keys, lane);
            if (live && e >= (M & ~3)) {
              float xt[P];
#pragma unroll
              for (int p = 0; p < P; ++p) xt[p] = x[p];
              mp_tail<P>(xt, e, G, seed1, seed2);
#pragma unroll
              for (int p = 0; p < P; ++p) x[p] = xt[p];
            }
          }
          // births: slots [M, M + new) in population order, row p = 1/Nc, ID (g, p, slot - offset_p + 1)
          const int Mn = kk + 1 < ngen ? s_gen[kk + 1].M : static_cast<int>(end);
          if (e >= M && e < Mn && e < cap) {
            const int r = e - M;
            int p = 0;
            while (p + 1 < P && r >= table[kk].new_offset[p + 1]) ++p;
            const float f = table[kk].new_freq[p];
#pragma unroll
            for (int pp = 0; pp < P; ++pp) x[pp] = (pp == p) ? f : 0.f;
            id_gp[e] = G.generation | (p << 24);
            id_tid[e] = r - table[kk].new_offset[p] + 1;
          }
        }
        if (!SMALL) {
#pragma unroll
          for (int p = 0; p < P; ++p) s_x[p][local] = x[p];
          here |= (mp_living<P>(x) ? 1u : 0u) << i;
        }
      }
      first = false;
      k = k1;
      if (SMALL || k + 2 > ngen || !lost_stays || s_gen[k].M < tile_first + kTile) continue;
      int at = mp_position<kThreads>(__popc(here), s_part[0], living);
      if (living <= kTile * 3 / 4) {
        packed = true;
#pragma unroll
        for (int i = 0; i < kSlots; ++i)
          if ((here >> i) & 1u) s_list[0][at++] = static_cast<unsigned short>(i * kThreads + threadIdx.x);
        __syncthreads();
        break;
      }
      __syncthreads();
    }
    // ---- the living slots, packed ----
    if (!SMALL && packed) {   // block-uniform
      int cur = 0, pstage = 3;
      while (living > 0) {
        const int k1 = min(ngen, k + pstage);
        int stays = 0;   // of this thread's slots, at positions t, t + 256, ...: how many still live
#pragma unroll 1
        for (int at = threadIdx.x; at < living; at += kThreads) {
          const int local = s_list[cur][at];
#pragma unroll
          for (int p = 0; p < P; ++p) x[p] = s_x[p][local];
#pragma unroll 1
          for (int kk = k; kk < k1; ++kk) {
            mp_generation<P, false>(x, true, tile_first + local, s_gen[kk], keys, lane);
            if (!mp_living<P>(x)) break;
          }
#pragma unroll
          for (int p = 0; p < P; ++p) s_x[p][local] = x[p];
          stays += mp_living<P>(x) ? 1 : 0;
        }
        k = k1;
        if (k >= ngen) break;   // block-uniform
        const int had = living;
        int to = mp_position<kThreads>(stays, s_part[cur ^ 1], living);
#pragma unroll 1
        for (int at = threadIdx.x; at < had; at += kThreads) {
          const int local = s_list[cur][at];
          unsigned any = 0;
#pragma unroll
          for (int p = 0; p < P; ++p) any |= __float_as_uint(s_x[p][local]);
          if (any) s_list[cur ^ 1][to++] = static_cast<unsigned short>(local);
        }
        __syncthreads();
        cur ^= 1;
        pstage += 1;
      }
      __syncthreads();
    }

    int kept = 0;
#pragma unroll 1
    for (int i = 0; i < kSlots; ++i) {
      const int local = i * kThreads + threadIdx.x, e = tile_first + local;
      bool keep = false;
      if (!SMALL) {
#pragma unroll
        for (int p = 0; p < P; ++p) x[p] = s_x[p][local];
      }
      if (e < Mw) {
        // keep unless lost in every alive population or fixed in every alive population, or preserved
        bool zero = true, one = true;
#pragma unroll
        for (int p = 0; p < P; ++p) {
          B[p * stride + e] = x[p];
          if ((alive >> p) & 1) {
            zero = zero && (x[p] <= 0.f);
            one = one && (x[p] >= 1.f);
          }
        }
        keep = !(zero || one);
        if (check_preserved && e < M0 && id_tid[e] < 0) keep = true;
      }
      if (compact) {
        const unsigned word = __ballot_sync(0xFFFFFFFFu, keep);
        if (lane == 0) flags[e >> 5] = word;
        kept += __popc(word);
      }
    }
    if (!SMALL && compact) {
      if (lane == 0) s_scan[threadIdx.x >> 5] = kept;
      __syncthreads();
      if (threadIdx.x == 0) {
        unsigned tot = 0;
#pragma unroll
        for (int w = 0; w < kThreads / 32; ++w) tot += s_scan[w];
        reinterpret_cast<unsigned short*>(tile_count)[t] = static_cast<unsigned short>(tot);   // the scan adds the halves
      }
      __syncthreads();
    }
  }
  // the last block to finish resets the scheduler for the next launch on this stream
  if (!SMALL && threadIdx.x == 0) {
    __threadfence();
    const int finished = atomicAdd(sched + 1, 1);
    if (finished == static_cast<int>(gridDim.x) - 1) {
      sched[0] = 0;
      sched[1] = 0;
    }
  }
}

// The compaction of a small window in one launch: a block counts the survivors before its tile from the flag
// words themselves (a few hundred words from L2), then moves its tile's.
template <int P>
__global__ void __launch_bounds__(256)
    compact_mp_kernel(const float* __restrict__ src, float* __restrict__ dst, long long stride,
                      const int* __restrict__ gp_src, const int* __restrict__ tid_src, int* __restrict__ gp_dst,
                      int* __restrict__ tid_dst, const unsigned* __restrict__ flags, int* __restrict__ d_count,
                      int slot_out, int preserve, unsigned long long* mail, unsigned tag) {
  __shared__ int s_sum[8];
  const int Mw = d_count[3];
  const int ntiles = max(1, (Mw + kTileSlots - 1) / kTileSlots), nwords = (Mw + 31) / 32;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int w0 = tile * (kTileSlots / 32);
    int sum = 0;
    for (int w = t; w < w0; w += 256) sum += __popc(flags[w]);
    sum = __reduce_add_sync(0xFFFFFFFFu, sum);
    if (lane == 0) s_sum[warp] = sum;
    __syncthreads();
    int before = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) before += s_sum[w];
    __syncthreads();
    const unsigned mine = w0 + lane < nwords ? flags[w0 + lane] : 0u;
    int incl = __popc(mine);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += y;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {   // lane l of word w holds slot 32 w + l
      const int w = i * 8 + warp;
      const unsigned word = __shfl_sync(0xFFFFFFFFu, mine, w);
      const int upto = __shfl_sync(0xFFFFFFFFu, incl, w) - __popc(word);
      if ((word >> lane) & 1u) {
        const int from = (w0 + w) * 32 + lane, to = before + upto + __popc(word & ((1u << lane) - 1u));
        const int id = tid_src[from];
#pragma unroll
        for (int p = 0; p < P; ++p) dst[p * stride + to] = src[p * stride + from];
        gp_dst[to] = gp_src[from];
        tid_dst[to] = preserve ? -abs(id) : id;
      }
    }
    if (tile == ntiles - 1 && t == 255) {   // lane 31 holds the tile's survivors
      d_count[slot_out] = before + incl;
      post_count(mail, tag, before + incl);
    }
  }
}

template <int P, bool SMALL>
static void launch_mp(Engine* e, const WindowMpLaunch& w) {
  constexpr int kThreads = MpShape<SMALL>::kThreads;
  // resident blocks per SM, queried once per form (thread-safe initialisation)
  static const int occupancy = [] {
    int o = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, window_mp_kernel<P, SMALL>, kThreads, 0) != cudaSuccess ||
        o < 1) {
      cudaGetLastError();
      o = 1;
    }
    return o;
  }();
  const int per_sm = e->blocks_per_sm > 0 ? std::min(e->blocks_per_sm, occupancy) : occupancy;
  const long long tiles = static_cast<long long>(w.tiles_bound) * (kTileSlots / MpShape<SMALL>::kTile);
  const int blocks = static_cast<int>(std::max(1ll, std::min<long long>(tiles, e->num_sms * per_sm)));
  window_mp_kernel<P, SMALL><<<blocks, kThreads, 0, e->stream>>>(
      w.A, w.B, w.stride, w.id_gp, w.id_tid, w.flags, w.tile_count, w.d_count, w.slot_in, w.slot_out, w.stride,
      w.table, w.ngen, w.births, w.compact, w.check_preserved, w.seed1, w.seed2, w.stats,
      philox_round_keys(w.seed1, w.seed2));
}

template <int P>
static void launch_mp_sized(Engine* e, const WindowMpLaunch& w) {
  if (w.small) launch_mp<P, true>(e, w);
  else launch_mp<P, false>(e, w);
}

template <int P>
static void launch_compact_mp(Engine* e, const WindowMpLaunch& w, float* dst, int* gp_dst, int* tid_dst, int preserve,
                              unsigned long long* mail, unsigned tag) {
  const int blocks = std::max(1, std::min(w.tiles_bound, e->num_sms * 8));
  compact_mp_kernel<P><<<blocks, 256, 0, e->stream>>>(w.B, dst, w.stride, w.id_gp, w.id_tid, gp_dst, tid_dst, w.flags,
                                                      w.d_count, w.slot_out, preserve, mail, tag);
}

gf_status window_mp_run(Engine* e, const WindowMpLaunch& w) {
  if (w.ngen < 1 || w.ngen > mp_max_window(w.P)) return fail(e, GF_ERR_INVALID_ARGUMENT, "window of %d generations", w.ngen);
  switch (w.P) {
    case 2: launch_mp_sized<2>(e, w); break;
    case 3: launch_mp_sized<3>(e, w); break;
    case 4: launch_mp_sized<4>(e, w); break;
    case 5: launch_mp_sized<5>(e, w); break;
    case 6: launch_mp_sized<6>(e, w); break;
    case 7: launch_mp_sized<7>(e, w); break;
    case 8: launch_mp_sized<8>(e, w); break;
    default: return fail(e, GF_ERR_INVALID_ARGUMENT, "multi-population window for %d populations", w.P);
  }
  GF_CUDA(e, cudaGetLastError());
  e->kernel_launches += 1;
  return GF_OK;
}

// The window ran small: its compaction.
gf_status compact_mp_run(Engine* e, const WindowMpLaunch& w, float* dst, int* gp_dst, int* tid_dst, bool preserve,
                         unsigned long long* mail, unsigned tag) {
  switch (w.P) {
    case 2: launch_compact_mp<2>(e, w, dst, gp_dst, tid_dst, preserve, mail, tag); break;
    case 3: launch_compact_mp<3>(e, w, dst, gp_dst, tid_dst, preserve, mail, tag); break;
    case 4: launch_compact_mp<4>(e, w, dst, gp_dst, tid_dst, preserve, mail, tag); break;
    case 5: launch_compact_mp<5>(e, w, dst, gp_dst, tid_dst, preserve, mail, tag); break;
    case 6: launch_compact_mp<6>(e, w, dst, gp_dst, tid_dst, preserve, mail, tag); break;
    case 7: launch_compact_mp<7>(e, w, dst, gp_dst, tid_dst, preserve, mail, tag); break;
    default: launch_compact_mp<8>(e, w, dst, gp_dst, tid_dst, preserve, mail, tag); break;
  }
  GF_CUDA(e, cudaGetLastError());
  e->kernel_launches += 1;
  return GF_OK;
}

}  // namespace gf
