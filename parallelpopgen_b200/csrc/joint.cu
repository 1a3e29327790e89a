// Joint site frequency spectrum of two populations: the expected number of sites whose sample of n_a
// chromosomes from population a holds i derived copies and whose sample of n_b chromosomes from
// population b holds j, over the mutation sites (each site's two population frequencies projected
// binomially and independently), plus the num_sites - M monomorphic sites at (0, 0).  The same for
// three populations: bin (i, j, k), with population c's sample of n_c holding k copies.
//
// The reference computes single-population marginals only (Spectrum::site_frequency_spectrum,
// spectrum.cu:213-294, whose projection of one frequency is C(n,k) p^k (1-p)^(n-k), spectrum.cu:90-139);
// this is the two-population form of the same projection.  For 1 <= i <= n_a - 1 the row sums equal the
// single-population SFS of population a.
//
// Work: M x (n_a + 1) x (n_b + 1) FP64 multiply-adds, organised as a GEMM with the mutations as the
// reduction dimension (JSFS = P_a^T P_b; with three populations the columns are the (j, k) pairs).  Two
// things keep it at the FP64 rate.  FP64 tensor-core fragments (gf_dmma.cuh) accumulate it: the CUDA cores'
// peak rate, with one instruction per 256 multiply-adds.  And the operands need no staging: with the
// levels in runs of eight, C(n, k) p^k q^(n-k) = W(k) * pmf(8r) * (p/q)^u for k = 8r + u, where W(k) =
// C(n, k) / C(n, 8r) does not depend on the mutation and is applied to the sums, so a fragment's element is
// one product of two values kept per mutation: the first level of its run and a power of p / q.  Block
// partials are reduced in a fixed order (deterministic).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "gf_dmma.cuh"
#include "gf_internal.h"

namespace gf {

constexpr int kJPart = 4;          // a warp owns up to 4 x 4 fragments (32 x 32 bins)
constexpr int kJWarps = 8;
constexpr int kJThreads = 32 * kJWarps;
constexpr int kJMaxN = 1023;
constexpr int kJMaxSmem = 112 * 1024;   // two blocks an SM

// How an output plane of (n_a + 1) x (n_b + 1)(n_c + 1) bins is shared out.
struct JointPlan {
  int row_tiles;          // fragment rows of the plane
  int tib, tjb;           // fragment rows / columns of a block's tile
  int wi, wj, wk;         // its warps: wi x wj parts of the tile, the k steps split wk ways
  int col_blocks;         // block tiles per row block
  int per_j;              // > 0: n_c + 1 exceeds a tile: per_j column blocks for each j
  int super;              // mutations prepared together (a multiple of 32)
  int rows;               // shared rows of super + 20 doubles
  int rows_b, rows_c;     // three populations: rows of b's and c's levels among them
  int smem;               // bytes
};

// One population's constants: C(n, k); W(k) = C(n, k) / C(n, 8 (k / 8)); and over whole runs
// C(n, 8r + 8) / C(n, 8r) and C(n, 8r - 8) / C(n, 8r).
struct JointTable {
  const double* c;
  const double* w;
  const double* up;
  const double* down;
  int n;
};

// One mutation's values for the runs r0 .. r0 + runs - 1 of population t: start(r) gets pmf(8r), pow[u] the
// power (p / q)^u.  The run nearest the mode is computed, the others follow from it run by run, up and down,
// by C(n, 8r +- 8) / C(n, 8r) * (p / q)^+-8: away from the mode the pmf only falls, so what underflows is below
// the smallest double, and the terms dropped with it (start below 5e-324, seven powers of p / q <= 2^24,
// W <= 1e21) below 1e-250.  A step adds about 1e-15 relative error.  Lost and fixed mutations are point
// masses.
template <typename Start>
__device__ __forceinline__ void mutation_values(float pf, int r0, int runs, const JointTable& t, double (&pow)[8],
                                                Start start) {
  if (!(pf > 0.f && pf < 1.f)) {
    const int k = pf >= 1.f ? t.n : 0;
#pragma unroll
    for (int u = 0; u < 8; ++u) pow[u] = u == (k & 7) ? 1.0 : 0.0;
    for (int r = 0; r < runs; ++r) start(r, r0 + r == k / 8 ? 1.0 / __ldg(t.w + k) : 0.0);
    return;
  }
  const double p = static_cast<double>(pf), q = 1.0 - p;
  const double pq_inv = 1.0 / (p * q);
  const double pq = p * p * pq_inv;
  pow[0] = 1.0;
  pow[1] = pq;
  pow[2] = pq * pq;
  pow[3] = pow[2] * pq;
  pow[4] = pow[2] * pow[2];
  pow[5] = pow[4] * pq;
  pow[6] = pow[4] * pow[2];
  pow[7] = pow[4] * pow[3];
  const double pq8 = pow[4] * pow[4];
  const int mode = min(t.n, static_cast<int>((t.n + 1) * p));
  const int m = min(max(mode / 8 - r0, 0), runs - 1);
  const int k = 8 * (r0 + m);
  const double at = binomial_pmf(__ldg(t.c + k), k, t.n, p, q);
  start(m, at);
  double v = at;
  for (int r = m + 1; r < runs; ++r) {
    v *= __ldg(t.up + r0 + r - 1) * pq8;
    start(r, v);
  }
  if (m > 0) {
    const double qp = q * q * pq_inv, qp2 = qp * qp, qp4 = qp2 * qp2, qp8 = qp4 * qp4;
    v = at;
    for (int r = m - 1; r >= 0; --r) {
      v *= __ldg(t.down + r0 + r + 1) * qp8;
      start(r, v);
    }
  }
}

// A warp's R x C fragments over the k steps [k0, k1) of a class, every nwk-th from wk.  a, b: the lane's
// mutation in the rows of run starts; ua, ub: its power row; off_b, off_c (THREE): its columns' rows of b's
// and c's levels.
template <bool THREE, int R, int C>
__device__ __forceinline__ void multiply_part(double (&acc)[kJPart][kJPart][2], const double* __restrict__ a,
                                              const double* __restrict__ ua, const double* __restrict__ b,
                                              const double* __restrict__ ub, const int (&off_b)[kJPart],
                                              const int (&off_c)[kJPart], int row, int k0, int k1, int nwk) {
#pragma unroll 2
  for (int ks = k0; ks < k1; ks += nwk) {
    double af[R], bf[C];
    const double u = ua[4 * ks];
#pragma unroll
    for (int r = 0; r < R; ++r) af[r] = a[r * row + 4 * ks] * u;
    if (THREE) {
#pragma unroll
      for (int c = 0; c < C; ++c) bf[c] = b[off_b[c] + 4 * ks] * b[off_c[c] + 4 * ks];
    } else {
      const double w = ub[4 * ks];
#pragma unroll
      for (int c = 0; c < C; ++c) bf[c] = b[c * row + 4 * ks] * w;
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = 0; c < C; ++c) dmma8x8x4(acc[r][c][0], acc[r][c][1], af[r], bf[c]);
  }
}

// THREE: a third population c; column (j, k) of the plane is j * (n_c + 1) + k.
//
// Per `super` mutations of the block's range: a stable sort by which of a and b have lost the mutation (a
// class then needs only fragment row 0 where a has, only the columns of j = 0 where b has: in simulated
// populations most mutations are private to one of them), the values of every mutation and population
// (mutation_values) into shared rows, then every warp multiplies its part over all k steps with no barrier
// between them.  Two blocks an SM, so that one prepares while the other multiplies.
//
// FP64-bound.  On a B200, 200,000 mutations (half private to one population), n = 100 x 80: 122 us (599 us for
// padded 128 x 128 tiles on the CUDA cores with an exp for every level; the fragments alone are 54 us at the
// FP64 tensor rate of 1.83e13 multiply-adds/s, the rest is mostly the preparation).  100,000 mutations, n = 20 x
// 16 x 12: 52 us (5,655 us with one padded tile per k).  Operands staged in shared memory for each chunk,
// whether by the same warps or by four writing warps, measured 168 and 200 us for the first.
template <bool THREE>
__global__ void __launch_bounds__(kJThreads, 2)
    joint_sfs_kernel(const float* __restrict__ fa, const float* __restrict__ fb, const float* __restrict__ fc, int M,
                     const JointTable ta, const JointTable tb, const JointTable tc, int per_block, const JointPlan P,
                     double* __restrict__ partial) {
  constexpr int NP = THREE ? 3 : 2;
  constexpr int kMaxGroups = 8;   // super <= 256
  extern __shared__ __align__(16) double s_mem[];
  // rows of `row` doubles, a mutation per column (rows 32 bytes apart modulo 128: a fragment's loads, eight
  // rows of four columns, fall into different banks)
  const int S = P.super, row = S + 20;
  double* const s_a = s_mem;                       // [tib] run starts of a
  double* const s_ua = s_a + P.tib * row;          // [8] powers of a
  double* const s_b = s_ua + 8 * row;              // two: [tjb] run starts of b; three: [rows_b + rows_c] levels
  double* const s_ub = s_b + P.tjb * row;          // two: [8] powers of b
  double* const s_c = s_b + P.rows_b * row;        // three: levels of c
  __shared__ unsigned s_mask[4][kMaxGroups];
  __shared__ int s_before[4][kMaxGroups];          // mutations of the class in earlier groups
  __shared__ int s_count[4];

  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int ncp = THREE ? tc.n + 1 : 1;
  const int NB = (tb.n + 1) * ncp;
  // the block's part of the plane
  const int rb = static_cast<int>(blockIdx.y) / P.col_blocks, cb = static_cast<int>(blockIdx.y) % P.col_blocks;
  const int i0 = rb * P.tib * 8;
  const int itiles = min(P.tib, P.row_tiles - rb * P.tib);
  int col0, width, k_lo = 0, nk = ncp;
  if (THREE && P.per_j > 0) {
    k_lo = (cb % P.per_j) * P.tjb * 8;
    col0 = (cb / P.per_j) * ncp + k_lo;
    width = min(P.tjb * 8, ncp - k_lo);
    nk = width;
  } else {
    col0 = cb * P.tjb * 8;
    width = min(P.tjb * 8, NB - col0);
  }
  const int jtiles = (width + 7) / 8;
  // three populations: the runs of b and c that the tile reaches
  const int j_lo = THREE ? col0 / ncp / 8 * 8 : col0;
  const int rj = THREE ? ((col0 + width - 1) / ncp - j_lo) / 8 + 1 : jtiles, rk = (nk + 7) / 8;
  // the warp's part of the tile
  const int wk = warp % P.wk, wj = (warp / P.wk) % P.wj, wi = warp / (P.wk * P.wj);
  const bool works = wi < P.wi;
  const int ti0 = itiles * wi / P.wi, ti1 = works ? itiles * (wi + 1) / P.wi : ti0;
  const int tj0 = jtiles * wj / P.wj, tj1 = jtiles * (wj + 1) / P.wj;
  const int g = lane >> 2, e = lane & 3;
  int off_b[kJPart], off_c[kJPart];
#pragma unroll
  for (int c = 0; c < kJPart; ++c) {
    const int x = col0 + min((tj0 + c) * 8 + g, width - 1);   // columns past the tile repeat its last one
    off_b[c] = THREE ? (x / ncp - j_lo) * row : 0;
    off_c[c] = THREE ? (P.rows_b + x % ncp - k_lo) * row : 0;
  }
  double acc[kJPart][kJPart][2];
#pragma unroll
  for (int r = 0; r < kJPart; ++r)
#pragma unroll
    for (int c = 0; c < kJPart; ++c) acc[r][c][0] = acc[r][c][1] = 0.0;

  const long long m0 = static_cast<long long>(blockIdx.x) * per_block;
  const long long m1 = min(static_cast<long long>(M), m0 + per_block);
  // of the two blocks of an SM (the grid's halves) the second begins with half a pass, so that they do not
  // prepare at the same time
  const bool second = (blockIdx.y * gridDim.x + blockIdx.x) * 2 >= gridDim.x * gridDim.y;
  int take = second ? S / 2 : S;
  for (long long base = m0; base < m1; base += take, take = S) {
    // ---- stable counting sort by class: bit 0 = lost in a, bit 1 = lost in b; a class starts at a
    // multiple of four columns (one k step), the columns between two classes hold zeros ----
    int cls = 4;
    float fr[NP] = {};
    if (tid < S) {
      if (tid < take && base + tid < m1) {
        fr[0] = fa[base + tid];
        fr[1] = fb[base + tid];
        if (THREE) fr[NP - 1] = fc[base + tid];
        cls = (fr[0] > 0.f ? 0 : 1) | (fr[1] > 0.f ? 0 : 2);
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const unsigned b = __ballot_sync(0xFFFFFFFFu, cls == c);
        if (lane == 0) s_mask[c][warp] = b;
      }
    }
    __syncthreads();   // also: every warp is done with the previous mutations' rows
    if (tid < 4) {
      int n = 0;
      for (int h = 0; h < S / 32; ++h) {
        s_before[tid][h] = n;
        n += __popc(s_mask[tid][h]);
      }
      s_count[tid] = n;
    }
    __syncthreads();
    int first[5], count[4];
    first[0] = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      count[c] = s_count[c];
      first[c + 1] = first[c] + (count[c] + 3) / 4 * 4;
    }
    // ---- values: a thread prepares its mutation for every population ----
    if (cls < 4) {
      const int c0 = cls == 0 ? first[0] : cls == 1 ? first[1] : cls == 2 ? first[2] : first[3];
      const int at = c0 + s_before[cls][warp] + __popc(s_mask[cls][warp] & ((1u << lane) - 1u));
      double pow[8];
      mutation_values(fr[0], i0 / 8, itiles, ta, pow, [&](int r, double v) { s_a[r * row + at] = v; });
#pragma unroll
      for (int u = 0; u < 8; ++u) s_ua[u * row + at] = pow[u];
      if (!THREE) {
        mutation_values(fr[1], col0 / 8, jtiles, tb, pow, [&](int r, double v) { s_b[r * row + at] = v; });
#pragma unroll
        for (int u = 0; u < 8; ++u) s_ub[u * row + at] = pow[u];
      } else {
        auto levels = [&](double* rows) {
          return [&pow, rows, row, at](int r, double v) {
#pragma unroll
            for (int u = 0; u < 8; ++u) rows[(8 * r + u) * row + at] = v * pow[u];
          };
        };
        mutation_values(fr[1], j_lo / 8, rj, tb, pow, levels(s_b));
        mutation_values(fr[NP - 1], k_lo / 8, rk, tc, pow, levels(s_c));
      }
    }
    // the zero columns: a's starts and every factor (zero times what an earlier pass left could be NaN)
    if (tid >= kJThreads - 16) {
      const int z = tid - (kJThreads - 16), c = z / 4;
      const int x = c == 0 ? first[0] + count[0] : c == 1 ? first[1] + count[1] : c == 2 ? first[2] + count[2] : first[3] + count[3];
      const int end = c == 0 ? first[1] : c == 1 ? first[2] : c == 2 ? first[3] : first[4];
      if (x + z % 4 < end)
        for (int r = 0; r < P.rows; ++r) s_mem[r * row + x + z % 4] = 0.0;
    }
    __syncthreads();

    // ---- every warp: its part, class by class ----
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
      const int k0 = (c == 0 ? first[0] : c == 1 ? first[1] : c == 2 ? first[2] : first[3]) / 4;
      const int k1 = (c == 0 ? first[1] : c == 1 ? first[2] : c == 2 ? first[3] : first[4]) / 4;
      const int gi = (c & 1) ? (i0 == 0 ? 1 : 0) : itiles;
      const int gj = (c & 2) ? (col0 < ncp ? min(jtiles, (ncp - col0 + 7) / 8) : 0) : jtiles;
      const int nri = min(ti1, gi) - ti0, nrj = min(tj1, gj) - tj0;
      if (nri <= 0 || nrj <= 0) continue;   // warp-uniform
      const double* const a = s_a + ti0 * row + e;
      const double* const ua = s_ua + g * row + e;
      const double* const b = THREE ? s_b + e : s_b + tj0 * row + e;
      const double* const ub = s_ub + g * row + e;
      switch (kJPart * (nri - 1) + nrj - 1) {
#define GF_PART(R, C)                                                                                        \
  case kJPart * (R - 1) + C - 1:                                                                             \
    multiply_part<THREE, R, C>(acc, a, ua, b, ub, off_b, off_c, row, k0 + wk, k1, P.wk);                     \
    break;
        GF_PART(1, 1) GF_PART(1, 2) GF_PART(1, 3) GF_PART(1, 4) GF_PART(2, 1) GF_PART(2, 2) GF_PART(2, 3) GF_PART(2, 4)
        GF_PART(3, 1) GF_PART(3, 2) GF_PART(3, 3) GF_PART(3, 4) GF_PART(4, 1) GF_PART(4, 2) GF_PART(4, 3) GF_PART(4, 4)
#undef GF_PART
      }
    }
  }

  // the wk partial accumulators of a part, added in order by its first warp
  if (P.wk > 1) {
    double* const mine = s_mem + (wi * P.wj + wj) * 32 * kJPart * kJPart * 2 + lane;
    for (int k = 1; k < P.wk; ++k) {
      __syncthreads();
      if (works && wk == k) {
#pragma unroll
        for (int r = 0; r < kJPart; ++r)
#pragma unroll
          for (int c = 0; c < kJPart; ++c) {
            mine[((r * kJPart + c) * 2) * 32] = acc[r][c][0];
            mine[((r * kJPart + c) * 2 + 1) * 32] = acc[r][c][1];
          }
      }
      __syncthreads();
      if (works && wk == 0) {
#pragma unroll
        for (int r = 0; r < kJPart; ++r)
#pragma unroll
          for (int c = 0; c < kJPart; ++c) {
            acc[r][c][0] += mine[((r * kJPart + c) * 2) * 32];
            acc[r][c][1] += mine[((r * kJPart + c) * 2 + 1) * 32];
          }
      }
    }
  }
  if (!works || wk != 0) return;
  double* const out = partial + static_cast<long long>(blockIdx.x) * (ta.n + 1) * NB;
#pragma unroll
  for (int r = 0; r < kJPart; ++r) {
    const int i = i0 + (ti0 + r) * 8 + g;
    if (ti0 + r >= ti1 || i > ta.n) continue;
    const double wa = __ldg(ta.w + i);
#pragma unroll
    for (int c = 0; c < kJPart; ++c) {
      if (tj0 + c >= tj1) continue;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int x = (tj0 + c) * 8 + 2 * e + h;
        if (x >= width) continue;
        const int j = (col0 + x) / ncp, k = (col0 + x) - j * ncp;
        double w = wa * __ldg(tb.w + j);
        if (THREE) w *= __ldg(tc.w + k);
        out[static_cast<long long>(i) * NB + col0 + x] = acc[r][c][h] * w;
      }
    }
  }
}

// out[bin] = sum of the partials, plus the monomorphic sites at bin 0.  A block takes 32 bins (one per
// lane); its 8 warps sum fixed, contiguous eighths of the partials, added in warp order.
constexpr int kJFinishWarps = 8;
__global__ void __launch_bounds__(32 * kJFinishWarps)
    joint_finish_kernel(const double* __restrict__ partial, int nblocks, long long bins, double extra0,
                        float* __restrict__ out) {
  __shared__ double s_sum[kJFinishWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long b = static_cast<long long>(blockIdx.x) * 32 + lane;
  const int per = (nblocks + kJFinishWarps - 1) / kJFinishWarps;
  const int k1 = min(nblocks, (warp + 1) * per);
  double s = 0.0;
  if (b < bins)
    for (int k = warp * per; k < k1; ++k) s += partial[k * bins + b];
  s_sum[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && b < bins) {
    double t = b == 0 ? extra0 : 0.0;
#pragma unroll
    for (int w = 0; w < kJFinishWarps; ++w) t += s_sum[w][lane];
    out[b] = static_cast<float>(t);
  }
}

// Largest number of bins of a three-population joint spectrum (the partial sums hold one copy per block).
constexpr long long kJMaxBins3 = 1ll << 24;

// The tables of one population (JointTable), one after the other: C(n, k) and W(k) for k = 0 .. n, and the
// two run ratios for r = 0 .. n / 8.
static size_t joint_table_size(int n) { return 2 * (n + 1) + 2 * (n / 8 + 1); }

static JointTable joint_table_at(const double* d, int n) {
  return {d, d + (n + 1), d + 2 * (n + 1), d + 2 * (n + 1) + n / 8 + 1, n};
}

static void joint_table(std::vector<double>& h, int n) {
  long double c = 1.0L;   // C(1023, 511) is about 3e306
  for (int k = 0; k <= n; ++k) {
    h.push_back(static_cast<double>(c));
    c *= static_cast<long double>(n - k) / (k + 1);
  }
  auto over = [n](int k, int steps) {   // C(n, k + steps) / C(n, k)
    long double v = 1.0L;
    for (int u = 0; u < steps; ++u) v *= static_cast<long double>(n - k - u) / (k + u + 1);
    return v;
  };
  for (int k = 0; k <= n; ++k) h.push_back(static_cast<double>(over(k / 8 * 8, k % 8)));
  for (int r = 0; r <= n / 8; ++r) h.push_back(8 * r + 8 <= n ? static_cast<double>(over(8 * r, 8)) : 0.0);
  for (int r = 0; r <= n / 8; ++r) h.push_back(r > 0 ? static_cast<double>(1.0L / over(8 * r - 8, 8)) : 0.0);
}

// Shares the plane out in equal blocks of at most eight parts of 32 x 32 bins (16 fragment rows, 32 columns
// at most), a warp for each; with fewer parts the k steps are split over two, four or eight times as many
// warps.  Mutations are prepared 256 at a time, fewer where their rows would not leave room for two blocks
// an SM (three populations of large samples).
static JointPlan joint_plan(int na, int nb, int nc, bool three) {
  JointPlan p{};
  const int ncp = three ? nc + 1 : 1;
  const int NB = (nb + 1) * ncp;
  p.row_tiles = (na + 8) / 8;
  const int row_blocks = (p.row_tiles + 15) / 16;
  p.tib = (p.row_tiles + row_blocks - 1) / row_blocks;
  p.wi = (p.tib + kJPart - 1) / kJPart;
  const int most = kJWarps / p.wi * kJPart;   // fragment columns of a tile
  if (three && ncp > most * 8) {
    const int tiles = (ncp + 7) / 8;
    p.per_j = (tiles + most - 1) / most;
    p.tjb = (tiles + p.per_j - 1) / p.per_j;
    p.col_blocks = (nb + 1) * p.per_j;
  } else {
    const int tiles = (NB + 7) / 8;
    p.col_blocks = (tiles + most - 1) / most;
    p.tjb = (tiles + p.col_blocks - 1) / p.col_blocks;
    p.col_blocks = (tiles + p.tjb - 1) / p.tjb;
  }
  p.wj = (p.tjb + kJPart - 1) / kJPart;
  p.wk = 1;
  while (p.wi * p.wj * p.wk * 2 <= kJWarps) p.wk *= 2;
  if (three) {
    auto runs = [](int n) { return (n + 7) / 8 * 8; };
    p.rows_b = runs(std::min(nb + 1, (p.per_j > 0 ? 1 : p.tjb * 8 / ncp + 2) + 7));   // from a multiple of 8
    p.rows_c = runs(std::min(ncp, p.per_j > 0 ? p.tjb * 8 : ncp));
  }
  p.rows = p.tib + 8 + (three ? p.rows_b + p.rows_c : p.tjb + 8);
  const size_t reduce = p.wk > 1 ? static_cast<size_t>(p.wi) * p.wj * 32 * kJPart * kJPart * 2 : 0;
  for (p.super = 256;; p.super /= 2) {
    p.smem = static_cast<int>(sizeof(double) * std::max(static_cast<size_t>(p.rows) * (p.super + 20), reduce));
    if (p.smem <= kJMaxSmem || p.super == 32) return p;   // with 32, 122 KB at most
  }
}

// d_fc == nullptr: two populations; else three (n_c >= 1).
gf_status joint_sfs_device(Engine* e, const float* d_fa, const float* d_fb, const float* d_fc, int M, int na, int nb,
                           int nc, float num_sites, float* d_out) {
  const bool three = d_fc != nullptr || nc > 0;
  if (na < 1 || nb < 1 || na > kJMaxN || nb > kJMaxN || (three && (nc < 1 || nc > kJMaxN)))
    return fail(e, GF_ERR_INVALID_ARGUMENT, "sample sizes %d, %d%s outside [1, %d]", na, nb, three ? " (or n_c)" : "",
                kJMaxN);
  if (M < 0) return fail(e, GF_ERR_INVALID_ARGUMENT, "negative mutation count");
  if (M > 0 && (!d_fa || !d_fb || (three && !d_fc))) return fail(e, GF_ERR_INVALID_ARGUMENT, "frequency rows are NULL");
  if (!d_out) return fail(e, GF_ERR_INVALID_ARGUMENT, "output is NULL");
  const long long bins = static_cast<long long>(na + 1) * (nb + 1) * (three ? nc + 1 : 1);
  if (three && bins > kJMaxBins3)
    return fail(e, GF_ERR_CAPACITY, "%lld bins exceed the three-population limit of %lld", bins, kJMaxBins3);
  const JointPlan plan = joint_plan(na, nb, nc, three);
  const int tiles = (plan.row_tiles + plan.tib - 1) / plan.tib * plan.col_blocks;
  // one wave of blocks over all tiles (two an SM); partials kept under 256 MB
  int nblocks = std::max(1, 2 * e->num_sms / tiles);
  nblocks = std::min<long long>(nblocks, std::max<long long>(1, (256ll << 20) / (bins * 8)));
  nblocks = std::min(nblocks, std::max(1, M / 64));
  int per_block = std::max(32, M / nblocks + (M % nblocks != 0));
  if (nblocks > 1) per_block = (per_block + 31) / 32 * 32;
  nblocks = std::max(1, M / per_block + (M % per_block != 0));

  double* d_tab = nullptr;
  double* d_partial = nullptr;
  std::vector<double> h;
  h.reserve(joint_table_size(na) + joint_table_size(nb) + joint_table_size(nc));
  joint_table(h, na);
  joint_table(h, nb);
  if (three) joint_table(h, nc);
  gf_status st = pool_alloc(e, reinterpret_cast<void**>(&d_tab), sizeof(double) * h.size());
  if (st != GF_OK) return st;
  st = pool_alloc(e, reinterpret_cast<void**>(&d_partial), sizeof(double) * bins * nblocks);
  if (st != GF_OK) {
    cudaFreeAsync(d_tab, e->stream);
    return st;
  }
  cudaError_t err = cudaMemcpyAsync(d_tab, h.data(), sizeof(double) * h.size(), cudaMemcpyHostToDevice, e->stream);
  if (err == cudaSuccess && M > 0) {
    const double* at = d_tab + joint_table_size(na);
    const JointTable ta = joint_table_at(d_tab, na), tb = joint_table_at(at, nb);
    const JointTable tc = joint_table_at(three ? at + joint_table_size(nb) : nullptr, three ? nc : 0);
    const auto kernel = three ? joint_sfs_kernel<true> : joint_sfs_kernel<false>;
    err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kJMaxSmem + 16 * 1024);
    if (err == cudaSuccess && tiles > 65535) err = cudaErrorInvalidConfiguration;
    if (err == cudaSuccess) {
      kernel<<<dim3(nblocks, tiles), kJThreads, plan.smem, e->stream>>>(d_fa, d_fb, d_fc, M, ta, tb, tc, per_block, plan,
                                                                      d_partial);
      err = cudaGetLastError();
      e->kernel_launches += 1;
    }
  }
  if (err == cudaSuccess) {
    joint_finish_kernel<<<static_cast<unsigned>((bins + 31) / 32), 32 * kJFinishWarps, 0, e->stream>>>(
        d_partial, M > 0 ? nblocks : 0, bins, static_cast<double>(num_sites) - M, d_out);
    err = cudaGetLastError();
    e->kernel_launches += 1;
  }
  cudaFreeAsync(d_partial, e->stream);
  cudaFreeAsync(d_tab, e->stream);
  if (err != cudaSuccess) return cuda_fail(e, err, "joint SFS");
  return GF_OK;
}

}  // namespace gf

using namespace gf;

extern "C" {

gf_status gf_joint_site_frequency_spectrum_device(gf_engine* g, const float* d_freq_a, const float* d_freq_b,
                                                  int32_t M, int32_t n_a, int32_t n_b, float num_sites,
                                                  float* d_out) {
  return guard_host(g, [&]() -> gf_status {
    if (!g) return GF_ERR_INVALID_ARGUMENT;
    Engine* e = &g->impl;
    GF_CUDA(e, cudaSetDevice(e->device));
    return joint_sfs_device(e, d_freq_a, d_freq_b, nullptr, M, n_a, n_b, 0, num_sites, d_out);
  });
}

gf_status gf_joint3_site_frequency_spectrum_device(gf_engine* g, const float* d_freq_a, const float* d_freq_b,
                                                   const float* d_freq_c, int32_t M, int32_t n_a, int32_t n_b,
                                                   int32_t n_c, float num_sites, float* d_out) {
  return guard_host(g, [&]() -> gf_status {
    if (!g) return GF_ERR_INVALID_ARGUMENT;
    Engine* e = &g->impl;
    if (n_c < 1) return fail(e, GF_ERR_INVALID_ARGUMENT, "sample size n_c %d below 1", n_c);
    GF_CUDA(e, cudaSetDevice(e->device));
    return joint_sfs_device(e, d_freq_a, d_freq_b, d_freq_c, M, n_a, n_b, n_c, num_sites, d_out);
  });
}

}  // extern "C"

namespace gf {

// Host rows in, host spectrum out (freq_c == nullptr: two populations).
static gf_status joint_sfs_host(Engine* e, const float* freq_a, const float* freq_b, const float* freq_c, int M,
                                int n_a, int n_b, int n_c, float num_sites, float* out) {
  const bool three = freq_c != nullptr || n_c > 0;
  if (M < 0 || (M > 0 && (!freq_a || !freq_b || (three && !freq_c))) || !out)
    return fail(e, GF_ERR_INVALID_ARGUMENT, "bad buffers");
  if (n_a < 1 || n_b < 1 || n_a > kJMaxN || n_b > kJMaxN || (three && (n_c < 1 || n_c > kJMaxN)))
    return fail(e, GF_ERR_INVALID_ARGUMENT, "sample sizes %d, %d%s outside [1, %d]", n_a, n_b, three ? " (or n_c)" : "",
                kJMaxN);
  const long long bins = static_cast<long long>(n_a + 1) * (n_b + 1) * (three ? n_c + 1 : 1);
  if (three && bins > kJMaxBins3)
    return fail(e, GF_ERR_CAPACITY, "%lld bins exceed the three-population limit of %lld", bins, kJMaxBins3);
  GF_CUDA(e, cudaSetDevice(e->device));
  const long long rows = three ? 3 : 2;
  float* d = nullptr;
  gf_status st = pool_alloc(e, reinterpret_cast<void**>(&d), sizeof(float) * (rows * std::max(M, 1) + bins));
  if (st != GF_OK) return st;
  float* d_fa = d;
  float* d_fb = d + std::max(M, 1);
  float* d_fc = three ? d + 2ll * std::max(M, 1) : nullptr;
  float* d_out = d + rows * std::max(M, 1);
  cudaError_t err = cudaSuccess;
  if (M > 0) {
    err = cudaMemcpyAsync(d_fa, freq_a, sizeof(float) * M, cudaMemcpyHostToDevice, e->stream);
    if (err == cudaSuccess) err = cudaMemcpyAsync(d_fb, freq_b, sizeof(float) * M, cudaMemcpyHostToDevice, e->stream);
    if (err == cudaSuccess && three)
      err = cudaMemcpyAsync(d_fc, freq_c, sizeof(float) * M, cudaMemcpyHostToDevice, e->stream);
  }
  if (err == cudaSuccess) {
    st = joint_sfs_device(e, d_fa, d_fb, d_fc, M, n_a, n_b, three ? n_c : 0, num_sites, d_out);
    if (st == GF_OK) err = cudaMemcpyAsync(out, d_out, sizeof(float) * bins, cudaMemcpyDeviceToHost, e->stream);
  }
  cudaFreeAsync(d, e->stream);
  if (err == cudaSuccess) err = cudaStreamSynchronize(e->stream);
  if (st != GF_OK) return st;
  if (err != cudaSuccess) return cuda_fail(e, err, "joint SFS transfer");
  return GF_OK;
}

}  // namespace gf

extern "C" {

gf_status gf_joint_site_frequency_spectrum(gf_engine* g, const float* freq_a, const float* freq_b, int32_t M,
                                           int32_t n_a, int32_t n_b, float num_sites, float* out) {
  return guard_host(g, [&]() -> gf_status {
    if (!g) return GF_ERR_INVALID_ARGUMENT;
    return joint_sfs_host(&g->impl, freq_a, freq_b, nullptr, M, n_a, n_b, 0, num_sites, out);
  });
}

gf_status gf_joint3_site_frequency_spectrum(gf_engine* g, const float* freq_a, const float* freq_b, const float* freq_c,
                                            int32_t M, int32_t n_a, int32_t n_b, int32_t n_c, float num_sites,
                                            float* out) {
  return guard_host(g, [&]() -> gf_status {
    if (!g) return GF_ERR_INVALID_ARGUMENT;
    if (n_c < 1) return fail(&g->impl, GF_ERR_INVALID_ARGUMENT, "sample size n_c %d below 1", n_c);
    return joint_sfs_host(&g->impl, freq_a, freq_b, freq_c, M, n_a, n_b, n_c, num_sites, out);
  });
}

}  // extern "C"
