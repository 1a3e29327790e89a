// Binomial projection of allele frequencies onto a sample of n (Spectrum::site_frequency_spectrum,
// spectrum.cu:90-139 of the reference): SFS_k = sum over items of count * C(n, k) p^k q^(n-k), k = 0 .. n, for
// the single-population spectra (spectrum.cu) and the batched replicates (batch.cu).
//
// With the levels in runs of B, C(n, k) p^k q^(n-k) = W(k) * pmf(B a) * (p/q)^b for k = B a + b, where W(k) =
// C(n, k) / C(n, B a) does not depend on the item: SFS_{Ba+b} = W(k) sum_i U_i[a] V_i[b] is a matrix product
// with the items as the reduction dimension, accumulated by FP64 tensor-core fragments (gf_dmma.cuh).  An
// item costs n multiply-adds and about n / B + B products to prepare (one exp every four levels before).
// Everything is double, in a fixed order: deterministic.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>

#include "gf_dmma.cuh"
#include "gf_project.h"

namespace gf {

constexpr int kProjMaxRuns = 64;

// For the runs a = 0 .. n / B: C(n, B a) (its logarithm when n > 1023, where it exceeds a double's range),
// C(n, B(a + 1)) / C(n, B a) and C(n, B(a - 1)) / C(n, B a).
struct ProjTable {
  double c[kProjMaxRuns];
  double up[kProjMaxRuns];
  double down[kProjMaxRuns];
  int n;
};

constexpr int kProjRow = 36;   // a shared row: 32 items, rows 32 bytes apart modulo 128 (fragment loads)

// Shape of a projection: fragments of TA x TB (runs x levels of a run), and the warps of a block.
template <int TA, int TB, int WARPS>
struct ProjShape {
  static constexpr int B = 8 * TB;
  static constexpr int ROWS = 8 * TA + B;
  static constexpr int WARP_DOUBLES = ROWS * kProjRow;
  static constexpr int SMEM = static_cast<int>(sizeof(double)) * (WARPS * WARP_DOUBLES + 3 * kProjMaxRuns);
  static_assert(WARP_DOUBLES >= 64 * TA * TB, "a warp's sums fit where its rows were");
  static_assert(SMEM <= 227 * 1024 - 8192, "shared memory");
};

// Block (x, y): every gridDim.x-th batch of 32 items of row y; writes the block's sums, without W, to
// partial[(y * gridDim.x + x) * (n + 2)], the number of items' mutations outside (0, 1) behind them.
//
// A warp gathers 32 items with a nonzero count and a frequency in (0, 1), prepares one per lane (runs U and
// powers V into its shared rows), then multiplies them; no barrier until the end, so the preparation of one
// warp (a chain of about 2,000 cycles) runs under the fragments of the others.
//
// FP64-bound: 36 us for the histogram of 2.7 M mutations over 262,145 counts at n = 1,000 on a B200 (303 us for
// one thread per four levels, each starting from an exp), of which the fragments are about 20; 0.93 ms for
// 512 replicates' rows of 9 M mutations in all at n = 100 (48.8 ms with an exp per mutation and level).
template <int TA, int TB, int WARPS>
__global__ void __launch_bounds__(32 * WARPS)
    project_kernel(const ProjSource src, const __grid_constant__ ProjTable tab, double* __restrict__ partial) {
  using S = ProjShape<TA, TB, WARPS>;
  constexpr int B = S::B;
  constexpr bool LARGE = 64 * TA * TB > 1024;
  extern __shared__ __align__(16) double s_proj[];
  __shared__ float s_qp[WARPS][64];
  __shared__ unsigned s_qc[WARPS][64];
  __shared__ unsigned s_out[WARPS];
  double* const s_c = s_proj;
  double* const s_up = s_c + kProjMaxRuns;
  double* const s_down = s_up + kProjMaxRuns;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* const s_u = s_down + kProjMaxRuns + warp * S::WARP_DOUBLES;
  double* const s_v = s_u + 8 * TA * kProjRow;
  const int n = tab.n, runs = n / B + 1;
  for (int a = threadIdx.x; a < runs; a += 32 * WARPS) {
    s_c[a] = tab.c[a];
    s_up[a] = tab.up[a];
    s_down[a] = tab.down[a];
  }
  for (int a = runs; a < 8 * TA; ++a) s_u[a * kProjRow + lane] = 0.0;
  __syncthreads();

  const bool direct = src.counts == nullptr || (src.mismatch && *src.mismatch != 0);
  const float* const freq = src.freq + (src.rep_base ? src.rep_base[blockIdx.y] : 0);
  const long long M = src.rep_M ? src.rep_M[blockIdx.y] : src.M;
  const long long classes = static_cast<long long>(src.Nc) + 1;
  const long long items = direct ? M : classes * (src.rounded ? 2 : 1);
  const float Nf = static_cast<float>(src.Nc);
  double acc[TA][TB][2];
#pragma unroll
  for (int r = 0; r < TA; ++r)
#pragma unroll
    for (int c = 0; c < TB; ++c) acc[r][c][0] = acc[r][c][1] = 0.0;
  unsigned outside = 0;
  int queued = 0;   // warp-uniform, below 32 between batches
  const long long stride = 32ll * WARPS * gridDim.x;
  for (long long i0 = 32ll * (warp * static_cast<long long>(gridDim.x) + blockIdx.x);; i0 += stride) {
    const bool more = i0 < items;   // warp-uniform
    if (more) {
      const long long i = i0 + lane;
      float p = 0.f;
      unsigned cnt = 0;
      if (i < items) {
        if (direct) {
          p = freq[i];
          cnt = 1;
        } else {
          cnt = src.counts[i];
          if (cnt) p = i < classes ? static_cast<float>(static_cast<int>(i)) / Nf
                                   : __fdiv_rn(static_cast<float>(static_cast<int>(i - classes)), Nf);
        }
      }
      const bool in = cnt && p > 0.f && p < 1.f;
      if (!in) outside += cnt;
      const unsigned b = __ballot_sync(0xFFFFFFFFu, in);
      if (in) {
        const int at = queued + __popc(b & ((1u << lane) - 1u));
        s_qp[warp][at] = p;
        s_qc[warp][at] = cnt;
      }
      queued += __popc(b);
      __syncwarp();
    }
    if (queued >= 32 || (!more && queued > 0)) {
      const bool live = lane < queued;
      const double p = live ? static_cast<double>(s_qp[warp][lane]) : 0.5;
      const double cnt = live ? static_cast<double>(s_qc[warp][lane]) : 0.0;
      // the rest of the queue moves to its front
      const int rest = queued - 32;
      if (lane < rest) {
        const float qp = s_qp[warp][32 + lane];
        const unsigned qc = s_qc[warp][32 + lane];
        s_qp[warp][lane] = qp;
        s_qc[warp][lane] = qc;
      }
      queued = max(rest, 0);
      const double q = 1.0 - p;
      const double inv = 1.0 / (p * q);
      const double r = p * p * inv;             // p / q
      const double r2 = r * r, r4 = r2 * r2;
      double v[4] = {1.0, r, r2, r2 * r};
#pragma unroll
      for (int b = 0; b < B; b += 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          s_v[(b + j) * kProjRow + lane] = v[j];
          v[j] *= r4;
        }
      }
      double rB = r4;
#pragma unroll
      for (int b = 4; b < B; b *= 2) rB *= rB;
      const double s = q * q * inv, s2 = s * s;
      double sB = s2 * s2;
#pragma unroll
      for (int b = 4; b < B; b *= 2) sB *= sB;
      // the run nearest the mode, then the others run by run, up and down together: away from the mode the
      // pmf only falls, so what underflows (and the terms dropped with it, at most 1e-70) is far below the
      // smallest float of the output
      const int m = min(n, static_cast<int>((n + 1) * p)) / B;
      const int k = B * m;
      double hi = LARGE ? exp(s_c[m] + k * log(p) + (n - k) * log1p(-p)) : binomial_pmf(s_c[m], k, n, p, q);
      hi *= cnt;
      double lo = hi;
      s_u[m * kProjRow + lane] = hi;
      const int far = max(m, runs - 1 - m);
      for (int d = 1; d <= far; ++d) {
        if (m + d < runs) {
          hi *= s_up[m + d - 1] * rB;
          s_u[(m + d) * kProjRow + lane] = hi;
        }
        if (m >= d) {
          lo *= s_down[m - d + 1] * sB;
          s_u[(m - d) * kProjRow + lane] = lo;
        }
      }
      __syncwarp();
      const double* const ua = s_u + (lane >> 2) * kProjRow + (lane & 3);
      const double* const vb = s_v + (lane >> 2) * kProjRow + (lane & 3);
#pragma unroll 2
      for (int ks = 0; ks < 8; ++ks) {
        double af[TA], bf[TB];
#pragma unroll
        for (int x = 0; x < TA; ++x) af[x] = ua[8 * x * kProjRow + 4 * ks];
#pragma unroll
        for (int x = 0; x < TB; ++x) bf[x] = vb[8 * x * kProjRow + 4 * ks];
#pragma unroll
        for (int x = 0; x < TA; ++x)
#pragma unroll
          for (int y = 0; y < TB; ++y) dmma8x8x4(acc[x][y][0], acc[x][y][1], af[x], bf[y]);
      }
      __syncwarp();
    }
    if (!more) break;
  }
  // the block's sums: the warps' in order, level by level
  {
    double* const mine = s_u;
    const int a = lane >> 2, b = 2 * (lane & 3);
#pragma unroll
    for (int x = 0; x < TA; ++x)
#pragma unroll
      for (int y = 0; y < TB; ++y) {
        mine[(8 * x + a) * B + 8 * y + b] = acc[x][y][0];
        mine[(8 * x + a) * B + 8 * y + b + 1] = acc[x][y][1];
      }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) outside += __shfl_xor_sync(0xFFFFFFFFu, outside, o);
    if (lane == 0) s_out[warp] = outside;
  }
  __syncthreads();
  double* const out = partial + (static_cast<long long>(blockIdx.y) * gridDim.x + blockIdx.x) * (n + 2);
  const double* const sums = s_down + kProjMaxRuns;
  for (int k = threadIdx.x; k <= n; k += 32 * WARPS) {
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) t += sums[w * S::WARP_DOUBLES + k];
    out[k] = t;
  }
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    for (int w = 0; w < WARPS; ++w) t += s_out[w];
    out[n + 1] = static_cast<double>(t);
  }
}

// Fixed-order reduction of the partials of row y into float bins, with W(k) applied; k == n and every mutation
// outside (0, 1) fold into bin 0, plus the sites without a mutation (spectrum.cu:130-138).  A block takes 32
// levels (one per lane); its 8 warps sum fixed, contiguous eighths of the partials, added in warp order.
// rep_L: row y holds rep_M[y] mutations of rep_L[y] sites (null: extra0).
constexpr int kFinishWarps = 8;
__global__ void __launch_bounds__(32 * kFinishWarps)
    project_finish_kernel(const double* __restrict__ partial, int parts, int n, int B, double extra0,
                          const int* __restrict__ rep_M, const float* __restrict__ rep_L, float* __restrict__ out) {
  __shared__ double s_sum[kFinishWarps][32];
  __shared__ double s_top[kFinishWarps][2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k = blockIdx.x * 32 + lane;
  const double* const p = partial + static_cast<long long>(blockIdx.y) * parts * (n + 2);
  const int per = (parts + kFinishWarps - 1) / kFinishWarps;
  const int b0 = min(parts, warp * per), b1 = min(parts, b0 + per);
  double s = 0.0;
  if (k < n)
    for (int b = b0; b < b1; ++b) s += p[static_cast<long long>(b) * (n + 2) + k];
  s_sum[warp][lane] = s;
  if (blockIdx.x == 0 && lane < 2) {   // level n and the count outside (0, 1)
    double t = 0.0;
    for (int b = b0; b < b1; ++b) t += p[static_cast<long long>(b) * (n + 2) + n + lane];
    s_top[warp][lane] = t;
  }
  __syncthreads();
  if (warp != 0 || k >= n) return;
  auto weight = [n, B](int level) {   // C(n, level) / C(n, B (level / B)): at most 31 factors of at most 2047 each
    const int k0 = level / B * B;
    double num = 1.0, den = 1.0;
    for (int u = k0; u < level; ++u) {
      num *= n - u;
      den *= u + 1;
    }
    return num / den;
  };
  double t = 0.0;
#pragma unroll
  for (int w = 0; w < kFinishWarps; ++w) t += s_sum[w][lane];
  t *= weight(k);
  if (k == 0) {
    double top = 0.0, outside = 0.0;
#pragma unroll
    for (int w = 0; w < kFinishWarps; ++w) {
      top += s_top[w][0];
      outside += s_top[w][1];
    }
    if (rep_L) extra0 = static_cast<double>(rep_L[blockIdx.y] - rep_M[blockIdx.y]);
    t += top * weight(n) + outside + extra0;
  }
  out[static_cast<long long>(blockIdx.y) * n + k] = static_cast<float>(t);
}

// ------------------------------------------------------------------------------------------------
// host
// ------------------------------------------------------------------------------------------------
// Levels of a run for a sample of n: 8, 16 or 32, the split with the fewest values to prepare per item.
static int project_run(int n) { return n + 1 <= 64 ? 8 : n + 1 <= 256 ? 16 : 32; }

static ProjTable project_table(int n) {
  ProjTable t{};
  t.n = n;
  const int B = project_run(n);
  long double c = 1.0L;   // C(2047, 1023) is about 1e614
  for (int a = 0; a <= n / B; ++a) {
    t.c[a] = static_cast<double>(n > 1023 ? std::log(c) : c);
    if (B * a + B > n) break;
    long double up = 1.0L;
    for (int k = B * a; k < B * a + B; ++k) up *= static_cast<long double>(n - k) / (k + 1);
    t.up[a] = static_cast<double>(up);
    t.down[a + 1] = static_cast<double>(1.0L / up);
    c *= up;
  }
  return t;
}

// Runs f(shape, kernel, warps, resident blocks an SM) for the shape that holds a sample of n (f returns a
// cudaError_t or an int).
template <typename F>
static auto with_shape(int n, F f) {
  const int levels = n + 1;
  if (levels <= 64) return f(ProjShape<1, 1, 16>{}, project_kernel<1, 1, 16>, 16, 2);
  if (levels <= 128) return f(ProjShape<1, 2, 12>{}, project_kernel<1, 2, 12>, 12, 2);
  if (levels <= 256) return f(ProjShape<2, 2, 10>{}, project_kernel<2, 2, 10>, 10, 2);
  if (levels <= 512) return f(ProjShape<2, 4, 16>{}, project_kernel<2, 4, 16>, 16, 1);
  if (levels <= 1024) return f(ProjShape<4, 4, 12>{}, project_kernel<4, 4, 12>, 12, 1);
  return f(ProjShape<8, 4, 7>{}, project_kernel<8, 4, 7>, 7, 1);
}

int project_parts(int n, long long items, int rows, int num_sms) {
  return with_shape(n, [&](auto, auto, int warps, int resident) {
    const long long want = (items + 32 * warps - 1) / (32 * warps);
    const long long most = std::max(1, num_sms * resident / std::max(rows, 1));
    return static_cast<int>(std::max(1ll, std::min(want, most)));
  });
}

// The kernel of a sample of n.  A process's first projection loads the one it needs: with the kernels of all sizes
// its first spectrum took 1.61 ms (n = 1,000) and 1.87 ms (n = 100) on a B200, with one 1.29 and 0.93.
static cudaError_t shape_ready(int n) {
  static std::atomic<unsigned> done[64] = {};   // per device, a bit a shape
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  int shape = 0;
  for (int most = 64; shape < 5 && n + 1 > most; most *= 2) ++shape;
  const unsigned bit = 1u << shape;
  if (dev >= 0 && dev < 64 && (done[dev] & bit)) return cudaSuccess;
  err = with_shape(n, [](auto s, auto kernel, int, int) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, decltype(s)::SMEM);
  });
  if (err == cudaSuccess && dev >= 0 && dev < 64) done[dev] |= bit;
  return err;
}

cudaError_t project_ready() {
  for (int n : {1, 64, 128, 256, 512, 1024}) {
    const cudaError_t err = shape_ready(n);
    if (err != cudaSuccess) return err;
  }
  cudaFuncAttributes at;
  return cudaFuncGetAttributes(&at, project_finish_kernel);
}

cudaError_t project_rows(const ProjSource& src, int n, int rows, int parts, double extra0, const float* rep_L,
                         double* scratch, float* out, cudaStream_t stream) {
  cudaError_t err = shape_ready(n);
  if (err != cudaSuccess) return err;
  const ProjTable tab = project_table(n);
  err = with_shape(n, [&](auto shape, auto kernel, int warps, int) {
    kernel<<<dim3(parts, rows), 32 * warps, decltype(shape)::SMEM, stream>>>(src, tab, scratch);
    return cudaGetLastError();
  });
  if (err != cudaSuccess) return err;
  project_finish_kernel<<<dim3((n + 31) / 32, rows), 32 * kFinishWarps, 0, stream>>>(
      scratch, parts, n, project_run(n), extra0, src.rep_M, rep_L, out);
  return cudaGetLastError();
}

}  // namespace gf
