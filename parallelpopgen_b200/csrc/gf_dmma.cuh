// FP64 building blocks of the spectrum projections: the tensor-core fragment D (8 x 8) += A (8 x 4) * B (4 x 8)
// and the binomial pmf at one level.
//
// Fragments (one warp): lane holds A[row = lane / 4][k = lane % 4], B[k = lane % 4][col = lane / 4] and
// D[row = lane / 4][col = 2 (lane % 4) + {0, 1}].
#pragma once

#include <cuda_runtime.h>

namespace gf {

__device__ __forceinline__ void dmma8x8x4(double& d0, double& d1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// Smallest row length >= n (in doubles) whose rows are 32 bytes apart modulo the 128 bytes of a
// shared-memory wavefront: the four k rows of a fragment load then fall into different banks.
__host__ __device__ constexpr int dmma_row(int n) { return (n + 11) / 16 * 16 + 4; }

// x = m 2^e with m in (1/2, 1] (x > 0 and normal).
__device__ __forceinline__ double split_exponent(double x, int& e) {
  const int hi = __double2hiint(x);
  double m = __hiloint2double((hi & 0x000FFFFF) | 0x3FE00000, __double2loint(x));   // [1/2, 1)
  e = (hi >> 20) - 1022;
  if (m == 0.5) {
    m = 1.0;
    e -= 1;
  }
  return m;
}

// c p^k q^(n-k), n <= 1023, by repeated squaring of the mantissas, the exponents apart: m_p^k m_q^(n-k) >= 2^-1023
// and C(n, k) <= 2^1020 stay in range.  About n * 1e-16 relative error, as k log p + (n - k) log q has, in a
// third of the dependent operations of two logarithms and an exp.
__device__ __forceinline__ double binomial_pmf(double c, int k, int n, double p, double q) {
  int ep, eq;
  double bp = split_exponent(p, ep), bq = split_exponent(q, eq);
  const int kq = n - k;
  double vp = 1.0, vq = 1.0;
  for (int bit = 1; bit <= n; bit <<= 1) {   // uniform
    vp = (k & bit) ? vp * bp : vp;
    vq = (kq & bit) ? vq * bq : vq;
    bp *= bp;
    bq *= bq;
  }
  return ldexp(c * vp * vq, ep * k + eq * kq);
}

}  // namespace gf
