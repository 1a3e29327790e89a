// FP64 tensor-core building block of the spectrum projections: D (8 x 8) += A (8 x 4) * B (4 x 8).
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

}  // namespace gf
