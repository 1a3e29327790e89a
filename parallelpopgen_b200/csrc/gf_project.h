// Binomial projection of allele frequencies onto a sample of n (project.cu), for the single-population spectra
// (spectrum.cu) and the batched replicates (batch.cu).
#pragma once

#include <cuda_runtime.h>

namespace gf {

constexpr int kProjMaxSample = 2047;

// Items: the mutations of one row, or the classes of a histogram of it, or one row per replicate.
struct ProjSource {
  const float* freq = nullptr;          // the row (direct items)
  int M = 0;
  const unsigned* counts = nullptr;     // histogram: [0, Nc] of j / Nc in the device's division, then the
  int Nc = 0;                           // same of the correctly rounded quotients that differ from it
  int rounded = 0;                      // 1: the second half exists
  const unsigned* mismatch = nullptr;   // != 0: some frequency is on neither grid, so the row is projected
  const long long* rep_base = nullptr;  // replicate y: its row at freq + rep_base[y], rep_M[y] long
  const int* rep_M = nullptr;
};

// Blocks per row of a projection of at most `items` items in each of `rows` rows: one wave of resident blocks,
// at least one batch of 32 items a warp.
int project_parts(int n, long long items, int rows, int num_sms);

// Doubles of scratch of a projection.
inline size_t project_scratch(int n, int parts, int rows) {
  return static_cast<size_t>(rows) * parts * (n + 2);
}

// Projects `rows` rows onto samples of n: out[y * n + k].  Bin 0 also takes extra0, or, where rep_L is given,
// replicate y's sites without a mutation, rep_L[y] - rep_M[y].  Two launches on `stream`.
cudaError_t project_rows(const ProjSource& src, int n, int rows, int parts, double extra0, const float* rep_L,
                         double* scratch, float* out, cudaStream_t stream);

// Loads the kernels of every sample size and sets their shared-memory limits on the current device (idempotent); without
// it a size is set up by its first projection.
cudaError_t project_ready();

}  // namespace gf
