// Spectrum: population frequency histogram and binomially projected site frequency spectrum
// (Spectrum::population_frequency_histogram / site_frequency_spectrum, spectrum.cu:74-294 of the
// reference).
//
// The histogram counts allele counts j = round(Nc * p) over j in [0, Nc] (population_hist, spectrum.cu:74-83),
// with a block-private shared-memory histogram for the low-count bins -- where a neutral SFS puts most of
// its mass -- and global atomics above them.
//
// The SFS projects either every mutation of the row, or, where the row holds more mutations than a
// quarter of its possible frequencies, the classes of its histogram: sum_i f(p_i) = sum_j c_j f(p_j).  This is
// exact because engine frequencies are float(j) / Nc, in the division of the device's fast-math code or
// (mutations born in the last generation, rows made on a host) the correctly rounded one: the histogram
// kernel counts the two apart and flags any other frequency, in which case the projection takes the row's
// mutations after all -- decided on the device, so nothing waits for the flag.  Terms are evaluated in
// double precision and reduced in a fixed order, so the result is deterministic (the reference's float
// atomics are not, spectrum.cu:271-272).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "gf_internal.h"
#include "gf_project.h"

namespace gf {

constexpr int kHistThreads = 512;
constexpr int kHistBins = 4096;   // low counts with a shared counter per block

// counts[j] for j in [0, Nc].  SPLIT: only the frequencies equal to float(j) / Nc in the device's division;
// where `rounded`, counts[Nc + 1 + j] those equal to the correctly rounded quotient alone; mismatch[0] != 0
// if some frequency is neither.
//
// 16 KB (SPLIT: 32 KB) of counters a block, four blocks an SM: a neutral row of 2.7 M mutations over 262,145
// counts takes 20 us, and took 37 with 160 KB of counters (zeroing and flushing 40,960 of them per block was most of
// the difference).
template <bool SPLIT>
__global__ void __launch_bounds__(kHistThreads)
    hist_kernel(const float* __restrict__ freq, int M, int Nc, unsigned* __restrict__ counts, int rounded,
                unsigned* __restrict__ mismatch) {
  __shared__ unsigned s_bins[SPLIT ? 2 * kHistBins : kHistBins];
  const int bins = min(kHistBins, Nc + 1);
  for (int b = threadIdx.x; b < (SPLIT ? 2 * kHistBins : kHistBins); b += kHistThreads) s_bins[b] = 0;
  __syncthreads();
  unsigned bad = 0;
  const float Nf = static_cast<float>(Nc);
  const long long step = static_cast<long long>(kHistThreads) * gridDim.x;
  for (long long i = static_cast<long long>(blockIdx.x) * kHistThreads + threadIdx.x; i < M; i += step) {
    const float p = freq[i];
    int j = static_cast<int>(round(Nc * p));
    if (j < 0) j = 0;
    if (j > Nc) j = Nc;
    int half = 0;
    if (SPLIT && static_cast<float>(j) / Nf != p) {
      if (rounded && __fdiv_rn(static_cast<float>(j), Nf) == p) half = 1;
      else bad = 1;
    }
    if (j < bins) {
      // warp-aggregated: one shared atomic per distinct bin in the warp
      const int key = half * kHistBins + j;
      const unsigned active = __activemask();
      const unsigned peers = __match_any_sync(active, key);
      const int leader = __ffs(peers) - 1;
      if ((threadIdx.x & 31) == leader) atomicAdd(&s_bins[key], __popc(peers));
    } else {
      atomicAdd(&counts[half * (static_cast<long long>(Nc) + 1) + j], 1u);
    }
  }
  if (SPLIT && bad) atomicOr(mismatch, 1u);
  __syncthreads();
  for (int b = threadIdx.x; b < bins; b += kHistThreads) {
    const unsigned v = s_bins[b];
    if (v) atomicAdd(&counts[b], v);
    if (SPLIT) {
      const unsigned w = s_bins[kHistBins + b];
      if (w) atomicAdd(&counts[static_cast<long long>(Nc) + 1 + b], w);
    }
  }
}

// population_frequency_histogram output: out[k] = count of k (k in [1, Nc)), out[0] = count of 0,
// of Nc (fixed folds into 0) and of the (num_sites - M) monomorphic sites, in uint32 arithmetic as
// the reference accumulates it (spectrum.cu:78-82).
__global__ void hist_to_float_kernel(const unsigned* __restrict__ counts, int Nc, unsigned extra0, float* __restrict__ out) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < Nc; k += blockDim.x * gridDim.x) {
    unsigned v = counts[k];
    if (k == 0) v = v + counts[Nc] + extra0;
    out[k] = static_cast<float>(v);
  }
}

// ------------------------------------------------------------------------------------------------
// host drivers
// ------------------------------------------------------------------------------------------------
static size_t al256(size_t v) { return (v + 255) / 256 * 256; }

static int hist_blocks(int M) { return std::max(1, std::min(148 * 4, M / (4 * kHistThreads) + 1)); }

gf_status population_histogram_device(Engine* e, const float* d_freq, int M, int Nc, float num_sites, float* d_out) {
  if (Nc <= 0) return fail(e, GF_ERR_INVALID_ARGUMENT, "Nchrom_e must be > 0");
  if (M < 0) return fail(e, GF_ERR_INVALID_ARGUMENT, "num_mutations < 0");
  const size_t bytes = sizeof(unsigned) * (static_cast<size_t>(Nc) + 1);
  gf_status st = ensure_scratch(e, &e->spec_scratch, &e->spec_scratch_bytes, bytes);
  if (st != GF_OK) return st;
  unsigned* counts = static_cast<unsigned*>(e->spec_scratch);
  GF_CUDA(e, cudaMemsetAsync(counts, 0, bytes, e->stream));
  if (M > 0) {
    hist_kernel<false><<<hist_blocks(M), kHistThreads, 0, e->stream>>>(d_freq, M, Nc, counts, 0, nullptr);
    GF_CUDA(e, cudaGetLastError());
    e->kernel_launches += 1;
  }
  const unsigned extra0 = static_cast<unsigned>(static_cast<int>(num_sites) - M);
  hist_to_float_kernel<<<std::max(1, std::min(1024, (Nc + 255) / 256)), 256, 0, e->stream>>>(counts, Nc, extra0, d_out);
  GF_CUDA(e, cudaGetLastError());
  e->kernel_launches += 1;
  return GF_OK;
}

// Whether a row's histogram is projected instead of its mutations.  A mutation costs the projection about
// 64 ns / 1,000 (n = 1,000) and the histogram a tenth of that, and a neutral row of M = Nc / 4 mutations holds
// about half as many distinct frequencies; below that the two are level and the row itself is one launch
// less.
static bool project_histogram(int M, int Nc) { return M > Nc / 4; }

gf_status site_frequency_spectrum_device(Engine* e, const float* d_freq, int M, int Nc, int n, float num_sites,
                                         float* d_out) {
  if (n <= 0 || n >= Nc)
    return fail(e, GF_ERR_INVALID_ARGUMENT, "sample_size %d out of range [1, population_size %d)", n, Nc);
  if (M < 0) return fail(e, GF_ERR_INVALID_ARGUMENT, "num_mutations < 0");
  if (n > kProjMaxSample) return fail(e, GF_ERR_CAPACITY, "sample_size %d above the supported %d", n, kProjMaxSample);
  const bool hist = project_histogram(M, Nc);
  const size_t count_bytes = hist ? al256(sizeof(unsigned) * (2 * (static_cast<size_t>(Nc) + 1) + 1)) : 0;
  const int parts = project_parts(n, M, 1, e->num_sms);
  gf_status st = ensure_scratch(e, &e->spec_scratch, &e->spec_scratch_bytes,
                                count_bytes + sizeof(double) * project_scratch(n, parts, 1));
  if (st != GF_OK) return st;
  double* partial = reinterpret_cast<double*>(static_cast<char*>(e->spec_scratch) + count_bytes);
  ProjSource src;
  src.freq = d_freq;
  src.M = M;
  if (hist) {
    unsigned* counts = static_cast<unsigned*>(e->spec_scratch);
    unsigned* mismatch = counts + 2 * (static_cast<size_t>(Nc) + 1);
    GF_CUDA(e, cudaMemsetAsync(counts, 0, count_bytes, e->stream));
    hist_kernel<true><<<hist_blocks(M), kHistThreads, 0, e->stream>>>(d_freq, M, Nc, counts, 1, mismatch);
    GF_CUDA(e, cudaGetLastError());
    e->kernel_launches += 1;
    src.counts = counts;
    src.Nc = Nc;
    src.rounded = 1;
    src.mismatch = mismatch;
  }
  GF_CUDA(e, project_rows(src, n, 1, parts, static_cast<double>(num_sites - M), nullptr, partial, d_out, e->stream));
  e->kernel_launches += 2;
  return GF_OK;
}

static gf_status stage_input(Engine* e, const float* h_freq, int M, const float** d_freq) {
  gf_status st = ensure_scratch(e, reinterpret_cast<void**>(&e->spec_in), &e->spec_in_bytes,
                                sizeof(float) * std::max(M, 1));
  if (st != GF_OK) return st;
  if (M > 0) GF_CUDA(e, cudaMemcpyAsync(e->spec_in, h_freq, sizeof(float) * M, cudaMemcpyHostToDevice, e->stream));
  *d_freq = e->spec_in;
  return GF_OK;
}

}  // namespace gf

using namespace gf;

extern "C" {

gf_status gf_population_histogram_device(gf_engine* g, const float* d_freq, int32_t M, int32_t Nc, float L, float* d_out) {
  return guard_host(g, [&]() -> gf_status {
    if (!g) return GF_ERR_INVALID_ARGUMENT;
    Engine* e = &g->impl;
    GF_CUDA(e, cudaSetDevice(e->device));
    return population_histogram_device(e, d_freq, M, Nc, L, d_out);
  });
}

gf_status gf_site_frequency_spectrum_device(gf_engine* g, const float* d_freq, int32_t M, int32_t Nc, int32_t n, float L,
                                            float* d_out) {
  return guard_host(g, [&]() -> gf_status {
    if (!g) return GF_ERR_INVALID_ARGUMENT;
    Engine* e = &g->impl;
    GF_CUDA(e, cudaSetDevice(e->device));
    return site_frequency_spectrum_device(e, d_freq, M, Nc, n, L, d_out);
  });
}

gf_status gf_population_histogram(gf_engine* g, const float* freq, int32_t M, int32_t Nc, float L, float* out) {
  return guard_host(g, [&]() -> gf_status {
    if (!g) return GF_ERR_INVALID_ARGUMENT;
    Engine* e = &g->impl;
    if (!out || (M > 0 && !freq)) return fail(e, GF_ERR_INVALID_ARGUMENT, "NULL buffer");
    GF_CUDA(e, cudaSetDevice(e->device));
    const float* d_freq = nullptr;
    gf_status st = stage_input(e, freq, M, &d_freq);
    if (st != GF_OK) return st;
    st = ensure_scratch(e, reinterpret_cast<void**>(&e->spec_out), &e->spec_out_bytes, sizeof(float) * std::max(Nc, 1));
    if (st != GF_OK) return st;
    st = population_histogram_device(e, d_freq, M, Nc, L, e->spec_out);
    if (st != GF_OK) return st;
    GF_CUDA(e, cudaMemcpyAsync(out, e->spec_out, sizeof(float) * Nc, cudaMemcpyDeviceToHost, e->stream));
    GF_CUDA(e, cudaStreamSynchronize(e->stream));
    return GF_OK;
  });
}

gf_status gf_site_frequency_spectrum(gf_engine* g, const float* freq, int32_t M, int32_t Nc, int32_t n, float L, float* out) {
  return guard_host(g, [&]() -> gf_status {
    if (!g) return GF_ERR_INVALID_ARGUMENT;
    Engine* e = &g->impl;
    if (!out || (M > 0 && !freq)) return fail(e, GF_ERR_INVALID_ARGUMENT, "NULL buffer");
    GF_CUDA(e, cudaSetDevice(e->device));
    const float* d_freq = nullptr;
    gf_status st = stage_input(e, freq, M, &d_freq);
    if (st != GF_OK) return st;
    st = ensure_scratch(e, reinterpret_cast<void**>(&e->spec_out), &e->spec_out_bytes, sizeof(float) * std::max(n, 1));
    if (st != GF_OK) return st;
    st = site_frequency_spectrum_device(e, d_freq, M, Nc, n, L, e->spec_out);
    if (st != GF_OK) return st;
    GF_CUDA(e, cudaMemcpyAsync(out, e->spec_out, sizeof(float) * n, cudaMemcpyDeviceToHost, e->stream));
    GF_CUDA(e, cudaStreamSynchronize(e->stream));
    return GF_OK;
  });
}

}  // extern "C"

// ==================================================================================================
// SFS without allocation.
//
// For callers that must not allocate device memory: code running inside a framework that owns the
// GPU's memory budget (a caching allocator or a pre-reserved pool, where a library's own cudaMalloc
// would bypass the budget and can fail mid-run), and code on a latency-critical path, where
// cudaMalloc / cudaFree would synchronize the device and stall work queued on other streams.  This
// entry point takes its scratch from one file-scope __device__ array instead of engine-owned
// allocations, and needs no gf_engine.
//
// The array is part of the library image: every GPU that loads libgofish_b200.so holds it
// (GF_NOALLOC_SCRATCH_BYTES, about 6.3 MB) until the process exits.  All calls on a device share it
// and it keeps the previous call's contents, so calls whose GPU work overlaps (concurrent streams, or
// several host threads) race and must be serialized by the caller.
// ==================================================================================================

#include <mutex>

namespace gf {

// Scratch of gf_site_frequency_spectrum_noalloc: [counts | mismatch | spare | partials]
constexpr size_t kNoAllocCountsOff = 0;
constexpr size_t kNoAllocFlagsOff = (sizeof(unsigned) * (GF_NOALLOC_MAX_NCHROM + 1) + 255) / 256 * 256;
constexpr size_t kNoAllocPartialOff = kNoAllocFlagsOff + 256;
constexpr size_t kNoAllocBytes = GF_NOALLOC_SCRATCH_BYTES;
constexpr int kNoAllocMaxBlocks = static_cast<int>((kNoAllocBytes - kNoAllocPartialOff) / (sizeof(double) * (GF_NOALLOC_MAX_SAMPLE + 2)));
static_assert(kNoAllocMaxBlocks >= 148, "a block per SM fits the scratch");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

// Per-device set-up, done once per device by the first call on it (with that device current): the
// scratch array's device address (in host code the array's name only stands for the symbol; kernels
// must be given this address), and the kernels of every sample size loaded with their shared-memory limits.
// Under lazy module loading this first call may also load the module, which is when the array takes its
// device memory.  The cached set-up does not survive cudaDeviceReset.
static gf_status noalloc_scratch(int device, unsigned char** out) {
  static std::mutex mu;
  static unsigned char* addr[64] = {nullptr};
  if (device < 0 || device >= 64) return GF_ERR_NO_DEVICE;
  std::lock_guard<std::mutex> lock(mu);
  if (!addr[device]) {
    void* p = nullptr;
    cudaError_t err = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    cudaFuncAttributes at;
    if (err == cudaSuccess && p) err = cudaFuncGetAttributes(&at, hist_kernel<true>);
    if (err == cudaSuccess && p) err = project_ready();
    if (err != cudaSuccess || !p) {
      cudaGetLastError();
      return GF_ERR_CUDA;
    }
    addr[device] = static_cast<unsigned char*>(p);
  }
  *out = addr[device];
  return GF_OK;
}

#define GF_NA_CUDA(call)                     \
  do {                                       \
    if ((call) != cudaSuccess) {             \
      cudaGetLastError();                    \
      return GF_ERR_CUDA;                    \
    }                                        \
  } while (0)

}  // namespace gf

extern "C" {

gf_status gf_site_frequency_spectrum_noalloc(const float* d_freq, int32_t M, int32_t Nc, int32_t n, float num_sites,
                                             float* d_out, void* cuda_stream) {
  using namespace gf;
  if (!d_out || (M > 0 && !d_freq) || M < 0) return GF_ERR_INVALID_ARGUMENT;
  if (n <= 0 || n >= Nc) return GF_ERR_INVALID_ARGUMENT;
  if (Nc > GF_NOALLOC_MAX_NCHROM || n > GF_NOALLOC_MAX_SAMPLE) return GF_ERR_CAPACITY;
  int device = 0;
  GF_NA_CUDA(cudaGetDevice(&device));
  unsigned char* base = nullptr;
  const gf_status st = noalloc_scratch(device, &base);
  if (st != GF_OK) return st;
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  unsigned* counts = reinterpret_cast<unsigned*>(base + kNoAllocCountsOff);
  unsigned* mismatch = reinterpret_cast<unsigned*>(base + kNoAllocFlagsOff);
  double* partial = reinterpret_cast<double*>(base + kNoAllocPartialOff);
  // the array keeps the previous call's contents: what is accumulated into starts from zero here.  Both
  // halves of the histogram where they fit, else rows of rounded quotients are projected one by one.
  const size_t classes = static_cast<size_t>(Nc) + 1;
  const int rounded = 2 * classes <= GF_NOALLOC_MAX_NCHROM + 1 ? 1 : 0;
  ProjSource src;
  src.freq = d_freq;
  src.M = M;
  if (project_histogram(M, Nc)) {
    GF_NA_CUDA(cudaMemsetAsync(counts, 0, sizeof(unsigned) * classes * (rounded ? 2 : 1), stream));
    GF_NA_CUDA(cudaMemsetAsync(mismatch, 0, sizeof(unsigned), stream));
    hist_kernel<true><<<hist_blocks(M), kHistThreads, 0, stream>>>(d_freq, M, Nc, counts, rounded, mismatch);
    GF_NA_CUDA(cudaGetLastError());
    src.counts = counts;
    src.Nc = Nc;
    src.rounded = rounded;
    src.mismatch = mismatch;
  }
  const int parts = std::min(kNoAllocMaxBlocks, project_parts(n, M, 1, 148));
  GF_NA_CUDA(project_rows(src, n, 1, parts, static_cast<double>(num_sites - M), nullptr, partial, d_out, stream));
  return GF_OK;
}
}  // extern "C"
