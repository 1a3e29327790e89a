// SFS surrogate network on sm_100a tensor cores: a bf16 GEMM built on TMA + tcgen05 with the
// accumulator in tensor memory, fused epilogues (bias + GELU forward, the loss and its gradient, GELU'
// backward with bias gradients), and one kernel for the weight gradients of all layers and Adam.
//
// Every GEMM is C[M][N] = A[M][K] * B[N][K]^T with both operands K-contiguous:
//   forward   Z_l  = Y_{l-1} W_l^T          A = Y_{l-1} [batch][in]      B = W_l   [out][in]
//   input     dY_{l-1} = dZ_l W_l           A = dZ_l    [batch][out]     B = W_l^T [in][out]
//   weights   dW_l = dZ_l^T Y_{l-1}         A = dZ_l^T  [out][batch]     B = Y_{l-1}^T [in][batch]
// so the forward epilogue writes each activation twice (row-major and transposed), the backward
// epilogue does the same for dZ, and Adam keeps bf16 copies of W and W^T.  Layer 1's six inputs are
// zero-padded to 64 columns and layer 5's 99 outputs to 128 rows; padding stays exactly zero.
//
// The reference has no network (3P answers every SFS query by simulation, go_fish.cuh:280 and
// spectrum.h:90); this file serves the surrogate that stands in for those calls.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <exception>
#include <mutex>
#include <new>
#include <string>
#include <thread>
#include <utility>
#include <vector>

#include "gf_surrogate.h"
#include "gf_umma.cuh"

namespace gfm {

constexpr int BM = 128;       // tile rows = tensor-memory lanes
constexpr int BK = 64;        // K per pipeline stage: one 128-byte swizzle row of bf16
constexpr long long WAIT_LIMIT = 1ll << 31;   // SM cycles (about a second) before a wait gives up
constexpr long long INJECT_WAIT_LIMIT = 1ll << 22;   // the same under fault injection (about 2 ms)
constexpr int HID = GF_MLP_HIDDEN;
constexpr int IN_PAD = 64;
constexpr int OUT_PAD = 128;
constexpr int MAX_SPLITS = 16;

enum Epi : int {
  EPI_STORE_F32 = 0,     // C (fp32)
  EPI_FWD_GELU = 1,      // Z = acc + bias (fp32), Y = GELU(Z) (bf16) and Y^T (bf16)
  EPI_BWD_GELU = 3,      // dZ = acc * GELU'(Z) (bf16) and dZ^T (bf16), bias partials
  EPI_FWD_GELU_INFER = 5,// Y = GELU(acc + bias) (bf16) only
  EPI_FWD_OUT = 6,       // out = acc + bias written straight to the caller's [rows][99] array
  EPI_FWD_LOSS = 7       // dOut = 2 (acc + bias - target) / (rows * 99) (bf16) and dOut^T, the tile's column sums
                         // of it (layer 5's bias gradient) and its loss
};

struct EpiArgs {
  const float* bias;         // [N]
  const float* z;            // forward pre-activation read by the backward epilogue
  long long ldz;
  float* bias_part;          // [M / 128][ld_bias_part] column sums of the backward output
  long long ld_bias_part;
  float* out;                // caller's output [rows][out_cols] (EPI_FWD_OUT)
  int out_cols;
  const float* target;       // [rows][99], row idx[i] for output row i where idx is given (EPI_FWD_LOSS)
  const long long* idx;
  float* loss_part;          // [M / 128] (EPI_FWD_LOSS)
  int batch;
  int* fault;                // set when a bounded wait ran out
};

// Epilogue warps of an N tile: two per tensor-memory lane quarter, one where a quarter has a single 32-column
// chunk.
__host__ __device__ constexpr int epi_warps(int BN) { return BN >= 64 ? 8 : 4; }
__host__ __device__ constexpr int gemm_threads(int BN) { return 64 + 32 * epi_warps(BN); }   // TMA warp, MMA warp, epilogue warps

// Programmatic dependent launch: a training step's kernels follow one another on one stream, and each may set
// up its barriers and tensor memory while the one before it still runs, then waits here for its results.
// (Without the launch attribute both are no-ops.)
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_next() { asm volatile("griddepcontrol.launch_dependents;"); }
constexpr int SMEM_LIMIT = 232448;                  // dynamic shared memory per CTA on sm_100

// Per-epilogue-warp staging of one 32 x 32 output chunk, double-buffered: fp32 rows with the 128-byte
// swizzle, bf16 rows with the 64-byte swizzle, bf16 transposed rows unswizzled -- the layouts the
// output tensor maps expect, and conflict-free for the row-per-lane writes.  Only the outputs the
// epilogue writes get space.
template <int BN, int EPI>
struct Stage {
  static constexpr bool F32 = EPI == EPI_STORE_F32 || EPI == EPI_FWD_GELU;
  static constexpr bool BF16 = EPI == EPI_FWD_GELU || EPI == EPI_FWD_GELU_INFER || EPI == EPI_BWD_GELU ||
                               EPI == EPI_FWD_LOSS;
  static constexpr bool T = EPI == EPI_FWD_GELU || EPI == EPI_BWD_GELU || EPI == EPI_FWD_LOSS;
  static constexpr int BUFFERS = BN >= 128 ? 2 : 1;   // a warp has one chunk per tile below that
  static constexpr int F32_OFF = 0;
  static constexpr int BF16_OFF = F32 ? 4096 : 0;
  static constexpr int T_OFF = BF16_OFF + (BF16 ? 2048 : 0);
  static constexpr int BUF = ((T_OFF + (T ? 2048 : 0)) + 1023) / 1024 * 1024;
  static constexpr int WARP = BUFFERS * BUF;
};

template <int BN, int EPI>
struct Smem {
  // narrow training tiles load two K blocks with one TMA box (a 3-D map of K blocks): half the loads, which is
  // what their short K loops wait for (128-wide tiles have no room for it beside their staging)
  static constexpr int KS = BN < 128 && (EPI == EPI_FWD_GELU || EPI == EPI_BWD_GELU) ? 2 : 1;
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = KS * (A_BYTES + B_BYTES);
  static constexpr int BIAS_FLOATS = 512;   // the bias vector of the whole output width
  // EPI_FWD_OUT stages a whole 128-row tile of the caller's [rows][99] output (one contiguous span)
  // EPI_FWD_LOSS keeps a tile's targets, then its residuals, in rows of 99 floats
  static constexpr int OUT_TILE =
      EPI == EPI_FWD_OUT || EPI == EPI_FWD_LOSS ? (BM * GF_MLP_OUTPUTS * 4 + 1023) / 1024 * 1024 : 0;
  static constexpr int STAGING = epi_warps(BN) * Stage<BN, EPI>::WARP;
  static constexpr int EXTRA = STAGING + OUT_TILE + 256 + 2 * 4 * 32 * 4 + 4 * BIAS_FLOATS + 1024;
  // narrow tiles: two stages of two blocks, so that the next kernel's CTA fits beside this one's
  static constexpr int STAGES = BN == 32                                  ? 2
                                : (4 * STAGE_BYTES + EXTRA <= SMEM_LIMIT) ? 4
                                : (3 * STAGE_BYTES + EXTRA <= SMEM_LIMIT) ? 3
                                                                          : 2;
  static constexpr int STG_OFFSET = STAGES * STAGE_BYTES;
  static constexpr int BAR_OFFSET = STG_OFFSET + STAGING + OUT_TILE;
  static constexpr int OUT_OFFSET = BAR_OFFSET - OUT_TILE;
  static constexpr int BIAS_OFFSET = BAR_OFFSET + 256 + 2 * 4 * 32 * 4;
  static constexpr int BYTES = BIAS_OFFSET + 4 * BIAS_FLOATS + 1024;   // + barriers, reductions, bias, alignment
  static_assert(BYTES <= SMEM_LIMIT, "shared memory");
};

// GELU in its tanh form, 0.5 z (1 + tanh(sqrt(2/pi) (z + 0.044715 z^3))), on the hardware tanh.
constexpr float GELU_C = 0.7978845608028654f;
constexpr float GELU_A = 0.044715f;

__device__ __forceinline__ float tanh_hw(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Written as tanh(z (c + c a z^2)) and (z/2) t + z/2: six instructions, one of them on the MUFU pipe.
// The fused forward's epilogue is bound by instruction issue, and this form issues two fewer than
// c (z + a z^3) and (z/2)(1 + t).
__device__ __forceinline__ float gelu(float z) {
  const float t = tanh_hw(z * fmaf(GELU_C * GELU_A, z * z, GELU_C));
  const float hz = 0.5f * z;
  return fmaf(hz, t, hz);
}

__device__ __forceinline__ float gelu_grad(float z) {
  const float z2 = z * z;
  const float t = tanh_hw(GELU_C * fmaf(GELU_A * z, z2, z));
  return 0.5f * (1.f + t) + 0.5f * z * (1.f - t * t) * GELU_C * fmaf(3.f * GELU_A, z2, 1.f);
}

// row `r` of a 32 x 32 fp32 chunk, 128-byte swizzle (16-byte unit q of row r sits at q ^ (r % 8))
__device__ __forceinline__ void stage_f32_row(uint8_t* buf, int r, const float* v) {
#pragma unroll
  for (int q = 0; q < 8; ++q)
    *reinterpret_cast<float4*>(buf + r * 128 + ((q ^ (r & 7)) << 4)) =
        make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
}

// row `r` of a 32 x 32 bf16 chunk, 64-byte swizzle (16-byte unit q of row r sits at q ^ ((r / 2) % 4))
__device__ __forceinline__ void stage_bf16_row(uint8_t* buf, int r, const float* v) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t w[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      __nv_bfloat162 p = __floats2bfloat162_rn(v[q * 8 + 2 * t], v[q * 8 + 2 * t + 1]);
      w[t] = *reinterpret_cast<uint32_t*>(&p);
    }
    *reinterpret_cast<uint4*>(buf + r * 64 + ((q ^ ((r >> 1) & 3)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// column `r` of the transposed chunk: element (j, r) at j * 64 + 2 r
__device__ __forceinline__ void stage_bf16_col(uint8_t* buf, int r, const float* v) {
#pragma unroll
  for (int j = 0; j < 32; ++j) *reinterpret_cast<__nv_bfloat16*>(buf + j * 64 + 2 * r) = __float2bfloat16_rn(v[j]);
}

// Persistent tensor-core GEMM: CTAs stride over 128 x BN output tiles (N fastest, then M).  Warp 0 streams A/B
// K-blocks with TMA into a ring of two to four stages, warp 1 issues tcgen05 MMAs into one of two tensor-memory
// accumulators, four (32-wide tiles) or eight epilogue warps drain the other one (tcgen05.ld -> registers ->
// swizzled shared staging -> TMA store), so a tile's epilogue overlaps the next tile's MMAs.
template <int BN, int EPI>
__global__ void __launch_bounds__(gemm_threads(BN), BN == 32 ? 2 : 1)   // 2: the next kernel's CTA beside it
umma_gemm_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                 const __grid_constant__ CUtensorMap tma_c, const __grid_constant__ CUtensorMap tma_y,
                 const __grid_constant__ CUtensorMap tma_yt, int m_tiles, int n_tiles, int k_blocks, EpiArgs ep,
                 long long wait_limit, int inject) {
  using L = Smem<BN, EPI>;
  using SG = Stage<BN, EPI>;
  constexpr int STAGES = L::STAGES;
  constexpr int EPI_WARPS = epi_warps(BN);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::BAR_OFFSET);
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;      // accumulator ready (MMA -> epilogue)
  uint64_t* tempty = tfull + 2;          // accumulator drained (epilogue -> MMA)
  uint64_t* drain = tempty + 2;           // MMA completion before tensor memory is released (abort path)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  int* timed_out = reinterpret_cast<int*>(tmem_slot + 1);
  int* epi_fail = timed_out + 1;         // the epilogue warps' joint verdict (sticky)
  int* consumed_s = timed_out + 2;       // K-blocks the MMA thread received (for the drain)
  float* red = reinterpret_cast<float*>(smem + L::BAR_OFFSET + 256);   // [2 halves][4 quarters][32]
  float* s_bias = reinterpret_cast<float*>(smem + L::BIAS_OFFSET);
  volatile int* abort_flag = timed_out;
  constexpr bool HAS_BIAS = EPI == EPI_FWD_GELU || EPI == EPI_FWD_GELU_INFER || EPI == EPI_FWD_OUT ||
                            EPI == EPI_FWD_LOSS;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles = m_tiles * n_tiles;
  // Bounded waits.  The producer and MMA threads stop issuing work as soon as any wait of the CTA has
  // run out (`wait`); the epilogue warps wait on the barrier alone and then agree on the outcome, so
  // all of them leave the tile loop together.  An aborted CTA never touches unsynchronised data: it
  // drains what it issued and releases tensor memory.
  auto wait = [&](uint64_t* bar, uint32_t parity) { return mbar_wait_warp(bar, parity, wait_limit, abort_flag); };

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_b);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], EPI_WARPS);
    }
    mbar_init(drain, 1);
    *timed_out = 0;
    *epi_fail = 0;
    *consumed_s = 0;
    mbar_fence_init();
  }
  __syncwarp();
  if (warp == 1) tmem_alloc(tmem_slot, 2 * BN);
  grid_launch_next();
  grid_wait();   // from here on: what the kernels before this one wrote
  if constexpr (HAS_BIAS) {
    for (int i = threadIdx.x; i < n_tiles * BN && i < L::BIAS_FLOATS; i += blockDim.x) s_bias[i] = ep.bias[i];
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  bool late = false;
  int issued = 0;   // K-blocks the producer issued (for the drain after a timeout)

  // warps 0 and 1 stay converged and elect the lane that issues, which keeps the operands in uniform registers
  if (warp == 0) {
    int s = 0;
    uint32_t phase = 1;
    for (int tile = blockIdx.x; tile < tiles && !late; tile += gridDim.x) {
      const int nt = tile % n_tiles, mt = tile / n_tiles;
      for (int kb = 0; kb < k_blocks; kb += L::KS) {
        if (!wait(&empty[s], phase)) {
          late = true;
          break;
        }
        uint8_t* a = smem + s * L::STAGE_BYTES;
        if (elect_one()) {
          if constexpr (L::KS == 1) {
            mbar_arrive_expect_tx(&full[s], L::STAGE_BYTES);
            tma_load_2d(a, &tma_a, kb * BK, mt * BM, &full[s]);
            tma_load_2d(a + L::A_BYTES, &tma_b, kb * BK, nt * BN, &full[s]);
          } else {   // the maps' boxes hold min(KS, k_blocks) K blocks
            mbar_arrive_expect_tx(&full[s], min(L::KS, k_blocks) * (L::A_BYTES + L::B_BYTES));
            tma_load_3d(a, &tma_a, 0, mt * BM, kb, &full[s]);
            tma_load_3d(a + L::KS * L::A_BYTES, &tma_b, 0, nt * BN, kb, &full[s]);
          }
        }
        __syncwarp();
        ++issued;
        if (++s == STAGES) {
          s = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = bf16_idesc(BM, BN);
    const uint64_t desc = sw128_kmajor_desc(smem_u32(smem));
    int s = 0, received = 0, local = 0;
    uint32_t phase = 0;
    for (int tile = blockIdx.x; tile < tiles && !late; tile += gridDim.x, ++local) {
      const int acc = local & 1;
      const uint32_t use = static_cast<uint32_t>(local >> 1);
      if (!wait(&tempty[acc], (use & 1) ^ 1)) {
        late = true;
        break;
      }
      tc_fence_after();
      const uint32_t d = tmem + static_cast<uint32_t>(acc * BN);
      for (int kb = 0; kb < k_blocks; kb += L::KS) {
        if (!wait(&full[s], phase)) {
          late = true;
          break;
        }
        ++received;
        tc_fence_after();
        // descriptor addresses count 16 bytes
        const uint64_t a = desc + s * (L::STAGE_BYTES >> 4), b = a + (L::KS * L::A_BYTES >> 4);
        if (elect_one()) {
#pragma unroll
          for (int h = 0; h < L::KS; ++h) {
            if (kb + h < k_blocks) {
#pragma unroll
              for (int kk = 0; kk < BK / 16; ++kk)
                umma_bf16(d, a + h * (L::A_BYTES >> 4) + 2 * kk, b + h * (L::B_BYTES >> 4) + 2 * kk, idesc,
                          (kb | h | kk) != 0);
            }
          }
          umma_commit(&empty[s]);
        }
        __syncwarp();
        if (++s == STAGES) {
          s = 0;
          phase ^= 1;
        }
      }
      if (late) break;
      // fault injection for tests: withhold the first accumulator hand-off
      if (!((inject & 1) && local == 0) && elect_one()) umma_commit(&tfull[acc]);
      __syncwarp();
    }
    if (lane == 0) *consumed_s = received;
    __syncwarp();
  } else {
    // epilogue warps: TMEM lane quarter = warp % 4; the two warps of a quarter take alternate
    // 32-column chunks
    const int qd = warp & 3;
    const int ew = warp - 2;
    const int half = ew >> 2;
    uint8_t* stg = smem + L::STG_OFFSET + ew * SG::WARP;
    // the forward pre-activations of 32 columns of a row (EPI_BWD_GELU), read while the MMAs run where the warp
    // has a single chunk per tile
    float4 z[EPI == EPI_BWD_GELU ? 8 : 1];
    auto load_z = [&](float4* to, int r, int n) {
      const float4* zp = reinterpret_cast<const float4*>(ep.z + static_cast<long long>(r) * ep.ldz + n);
#pragma unroll
      for (int q = 0; q < 8; ++q) to[q] = __ldg(zp + q);
    };
    int chunk = 0, local = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++local) {
      const int nt = tile % n_tiles, mt = tile / n_tiles;
      const int acc = local & 1;
      const uint32_t use = static_cast<uint32_t>(local >> 1);
      if constexpr (EPI == EPI_BWD_GELU && SG::BUFFERS == 1) load_z(z, mt * BM + qd * 32 + lane, nt * BN + 32 * half);
      if constexpr (EPI == EPI_FWD_LOSS) {
        // the tile's targets, coalesced row by row, while its MMAs run (the barrier below orders them); a lane
        // holds one of the warp's row indices, so that the rows' loads do not wait for one another
        constexpr int ROWS = BM / EPI_WARPS;
        float* s_t = reinterpret_cast<float*>(smem + L::OUT_OFFSET) + ew * ROWS * GF_MLP_OUTPUTS;
        const long long r0 = static_cast<long long>(mt) * BM + ew * ROWS;
        const long long mine = lane < ROWS ? (ep.idx ? ep.idx[r0 + lane] : r0 + lane) : 0;
#pragma unroll 8
        for (int r = 0; r < ROWS; ++r) {
          const float* from = ep.target + __shfl_sync(0xffffffffu, mine, r) * GF_MLP_OUTPUTS;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (32 * j + lane < GF_MLP_OUTPUTS) s_t[r * GF_MLP_OUTPUTS + 32 * j + lane] = __ldg(from + 32 * j + lane);
        }
      }
      if (lane == 0 && !mbar_wait(&tfull[acc], use & 1, wait_limit)) atomicOr(epi_fail, 1);
      named_barrier_sync(4, 32 * EPI_WARPS);     // every epilogue warp has its verdict in epi_fail
      if (*reinterpret_cast<volatile int*>(epi_fail)) {
        late = true;
        break;
      }
      __syncwarp();
      tc_fence_after();
      const int row0 = mt * BM + qd * 32;        // first output row of this warp
      const int row = row0 + lane;
      float* s_out = reinterpret_cast<float*>(smem + L::OUT_OFFSET);
      if constexpr (EPI == EPI_FWD_OUT) {
        // the previous tile's bulk store has read the staging tile
        if (ew == 0 && lane == 0) bulk_wait_read<0>();
        named_barrier_sync(3, 32 * EPI_WARPS);
      }
      const uint32_t tbase = tmem + (static_cast<uint32_t>(qd * 32) << 16) + static_cast<uint32_t>(acc * BN);
#pragma unroll 1
      for (int c0 = 32 * half; c0 < BN; c0 += 64, ++chunk) {
        const int n = nt * BN + c0;
        uint8_t* buf = stg + (chunk % SG::BUFFERS) * SG::BUF;
        if (lane == 0) bulk_wait_read<SG::BUFFERS - 1>();     // the store that last used this buffer has read it
        __syncwarp();
        float v[32];
        tmem_ld_32cols(tbase + c0, v);
        if constexpr (EPI == EPI_STORE_F32) {
          stage_f32_row(buf + SG::F32_OFF, lane, v);
        } else if constexpr (EPI == EPI_FWD_OUT) {
          // row stride 99 words: lanes (rows) hit distinct banks
          float* o = s_out + (qd * 32 + lane) * GF_MLP_OUTPUTS;
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (n + j < GF_MLP_OUTPUTS) o[n + j] = v[j] + s_bias[n + j];
        } else if constexpr (EPI == EPI_FWD_GELU || EPI == EPI_FWD_GELU_INFER) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] += s_bias[n + j];
          if constexpr (EPI == EPI_FWD_GELU) stage_f32_row(buf + SG::F32_OFF, lane, v);
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = gelu(v[j]);
          stage_bf16_row(buf + SG::BF16_OFF, lane, v);
          if constexpr (EPI == EPI_FWD_GELU) stage_bf16_col(buf + SG::T_OFF, lane, v);
        } else if constexpr (EPI == EPI_FWD_LOSS) {
          const float scale = 2.f / (static_cast<float>(ep.batch) * GF_MLP_OUTPUTS);
          float* d = s_out + (qd * 32 + lane) * GF_MLP_OUTPUTS;   // targets in, residuals out
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            if (n + j < GF_MLP_OUTPUTS) {
              const float r = v[j] + s_bias[n + j] - d[n + j];
              d[n + j] = r;
              v[j] = scale * r;
            } else {
              v[j] = 0.f;
            }
          }
          stage_bf16_row(buf + SG::BF16_OFF, lane, v);
          stage_bf16_col(buf + SG::T_OFF, lane, v);
        } else if constexpr (EPI == EPI_BWD_GELU) {
          if constexpr (SG::BUFFERS > 1) load_z(z, row, n);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            v[4 * q] *= gelu_grad(z[q].x);
            v[4 * q + 1] *= gelu_grad(z[q].y);
            v[4 * q + 2] *= gelu_grad(z[q].z);
            v[4 * q + 3] *= gelu_grad(z[q].w);
          }
          stage_bf16_row(buf + SG::BF16_OFF, lane, v);
          stage_bf16_col(buf + SG::T_OFF, lane, v);
          // column sums over the tile's 128 rows (fixed order: lanes, then quarters 0..3); the four
          // warps of a half work on the same chunk and meet at their own named barrier
          // lanes: the sums of a butterfly over all 32 columns, but each step keeps only the half of the columns
          // that this lane's bit selects and sends the other (31 shuffles in place of 160), so lane j ends with
          // column j
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            const bool upper = (lane & o) != 0;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              if (j >= o) break;
              const float keep = upper ? v[j + o] : v[j], send = upper ? v[j] : v[j + o];
              v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
          }
          const float mine = v[0];
          float* rh = red + half * 128;
          rh[qd * 32 + lane] = mine;
          named_barrier_sync(1 + half, 128);
          if (qd == 0) {
            const float t = ((rh[lane] + rh[32 + lane]) + rh[64 + lane]) + rh[96 + lane];
            ep.bias_part[mt * ep.ld_bias_part + n + lane] = t;
          }
          named_barrier_sync(1 + half, 128);
        }
        if constexpr (EPI == EPI_FWD_OUT) continue;   // written directly
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          if constexpr (SG::F32) tma_store_2d(&tma_c, n, row0, buf + SG::F32_OFF);
          if constexpr (SG::BF16) tma_store_2d(&tma_y, n, row0, buf + SG::BF16_OFF);
          if constexpr (SG::T) tma_store_2d(&tma_yt, row0, n, buf + SG::T_OFF);
          bulk_commit();
        }
      }
      if constexpr (EPI == EPI_FWD_OUT) {
        // rows [mt*128, mt*128 + 128) of a [rows][99] array are one contiguous span
        fence_proxy_async_smem();
        named_barrier_sync(3, 32 * EPI_WARPS);
        if (ew == 0 && lane == 0) {
          bulk_store_1d(ep.out + static_cast<long long>(mt) * BM * GF_MLP_OUTPUTS, s_out, BM * GF_MLP_OUTPUTS * 4);
          bulk_commit();
        }
      }
      if constexpr (EPI == EPI_FWD_LOSS) {
        // sums over the tile in a fixed order: a column's rows 0 .. 127, a row's columns, then the rows
        named_barrier_sync(3, 32 * EPI_WARPS);   // every residual is in place
        const int et = threadIdx.x - 64;
        if (et < BM) {
          float l = 0.f;
          const float* d = s_out + et * GF_MLP_OUTPUTS;
#pragma unroll 11
          for (int j = 0; j < GF_MLP_OUTPUTS; ++j) l += d[j] * d[j];
          red[et] = l;
        } else if (et - BM < GF_MLP_OUTPUTS) {
          const float scale = 2.f / (static_cast<float>(ep.batch) * GF_MLP_OUTPUTS);
          const int j = et - BM;
          float t = 0.f;
#pragma unroll 16
          for (int i = 0; i < BM; ++i) t += scale * s_out[i * GF_MLP_OUTPUTS + j];
          ep.bias_part[mt * ep.ld_bias_part + j] = t;
        }
        named_barrier_sync(3, 32 * EPI_WARPS);
        if (et == 0) {
          float t = 0.f;
#pragma unroll 16
          for (int i = 0; i < BM; ++i) t += red[i];
          ep.loss_part[mt] = t / (static_cast<float>(ep.batch) * GF_MLP_OUTPUTS);
        }
        named_barrier_sync(3, 32 * EPI_WARPS);   // before the next tile's targets
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[acc]);
    }
    if (lane == 0) bulk_wait_all();
    __syncwarp();
  }

  tc_fence_before();
  if (late) *abort_flag = 1;
  __syncthreads();
  if (*abort_flag) {
    // a wait ran out: let every load and MMA this CTA issued finish before its shared and tensor
    // memory are released (each wait again bounded)
    if (threadIdx.x == 0) {
      // loads issued but never received by the MMA thread are still landing
      for (int it = *consumed_s; it < issued; ++it) mbar_wait(&full[it % STAGES], (it / STAGES) & 1, wait_limit);
      if (ep.fault) atomicOr(ep.fault, 1);
    } else if (warp == 1) {
      if (elect_one()) umma_commit(drain);   // arrives once every MMA that lane issued has completed
      mbar_wait(drain, 0, wait_limit);
    }
    __syncthreads();
  }
  if (warp == 1) tmem_dealloc(tmem, 2 * BN);
}

// ---------------------------------------------------------------------------------------------
// Fused inference forward: all five layers of a 128-row tile in one CTA, the activations on chip, the
// MMAs of two CTAs paired
//
// The layered path writes each hidden activation (batch x 512 bf16) to memory and reads it back in
// the next layer's GEMM.  Here a CTA keeps its tile's activation H (128 x 512 bf16 = 128 KB) in
// shared memory, in the 128-byte-swizzled K-major layout the MMA reads (eight 64-column K blocks of
// 16 KB), and the layer's fp32 accumulator (128 x 512) in all 512 tensor-memory columns: N half 0
// in region A (columns 0-255), N half 1 in region B (256-511).  Two neighbouring tiles run on a cluster
// of two CTAs: warp 1 of the even one issues MMAs of M = 256 over both (A = each CTA's H, B = weight K
// blocks of which each CTA holds half the rows, streamed by its warp 0 through a ring of six from L2,
// where every CTA finds the 1.3 MB of weights), warp 1 of the odd one reports what has landed there.  16
// epilogue warps a CTA drain the accumulators (bias, GELU, bf16) back into H for the next layer,
// overlapped with the MMAs: region A while N half 1 accumulates (staged in tensor memory, since H is
// still being read), region B, two K blocks at a time, while the next layer's first K blocks accumulate.
// The last layer's epilogue writes acc + bias to the caller's [batch][99] array.  Each layer's MMAs run
// in the order of the layered GEMMs (N halves of 256, K blocks 0..7, four 16-wide slices each; layer 5
// one 128-wide N tile), so the outputs are bit-identical to the layered path.
//
// A layer takes about 11,000 cycles, of which the MMAs 8,400 at their peak rate and the two epilogues 3,800 +
// 3,200: they share tensor memory and shared memory, and each slows the other down.  32,768 rows (256 tiles,
// two rounds of 74 pairs) take 62.5 us; with single-lane producer and issue code on single CTAs it was 86.4,
// a K block taking 940 cycles to issue.  By step: pairs alone 89.5, converged producer and issue warps 71.9,
// region B in two parts and the bias from L1 65.8, a ring of single K blocks 64.2, epilogue warps that wait
// each for themselves 62.5; region B in four parts is slower again (64.4).
// ---------------------------------------------------------------------------------------------
constexpr int FF_EPI_WARPS = 16;                          // four per tensor-memory lane quarter
constexpr int FF_THREADS = 64 + 32 * FF_EPI_WARPS;        // TMA warp, MMA warp, 16 epilogue warps
constexpr int FF_WSTAGES = 6;
constexpr int FF_KB_BYTES = BM * BK * 2;                  // one 128 x 64 bf16 K block of H: 16 KB
constexpr int FF_H_BYTES = BM * HID * 2;                  // H: 128 KB
constexpr int FF_WSTAGE_BYTES = 128 * BK * 2;             // this CTA's 128 rows of a 256-row x 64 weight block: 16 KB
constexpr int FF_BAR_OFFSET = FF_H_BYTES + FF_WSTAGES * FF_WSTAGE_BYTES;
constexpr int FF_ALIGN_SLACK = 256;   // dynamic shared memory starts 1024-aligned when a kernel has no static
                                      // shared memory; up to this much misalignment is absorbed, more is a fault
constexpr int FF_SMEM = FF_BAR_OFFSET + 256 + FF_ALIGN_SLACK;   // + barriers and flags
static_assert(FF_SMEM <= SMEM_LIMIT, "fused forward shared memory");
constexpr int FF_LOADS_PER_TILE = 2 + 3 * 16 + 8;           // weight blocks streamed per tile
constexpr int kFfStoreThread = 64;                         // the epilogue thread that issues the output stores
static_assert(BM * GF_MLP_OUTPUTS * 4 <= 4 * FF_KB_BYTES, "staged outputs fit in H's K blocks 1-4");

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(FF_THREADS, 1)
fused_forward_kernel(const __grid_constant__ CUtensorMap tma_x, const __grid_constant__ CUtensorMap tma_w1,
                     const __grid_constant__ CUtensorMap tma_w2, const __grid_constant__ CUtensorMap tma_w3,
                     const __grid_constant__ CUtensorMap tma_w4, const __grid_constant__ CUtensorMap tma_w5,
                     const float* __restrict__ b1, const float* __restrict__ b2, const float* __restrict__ b3,
                     const float* __restrict__ b4, const float* __restrict__ b5, float* __restrict__ out,
                     int batch, int m_tiles, long long wait_limit, int inject, int* fault) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  if (smem - smem_raw > FF_ALIGN_SLACK) {   // the layout would not fit (the same in both CTAs)
    if (threadIdx.x == 0 && fault) atomicOr(fault, 1);
    return;
  }
  uint8_t* H = smem;
  uint8_t* W = smem + FF_H_BYTES;
  uint64_t* wfull = reinterpret_cast<uint64_t*>(smem + FF_BAR_OFFSET);
  uint64_t* wempty = wfull + FF_WSTAGES;
  uint64_t* xfull = wempty + FF_WSTAGES;   // the tile's inputs have landed in H's first K block
  uint64_t* accA = xfull + 1;              // N half 0 (region A) accumulated (MMA -> epilogue)
  uint64_t* accB = accA + 1;               // N half 1 (region B) accumulated: the layer's MMAs are done
  uint64_t* hlo = accB + 1;                // H's K blocks 0-3 written, region A drained (epilogue -> MMA)
  uint64_t* hmid = hlo + 1;                // H's K blocks 4-5 written (epilogue -> MMA)
  uint64_t* hhi = hmid + 1;                // H's K blocks 6-7 written, region B drained (epilogue -> MMA)
  uint64_t* hfree = hhi + 1;               // the tile's last MMAs have read H (MMA -> producer)
  uint64_t* staged = hfree + 1;            // the tile's output rows are staged (epilogue -> its storing thread)
  uint64_t* sread = staged + 1;            // ... and have been read by the store (storing thread -> epilogue)
  uint64_t* drain = sread + 1;             // MMA completion before tensor memory is released (abort)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  int* flags = reinterpret_cast<int*>(tmem_slot + 1);
  volatile int* abort_flag = flags;        // [0] a wait ran out; [2], [3] consumed
  int* consumed_s = flags + 2;             // weight blocks the MMA thread received (for the drain)
  int* x_consumed_s = flags + 3;           // input tiles the MMA thread received

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  // a pair's tiles are neighbours; past the last one the odd CTA works on rows that nobody reads
  const int tiles_up = m_tiles + (m_tiles & 1);
  auto wait = [&](uint64_t* bar, uint32_t parity) { return mbar_wait_warp(bar, parity, wait_limit, abort_flag); };

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tma_x);
    for (int s = 0; s < FF_WSTAGES; ++s) {
      mbar_init(&wfull[s], 2 - rank);   // in the even CTA also told of the other one's block
      mbar_init(&wempty[s], 1);
    }
    mbar_init(xfull, 2 - rank);
    mbar_init(accA, 1);
    mbar_init(accB, 1);
    mbar_init(hlo, 2 * FF_EPI_WARPS);   // in the even CTA, from both
    mbar_init(hmid, 2 * FF_EPI_WARPS);
    mbar_init(hhi, 2 * FF_EPI_WARPS);
    mbar_init(hfree, 1);
    mbar_init(staged, FF_EPI_WARPS);
    mbar_init(sread, 1);
    mbar_init(drain, 1);
    flags[0] = flags[1] = flags[2] = flags[3] = 0;
    mbar_fence_init();
  }
  __syncwarp();
  if (warp == 1) tmem_alloc_pair(tmem_slot, 512);
  tc_fence_before();
  cluster_sync();   // both CTAs' barriers are there
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  bool late = false;
  int issued = 0, x_issued = 0;

  // Warps 0 and 1 stay converged, with one elected lane to issue: as single-lane code the producer took 500 to
  // 1,000 cycles a box and the MMA issue 680 a K block, more than the tensor cores need.
  if (warp == 0) {
    // ---- producer: the tile's inputs, then its weights in the order the MMAs use them ----
    int s = 0, local = 0;
    uint32_t phase = 1;
    auto load = [&](const CUtensorMap& map, int n0, int kb, int bytes) -> bool {
      if (!wait(&wempty[s], phase)) return false;
      if (elect_one()) {
        mbar_arrive_expect_tx(&wfull[s], bytes);
        tma_load_2d(W + s * FF_WSTAGE_BYTES, &map, kb * BK, n0, &wfull[s]);
      }
      __syncwarp();
      ++issued;
      if (++s == FF_WSTAGES) {
        s = 0;
        phase ^= 1;
      }
      return true;
    };
    for (int tile = blockIdx.x; tile < tiles_up && !late; tile += gridDim.x, ++local) {
      if (local > 0 && !wait(hfree, (local - 1) & 1)) {   // the previous tile's MMAs are done with H
        late = true;
        break;
      }
      if (elect_one()) {
        mbar_arrive_expect_tx(xfull, FF_KB_BYTES);
        tma_load_2d(H, &tma_x, 0, tile * BM, xfull);
      }
      __syncwarp();
      ++x_issued;
      // this CTA's 128 (layer 5: 64) rows of each block
      const int row = static_cast<int>(rank) * BM;
      late = !load(tma_w1, row, 0, FF_KB_BYTES) || !load(tma_w1, 256 + row, 0, FF_KB_BYTES);
      for (int n0 = row; n0 < HID && !late; n0 += 256)
        for (int kb = 0; kb < 8 && !late; ++kb) late = !load(tma_w2, n0, kb, FF_WSTAGE_BYTES);
      for (int n0 = row; n0 < HID && !late; n0 += 256)
        for (int kb = 0; kb < 8 && !late; ++kb) late = !load(tma_w3, n0, kb, FF_WSTAGE_BYTES);
      for (int n0 = row; n0 < HID && !late; n0 += 256)
        for (int kb = 0; kb < 8 && !late; ++kb) late = !load(tma_w4, n0, kb, FF_WSTAGE_BYTES);
      for (int kb = 0; kb < 8 && !late; ++kb) late = !load(tma_w5, row / 2, kb, FF_WSTAGE_BYTES / 2);
    }
  } else if (warp == 1 && rank == 1) {
    // ---- the odd CTA tells the even one's MMA warp what has landed here ----
    int s = 0, got = 0, local = 0;
    uint32_t phase = 0;
    for (int tile = blockIdx.x; tile < tiles_up && !late; tile += gridDim.x, ++local) {
      if (!wait(xfull, local & 1)) {
        late = true;
        break;
      }
      if (lane == 0) {
        *x_consumed_s = local + 1;
        mbar_arrive_remote(xfull, 0);
      }
      __syncwarp();
      for (int i = 0; i < FF_LOADS_PER_TILE; ++i) {
        if (!wait(&wfull[s], phase)) {
          late = true;
          break;
        }
        ++got;
        if (lane == 0) mbar_arrive_remote(&wfull[s], 0);
        __syncwarp();
        if (++s == FF_WSTAGES) {
          s = 0;
          phase ^= 1;
        }
      }
    }
    if (lane == 0) *consumed_s = got;
    __syncwarp();
  } else if (warp == 1) {
    // ---- MMA issue (the even CTA) ----
    constexpr uint32_t idesc256 = bf16_idesc(2 * BM, 256);
    constexpr uint32_t idesc128 = bf16_idesc(2 * BM, OUT_PAD);
    int got = 0, local = 0, lo_waits = 0, hi_waits = 0, xs = 0;
    const uint64_t h_desc = sw128_kmajor_desc(smem_u32(H)), w_desc = sw128_kmajor_desc(smem_u32(W));
    int s = 0;
    uint32_t phase = 0;
    // the four MMAs of the next weight block (ring slot s): A = H's K block kb.  Descriptor addresses count 16 bytes.
    auto stage = [&](int kb, uint32_t d, uint32_t idesc) -> bool {
      if (!wait(&wfull[s], phase)) return false;
      tc_fence_after();
      const uint64_t a = h_desc + kb * (FF_KB_BYTES >> 4), w = w_desc + s * (FF_WSTAGE_BYTES >> 4);
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < BK / 16; ++kk) umma_bf16_pair(d, a + 2 * kk, w + 2 * kk, idesc, (kb | kk) != 0);
        umma_commit_pair(&wempty[s]);
      }
      __syncwarp();
      ++got;
      if (++s == FF_WSTAGES) {
        s = 0;
        phase ^= 1;
      }
      return true;
    };
    auto commit = [&](uint64_t* bar) {
      if (elect_one()) umma_commit_pair(bar);
      __syncwarp();
    };
    for (int tile = blockIdx.x; tile < tiles_up && !late; tile += gridDim.x, ++local) {
      if (!wait(xfull, local & 1)) {
        late = true;
        break;
      }
      ++xs;
      for (int layer = 0; layer < GF_MLP_LAYERS; ++layer) {
        // region A drained (by the previous layer's staging copy, or the previous tile's output) and,
        // from the second layer on, H's K blocks 0-3 written
        if (local > 0 || layer > 0) {
          if (!wait(hlo, lo_waits & 1)) {
            late = true;
            break;
          }
          ++lo_waits;
        }
        tc_fence_after();
        // N half 0 (the output layer's only N tile) into region A; K blocks 4-7 once H's K blocks 4-7
        // are written (which also means region B is drained)
        const int kblocks = layer == 0 ? 1 : 8;
        for (int kb = 0; kb < kblocks && !late; ++kb) {
          if (kb == 4 || kb == 6) {
            if (!wait(kb == 4 ? hmid : hhi, hi_waits & 1)) {
              late = true;
              break;
            }
            if (kb == 6) ++hi_waits;
            tc_fence_after();
          }
          late = !stage(kb, tmem, layer == 4 ? idesc128 : idesc256);
        }
        if (late) break;
        // fault injection for tests: withhold the first accumulator hand-off
        if (!((inject & 1) && local == 0 && layer == 0)) commit(accA);
        if (layer < 4) {
          // N half 1 into region B, while the epilogue drains region A
          for (int kb = 0; kb < kblocks && !late; ++kb) late = !stage(kb, tmem + 256, idesc256);
          if (late) break;
          commit(accB);   // also: every MMA of the layer has read H
        }
      }
      if (late) break;
      commit(hfree);
    }
    if (lane == 0) {
      *consumed_s = got;
      *x_consumed_s = xs;
    }
    __syncwarp();
  } else {
    // ---- epilogue: lane quarter qd of tensor memory, column group cg of each N half ----
    // A hidden layer's N half 0 (region A, tensor-memory columns 0-255) is drained while the MMAs of
    // N half 1 run: bias + GELU, rounded to bf16 pairs and stored back into the first half of the
    // warp's own region-A columns (H is still being read).  Once every MMA of the layer is done, the
    // staged half is copied into H's K blocks 0-3, which releases region A and lets the next layer's
    // MMAs start on K blocks 0-3 while N half 1 (region B) is drained straight into K blocks 4-7.
    const int qd = warp & 3;
    const int cg = (warp - 2) >> 2;
    const int r = qd * 32 + lane;                 // row within the tile
    float* s_out = reinterpret_cast<float*>(H + FF_KB_BYTES);   // the last layer's staged outputs
    const uint32_t tlane = tmem + (static_cast<uint32_t>(qd * 32) << 16);
    int a_waits = 0, b_waits = 0;
    const float* bias = b1;
    // every warp waits for the MMA hand-off itself: nothing in the epilogue waits for all of its warps
    auto handoff = [&](uint64_t* bar, int& n) -> bool {
      const bool ok = wait(bar, n & 1);
      ++n;
      __syncwarp();
      tc_fence_after();
      return ok;
    };
    // bias + GELU of the 32 accumulator columns at tensor-memory column tcol (output columns c0 ..
    // c0 + 31), rounded to 16 bf16 pairs
    auto gelu_pack = [&](uint32_t tcol, int c0, uint32_t (&w)[16]) {
      float v[32];
      tmem_ld_32cols(tlane + tcol, v);
      const float4* b4v = reinterpret_cast<const float4*>(bias + c0);
#pragma unroll
      for (int q4 = 0; q4 < 8; ++q4) {
        const float4 bb = __ldg(b4v + q4);
        v[4 * q4] = gelu(v[4 * q4] + bb.x);
        v[4 * q4 + 1] = gelu(v[4 * q4 + 1] + bb.y);
        v[4 * q4 + 2] = gelu(v[4 * q4 + 2] + bb.z);
        v[4 * q4 + 3] = gelu(v[4 * q4 + 3] + bb.w);
      }
#pragma unroll
      for (int t = 0; t < 16; ++t) {
        __nv_bfloat162 pr = __floats2bfloat162_rn(v[2 * t], v[2 * t + 1]);
        w[t] = *reinterpret_cast<uint32_t*>(&pr);
      }
    };
    // row r, output columns c0 .. c0+31 of H: K block c0 / 64, 16-byte units (c0 % 64) / 8 + q, placed
    // at unit ^ (r % 8) of the row (128-byte swizzle)
    auto store_h = [&](int c0, const uint32_t (&w)[16]) {
      uint8_t* rowp = H + (c0 >> 6) * FF_KB_BYTES + r * 128;
      const int u0 = (c0 & 63) >> 3;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        *reinterpret_cast<uint4*>(rowp + (((u0 + q) ^ (r & 7)) << 4)) =
            make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
    };
    int local = 0;
    for (int tile = blockIdx.x; tile < tiles_up; tile += gridDim.x, ++local) {
      bool stop = false;
      for (int layer = 0; layer < GF_MLP_LAYERS; ++layer) {
        bias = layer == 0 ? b1 : layer == 1 ? b2 : layer == 2 ? b3 : layer == 3 ? b4 : b5;   // 16-byte aligned, in L1
        if (!handoff(accA, a_waits)) {
          stop = true;
          break;
        }
        if (layer < 4) {
          // N half 0: output columns cg*64 .. cg*64+63, staged as bf16 pairs in tensor-memory columns
          // cg*64 .. cg*64+31 (each chunk's pairs land on columns this warp has already read)
#pragma unroll 1
          for (int h = 0; h < 2; ++h) {
            uint32_t w[16];
            gelu_pack(cg * 64 + 32 * h, cg * 64 + 32 * h, w);
            tmem_st_16cols(tlane + cg * 64 + 16 * h, w);
          }
          tmem_st_wait();
          // the previous tile's output store has read its staging rows before this tile writes H
          if (layer == 0 && local > 0) {
            if (threadIdx.x == kFfStoreThread) {
              bulk_wait_read<0>();
              mbar_arrive(sread);
            }
            __syncwarp();
            if (!wait(sread, (local - 1) & 1)) {
              stop = true;
              break;
            }
          }
          if (!handoff(accB, b_waits)) {   // every MMA of the layer is done with H
            stop = true;
            break;
          }
          {
            float v[32];
            tmem_ld_32cols(tlane + cg * 64, v);
            uint32_t w0[16], w1[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              w0[j] = __float_as_uint(v[j]);
              w1[j] = __float_as_uint(v[16 + j]);
            }
            store_h(cg * 64, w0);
            store_h(cg * 64 + 32, w1);
          }
          fence_proxy_async_smem();   // H is read by the tensor cores (async proxy)
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_remote(hlo, 0);   // H's K blocks 0-3 written, region A drained
          // N half 1 straight into H, K blocks 4-5 before 6-7, so that the MMAs can follow
#pragma unroll 1
          for (int h = 0; h < 2; ++h) {
            uint32_t w[16];
            const int c0 = 256 + 128 * h + 32 * cg;
            gelu_pack(c0, c0, w);
            store_h(c0, w);
            fence_proxy_async_smem();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(h == 0 ? hmid : hhi, 0);   // K blocks 4-5; 6-7, region B drained
          }
        } else {
          // layer 5: 128 padded outputs, one 32-column chunk per warp.  The first 99 of each row are
          // staged in H's K blocks 1-4 (row stride 99 words: the lanes' rows fall in distinct banks), and
          // the tile's rows, one contiguous span of the caller's [batch][99] array, leave in one bulk
          // store.  K block 0 may already be receiving the next tile's inputs; blocks 1-7 are next
          // written by the next tile's first epilogue, which waits until this store has read them.
          const int c0 = cg * 32;
          float v[32];
          tmem_ld_32cols(tlane + c0, v);
          float* o = s_out + r * GF_MLP_OUTPUTS;
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (c0 + j < GF_MLP_OUTPUTS) o[c0 + j] = v[j] + __ldg(bias + c0 + j);
          fence_proxy_async_smem();   // the staged rows are read by the bulk copy (async proxy)
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            mbar_arrive_remote(hlo, 0);   // region A drained: the next tile's first MMAs may write it
            mbar_arrive(staged);
          }
          if (threadIdx.x == kFfStoreThread) {
            if (!mbar_wait(staged, local & 1, wait_limit)) {
              *abort_flag = 1;
            } else if (tile < m_tiles) {
              // batch is a multiple of 128 (checked by the caller): the tile's rows are all in range
              bulk_store_1d(out + static_cast<long long>(tile) * BM * GF_MLP_OUTPUTS, s_out,
                            BM * GF_MLP_OUTPUTS * 4);
              bulk_commit();
            }
          }
          __syncwarp();
        }
      }
      if (stop) {
        late = true;
        break;
      }
    }
    if (threadIdx.x == kFfStoreThread) bulk_wait_all();   // the outputs are written before the CTA exits
  }

  tc_fence_before();
  if (late) *abort_flag = 1;
  __syncthreads();
  if (*abort_flag) {
    // a wait ran out: every load and MMA this CTA issued completes before its shared and tensor memory
    // are released (each wait again bounded)
    if (threadIdx.x == 0) {
      for (int it = *consumed_s; it < issued; ++it)
        mbar_wait(&wfull[it % FF_WSTAGES], (it / FF_WSTAGES) & 1, wait_limit);
      for (int x = *x_consumed_s; x < x_issued; ++x) mbar_wait(xfull, x & 1, wait_limit);
      if (fault) atomicOr(fault, 1);
    } else if (warp == 1 && rank == 0) {
      if (elect_one()) umma_commit_pair(drain);
      mbar_wait(drain, 0, wait_limit);
    }
    __syncthreads();
  }
  cluster_sync();   // the other CTA's MMAs, commits and arrivals are done with this one
  if (warp == 1) tmem_dealloc_pair(tmem, 512);
}

// ---------------------------------------------------------------------------------------------
// small kernels
// ---------------------------------------------------------------------------------------------

// Host queries: parameters [rows][6] doubles -> X0, the batch's rows past them zero, in the host encoding's
// arithmetic (double, rounded to fp32, then to bf16).
__global__ void query_encode_kernel(const double* __restrict__ params, int rows, int batch, const gf_mlp_scaling s,
                                    __nv_bfloat16* __restrict__ x0) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= batch) return;
  float v[8] = {};
  if (b < rows) {
#pragma unroll
    for (int j = 0; j < GF_MLP_INPUTS; ++j) {
      const double p = params[static_cast<long long>(b) * GF_MLP_INPUTS + j];
      const double lo = j == 1 ? s.asinh_low : s.low[j], hi = j == 1 ? s.asinh_high : s.high[j];
      const double at = j == 1 ? asinh(p / s.asinh_scale) : p;
      v[j] = static_cast<float>(2.0 * (at - lo) / (hi - lo) - 1.0);
    }
  }
  uint32_t w[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    __nv_bfloat162 p = __floats2bfloat162_rn(v[2 * t], v[2 * t + 1]);
    w[t] = *reinterpret_cast<uint32_t*>(&p);
  }
  *reinterpret_cast<uint4*>(x0 + static_cast<long long>(b) * IN_PAD) = make_uint4(w[0], w[1], w[2], w[3]);
}

// Outputs [rows][99] -> normalised spectra in double, a warp a row: the copy to the host, 792 bytes a row, is what
// a query waits for, and the exponentials (270 us on the host at 4,096 rows, 475 more for the sums and quotients)
// are a microsecond here.  The network's fault word goes to the host with them (host_fault, page-locked): outputs
// of a pass that gave up are not spectra.
__global__ void query_spectra_kernel(const float* __restrict__ y, int rows, const gf_mlp_scaling s,
                                     double* __restrict__ out, const int* __restrict__ fault, int* host_fault) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *host_fault = *fault;
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (row >= rows) return;   // warp-uniform
  double e[4];
  double sum = 0.0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int j = 32 * i + lane;
    e[i] = 0.0;
    if (j < GF_MLP_OUTPUTS)
      e[i] = exp(__dadd_rn(__dmul_rn(static_cast<double>(y[static_cast<long long>(row) * GF_MLP_OUTPUTS + j]), s.std[j]),
                           s.mean[j]));
    sum += e[i];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int j = 32 * i + lane;
    if (j < GF_MLP_OUTPUTS) out[static_cast<long long>(row) * GF_MLP_OUTPUTS + j] = e[i] / sum;
  }
}

// Inputs [batch][6] fp32 (row idx[i] for batch row i where idx is given) -> X0 [cap][64] bf16 (one 16-byte
// store of columns 0..7 per row; columns 8..63 stay zero) and, for training, X0^T [64][cap].
__global__ void encode_inputs_kernel(const float* __restrict__ x, const long long* __restrict__ idx, int batch,
                                     __nv_bfloat16* __restrict__ x0, __nv_bfloat16* __restrict__ x0t, long long cap,
                                     int transposed) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  grid_launch_next();
  grid_wait();   // the kernels before this one have read X0
  if (b >= batch) return;
  const long long from = idx ? idx[b] : b;
  float v[8];
#pragma unroll
  for (int j = 0; j < GF_MLP_INPUTS; ++j) v[j] = x[from * GF_MLP_INPUTS + j];
  v[6] = 0.f;
  v[7] = 0.f;
  uint32_t w[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    __nv_bfloat162 p = __floats2bfloat162_rn(v[2 * t], v[2 * t + 1]);
    w[t] = *reinterpret_cast<uint32_t*>(&p);
  }
  *reinterpret_cast<uint4*>(x0 + static_cast<long long>(b) * IN_PAD) = make_uint4(w[0], w[1], w[2], w[3]);
  if (transposed) {
#pragma unroll
    for (int j = 0; j < GF_MLP_INPUTS; ++j) x0t[j * cap + b] = __float2bfloat16_rn(v[j]);
  }
}

// ---------------------------------------------------------------------------------------------
// The end of a training step: the weight gradients of all layers, then Adam, in one launch
// ---------------------------------------------------------------------------------------------
// dW_l = dZ_l^T Y_{l-1} has few output tiles (108 of 128 x 64 over the five layers) and the batch as its
// reduction dimension.  A CTA owns one tile of one layer: the batch is cut into `splits` parts, each
// accumulated on its own in one of two tensor-memory accumulators and added up in registers in order (the
// sum, rounding included, of gradient slices reduced in a fixed order), and the tile's master weights,
// moments and bf16 copies are updated from the registers.  The gradient itself is only written where the
// caller asked for it.  Further blocks do the biases (partials summed in tile order) and the loss.
//
// At a batch of 1,024 the five GEMMs, their reduction over 27 MB of slices and Adam took 29 + 10 + 17 us in seven
// launches; here they take one of 13 us.
constexpr int DW_BN = 64;
constexpr int DW_EPI_WARPS = 8;
constexpr int DW_THREADS = 64 + 32 * DW_EPI_WARPS;
constexpr int DW_KS = 2;   // K blocks a stage, one TMA box each for A and B (batches are a multiple of 128 rows)
constexpr int DW_STAGES = 4;
constexpr int DW_A_BYTES = BM * BK * 2, DW_B_BYTES = DW_BN * BK * 2;
constexpr int DW_STAGE_BYTES = DW_KS * (DW_A_BYTES + DW_B_BYTES);
constexpr int DW_BAR_OFFSET = DW_STAGES * DW_STAGE_BYTES;
constexpr int DW_PIECE_ROW = 36;    // floats: rows 16 bytes apart modulo 128
constexpr int DW_TPIECE_ROW = 34;   // bf16
static_assert(DW_EPI_WARPS * 32 * (4 * DW_PIECE_ROW + 2 * DW_TPIECE_ROW) <= DW_BAR_OFFSET, "the pieces fit in the ring");
constexpr int DW_SMEM = DW_BAR_OFFSET + 256 + 1024;   // + barriers and flags, alignment

struct AdamArgs {
  float lr, beta1, beta2, eps, bc1, bc2, decay;
};

// Adam (with optional decoupled weight decay) of one master value.
__device__ __forceinline__ float adam_update(float w, float& m_io, float& v_io, float g, const AdamArgs& a) {
  // the products contracted as one kernel over all parameters had them, spelled out
  const float m = __fmaf_rn(1.f - a.beta1, g, __fmul_rn(a.beta1, m_io));
  const float v = __fmaf_rn(__fmul_rn(1.f - a.beta2, g), g, __fmul_rn(a.beta2, v_io));
  m_io = m;
  v_io = v;
  w -= a.lr * a.decay * w;
  w -= a.lr * (m / a.bc1) / (sqrtf(v / a.bc2) + a.eps);
  return w;
}

struct DwLayer {
  CUtensorMap a, b;        // dZ^T [out][batch], Y^T [in][batch]
  float *w, *m, *v, *g;    // [rows][cols]
  __nv_bfloat16 *wb, *wt;  // [rows][cols], [cols][rows]
  float *bias, *bm, *bv, *bg;
  const float* bias_part;  // [batch / 128][rows]
  int rows, cols, rows_true, cols_true;
  int splits;              // of the batch's K blocks
  int first;               // the layer's first tile in the grid
};

struct DwArgs {
  DwLayer layer[GF_MLP_LAYERS];
  AdamArgs adam;
  int tiles, k_blocks;     // tiles of all layers; 64-row K blocks of the batch
  int update;              // 1: Adam; 0: write the gradients
  int batch_tiles;
  const float* loss_part;
  float *loss, *loss_out;  // loss_out: the caller's, may be null
  int* fault;
  long long wait_limit;
};

__global__ void __launch_bounds__(DW_THREADS, 1) weight_update_kernel(const __grid_constant__ DwArgs A) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  if (static_cast<int>(blockIdx.x) >= A.tiles) {   // block-uniform: biases and loss
    grid_launch_next();
    grid_wait();
    int i = (static_cast<int>(blockIdx.x) - A.tiles) * DW_THREADS + threadIdx.x;
    if (i == 0) {
      float s = 0.f;
      for (int t = 0; t < A.batch_tiles; ++t) s += A.loss_part[t];
      *A.loss = s;
      if (A.loss_out) *A.loss_out = s;
    }
    int l = 0;
    while (l < GF_MLP_LAYERS && i >= A.layer[l].rows) i -= A.layer[l++].rows;
    if (l == GF_MLP_LAYERS || i >= A.layer[l].rows_true) return;
    const DwLayer& L = A.layer[l];
    float g = 0.f;
    for (int t = 0; t < A.batch_tiles; ++t) g += L.bias_part[t * L.rows + i];
    if (A.update) {
      float m = L.bm[i], v = L.bv[i];
      L.bias[i] = adam_update(L.bias[i], m, v, g, A.adam);
      L.bm[i] = m;
      L.bv[i] = v;
    } else {
      L.bg[i] = g;
    }
    return;
  }
  int l = 0;
  while (l + 1 < GF_MLP_LAYERS && static_cast<int>(blockIdx.x) >= A.layer[l + 1].first) ++l;
  const DwLayer& L = A.layer[l];
  const int n_tiles = L.cols / DW_BN;
  const int tile = static_cast<int>(blockIdx.x) - L.first;
  const int nt = tile % n_tiles, mt = tile / n_tiles;
  const int per_split = A.k_blocks / L.splits;

  uint64_t* full = reinterpret_cast<uint64_t*>(smem + DW_BAR_OFFSET);
  uint64_t* empty = full + DW_STAGES;
  uint64_t* tfull = empty + DW_STAGES;
  uint64_t* tempty = tfull + 2;
  uint64_t* drain = tempty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  int* timed_out = reinterpret_cast<int*>(tmem_slot + 1);
  int* epi_fail = timed_out + 1;
  int* consumed_s = timed_out + 2;
  volatile int* abort_flag = timed_out;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto wait = [&](uint64_t* bar, uint32_t parity) { return mbar_wait_warp(bar, parity, A.wait_limit, abort_flag); };
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&L.a);
    tma_prefetch_desc(&L.b);
    for (int s = 0; s < DW_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], DW_EPI_WARPS);
    }
    mbar_init(drain, 1);
    timed_out[0] = timed_out[1] = timed_out[2] = 0;
    mbar_fence_init();
  }
  __syncwarp();
  if (warp == 1) tmem_alloc(tmem_slot, 2 * DW_BN);
  grid_launch_next();
  grid_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  bool late = false;
  int issued = 0;

  if (warp == 0) {
    int s = 0;
    uint32_t phase = 1;
    for (; issued < A.k_blocks / DW_KS; ++issued) {
      if (!wait(&empty[s], phase)) {
        late = true;
        break;
      }
      uint8_t* a = smem + s * DW_STAGE_BYTES;
      if (elect_one()) {
        mbar_arrive_expect_tx(&full[s], DW_STAGE_BYTES);
        tma_load_3d(a, &L.a, 0, mt * BM, issued * DW_KS, &full[s]);
        tma_load_3d(a + DW_KS * DW_A_BYTES, &L.b, 0, nt * DW_BN, issued * DW_KS, &full[s]);
      }
      __syncwarp();
      if (++s == DW_STAGES) {
        s = 0;
        phase ^= 1;
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = bf16_idesc(BM, DW_BN);
    const uint64_t desc = sw128_kmajor_desc(smem_u32(smem));
    int s = 0, h = 0, received = 0;   // a split may end within a stage
    uint32_t phase = 0;
    for (int sp = 0; sp < L.splits && !late; ++sp) {
      const int acc = sp & 1;
      if (!wait(&tempty[acc], ((sp >> 1) & 1) ^ 1)) {
        late = true;
        break;
      }
      tc_fence_after();
      for (int kb = 0; kb < per_split; ++kb) {
        if (h == 0) {
          if (!wait(&full[s], phase)) {
            late = true;
            break;
          }
          ++received;
          tc_fence_after();
        }
        const uint64_t a = desc + s * (DW_STAGE_BYTES >> 4) + h * (DW_A_BYTES >> 4);
        const uint64_t b = desc + s * (DW_STAGE_BYTES >> 4) + (DW_KS * DW_A_BYTES >> 4) + h * (DW_B_BYTES >> 4);
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk)
            umma_bf16(tmem + acc * DW_BN, a + 2 * kk, b + 2 * kk, idesc, (kb | kk) != 0);
          if (h == DW_KS - 1) umma_commit(&empty[s]);
        }
        __syncwarp();
        if (++h == DW_KS) {
          h = 0;
          if (++s == DW_STAGES) {
            s = 0;
            phase ^= 1;
          }
        }
      }
      if (late) break;
      if (elect_one()) umma_commit(&tfull[acc]);
      __syncwarp();
    }
    if (lane == 0) *consumed_s = received;
    __syncwarp();
  } else {
    // epilogue warps: one 32 x 32 piece each (tensor-memory lane quarter, column half)
    const int qd = warp & 3, half = (warp - 2) >> 2;
    const int c0 = nt * DW_BN + 32 * half;
    const uint32_t tbase = tmem + (static_cast<uint32_t>(qd * 32) << 16) + static_cast<uint32_t>(32 * half);
    float g[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) g[j] = 0.f;
    for (int sp = 0; sp < L.splits; ++sp) {
      const int acc = sp & 1;
      if (lane == 0 && !mbar_wait(&tfull[acc], (sp >> 1) & 1, A.wait_limit)) atomicOr(epi_fail, 1);
      named_barrier_sync(4, 32 * DW_EPI_WARPS);
      if (*reinterpret_cast<volatile int*>(epi_fail)) {
        late = true;
        break;
      }
      __syncwarp();
      tc_fence_after();
      float v[32];
      tmem_ld_32cols(tbase + acc * DW_BN, v);
#pragma unroll
      for (int j = 0; j < 32; ++j) g[j] += v[j];
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[acc]);
    }
    if (!late) {
      // every MMA and load of the tile is done (the last hand-off), so the ring is free: the 32 x 32 piece goes
      // through it, to be updated in rows of eight float4 (four rows a warp instruction, each 128 contiguous
      // bytes of every array)
      float* const piece = reinterpret_cast<float*>(smem) + (warp - 2) * 32 * DW_PIECE_ROW;
      __nv_bfloat16* const tpiece = reinterpret_cast<__nv_bfloat16*>(smem + DW_EPI_WARPS * 32 * DW_PIECE_ROW * 4) +
                                    (warp - 2) * 32 * DW_TPIECE_ROW;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        *reinterpret_cast<float4*>(piece + lane * DW_PIECE_ROW + 4 * q) =
            make_float4(g[4 * q], g[4 * q + 1], g[4 * q + 2], g[4 * q + 3]);
      __syncwarp();
      const int row0 = mt * BM + qd * 32, c = 4 * (lane & 7);
      const int valid = L.cols_true - c0 - c;   // of this lane's four columns
      if (valid > 0) {
#pragma unroll 4
        for (int it = 0; it < 8; ++it) {
          const int r = 4 * it + (lane >> 3);
          if (row0 + r >= L.rows_true) continue;
          const long long at = static_cast<long long>(row0 + r) * L.cols + c0 + c;
          const float4 gv = *reinterpret_cast<const float4*>(piece + r * DW_PIECE_ROW + c);
          if (!A.update) {   // columns past cols_true: their gradient is an exact zero
            *reinterpret_cast<float4*>(L.g + at) = gv;
            continue;
          }
          // columns past cols_true stay zero: zero weight, moments and gradient
          float4 w = *reinterpret_cast<const float4*>(L.w + at);
          float4 m = *reinterpret_cast<const float4*>(L.m + at);
          float4 v = *reinterpret_cast<const float4*>(L.v + at);
          w.x = adam_update(w.x, m.x, v.x, gv.x, A.adam);
          w.y = adam_update(w.y, m.y, v.y, gv.y, A.adam);
          w.z = adam_update(w.z, m.z, v.z, gv.z, A.adam);
          w.w = adam_update(w.w, m.w, v.w, gv.w, A.adam);
          *reinterpret_cast<float4*>(L.w + at) = w;
          *reinterpret_cast<float4*>(L.m + at) = m;
          *reinterpret_cast<float4*>(L.v + at) = v;
          const __nv_bfloat16 b[4] = {__float2bfloat16_rn(w.x), __float2bfloat16_rn(w.y), __float2bfloat16_rn(w.z),
                                      __float2bfloat16_rn(w.w)};
          *reinterpret_cast<uint2*>(L.wb + at) =
              make_uint2(static_cast<uint32_t>(__bfloat16_as_ushort(b[0])) | static_cast<uint32_t>(__bfloat16_as_ushort(b[1])) << 16,
                         static_cast<uint32_t>(__bfloat16_as_ushort(b[2])) | static_cast<uint32_t>(__bfloat16_as_ushort(b[3])) << 16);
#pragma unroll
          for (int e = 0; e < 4; ++e) tpiece[(c + e) * DW_TPIECE_ROW + r] = b[e];
        }
      }
      __syncwarp();
      if (A.update) {   // the transposed copy: column c0 + j of the piece, a row a lane
        const int rows = min(32, L.rows_true - row0), cols = min(32, L.cols_true - c0);
        if (lane < rows) {
#pragma unroll 8
          for (int j = 0; j < cols; ++j)
            L.wt[static_cast<long long>(c0 + j) * L.rows + row0 + lane] = tpiece[j * DW_TPIECE_ROW + lane];
        }
      }
    }
  }

  tc_fence_before();
  if (late) *abort_flag = 1;
  __syncthreads();
  if (*abort_flag) {   // as in umma_gemm_kernel: what was issued lands before its memory is released
    if (threadIdx.x == 0) {
      for (int it = *consumed_s; it < issued; ++it) mbar_wait(&full[it % DW_STAGES], (it / DW_STAGES) & 1, A.wait_limit);
      if (A.fault) atomicOr(A.fault, 1);
    } else if (warp == 1) {
      if (elect_one()) umma_commit(drain);
      mbar_wait(drain, 0, A.wait_limit);
    }
    __syncthreads();
  }
  if (warp == 1) tmem_dealloc(tmem, 2 * DW_BN);
}

// One parameter tensor (padded shape rows x cols).
struct ParamSlot {
  float* w;
  __nv_bfloat16* wb;     // bf16 copy [rows][cols]
  __nv_bfloat16* wt;     // bf16 transposed copy [cols][rows]
  int rows, cols;
  long long offset;      // first element in the concatenated index space
};

struct ParamTable {
  ParamSlot s[GF_MLP_LAYERS];
  long long total;
};

__device__ __forceinline__ int find_slot(const ParamTable& t, long long i) {
  int k = 0;
#pragma unroll 1
  while (k + 1 < GF_MLP_LAYERS && t.s[k + 1].offset <= i) ++k;
  return k;
}

// bf16 copies of the master weights (after set_params).
__global__ void refresh_bf16_kernel(const __grid_constant__ ParamTable t) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < t.total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const ParamSlot& p = t.s[find_slot(t, i)];
    const long long e = i - p.offset;
    const int r = static_cast<int>(e / p.cols), c = static_cast<int>(e % p.cols);
    const __nv_bfloat16 b = __float2bfloat16_rn(p.w[e]);
    p.wb[e] = b;
    p.wt[static_cast<long long>(c) * p.rows + r] = b;
  }
}


// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

// Operand map: row-major bf16 [rows][cols] (cols contiguous), box box_rows x 64, 128-byte swizzle
// (the layout the UMMA matrix descriptors name).
bool make_map(CUtensorMap* m, const void* base, long long rows, long long cols, int box_rows) {
  auto fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(cols) * 2};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(BK), static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The same matrix as K blocks [cols / 64][rows][64], box `blocks` x box_rows x 64: a load lands as `blocks` tiles
// one after the other.
bool make_map_blocks(CUtensorMap* m, const void* base, long long rows, long long cols, int box_rows, int blocks) {
  auto fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[3] = {BK, static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(cols / BK)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(cols) * 2, BK * 2};
  cuuint32_t box[3] = {BK, static_cast<cuuint32_t>(box_rows), static_cast<cuuint32_t>(blocks)};
  cuuint32_t estr[3] = {1, 1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Output map of a row-major [rows][cols] matrix with 32 x 32 boxes, in the staging layout of the
// epilogue: fp32 with the 128-byte swizzle, bf16 with the 64-byte swizzle, or (transposed outputs) bf16
// unswizzled.
enum OutKind { OUT_F32 = 0, OUT_BF16 = 1, OUT_BF16_T = 2 };
bool make_out_map(CUtensorMap* m, const void* base, long long rows, long long cols, OutKind kind) {
  auto fn = encode_fn();
  if (!fn) return false;
  const int esize = kind == OUT_F32 ? 4 : 2;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(cols) * esize};
  cuuint32_t box[2] = {32, 32};
  cuuint32_t estr[2] = {1, 1};
  const CUtensorMapSwizzle sw = kind == OUT_F32    ? CU_TENSOR_MAP_SWIZZLE_128B
                                : kind == OUT_BF16 ? CU_TENSOR_MAP_SWIZZLE_64B
                                                   : CU_TENSOR_MAP_SWIZZLE_NONE;
  return fn(m, kind == OUT_F32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
            const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// SM count of the current device (cached per device)
int sm_count() {
  static std::atomic<int> counts[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 148;
  if (counts[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = 148;
    }
    counts[dev] = n;
  }
  return counts[dev];
}

// Launches with the dependent-launch attribute (grid_wait): the kernel may start once every block of the one
// before it on the stream has called grid_launch_next.
template <typename... P, typename... A>
cudaError_t launch_dependent(void (*kernel)(P...), int grid, int threads, int smem, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

// Sets a kernel's dynamic shared-memory limit, once per device.
template <typename Kernel>
cudaError_t allow_smem(Kernel kernel, int bytes, std::atomic<bool>* done) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && done[dev]) return cudaSuccess;
  const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (err == cudaSuccess && dev >= 0 && dev < 64) done[dev] = true;
  return err;
}

// Outputs the epilogue does not write get the A map in their slot (never used).  `step`: a kernel of a training
// step, launched dependently.
template <int BN, int EPI>
cudaError_t launch_gemm(const CUtensorMap& a, const CUtensorMap& b, const CUtensorMap* c, const CUtensorMap* y,
                        const CUtensorMap* yt, int M, int N, int K, const EpiArgs& ep, cudaStream_t stream,
                        int inject = 0, bool step = false) {
  static std::atomic<bool> attr_set[64] = {};
  const cudaError_t err = allow_smem(umma_gemm_kernel<BN, EPI>, Smem<BN, EPI>::BYTES, attr_set);
  if (err != cudaSuccess) return err;
  const int m_tiles = M / BM, n_tiles = N / BN;
  const int grid = std::min(m_tiles * n_tiles, sm_count());
  const long long limit = inject ? INJECT_WAIT_LIMIT : WAIT_LIMIT;
  if (step)
    return launch_dependent(umma_gemm_kernel<BN, EPI>, grid, gemm_threads(BN), Smem<BN, EPI>::BYTES, stream, a, b,
                            c ? *c : a, y ? *y : a, yt ? *yt : a, m_tiles, n_tiles, K / BK, ep, limit, inject);
  umma_gemm_kernel<BN, EPI><<<grid, gemm_threads(BN), Smem<BN, EPI>::BYTES, stream>>>(
      a, b, c ? *c : a, y ? *y : a, yt ? *yt : a, m_tiles, n_tiles, K / BK, ep, limit, inject);
  return cudaGetLastError();
}

// N tile of a training GEMM with 512 output columns: the widest that still gives every SM a tile, down to 32.
// At a batch of 1,024 (8 x 512 / N tiles) a forward layer takes 10 us with N = 128 and 32 CTAs, whose epilogues
// are most of it.
int train_tile(int batch) {
  const int m_tiles = batch / BM;
  if (m_tiles * (HID / 128) >= sm_count()) return 128;
  return m_tiles * (HID / 64) >= sm_count() ? 64 : 32;
}

template <int EPI>
cudaError_t launch_train_gemm(int bn, const CUtensorMap& a, const CUtensorMap& a128, const CUtensorMap* b, const CUtensorMap* c,
                              const CUtensorMap* y, const CUtensorMap* yt, int M, int K, const EpiArgs& ep,
                              cudaStream_t stream) {
  if (bn == 128) return launch_gemm<128, EPI>(a128, b[2], c, y, yt, M, HID, K, ep, stream, 0, true);
  if (bn == 64) return launch_gemm<64, EPI>(a, b[1], c, y, yt, M, HID, K, ep, stream, 0, true);
  return launch_gemm<32, EPI>(a, b[0], c, y, yt, M, HID, K, ep, stream, 0, true);
}

cudaError_t launch_fused_forward(const CUtensorMap& x, const CUtensorMap* w,
                                 float* const* bias, float* out, int batch, cudaStream_t stream, int inject,
                                 int* fault) {
  static std::atomic<bool> attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && !attr_set[dev]) {
    cudaError_t err = cudaFuncSetAttribute(fused_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FF_SMEM);
    if (err != cudaSuccess) return err;
    attr_set[dev] = true;
  }
  const int m_tiles = batch / BM;
  const int pairs = std::min((m_tiles + 1) / 2, sm_count() / 2);
  const int grid = 2 * pairs;
  fused_forward_kernel<<<grid, FF_THREADS, FF_SMEM, stream>>>(
      x, w[0], w[1], w[2], w[3], w[4], bias[0], bias[1], bias[2], bias[3], bias[4], out, batch, m_tiles,
      inject ? INJECT_WAIT_LIMIT : WAIT_LIMIT, inject, fault);
  return cudaGetLastError();
}

// Parts of the batch a layer's weight gradient is summed over (each a whole number of 64-row K blocks), from
// the count of its 128-wide output tiles: the order of the sum, and so its rounding, depends on it.
int choose_splits(int tiles, int K) {
  const int kblocks = K / BK;
  int s = 1;
  while (s < MAX_SPLITS && tiles * s < 148 && kblocks % (2 * s) == 0 && kblocks / (2 * s) >= 2) s *= 2;
  return s;
}

}  // namespace gfm

using namespace gfm;

struct gf_mlp {
  int device = 0;
  cudaStream_t stream = nullptr;
  gf_mlp_config cfg{};
  long long cap = 0;
  long long step = 0;
  std::string error;

  // layer geometry (padded): out x in
  int rows[GF_MLP_LAYERS] = {HID, HID, HID, HID, OUT_PAD};
  int cols[GF_MLP_LAYERS] = {IN_PAD, HID, HID, HID, HID};
  int rows_true[GF_MLP_LAYERS] = {HID, HID, HID, HID, GF_MLP_OUTPUTS};
  int cols_true[GF_MLP_LAYERS] = {GF_MLP_INPUTS, HID, HID, HID, HID};

  // parameters (fp32 master, Adam moments, gradient) -- one allocation each, weights then biases
  float* w[GF_MLP_LAYERS] = {};
  float* b[GF_MLP_LAYERS] = {};
  float* m_all = nullptr;
  float* v_all = nullptr;
  float* g_all = nullptr;
  float* w_all = nullptr;
  __nv_bfloat16* wb[GF_MLP_LAYERS] = {};
  __nv_bfloat16* wt[GF_MLP_LAYERS] = {};
  long long off_w[GF_MLP_LAYERS] = {}, off_b[GF_MLP_LAYERS] = {};
  long long n_params_padded = 0;

  // activations
  __nv_bfloat16 *x0 = nullptr, *x0t = nullptr;
  float* z[4] = {};
  __nv_bfloat16 *y[4] = {}, *yt[4] = {};
  __nv_bfloat16 *dout = nullptr, *doutt = nullptr;
  __nv_bfloat16 *dz[4] = {}, *dzt[4] = {};
  float* bpart[GF_MLP_LAYERS] = {};
  float* loss_part = nullptr;
  float* loss = nullptr;
  int* fault = nullptr;

  // host queries (gf_mlp_predict): rows at a time; device parameters, outputs and
  // spectra; the page-locked ring (one chunk's parameters and the fault word behind it), an event a chunk of it
  long long q_rows = 0;
  double *q_params = nullptr, *q_spec = nullptr;
  float* q_out = nullptr;
  double* q_ring = nullptr;
  cudaEvent_t q_done[4] = {};
  std::mutex querying;    // one host query at a time: held from its parameters to its spectra
  std::mutex enqueueing;  // a pass reads the inputs that were encoded just before it

  // tensor maps
  CUtensorMap fwd_a[GF_MLP_LAYERS], fwd_b[GF_MLP_LAYERS];     // A = input activations, B = W
  CUtensorMap fwd_b256[4];                                    // B = W in 256-row boxes (inference tiles)
  CUtensorMap fwd_pair[GF_MLP_LAYERS];                        // B = W in boxes of a paired CTA's half of the rows
  // training: A = input activations, B = W_l in 32-, 64- and 128-row boxes; A = dZ_l (dOut), B = W_l^T likewise
  // (l >= 2); two K blocks a box for tiles of 32 and 64 columns
  CUtensorMap train_a[4], train_b[4][3];
  CUtensorMap bwd_a[GF_MLP_LAYERS], bwd_a128[GF_MLP_LAYERS], bwd_b[GF_MLP_LAYERS][3];
  CUtensorMap dw_a[GF_MLP_LAYERS], dw_b[GF_MLP_LAYERS];       // A = dZ_l^T, B = Y_{l-1}^T
  CUtensorMap out_z[4], out_y[4], out_yt[4];                  // forward outputs of the hidden layers
  CUtensorMap out_dout, out_doutt;                            // dOut, dOut^T
  CUtensorMap out_dz[4], out_dzt[4];                          // backward outputs dZ, dZ^T

  std::vector<void*> allocations;
  int inject = 0;   // fault injection armed for the next forward pass (tests)
  int fused = 1;    // inference runs the fused five-layer kernel (0: one GEMM per layer)
};

namespace {

gf_status mlp_fail(gf_mlp* m, gf_status st, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  if (m) m->error = buf;
  return st;
}

#define MLP_CUDA(m, call)                                                                         \
  do {                                                                                            \
    cudaError_t _e = (call);                                                                      \
    if (_e != cudaSuccess) return mlp_fail((m), GF_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(_e)); \
  } while (0)

template <class T>
gf_status alloc(gf_mlp* m, T** p, long long count) {
  void* q = nullptr;
  if (cudaMalloc(&q, static_cast<size_t>(count) * sizeof(T)) != cudaSuccess) {
    cudaGetLastError();
    return mlp_fail(m, GF_ERR_OUT_OF_MEMORY, "device allocation of %lld bytes failed",
                    static_cast<long long>(count * sizeof(T)));
  }
  m->allocations.push_back(q);
  *p = static_cast<T*>(q);
  if (cudaMemsetAsync(q, 0, static_cast<size_t>(count) * sizeof(T), m->stream) != cudaSuccess)
    return mlp_fail(m, GF_ERR_CUDA, "memset failed");
  return GF_OK;
}

ParamTable param_table(gf_mlp* m) {
  ParamTable t{};
  for (int l = 0; l < GF_MLP_LAYERS; ++l) {
    t.s[l] = {m->w[l], m->wb[l], m->wt[l], m->rows[l], m->cols[l], t.total};
    t.total += static_cast<long long>(m->rows[l]) * m->cols[l];
  }
  return t;
}

gf_status check_batch(gf_mlp* m, int batch) {
  if (batch <= 0 || batch % BM != 0 || batch > m->cap)
    return mlp_fail(m, GF_ERR_INVALID_ARGUMENT, "batch %d must be a positive multiple of %d and at most %lld",
                    batch, BM, m->cap);
  return GF_OK;
}

// Inference: writes Y only, on 128 x 256 tiles (or keeps it on chip, fused), and the last layer writes the
// caller's [batch][99] array.
gf_status run_forward_encoded(gf_mlp* m, int batch, float* d_out) {
  if (m->fused) {
    cudaError_t err = launch_fused_forward(m->fwd_a[0], m->fwd_pair, m->b, d_out, batch, m->stream,
                                           m->inject, m->fault);
    m->inject = 0;
    if (err != cudaSuccess) return mlp_fail(m, GF_ERR_CUDA, "fused forward: %s", cudaGetErrorString(err));
    return GF_OK;
  }
  for (int l = 0; l < GF_MLP_LAYERS; ++l) {
    EpiArgs ep{};
    ep.bias = m->b[l];
    ep.fault = m->fault;
    cudaError_t err;
    if (l < 4) {
      err = launch_gemm<256, EPI_FWD_GELU_INFER>(m->fwd_a[l], m->fwd_b256[l], nullptr, &m->out_y[l], nullptr, batch, HID,
                                                 m->cols[l], ep, m->stream, l == 0 ? m->inject : 0);
      if (l == 0) m->inject = 0;
    } else {
      ep.out = d_out;
      ep.out_cols = GF_MLP_OUTPUTS;
      err = launch_gemm<128, EPI_FWD_OUT>(m->fwd_a[l], m->fwd_b[l], nullptr, nullptr, nullptr, batch, OUT_PAD, HID, ep,
                                          m->stream);
    }
    if (err != cudaSuccess) return mlp_fail(m, GF_ERR_CUDA, "forward GEMM %d: %s", l + 1, cudaGetErrorString(err));
  }
  return GF_OK;
}

gf_status run_forward(gf_mlp* m, const float* d_inputs, int batch, float* d_out) {
  std::lock_guard<std::mutex> lock(m->enqueueing);
  encode_inputs_kernel<<<(batch + 255) / 256, 256, 0, m->stream>>>(d_inputs, nullptr, batch, m->x0, m->x0t, m->cap, 0);
  MLP_CUDA(m, cudaGetLastError());
  return run_forward_encoded(m, batch, d_out);
}

// Buffers of gf_mlp_predict: at most kQueryRows rows are on the device at once, and their
// spectra come back in chunks through a page-locked ring of four, each copied to the caller while others are on
// their way.  The ring is short because page-locking 3 MB takes longer than several queries.
constexpr long long kQueryRows = 64 * BM;
constexpr int kQueryChunk = 256, kQueryRing = 4;
constexpr size_t kQueryChunkDoubles = static_cast<size_t>(kQueryChunk) * GF_MLP_OUTPUTS;

gf_status query_buffers(gf_mlp* m) {
  if (m->q_rows) return GF_OK;
  const long long rows = std::min(m->cap, kQueryRows);
  const size_t par = rows * GF_MLP_INPUTS * sizeof(double), spec = rows * GF_MLP_OUTPUTS * sizeof(double);
  if (!m->q_params) {
    void* d = nullptr;
    MLP_CUDA(m, cudaMalloc(&d, par + spec + rows * GF_MLP_OUTPUTS * sizeof(float)));
    m->allocations.push_back(d);
    m->q_params = static_cast<double*>(d);
    m->q_spec = m->q_params + rows * GF_MLP_INPUTS;
    m->q_out = reinterpret_cast<float*>(m->q_spec + rows * GF_MLP_OUTPUTS);
  }
  if (!m->q_ring)
    MLP_CUDA(m, cudaMallocHost(&m->q_ring, (kQueryRing * kQueryChunkDoubles + kQueryChunk * GF_MLP_INPUTS + 1) * sizeof(double)));
  static_assert(kQueryRing == sizeof(m->q_done) / sizeof(m->q_done[0]), "an event a chunk of the ring");
  for (cudaEvent_t& ev : m->q_done)
    if (!ev) MLP_CUDA(m, cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
  m->q_rows = rows;
  return GF_OK;
}

// The copy of chunk c of n rows' spectra into the ring.
cudaError_t issue_chunk(gf_mlp* m, int n, int c) {
  const size_t rows = std::min(kQueryChunk, n - c * kQueryChunk);
  const cudaError_t err =
      cudaMemcpyAsync(m->q_ring + (c % kQueryRing) * kQueryChunkDoubles, m->q_spec + c * kQueryChunkDoubles,
                      rows * GF_MLP_OUTPUTS * sizeof(double), cudaMemcpyDeviceToHost, m->stream);
  return err != cudaSuccess ? err : cudaEventRecord(m->q_done[c % kQueryRing], m->stream);
}

// Chunks c = first, first + step, ... to the caller, each once it has arrived, its place in the ring then taken by
// the chunk that follows it there (step divides the ring, so that one is this thread's too).
cudaError_t take_chunks(gf_mlp* m, int n, int first, int step, double* spectra) {
  for (int c = first; c * kQueryChunk < n; c += step) {
    cudaError_t err = cudaEventSynchronize(m->q_done[c % kQueryRing]);
    if (err != cudaSuccess) return err;
    const size_t rows = std::min(kQueryChunk, n - c * kQueryChunk);
    std::memcpy(spectra + c * kQueryChunkDoubles, m->q_ring + (c % kQueryRing) * kQueryChunkDoubles,
                rows * GF_MLP_OUTPUTS * sizeof(double));
    if ((c + kQueryRing) * kQueryChunk < n && (err = issue_chunk(m, n, c + kQueryRing)) != cudaSuccess) return err;
  }
  return cudaSuccess;
}

gf_status run_predict(gf_mlp* m, const double* params, long long rows, const gf_mlp_scaling& s, double* spectra) {
  gf_status st = query_buffers(m);
  if (st != GF_OK) return st;
  double* const h_params = m->q_ring + kQueryRing * kQueryChunkDoubles;
  int* const h_fault = reinterpret_cast<int*>(h_params + kQueryChunk * GF_MLP_INPUTS);
  for (long long r0 = 0; r0 < rows; r0 += m->q_rows) {
    const int n = static_cast<int>(std::min(m->q_rows, rows - r0)), batch = (n + BM - 1) / BM * BM;
    double* const to = spectra + r0 * GF_MLP_OUTPUTS;
    const size_t bytes = static_cast<size_t>(n) * GF_MLP_INPUTS * sizeof(double);
    // a single chunk's parameters and spectra cross the bus in the kernels themselves: two copies less to wait for
    const bool direct = n <= kQueryChunk;
    if (direct) std::memcpy(h_params, params + r0 * GF_MLP_INPUTS, bytes);
    else
      MLP_CUDA(m, cudaMemcpyAsync(m->q_params, params + r0 * GF_MLP_INPUTS, bytes, cudaMemcpyHostToDevice, m->stream));
    {
      std::lock_guard<std::mutex> lock(m->enqueueing);
      query_encode_kernel<<<(batch + 127) / 128, 128, 0, m->stream>>>(direct ? h_params : m->q_params, n, batch, s, m->x0);
      MLP_CUDA(m, cudaGetLastError());
      if ((st = run_forward_encoded(m, batch, m->q_out)) != GF_OK) return st;
    }
    query_spectra_kernel<<<(n + 7) / 8, 256, 0, m->stream>>>(m->q_out, n, s, direct ? m->q_ring : m->q_spec, m->fault,
                                                             h_fault);
    MLP_CUDA(m, cudaGetLastError());
    const int chunks = (n + kQueryChunk - 1) / kQueryChunk;
    if (direct) MLP_CUDA(m, cudaEventRecord(m->q_done[0], m->stream));
    else
      for (int c = 0; c < std::min(chunks, kQueryRing); ++c) MLP_CUDA(m, issue_chunk(m, n, c));
    // one thread copies 17 GB/s, a third of the bus: from eight chunks on two of them do, from sixteen four
    const int threads = chunks >= 16 ? 4 : chunks >= 8 ? 2 : 1;
    cudaError_t err[kQueryRing] = {};
    std::thread helper[kQueryRing];
    int started = 1;
    try {
      for (; started < threads; ++started)
        helper[started] = std::thread([=, &err] {
          err[started] = cudaSetDevice(m->device);
          if (err[started] == cudaSuccess) err[started] = take_chunks(m, n, started, threads, to);
        });
    } catch (const std::exception&) {   // no thread or no memory for it: this one takes the shares left over
    }
    err[0] = take_chunks(m, n, 0, threads, to);
    for (int t = started; t < threads && err[0] == cudaSuccess; ++t) err[0] = take_chunks(m, n, t, threads, to);
    for (int t = 1; t < started; ++t) helper[t].join();
    for (const cudaError_t e : err) MLP_CUDA(m, e);
    if (*h_fault) return gf_mlp_check(m);   // written by the kernel whose spectra have arrived
  }
  return GF_OK;
}

// Forward (Z, Y, Y^T of the hidden layers, dOut, dOut^T and the loss from the last), backward (dZ, dZ^T), then the
// weight gradients with Adam (adam) or into g_all (null): eleven launches, each starting under the tail of
// the one before (grid_wait).  idx: the batch's rows of d_inputs and d_targets (null: the first `batch`).
//
// Latency-bound at small batches: a chain of eleven kernels whose K loops are 1 to 8 blocks long.  At 1,024 a step
// takes 76 us; with single-lane producer and issue code 88, with one K block a TMA box as well 97, without the
// overlapped launches 107; in 23 separate launches it was 230 us of kernels.  At 128: 68 us, at 4,096: 120.
gf_status run_step(gf_mlp* m, const float* d_inputs, const float* d_targets, const long long* idx, int batch,
                   const AdamArgs* adam, float* d_loss) {
  std::lock_guard<std::mutex> lock(m->enqueueing);
  cudaError_t err = launch_dependent(encode_inputs_kernel, (batch + 255) / 256, 256, 0, m->stream, d_inputs, idx, batch,
                                     m->x0, m->x0t, m->cap, 1);
  if (err != cudaSuccess) return mlp_fail(m, GF_ERR_CUDA, "encoding the inputs: %s", cudaGetErrorString(err));
  const int bn = train_tile(batch);
  for (int l = 0; l < GF_MLP_LAYERS; ++l) {
    EpiArgs ep{};
    ep.bias = m->b[l];
    ep.fault = m->fault;
    if (l < 4) {
      err = launch_train_gemm<EPI_FWD_GELU>(bn, m->train_a[l], m->fwd_a[l], m->train_b[l], &m->out_z[l], &m->out_y[l],
                                            &m->out_yt[l], batch, m->cols[l], ep, m->stream);
    } else {
      ep.target = d_targets;
      ep.idx = idx;
      ep.batch = batch;
      ep.loss_part = m->loss_part;
      ep.bias_part = m->bpart[4];
      ep.ld_bias_part = OUT_PAD;
      err = launch_gemm<128, EPI_FWD_LOSS>(m->fwd_a[l], m->fwd_b[l], nullptr, &m->out_dout, &m->out_doutt, batch,
                                           OUT_PAD, HID, ep, m->stream, 0, true);
    }
    if (err != cudaSuccess) return mlp_fail(m, GF_ERR_CUDA, "forward GEMM %d: %s", l + 1, cudaGetErrorString(err));
  }
  for (int l = GF_MLP_LAYERS - 1; l > 0; --l) {
    // input gradient of layer l+1 = output gradient of layer l, times GELU'(Z_l)
    EpiArgs ep{};
    ep.z = m->z[l - 1];
    ep.ldz = HID;
    ep.bias_part = m->bpart[l - 1];
    ep.ld_bias_part = HID;
    ep.fault = m->fault;
    err = launch_train_gemm<EPI_BWD_GELU>(bn, m->bwd_a[l], m->bwd_a128[l], m->bwd_b[l], nullptr, &m->out_dz[l - 1],
                                          &m->out_dzt[l - 1], batch, m->rows[l], ep, m->stream);
    if (err != cudaSuccess)
      return mlp_fail(m, GF_ERR_CUDA, "input-gradient GEMM %d: %s", l + 1, cudaGetErrorString(err));
  }
  static std::atomic<bool> attr_set[64] = {};
  err = allow_smem(weight_update_kernel, DW_SMEM, attr_set);
  DwArgs A{};
  int biases = 0;
  for (int l = 0; l < GF_MLP_LAYERS; ++l) {
    DwLayer& L = A.layer[l];
    L.a = m->dw_a[l];
    L.b = m->dw_b[l];
    L.w = m->w[l];
    L.m = m->m_all + m->off_w[l];
    L.v = m->v_all + m->off_w[l];
    L.g = m->g_all + m->off_w[l];
    L.wb = m->wb[l];
    L.wt = m->wt[l];
    L.bias = m->b[l];
    L.bm = m->m_all + m->off_b[l];
    L.bv = m->v_all + m->off_b[l];
    L.bg = m->g_all + m->off_b[l];
    L.bias_part = m->bpart[l];
    L.rows = m->rows[l];
    L.cols = m->cols[l];
    L.rows_true = m->rows_true[l];
    L.cols_true = m->cols_true[l];
    L.splits = choose_splits((L.rows / BM) * (L.cols % 128 == 0 ? L.cols / 128 : L.cols / 64), batch);
    L.first = A.tiles;
    A.tiles += (L.rows / BM) * (L.cols / DW_BN);
    biases += L.rows;
  }
  if (adam) A.adam = *adam;
  A.update = adam ? 1 : 0;
  A.k_blocks = batch / BK;
  A.batch_tiles = batch / BM;
  A.loss_part = m->loss_part;
  A.loss = m->loss;
  A.loss_out = d_loss;
  A.fault = m->fault;
  A.wait_limit = WAIT_LIMIT;
  if (err == cudaSuccess)
    err = launch_dependent(weight_update_kernel, A.tiles + (biases + DW_THREADS - 1) / DW_THREADS, DW_THREADS, DW_SMEM,
                           m->stream, A);
  if (err != cudaSuccess) return mlp_fail(m, GF_ERR_CUDA, "weight gradients: %s", cudaGetErrorString(err));
  return GF_OK;
}

// Gradient step with the network's current learning rate.
gf_status run_train_step(gf_mlp* m, const float* d_inputs, const float* d_targets, const long long* idx, int batch,
                         float* d_loss) {
  const long long step = m->step + 1;
  const double bc1 = 1.0 - std::pow(static_cast<double>(m->cfg.beta1), static_cast<double>(step));
  const double bc2 = 1.0 - std::pow(static_cast<double>(m->cfg.beta2), static_cast<double>(step));
  const AdamArgs adam{m->cfg.lr, m->cfg.beta1, m->cfg.beta2, m->cfg.eps, static_cast<float>(bc1), static_cast<float>(bc2),
                      m->cfg.weight_decay};
  gf_status st = run_step(m, d_inputs, d_targets, idx, batch, &adam, d_loss);
  if (st == GF_OK) m->step = step;
  return st;
}

}  // namespace

extern "C" {

int64_t gf_mlp_param_count(void) {
  int64_t n = 0;
  const int r[GF_MLP_LAYERS] = {HID, HID, HID, HID, GF_MLP_OUTPUTS};
  const int c[GF_MLP_LAYERS] = {GF_MLP_INPUTS, HID, HID, HID, HID};
  for (int l = 0; l < GF_MLP_LAYERS; ++l) n += static_cast<int64_t>(r[l]) * c[l] + r[l];
  return n;
}

const char* gf_mlp_last_error(const gf_mlp* mlp) { return mlp ? mlp->error.c_str() : "null network"; }

gf_status gf_mlp_create(int32_t device, void* stream, const gf_mlp_config* config, gf_mlp** out) {
  if (!out || !config) return GF_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
    cudaGetLastError();
    return GF_ERR_NO_DEVICE;
  }
  if (config->batch_capacity <= 0 || config->batch_capacity % BM != 0) return GF_ERR_INVALID_ARGUMENT;
  if (!encode_fn()) return GF_ERR_CUDA;
  auto* m = new (std::nothrow) gf_mlp();
  if (!m) return GF_ERR_OUT_OF_MEMORY;
  m->device = device;
  m->cfg = *config;
  m->cap = config->batch_capacity;
  if (cudaSetDevice(device) != cudaSuccess) {
    delete m;
    return GF_ERR_CUDA;
  }
  m->stream = static_cast<cudaStream_t>(stream);
  gf_status st = GF_OK;
#define MLP_TRY(x)            \
  do {                        \
    st = (x);                 \
    if (st != GF_OK) goto bad; \
  } while (0)
  {
    long long off = 0;
    for (int l = 0; l < GF_MLP_LAYERS; ++l) {
      m->off_w[l] = off;
      off += static_cast<long long>(m->rows[l]) * m->cols[l];
    }
    for (int l = 0; l < GF_MLP_LAYERS; ++l) {
      m->off_b[l] = off;
      off += m->rows[l];
    }
    m->n_params_padded = off;
    MLP_TRY(alloc(m, &m->w_all, off));
    MLP_TRY(alloc(m, &m->m_all, off));
    MLP_TRY(alloc(m, &m->v_all, off));
    MLP_TRY(alloc(m, &m->g_all, off));
    for (int l = 0; l < GF_MLP_LAYERS; ++l) {
      m->w[l] = m->w_all + m->off_w[l];
      m->b[l] = m->w_all + m->off_b[l];
      const long long n = static_cast<long long>(m->rows[l]) * m->cols[l];
      MLP_TRY(alloc(m, &m->wb[l], n));
      MLP_TRY(alloc(m, &m->wt[l], n));
      MLP_TRY(alloc(m, &m->bpart[l], (m->cap / BM) * m->rows[l]));
    }
    const long long cap = m->cap;
    MLP_TRY(alloc(m, &m->x0, cap * IN_PAD));
    MLP_TRY(alloc(m, &m->x0t, cap * IN_PAD));
    for (int l = 0; l < 4; ++l) {
      MLP_TRY(alloc(m, &m->z[l], cap * HID));
      MLP_TRY(alloc(m, &m->y[l], cap * HID));
      MLP_TRY(alloc(m, &m->yt[l], cap * HID));
      MLP_TRY(alloc(m, &m->dz[l], cap * HID));
      MLP_TRY(alloc(m, &m->dzt[l], cap * HID));
    }
    MLP_TRY(alloc(m, &m->dout, cap * OUT_PAD));
    MLP_TRY(alloc(m, &m->doutt, cap * OUT_PAD));
    MLP_TRY(alloc(m, &m->loss_part, cap / BM));
    MLP_TRY(alloc(m, &m->loss, 1));
    MLP_TRY(alloc(m, &m->fault, 1));

    bool ok = true;
    for (int l = 0; l < GF_MLP_LAYERS; ++l) {
      const void* in = l == 0 ? static_cast<const void*>(m->x0) : m->y[l - 1];
      const void* in_t = l == 0 ? static_cast<const void*>(m->x0t) : m->yt[l - 1];
      const void* g = l == 4 ? static_cast<const void*>(m->dout) : m->dz[l];
      const void* g_t = l == 4 ? static_cast<const void*>(m->doutt) : m->dzt[l];
      ok = ok && make_map(&m->fwd_a[l], in, cap, m->cols[l], BM);
      ok = ok && make_map(&m->fwd_b[l], m->wb[l], m->rows[l], m->cols[l], 128);
      ok = ok && make_map(&m->fwd_pair[l], m->wb[l], m->rows[l], m->cols[l], l < 4 ? 128 : OUT_PAD / 2);
      if (l < 4) ok = ok && make_map(&m->fwd_b256[l], m->wb[l], m->rows[l], m->cols[l], 256);
      if (l < 4) {
        const int two = std::min(2, m->cols[l] / BK);
        ok = ok && make_map_blocks(&m->train_a[l], in, cap, m->cols[l], BM, two);
        for (int w = 0; w < 2; ++w)
          ok = ok && make_map_blocks(&m->train_b[l][w], m->wb[l], m->rows[l], m->cols[l], 32 << w, two);
        ok = ok && make_map(&m->train_b[l][2], m->wb[l], m->rows[l], m->cols[l], 128);
      }
      if (l > 0) {   // layer 1's input gradient is never formed
        ok = ok && make_map_blocks(&m->bwd_a[l], g, cap, m->rows[l], BM, 2);
        ok = ok && make_map(&m->bwd_a128[l], g, cap, m->rows[l], BM);
        for (int w = 0; w < 2; ++w)
          ok = ok && make_map_blocks(&m->bwd_b[l][w], m->wt[l], m->cols[l], m->rows[l], 32 << w, 2);
        ok = ok && make_map(&m->bwd_b[l][2], m->wt[l], m->cols[l], m->rows[l], 128);
      }
      ok = ok && make_map_blocks(&m->dw_a[l], g_t, m->rows[l], cap, BM, DW_KS);
      ok = ok && make_map_blocks(&m->dw_b[l], in_t, m->cols[l], cap, DW_BN, DW_KS);
    }
    for (int l = 0; l < 4; ++l) {
      ok = ok && make_out_map(&m->out_z[l], m->z[l], cap, HID, OUT_F32);
      ok = ok && make_out_map(&m->out_y[l], m->y[l], cap, HID, OUT_BF16);
      ok = ok && make_out_map(&m->out_yt[l], m->yt[l], HID, cap, OUT_BF16_T);
      ok = ok && make_out_map(&m->out_dz[l], m->dz[l], cap, HID, OUT_BF16);
      ok = ok && make_out_map(&m->out_dzt[l], m->dzt[l], HID, cap, OUT_BF16_T);
    }
    ok = ok && make_out_map(&m->out_dout, m->dout, cap, OUT_PAD, OUT_BF16);
    ok = ok && make_out_map(&m->out_doutt, m->doutt, OUT_PAD, cap, OUT_BF16_T);
    if (!ok) {
      st = mlp_fail(m, GF_ERR_CUDA, "tensor map encoding failed");
      goto bad;
    }
    if (cudaStreamSynchronize(m->stream) != cudaSuccess) {
      st = GF_ERR_CUDA;
      goto bad;
    }
  }
#undef MLP_TRY
  if (query_buffers(m) != GF_OK) {   // the first query tries again, and reports it
    cudaGetLastError();
    m->error.clear();
  }
  *out = m;
  return GF_OK;
bad:
  for (void* p : m->allocations) cudaFree(p);
  delete m;
  return st == GF_OK ? GF_ERR_CUDA : st;
}

gf_status gf_mlp_destroy(gf_mlp* mlp) {
  if (!mlp) return GF_OK;
  cudaSetDevice(mlp->device);
  cudaStreamSynchronize(mlp->stream);
  for (void* p : mlp->allocations) cudaFree(p);
  if (mlp->q_ring) cudaFreeHost(mlp->q_ring);
  for (cudaEvent_t ev : mlp->q_done)
    if (ev) cudaEventDestroy(ev);
  delete mlp;
  return GF_OK;
}

gf_status gf_mlp_set_params(gf_mlp* m, const float* params, int64_t count) {
  if (!m || !params) return GF_ERR_INVALID_ARGUMENT;
  if (count != gf_mlp_param_count())
    return mlp_fail(m, GF_ERR_INVALID_ARGUMENT, "expected %lld parameters, got %lld",
                    static_cast<long long>(gf_mlp_param_count()), static_cast<long long>(count));
  MLP_CUDA(m, cudaSetDevice(m->device));
  std::vector<float> h;
  try {
    h.assign(m->n_params_padded, 0.f);
  } catch (const std::bad_alloc&) {
    return mlp_fail(m, GF_ERR_OUT_OF_MEMORY, "host allocation failed");
  }
  const float* p = params;
  for (int l = 0; l < GF_MLP_LAYERS; ++l) {
    for (int r = 0; r < m->rows_true[l]; ++r)
      for (int c = 0; c < m->cols_true[l]; ++c) h[m->off_w[l] + static_cast<long long>(r) * m->cols[l] + c] = *p++;
    for (int r = 0; r < m->rows_true[l]; ++r) h[m->off_b[l] + r] = *p++;
  }
  MLP_CUDA(m, cudaMemcpyAsync(m->w_all, h.data(), h.size() * sizeof(float), cudaMemcpyHostToDevice, m->stream));
  MLP_CUDA(m, cudaMemsetAsync(m->m_all, 0, h.size() * sizeof(float), m->stream));
  MLP_CUDA(m, cudaMemsetAsync(m->v_all, 0, h.size() * sizeof(float), m->stream));
  ParamTable t = param_table(m);
  refresh_bf16_kernel<<<2 * 148, 256, 0, m->stream>>>(t);
  MLP_CUDA(m, cudaGetLastError());
  MLP_CUDA(m, cudaStreamSynchronize(m->stream));
  m->step = 0;
  return GF_OK;
}

static gf_status unpad_to_host(gf_mlp* m, const float* d_all, float* out) {
  std::vector<float> h;
  try {
    h.resize(m->n_params_padded);
  } catch (const std::bad_alloc&) {
    return mlp_fail(m, GF_ERR_OUT_OF_MEMORY, "host allocation failed");
  }
  MLP_CUDA(m, cudaMemcpyAsync(h.data(), d_all, h.size() * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
  MLP_CUDA(m, cudaStreamSynchronize(m->stream));
  float* p = out;
  for (int l = 0; l < GF_MLP_LAYERS; ++l) {
    for (int r = 0; r < m->rows_true[l]; ++r)
      for (int c = 0; c < m->cols_true[l]; ++c) *p++ = h[m->off_w[l] + static_cast<long long>(r) * m->cols[l] + c];
    for (int r = 0; r < m->rows_true[l]; ++r) *p++ = h[m->off_b[l] + r];
  }
  return GF_OK;
}

gf_status gf_mlp_get_params(gf_mlp* m, float* params, int64_t count) {
  if (!m || !params) return GF_ERR_INVALID_ARGUMENT;
  if (count != gf_mlp_param_count()) return mlp_fail(m, GF_ERR_INVALID_ARGUMENT, "parameter count mismatch");
  MLP_CUDA(m, cudaSetDevice(m->device));
  return unpad_to_host(m, m->w_all, params);
}

gf_status gf_mlp_set_learning_rate(gf_mlp* m, float lr) {
  if (!m || !(lr >= 0.f)) return GF_ERR_INVALID_ARGUMENT;
  m->cfg.lr = lr;
  return GF_OK;
}

gf_status gf_mlp_forward(gf_mlp* m, const float* d_inputs, int32_t batch, float* d_outputs) {
  if (!m || !d_inputs || !d_outputs) return GF_ERR_INVALID_ARGUMENT;
  gf_status st = check_batch(m, batch);
  if (st != GF_OK) return st;
  MLP_CUDA(m, cudaSetDevice(m->device));
  if (reinterpret_cast<uintptr_t>(d_outputs) & 15)
    return mlp_fail(m, GF_ERR_INVALID_ARGUMENT, "d_outputs must be 16-byte aligned");
  return run_forward(m, d_inputs, batch, d_outputs);
}

gf_status gf_mlp_predict(gf_mlp* m, const double* params, int64_t rows, const gf_mlp_scaling* scaling,
                         double* spectra) {
  if (!m || rows < 0 || !scaling || (rows > 0 && (!params || !spectra))) return GF_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(m->querying);
  MLP_CUDA(m, cudaSetDevice(m->device));
  return run_predict(m, params, rows, *scaling, spectra);
}

gf_status gf_rows_inside(const double* params, int64_t rows, int32_t columns, const double* low, const double* high,
                         uint8_t* inside) {
  if (rows < 0 || columns < 0 || (rows > 0 && (!params || !low || !high || !inside))) return GF_ERR_INVALID_ARGUMENT;
  for (int64_t i = 0; i < rows; ++i) {
    bool in = true;
    for (int32_t j = 0; j < columns; ++j) in &= params[i * columns + j] >= low[j] && params[i * columns + j] <= high[j];
    inside[i] = in ? 1 : 0;
  }
  return GF_OK;
}

gf_status gf_mlp_gradients(gf_mlp* m, const float* d_inputs, const float* d_targets, int32_t batch, float* grads,
                           float* loss) {
  if (!m || !d_inputs || !d_targets) return GF_ERR_INVALID_ARGUMENT;
  gf_status st = check_batch(m, batch);
  if (st != GF_OK) return st;
  MLP_CUDA(m, cudaSetDevice(m->device));
  if ((st = run_step(m, d_inputs, d_targets, nullptr, batch, nullptr, nullptr)) != GF_OK) return st;
  if (loss) {
    MLP_CUDA(m, cudaMemcpyAsync(loss, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream));
  }
  if (grads) {
    if ((st = unpad_to_host(m, m->g_all, grads)) != GF_OK) return st;
  }
  MLP_CUDA(m, cudaStreamSynchronize(m->stream));
  return gf_mlp_check(m);
}

gf_status gf_mlp_train_step(gf_mlp* m, const float* d_inputs, const float* d_targets, int32_t batch,
                            float* d_loss) {
  if (!m || !d_inputs || !d_targets) return GF_ERR_INVALID_ARGUMENT;
  gf_status st = check_batch(m, batch);
  if (st != GF_OK) return st;
  MLP_CUDA(m, cudaSetDevice(m->device));
  return run_train_step(m, d_inputs, d_targets, nullptr, batch, d_loss);
}

gf_status gf_mlp_train_step_rows(gf_mlp* m, const float* d_inputs, const float* d_targets, const int64_t* d_rows,
                                 int32_t batch, float* d_loss) {
  if (!m || !d_inputs || !d_targets || !d_rows) return GF_ERR_INVALID_ARGUMENT;
  gf_status st = check_batch(m, batch);
  if (st != GF_OK) return st;
  MLP_CUDA(m, cudaSetDevice(m->device));
  static_assert(sizeof(long long) == sizeof(int64_t), "row indices");
  return run_train_step(m, d_inputs, d_targets, reinterpret_cast<const long long*>(d_rows), batch, d_loss);
}

gf_status gf_mlp_check(gf_mlp* m) {
  if (!m) return GF_ERR_INVALID_ARGUMENT;
  MLP_CUDA(m, cudaSetDevice(m->device));
  int f = 0;
  MLP_CUDA(m, cudaMemcpyAsync(&f, m->fault, sizeof(int), cudaMemcpyDeviceToHost, m->stream));
  MLP_CUDA(m, cudaStreamSynchronize(m->stream));
  if (f) {
    MLP_CUDA(m, cudaMemsetAsync(m->fault, 0, sizeof(int), m->stream));
    MLP_CUDA(m, cudaStreamSynchronize(m->stream));
    return mlp_fail(m, GF_ERR_DEVICE, "a tensor-core GEMM wait ran out of time");
  }
  return GF_OK;
}

gf_status gf_mlp_set_fused_inference(gf_mlp* m, int32_t enable) {
  if (!m || enable < 0 || enable > 1) return GF_ERR_INVALID_ARGUMENT;
  m->fused = enable;
  return GF_OK;
}

gf_status gf_mlp_inject_fault(gf_mlp* m, int32_t kind) {
  if (!m || kind < 0 || kind > 1) return GF_ERR_INVALID_ARGUMENT;
  m->inject = kind;
  return GF_OK;
}

gf_status gf_bf16_gemm(const void* d_a, const void* d_b, int32_t M, int32_t N, int32_t K, float* d_c,
                       void* stream) {
  if (!d_a || !d_b || !d_c || M <= 0 || N <= 0 || K <= 0 || M % BM || N % 64 || K % BK)
    return GF_ERR_INVALID_ARGUMENT;
  if ((reinterpret_cast<uintptr_t>(d_a) | reinterpret_cast<uintptr_t>(d_b) | reinterpret_cast<uintptr_t>(d_c)) & 15)
    return GF_ERR_INVALID_ARGUMENT;
  const int bn = N % 128 == 0 ? 128 : 64;
  CUtensorMap a, b, c;
  if (!make_map(&a, d_a, M, K, BM) || !make_map(&b, d_b, N, K, bn) || !make_out_map(&c, d_c, M, N, OUT_F32))
    return GF_ERR_CUDA;
  EpiArgs ep{};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t err = bn == 128 ? launch_gemm<128, EPI_STORE_F32>(a, b, &c, nullptr, nullptr, M, N, K, ep, s)
                              : launch_gemm<64, EPI_STORE_F32>(a, b, &c, nullptr, nullptr, M, N, K, ep, s);
  return err == cudaSuccess ? GF_OK : GF_ERR_CUDA;
}

}  // extern "C"
