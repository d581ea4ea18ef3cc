// surrogate.cu — training and inference kernels of the thermal model
// (surrogate.h) on the tcgen05 tensor cores, and the frame generators of the
// FE-coupled path that use it or the synthetic field it learns.
//
// Kernels:
//   mlp_step_kernel       training: forward, loss and backward through the
//                         activations of a 128-row tile, persistent; bf16
//                         operands in shared memory, FP32 accumulators in TMEM.
//   mlp_wgrad_kernel      training: weight gradients over pieces of the batch,
//                         operands MN-major straight from the row-major
//                         activations.
//   mlp_chain_kernel      training: bias and head gradients, column sums.
//   mlp_update_kernel     training: the pieces' sum and Adam.
//   mlp_infer_kernel      the whole network per 128-query tile, persistent:
//                         Fourier features written into shared memory, four
//                         MMA layers with their weights streamed by TMA while
//                         the previous epilogue runs, the head in FP32.
//   plus data generation and the frame
//   generators (multi-track field, model frames with fallback).
// Every wait (mbarrier) is bounded; a wait that runs out sets *error and the
// block returns after releasing its TMEM.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <chrono>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/amca3d.h"
#include "surrogate.h"
#include "thermal_field.cuh"
#include "umma.cuh"

namespace amca {
namespace sur {

using bf16 = __nv_bfloat16;
constexpr unsigned long long kWaitNs = 1000000000ull;  // 1 s: every mbarrier wait
constexpr int kErrWait = 1;

// 1 / (1 + e^-z), with e^-z = 2^(-z log2 e), by the approximate 2^x and 1/x
// instructions in their flushing form: a 2^x below 2^-126 leaves 1 + 2^x at 1
// either way. The instructions are specified to a relative error of 2^-22 and to
// 1 ulp; the rounded constant and product add |z| 2^-23 to that of e^-z, of which
// the result takes the part e^-z / (1 + e^-z). z below -80 counts as -80, so
// that every value stays finite: the result is then 1.8e-35, where the true one
// is between that and 0.
__device__ __forceinline__ float sigmoid(float z) {
  float e, s;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(-1.4426950408889634f * fmaxf(z, -80.0f)));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(1.0f + e));
  return s;
}
__device__ __forceinline__ float silu(float z) { return z * sigmoid(z); }
__device__ __forceinline__ float silu_grad(float z) {
  const float s = sigmoid(z);
  return s * (1.0f + z * (1.0f - s));
}

// Normalised inputs u = (raw - shift) * scale of one raw input.
__device__ __forceinline__ void normalise(const SurModelDev &m, const float raw[kSurIn], float u[kSurIn]) {
#pragma unroll
  for (int i = 0; i < kSurIn; ++i) u[i] = (raw[i] - m.in_shift[i]) * m.in_scale[i];
}

// Fourier matrix in shared memory, a row in 8 floats (two aligned loads).
constexpr int kFourierPad = 8;
__device__ __forceinline__ void load_fourier(const SurModelDev &m, float (*B)[kFourierPad]) {
  for (int i = threadIdx.x; i < kSurFreq * kSurIn; i += blockDim.x) B[i / kSurIn][i % kSurIn] = m.fourier[i];
}

// Phase of one input: sv = sin(2 pi f), cv = cos(2 pi f), f = sum_i B[i] u_i
// (FP32, i ascending).
__device__ __forceinline__ void phases(const float B[kFourierPad], const float u[kSurIn], float &sv, float &cv) {
  const float4 b = *(const float4 *)B;
  const float row[kSurIn] = {b.x, b.y, b.z, b.w, B[4]};
  float f = 0.0f;
#pragma unroll
  for (int i = 0; i < kSurIn; ++i) f = __fadd_rn(f, __fmul_rn(row[i], u[i]));
  sincospif(2.0f * f, &sv, &cv);
}

__device__ __forceinline__ uint8_t *align1024(uint8_t *p) {
  return (uint8_t *)(((uintptr_t)p + 1023) & ~(uintptr_t)1023);
}

// ---------------------------------------------------------------------------
// Training. A step is four kernels:
//   mlp_step_kernel    forward, loss and the pre-activation gradients dZ of a
//                      128-row tile, layer by layer in shared memory;
//   mlp_wgrad_kernel   weight gradients dZ_l^T X_l over pieces of the batch;
//   mlp_chain_kernel   bias and head gradients, column sums over the batch;
//   mlp_update_kernel  the sums over the pieces, and Adam.
// Only what the gradients contract over the whole batch goes through memory:
// the layer inputs X_l, the head's input and dZ_l, row-major bf16, 4.4 KB a
// row. The weight gradients read them as MN-major operands, so no transposed
// copy of an activation or a weight exists. Before (a GEMM per layer and
// direction, each epilogue storing a row-major and a transposed copy, the
// transposed one 2 bytes at a time, one-block-per-column bias and head sums):
// 505 us for a step of 32,768 rows; now 168 us (alone and from a cold cache:
// 88, 32, 31 and 22 us; the chains run beside the weight gradients, a step's
// set-up beside the update before it). Every sum keeps its order: the trained
// parameters are the same bits.
// ---------------------------------------------------------------------------
constexpr int kTrainThreads = 512, kTrainGroups = 4, kTrainCols = kSurHid / kTrainGroups;
constexpr uint32_t kTrainSmem = 64u * 1024u + 128u * 1024u + 1024u;

// Tensor maps of a training step: bf16 weights [out][in] (box 64 x 256), the
// batch's layer inputs (X[0]: features) and dZ, each [rows][columns].
struct TrainMaps {
  CUtensorMap W[kSurLayers], X_out[kSurLayers + 1], dZ_out[kSurLayers];  // boxes of 128 rows (X[4]: the head's input)
  CUtensorMap X_in[kSurLayers], dZ_in[kSurLayers];  // boxes of kWgradRows rows
};

struct StepArgs {
  int64_t n;                  // rows, a multiple of 128
  const float *raw, *target;  // samples: raw inputs (5 each) and normalised temperature
  uint64_t nsamples, start, perm;  // row q is sample (start + q) * perm mod nsamples
  uint4 *zs;                  // bf16 pre-activations of layers 0..2, in the order of the threads that use them
  float *pred, *loss;         // [n x 2] mu, s; [n]
  float2 *dpred;              // [n] dL/dmu, dL/ds
  float inv_batch, lambda_s;
  int *error;
};

__device__ __forceinline__ uint64_t sample_of(const StepArgs &a, uint64_t q) {
  const uint64_t i = a.start + q;
  if (__umul64hi(i, a.perm) == 0) return (i * a.perm) % a.nsamples;
  return (uint64_t)(((unsigned __int128)i * a.perm) % a.nsamples);
}

// Forward and backward of 128-row tiles, persistent, one block per SM. Shared
// memory: the tile's current activations or dZ (128 x 256 bf16) and one layer's
// weights (256 x 256 bf16, streamed by TMA while the previous epilogue runs;
// the backward pass reads the same [out][in] tiles as MN-major B operands). 512
// threads: warp w reads TMEM lanes 32 (w % 4) (its rows) and the 64-column group
// w / 4. Bound by instruction issue in the features and epilogues (39% of the
// slots) and by the MMAs between them (about 1.1 us a layer), which nothing
// overlaps: 105 us for 32,768 rows with __expf and __fdividef and the Fourier
// matrix in global memory, 88 with the two MUFU operations of sigmoid() and the
// matrix in shared memory.
__global__ void __launch_bounds__(kTrainThreads, 1)
    mlp_step_kernel(const __grid_constant__ TrainMaps tm, SurModelDev md, StepArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *H = align1024(smem_raw);
  uint8_t *Wsm = H + 64 * 1024;
  __shared__ __align__(8) uint64_t wbar, mbar;
  __shared__ uint32_t tmem_base;
  __shared__ int s_abort;
  __shared__ __align__(16) float s_bias[kSurLayers][kSurHid];
  __shared__ __align__(16) float s_wh[kSurOut][kSurHid];
  __shared__ float s_bh[kSurOut];
  __shared__ float s_head[kTrainGroups][128][2];
  __shared__ float s_in[128][kSurIn], s_y[128], s_dp[128][2];  // s_in: normalised inputs
  __shared__ __align__(16) float s_fourier[kSurFreq][kFourierPad];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q4 = warp & 3, grp = warp >> 2, row = q4 * 32 + lane;
  const int64_t ntiles = a.n / 128;
  const SurParamLayout L;

  if (threadIdx.x == 0) {
    umma::mbar_init(umma::smem_u32(&wbar), 1);
    umma::mbar_init(umma::smem_u32(&mbar), 1);
    umma::mbar_fence_init();
    s_abort = 0;
  }
  if (warp == 0) umma::tmem_alloc(umma::smem_u32(&tmem_base), 256);
  load_fourier(md, s_fourier);
  // the parameters may still be in the making (the previous step's update)
  umma::wait_prerequisites();
  for (int i = threadIdx.x; i < kSurLayers * kSurHid; i += blockDim.x)
    s_bias[i / kSurHid][i % kSurHid] = md.p[L.b[i / kSurHid] + i % kSurHid];
  for (int i = threadIdx.x; i < kSurOut * kSurHid; i += blockDim.x) s_wh[i / kSurHid][i % kSurHid] = md.p[L.Wh + i];
  if (threadIdx.x < kSurOut) s_bh[threadIdx.x] = md.p[L.bh + threadIdx.x];
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  const uint32_t tmem = tmem_base;
  const uint32_t trow = tmem + ((uint32_t)(q4 * 32) << 16);
  constexpr uint32_t id_fwd = umma::idesc_bf16_f32(128, kSurHid);
  constexpr uint32_t id_bwd = umma::idesc_bf16_f32(128, kSurHid, false, true);

  bool w_pending = false;  // thread 0: a weight load is in flight, and the phase it completes
  uint32_t wph = 0;
  auto load_w = [&](int l) {
    const int kbs = SurParamLayout::in_dim(l) / 64;
    const uint32_t bar = umma::smem_u32(&wbar);
    umma::mbar_expect_tx(bar, (uint32_t)kbs * 32u * 1024u);
    for (int kb = 0; kb < kbs; ++kb) umma::tma_load_2d(umma::smem_u32(Wsm + kb * 32 * 1024), &tm.W[l], bar, kb * 64, 0);
    w_pending = true;
  };
  auto weights_in = [&]() {
    if (!umma::mbar_wait(umma::smem_u32(&wbar), wph, kWaitNs)) return false;
    w_pending = false;
    wph ^= 1u;
    return true;
  };
  auto store_tile = [&](const CUtensorMap &t, int kbs, int64_t tile) {
    for (int kb = 0; kb < kbs; ++kb) umma::tma_store_2d(&t, umma::smem_u32(H + kb * 16 * 1024), kb * 64, (int)(tile * 128));
    umma::bulk_commit();
  };
  if (threadIdx.x == 0) load_w(0);
  uint32_t mph = 0;
  bool ok = true;
  // every MMA issued by thread 0 has completed (bounded), in all threads
  auto mma_done = [&]() {
    const bool mok = umma::mbar_wait(umma::smem_u32(&mbar), mph, kWaitNs);
    mph ^= 1u;
    ok = __syncthreads_and(mok ? 1 : 0) != 0 && !s_abort;
    umma::tc_fence_after();
    return ok;
  };
  // what was written to shared memory is visible to the tensor cores and TMA
  auto publish = [&]() {
    umma::fence_async_smem();
    umma::tc_fence_before();
    __syncthreads();
  };

  for (int64_t tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
    if (grp == 0) {
      const uint64_t i = sample_of(a, (uint64_t)(tile * 128 + row));
      float raw[kSurIn], u[kSurIn];
#pragma unroll
      for (int k = 0; k < kSurIn; ++k) raw[k] = a.raw[i * kSurIn + k];
      normalise(md, raw, u);
#pragma unroll
      for (int k = 0; k < kSurIn; ++k) s_in[row][k] = u[k];
      s_y[row] = a.target[i];
    }
    if (threadIdx.x == 0) umma::bulk_wait_read();  // the previous tile's last store has left H
    __syncthreads();
    {
      float u[kSurIn];
#pragma unroll
      for (int k = 0; k < kSurIn; ++k) u[k] = s_in[row][k];
      for (int j0 = grp * (kSurFreq / kTrainGroups); j0 < (grp + 1) * (kSurFreq / kTrainGroups); j0 += 8) {
        __align__(16) bf16 sb[8], cb[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          float sv, cv;
          phases(s_fourier[j0 + t], u, sv, cv);
          sb[t] = __float2bfloat16_rn(sv);
          cb[t] = __float2bfloat16_rn(cv);
        }
        *(uint4 *)(H + umma::sw128_offset(row, j0, 128)) = *(const uint4 *)sb;
        *(uint4 *)(H + umma::sw128_offset(row, kSurFreq + j0, 128)) = *(const uint4 *)cb;
      }
    }
    publish();
    if (threadIdx.x == 0) store_tile(tm.X_out[0], kSurEnc / 64, tile);
    uint4 *zt = a.zs + tile * (3 * (kTrainCols / 8) * kTrainThreads) + threadIdx.x;

    // --- forward ---
    for (int l = 0; l < kSurLayers; ++l) {
      if (threadIdx.x == 0) {
        if (!weights_in()) {
          s_abort = 1;
        } else {
          umma::tc_fence_after();
          const int kbs = SurParamLayout::in_dim(l) / 64;
          for (int kb = 0; kb < kbs; ++kb) {
            const uint32_t ha = umma::smem_u32(H + kb * 16 * 1024), wa = umma::smem_u32(Wsm + kb * 32 * 1024);
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma::mma_bf16(tmem, umma::sdesc_sw128(ha + 32u * k), umma::sdesc_sw128(wa + 32u * k), id_fwd,
                             (kb | k) != 0 ? 1u : 0u);
          }
        }
        umma::mma_commit(umma::smem_u32(&mbar));
        umma::bulk_wait_read();  // H may be rewritten once its store has read it
      }
      if (!mma_done()) break;
      // the weights are free again (the last layer's stay for the backward pass)
      if (threadIdx.x == 0 && l < kSurLayers - 1) load_w(l + 1);
      if (l < kSurLayers - 1) {
        for (int c0 = grp * kTrainCols; c0 < (grp + 1) * kTrainCols; c0 += 32) {
          float v[32];
          umma::tmem_ld32(trow + c0, v);
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            __align__(16) bf16 zb[8], hb[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) {
              const float z = v[j + t] + s_bias[l][c0 + j + t];
              zb[t] = __float2bfloat16_rn(z);
              hb[t] = __float2bfloat16_rn(silu(z));
            }
            zt[(l * (kTrainCols / 8) + (c0 % kTrainCols + j) / 8) * kTrainThreads] = *(const uint4 *)zb;
            *(uint4 *)(H + umma::sw128_offset(row, c0 + j, 128)) = *(const uint4 *)hb;
          }
        }
        publish();
        if (threadIdx.x == 0) store_tile(tm.X_out[l + 1], kSurHid / 64, tile);
      }
    }
    if (!ok) break;

    // --- head: mu and s are summed column by column in each half (groups 0, 1
    // and 2, 3), the second group of a half going on where the first ended ---
    float mu = 0.0f, s = 0.0f;
    for (int pass = 0; pass < 2; ++pass) {
      if ((grp & 1) == pass) {
        if (pass) {
          mu = s_head[grp - 1][row][0];
          s = s_head[grp - 1][row][1];
        }
        for (int c0 = grp * kTrainCols; c0 < (grp + 1) * kTrainCols; c0 += 32) {
          float v[32];
          umma::tmem_ld32(trow + c0, v);
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            __align__(16) bf16 hb[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) {
              const float h = silu(v[j + t] + s_bias[kSurLayers - 1][c0 + j + t]);
              hb[t] = __float2bfloat16_rn(h);
              mu = fmaf(h, s_wh[0][c0 + j + t], mu);
              s = fmaf(h, s_wh[1][c0 + j + t], s);
            }
            *(uint4 *)(H + umma::sw128_offset(row, c0 + j, 128)) = *(const uint4 *)hb;
          }
        }
        s_head[grp][row][0] = mu;
        s_head[grp][row][1] = s;
      }
      publish();
    }
    if (threadIdx.x == 0) {  // the head's input, for its gradients; read before dZ replaces it
      store_tile(tm.X_out[kSurLayers], kSurHid / 64, tile);
      umma::bulk_wait_read();
    }
    if (grp == 1) {
      mu = s_head[1][row][0] + s_head[3][row][0] + s_bh[0];
      s = s_head[1][row][1] + s_head[3][row][1] + s_bh[1];
      s = fminf(fmaxf(s, -12.0f), 4.0f);
      const float r = mu - s_y[row];
      const float e2 = __expf(-2.0f * s);
      // mean squared error on mu; the error head learns log |mu - y| (Gaussian
      // negative log-likelihood with mu held fixed), weighted by lambda_s
      const float dmu = r * a.inv_batch;
      const float ds = a.lambda_s * (1.0f - e2 * r * r) * a.inv_batch;
      const int64_t m = tile * 128 + row;
      *(float2 *)(a.pred + 2 * m) = make_float2(mu, s);
      a.loss[m] = 0.5f * r * r;
      s_dp[row][0] = dmu;
      s_dp[row][1] = ds;
      a.dpred[m] = make_float2(dmu, ds);
    }
    __syncthreads();
    {  // dZ of the last layer
      const float dmu = s_dp[row][0], ds = s_dp[row][1];
      for (int c0 = grp * kTrainCols; c0 < (grp + 1) * kTrainCols; c0 += 32) {
        float v[32];
        umma::tmem_ld32(trow + c0, v);
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
          __align__(16) bf16 gb[8];
#pragma unroll
          for (int t = 0; t < 8; ++t) {
            const float dh = dmu * s_wh[0][c0 + j + t] + ds * s_wh[1][c0 + j + t];
            gb[t] = __float2bfloat16_rn(dh * silu_grad(v[j + t] + s_bias[kSurLayers - 1][c0 + j + t]));
          }
          *(uint4 *)(H + umma::sw128_offset(row, c0 + j, 128)) = *(const uint4 *)gb;
        }
      }
    }
    publish();
    if (threadIdx.x == 0) store_tile(tm.dZ_out[kSurLayers - 1], kSurHid / 64, tile);

    // --- backward: dZ_{l-1} = (dZ_l W_l) SiLU'(z_{l-1}) ---
    for (int l = kSurLayers - 1; l > 0; --l) {
      if (threadIdx.x == 0) {
        if (l < kSurLayers - 1 && !weights_in()) {
          s_abort = 1;
        } else {
          umma::tc_fence_after();
          for (int k = 0; k < 16; ++k)
            umma::mma_bf16(tmem, umma::sdesc_sw128(umma::smem_u32(H + (k >> 2) * 16 * 1024) + 32u * (k & 3)),
                           umma::sdesc_sw128_mn(umma::smem_u32(Wsm) + 2048u * k, 32 * 1024), id_bwd, k != 0 ? 1u : 0u);
        }
        umma::mma_commit(umma::smem_u32(&mbar));
        umma::bulk_wait_read();
      }
      uint4 zq[kTrainCols / 8];  // in flight while the MMAs run
#pragma unroll
      for (int c = 0; c < kTrainCols / 8; ++c) zq[c] = zt[((l - 1) * (kTrainCols / 8) + c) * kTrainThreads];
      if (!mma_done()) break;
      if (threadIdx.x == 0) {
        if (l > 1) load_w(l - 1);
        else if (tile + gridDim.x < ntiles) load_w(0);
      }
#pragma unroll
      for (int h = 0; h < kTrainCols / 32; ++h) {
        const int c0 = grp * kTrainCols + 32 * h;
        float v[32];
        umma::tmem_ld32(trow + c0, v);
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
          const bf16 *zb = (const bf16 *)&zq[4 * h + j / 8];
          __align__(16) bf16 gb[8];
#pragma unroll
          for (int t = 0; t < 8; ++t)
            gb[t] = __float2bfloat16_rn(v[j + t] * silu_grad(__bfloat162float(zb[t])));
          *(uint4 *)(H + umma::sw128_offset(row, c0 + j, 128)) = *(const uint4 *)gb;
        }
      }
      publish();
      if (threadIdx.x == 0) store_tile(tm.dZ_out[l - 1], kSurHid / 64, tile);
    }
  }
  if (threadIdx.x == 0) {
    if (!ok) {
      atomicCAS(a.error, 0, kErrWait);
      if (w_pending) umma::mbar_wait(umma::smem_u32(&wbar), wph, kWaitNs);  // let a load in flight land
    }
    umma::bulk_wait();
  }
  umma::tc_fence_before();
  __syncthreads();
  if (warp == 0) umma::tmem_free(tmem, 256);
}

// Weight gradients of one piece of the batch: block (item, piece) computes rows
// 128 h .. +127 and `width` columns of dZ_l^T X_l over the piece's rows, both
// operands MN-major tiles of 32 rows loaded by TMA (4-stage ring). Two blocks
// per SM (96 KB and 256 TMEM columns each), so that one's stores run under the
// other's MMAs.
// The piece's sums go to memory as float4s in the order of the threads, which
// the update kernel reads back coalesced. The pieces are the longest equal
// ones that divide the batch into at most 64 of at least 512 rows (an odd
// number of rows / 128 divides into few or none); where that leaves SMs idle
// the columns are split too.
constexpr int kWgradThreads = 256, kWgradStages = 4, kWgradRows = 32;
constexpr uint32_t kWgradBox = kWgradRows * 128u;  // 64 columns of a stage's rows
constexpr uint32_t kWgradStage = (2u + 4u) * kWgradBox;
constexpr uint32_t kWgradSmem = kWgradStages * kWgradStage + 1024u;
// floats of a piece: the weights of row half h of layer l from wgrad_offset(2 l + h)
constexpr int64_t kPiece = (int64_t)kSurHid * (kSurEnc + 3 * kSurHid);
__host__ __device__ constexpr int64_t wgrad_offset(int lh) {
  return lh < 2 ? (int64_t)lh * 128 * kSurEnc : (int64_t)kSurHid * kSurEnc + (int64_t)(lh - 2) * 128 * kSurHid;
}
__host__ __device__ constexpr int wgrad_items(int width) {
  return 2 * (width < kSurEnc ? kSurEnc / width : 1) + 6 * (kSurHid / width);
}

__global__ void __launch_bounds__(kWgradThreads, 2)
    mlp_wgrad_kernel(const __grid_constant__ TrainMaps tm, int width, int per, float *partial, int *error) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = align1024(smem_raw);
  __shared__ __align__(8) uint64_t full[kWgradStages], empty[kWgradStages], done;
  __shared__ uint32_t tmem_base;
  __shared__ int s_abort;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // item: (layer, column slice, row half), the first layer's first
  const int n0 = 2 * (width < kSurEnc ? kSurEnc / width : 1), per_layer = 2 * (kSurHid / width);
  const int x = blockIdx.x, l = x < n0 ? 0 : 1 + (x - n0) / per_layer;
  const int in_layer = l == 0 ? x : (x - n0) % per_layer, h = in_layer & 1;
  const int N = min(width, SurParamLayout::in_dim(l)), col0 = (in_layer >> 1) * N;
  const int kb0 = blockIdx.y * per, nk = per;  // blocks of kWgradRows rows
  if (threadIdx.x == 0) {
    for (int s = 0; s < kWgradStages; ++s) {
      umma::mbar_init(umma::smem_u32(&full[s]), 1);
      umma::mbar_init(umma::smem_u32(&empty[s]), 1);
    }
    umma::mbar_init(umma::smem_u32(&done), 1);
    umma::mbar_fence_init();
    s_abort = 0;
  }
  if (warp == 0) umma::tmem_alloc(umma::smem_u32(&tmem_base), 256);
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  const uint32_t tmem = tmem_base;

  if (threadIdx.x == 0) {
    const uint32_t idesc = umma::idesc_bf16_f32(128, N, true, true);
    const uint32_t bytes = (2u + (uint32_t)(N / 64)) * kWgradBox;
    auto load = [&](int s, int kb) {
      const uint32_t sa = umma::smem_u32(smem + s * kWgradStage), bar = umma::smem_u32(&full[s]);
      const int r = (kb0 + kb) * kWgradRows;
      umma::mbar_expect_tx(bar, bytes);
      for (int c = 0; c < 2; ++c) umma::tma_load_2d(sa + c * kWgradBox, &tm.dZ_in[l], bar, h * 128 + c * 64, r);
      for (int c = 0; c < N / 64; ++c) umma::tma_load_2d(sa + (2 + c) * kWgradBox, &tm.X_in[l], bar, col0 + c * 64, r);
    };
    int loaded = 0;
    for (; loaded < kWgradStages && loaded < nk; ++loaded) load(loaded, loaded);
    bool ok = true;
    for (int kb = 0; kb < nk; ++kb) {
      const int s = kb % kWgradStages;
      if (!umma::mbar_wait(umma::smem_u32(&full[s]), (uint32_t)((kb / kWgradStages) & 1), kWaitNs)) {
        ok = false;
        break;
      }
      umma::tc_fence_after();
      const uint32_t sa = umma::smem_u32(smem + s * kWgradStage), sb = sa + 2u * kWgradBox;
#pragma unroll
      for (int k = 0; k < kWgradRows / 16; ++k)
        umma::mma_bf16(tmem, umma::sdesc_sw128_mn(sa + 2048u * k, kWgradBox),
                       umma::sdesc_sw128_mn(sb + 2048u * k, kWgradBox), idesc, (kb | k) != 0 ? 1u : 0u);
      umma::mma_commit(umma::smem_u32(&empty[s]));
      // refill the stage of the previous block (its MMAs were issued one iteration earlier)
      if (kb >= 1 && loaded < nk) {
        const int sp = (kb - 1) % kWgradStages;
        if (!umma::mbar_wait(umma::smem_u32(&empty[sp]), (uint32_t)(((kb - 1) / kWgradStages) & 1), kWaitNs)) {
          ok = false;
          break;
        }
        load(sp, loaded++);
      }
    }
    if (!ok) {
      s_abort = 1;
      atomicCAS(error, 0, kErrWait);
      // let every load still in flight land before the block exits
      for (int kb = 0; kb < loaded; ++kb)
        umma::mbar_wait(umma::smem_u32(&full[kb % kWgradStages]), (uint32_t)((kb / kWgradStages) & 1), kWaitNs);
    }
    umma::mma_commit(umma::smem_u32(&done));
  }
  const bool done_ok = umma::mbar_wait(umma::smem_u32(&done), 0, kWaitNs);
  const bool all_ok = __syncthreads_and(done_ok ? 1 : 0) != 0;
  if (!done_ok) atomicCAS(error, 0, kErrWait);
  umma::tc_fence_after();
  if (all_ok && !s_abort) {
    const int q = warp & 3, half = warp >> 2, row = q * 32 + lane;
    const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16);
    float4 *w = (float4 *)(partial + (int64_t)blockIdx.y * kPiece + wgrad_offset(2 * l + h));
    for (int c0 = half * (N / 2); c0 < (half + 1) * (N / 2); c0 += 32) {
      float v[32];
      umma::tmem_ld32(trow + c0, v);
#pragma unroll
      for (int j = 0; j < 32; j += 4)
        w[((col0 + c0 + j) / 4) * 128 + row] = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
    }
  }
  umma::tc_fence_before();
  __syncthreads();
  if (warp == 0) umma::tmem_free(tmem, 256);
  umma::wait_prerequisites();  // the update kernel, next in the stream, needs the chains too
}

// Column sums of the batch in 256 interleaved chains: chain t of column c adds
// rows t, t + 256, t + 512, ... in order. Sets 0..3 are the bias gradients
// (the rows of dZ_l), 4 and 5 the head's (rows of its input times dL/dmu and
// dL/ds), and the head's own biases (dL/dmu, dL/ds themselves) go to chainb.
// The update kernel adds the chains pairwise, t and t + 128 first. A thread has
// four columns, a warp 256 bytes of a row; 64 blocks a matrix read the batch
// once, most of it from L2 (one block per column over a transposed copy
// before).
constexpr int kChains = 256, kChainSets = kSurLayers + kSurOut, kChainThreads = 256, kChainCols = 4;
struct ChainArgs {
  const bf16 *dZ[kSurLayers], *H;
  const float2 *dpred;
  int64_t n;
  float *chain;   // [kChainSets][kChains][kSurHid]
  float *chainb;  // [kChains][kSurOut]
};

constexpr int kChainBatch = 16;  // rows whose loads are in flight before any is added

__global__ void __launch_bounds__(kChainThreads) mlp_chain_kernel(ChainArgs a) {
  umma::launch_dependents();  // the weight gradients need nothing of this kernel
  constexpr int per_row = kSurHid / kChainCols;  // threads on one row
  const int t = blockIdx.x * (kChainThreads / per_row) + threadIdx.x / per_row;
  const int c = threadIdx.x % per_row * kChainCols;
  const int set = blockIdx.y;
  const bool head = set == kSurLayers;
  const bf16 *src = (head ? a.H : set == 0 ? a.dZ[0] : set == 1 ? a.dZ[1] : set == 2 ? a.dZ[2] : a.dZ[3]) + c;
  float s0[kChainCols] = {}, s1[kChainCols] = {}, b0 = 0.0f, b1 = 0.0f;
  for (int64_t m0 = t; m0 < a.n; m0 += kChains * kChainBatch) {
    uint2 u[kChainBatch];
    float2 d[kChainBatch];
#pragma unroll
    for (int k = 0; k < kChainBatch; ++k) {
      const int64_t m = m0 + k * kChains;
      u[k] = m < a.n ? *(const uint2 *)(src + m * kSurHid) : make_uint2(0u, 0u);
    }
    if (head) {
#pragma unroll
      for (int k = 0; k < kChainBatch; ++k) {
        const int64_t m = m0 + k * kChains;
        d[k] = m < a.n ? a.dpred[m] : make_float2(0.0f, 0.0f);
      }
    }
#pragma unroll
    for (int k = 0; k < kChainBatch; ++k) {
      if (m0 + k * kChains >= a.n) break;
      const __nv_bfloat162 *b = (const __nv_bfloat162 *)&u[k];
      const float h[kChainCols] = {__low2float(b[0]), __high2float(b[0]), __low2float(b[1]), __high2float(b[1])};
      if (!head) {
#pragma unroll
        for (int i = 0; i < kChainCols; ++i) s0[i] += h[i];
      } else {
#pragma unroll
        for (int i = 0; i < kChainCols; ++i) {
          s0[i] += d[k].x * h[i];
          s1[i] += d[k].y * h[i];
        }
        b0 += d[k].x;
        b1 += d[k].y;
      }
    }
  }
  float *out = a.chain + ((int64_t)set * kChains + t) * kSurHid + c;
  *(float4 *)out = make_float4(s0[0], s0[1], s0[2], s0[3]);
  if (head) {
    *(float4 *)(out + kChains * kSurHid) = make_float4(s1[0], s1[1], s1[2], s1[3]);
    if (c == 0) *(float2 *)(a.chainb + kSurOut * t) = make_float2(b0, b1);
  }
}

// Gradients summed over the pieces in order, or from the chains. ADAM: then the
// parameter's Adam step and its bf16 copy; otherwise the gradient is stored.
// The first kWeightBlocks blocks have two weights per thread, the
// others 32 columns of a chain set (the last one the head's biases). Bound by
// reading the pieces (59 MB at 64 of them).
struct AdamArgs {
  float *p, *m, *v, *g;
  float lr, beta1, beta2, eps, bc1, bc2;
  bf16 *Wb[kSurLayers];
};

template <bool ADAM>
__device__ __forceinline__ float update_param(const AdamArgs &a, int64_t i, float g) {
  if (!ADAM) {
    a.g[i] = g;
    return 0.0f;
  }
  const float m = a.beta1 * a.m[i] + (1.0f - a.beta1) * g;
  const float v = a.beta2 * a.v[i] + (1.0f - a.beta2) * g * g;
  a.m[i] = m;
  a.v[i] = v;
  const float p = a.p[i] - a.lr * (m / a.bc1) / (sqrtf(v / a.bc2) + a.eps);
  a.p[i] = p;
  return p;
}

constexpr int kUpdateThreads = 256;
constexpr int kWeightBlocks = (int)(kPiece / 2 / kUpdateThreads);
constexpr int kUpdateBlocks = kWeightBlocks + kChainSets * kSurHid / 32 + 1;
static_assert(kPiece % (2 * kUpdateThreads) == 0, "whole blocks of weights");

// x[t] + x[t + 128], then + 64, ... + 8: the pairwise sum of the 32 chains
// t = w, w + 8, w + 16, ... (i-th value: t = w + 8 i)
template <int N>
__device__ __forceinline__ float pair_sum(const float *x) {
  if constexpr (N == 32) return x[0];
  else return pair_sum<2 * N>(x) + pair_sum<2 * N>(x + N);
}

template <bool ADAM>
__global__ void __launch_bounds__(kUpdateThreads)
    mlp_update_kernel(AdamArgs a, const float *partial, int pieces, const float *chain, const float *chainb) {
  umma::launch_dependents();  // the next step's blocks set up meanwhile
  const SurParamLayout L;
  if (blockIdx.x < kWeightBlocks) {
    const int i = blockIdx.x * kUpdateThreads + threadIdx.x;
    const float2 *src = (const float2 *)partial + i;
    float2 s = make_float2(0.0f, 0.0f);
    for (int z0 = 0; z0 < pieces; z0 += 16) {
      float2 q[16];
#pragma unroll
      for (int z = 0; z < 16; ++z)
        q[z] = z0 + z < pieces ? __ldcs(src + (z0 + z) * (kPiece / 2)) : make_float2(0.0f, 0.0f);
#pragma unroll
      for (int z = 0; z < 16; ++z) {
        if (z0 + z >= pieces) break;
        s.x += q[z].x;
        s.y += q[z].y;
      }
    }
    int lh = 0;
    while (lh + 1 < 2 * kSurLayers && 2 * i >= wgrad_offset(lh + 1)) ++lh;
    const int l = lh >> 1, K = l == 0 ? kSurEnc : kSurHid;
    const int o = 2 * i - (int)wgrad_offset(lh);  // ((column / 4) * 128 + row) * 4 + column % 4
    const int at = ((lh & 1) * 128 + (o >> 2) % 128) * K + (o >> 9) * 4 + (o & 3);
    const int64_t first = l == 0 ? 0 : L.W[1] + (l - 1) * (L.W[2] - L.W[1]);
    const float px = update_param<ADAM>(a, first + at, s.x), py = update_param<ADAM>(a, first + at + 1, s.y);
    if (ADAM) {
      bf16 *wb = l == 0 ? a.Wb[0] : l == 1 ? a.Wb[1] : l == 2 ? a.Wb[2] : a.Wb[3];
      *(__nv_bfloat162 *)(wb + at) = __floats2bfloat162_rn(px, py);
    }
    return;
  }
  __shared__ float red[8][32];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j = (blockIdx.x - kWeightBlocks) * 32 + lane;  // column of all chain sets
  const bool last = blockIdx.x == kUpdateBlocks - 1;
  const int set = j / kSurHid, c = j % kSurHid;
  const float *src = last ? chainb + lane : chain + (int64_t)set * kChains * kSurHid + c;
  const int stride = last ? kSurOut : kSurHid;
  float x[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) x[i] = !last || lane < kSurOut ? src[(w + 8 * i) * stride] : 0.0f;
  red[w][lane] = pair_sum<1>(x);
  __syncthreads();
  if (w != 0 || (last && lane >= kSurOut)) return;
  const float g = ((red[0][lane] + red[4][lane]) + (red[2][lane] + red[6][lane])) +
                  ((red[1][lane] + red[5][lane]) + (red[3][lane] + red[7][lane]));
  update_param<ADAM>(a, last ? L.bh + lane : set < kSurLayers ? L.b[0] + c + (set ? L.b[1] - L.b[0] + (set - 1) * (L.b[2] - L.b[1]) : 0)
                                                             : L.Wh + (set - kSurLayers) * kSurHid + c, g);
}

// bf16 copies of every layer's weights from the master parameters.
__global__ void refresh_bf16_kernel(AdamArgs a) {
  const SurParamLayout L;
  for (int l = 0; l < kSurLayers; ++l) {
    const int64_t n = (int64_t)kSurHid * SurParamLayout::in_dim(l);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
      a.Wb[l][i] = __float2bfloat16_rn(a.p[L.W[l] + i]);
  }
}

// acc[0] += sum of loss[0..n)
__global__ void accum_loss_kernel(const float *loss, int64_t n, double *acc) {
  __shared__ double red[256];
  double s = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    s += loss[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicAdd(acc, red[0]);
}

// Counter-based uniform draws: (seed, stream, index) -> [0, 1), splitmix64.
__host__ __device__ inline uint64_t mix64(uint64_t z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
__host__ __device__ inline double uniform01(uint64_t seed, uint64_t stream, uint64_t i) {
  return (double)(mix64(seed * 0x100000001b3ull ^ mix64(stream * 0x9e3779b97f4a7c15ull + i)) >> 11) * 0x1.0p-53;
}

// Training set: sample i is a point at a random offset from the source (the
// frames of a moving source present FE nodes at every offset), at a random
// power and speed, labelled with the FE field. A fraction `near` of the
// samples is drawn from the box around the melt pool, a fraction `shell` from
// that box until the field lies in [shell_lo, shell_hi] (the band around the
// mushy zone), the rest from the model's window.
struct DataSpec {
  uint64_t seed;
  double p_lo, p_hi, v_lo, v_hi;
  double win_lo[3], win_hi[3];    // along-track, lateral, depth window (m)
  double near_lo[3], near_hi[3];  // melt-pool box (m)
  double near;                    // fraction from the melt-pool box
  double shell_lo, shell_hi;      // temperature band (K) ...
  double shell;                   // ... fraction of the samples drawn from the box until inside it
  ScanSource src;                 // physics; power and speed are replaced per sample
  float t_shift, t_scale;
  int log_out;
};

__global__ void make_data_kernel(DataSpec ds, int64_t first, int64_t n, float *raw, float *target) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t i = (uint64_t)(first + q);
    ScanSource s = ds.src;
    s.ntracks = 1;
    s.power = ds.p_lo + (ds.p_hi - ds.p_lo) * uniform01(ds.seed, 0, i);
    s.speed = ds.v_lo + (ds.v_hi - ds.v_lo) * uniform01(ds.seed, 1, i);
    const double kind = uniform01(ds.seed, 2, i);
    const bool shell = kind < ds.shell, nr = shell || kind < ds.shell + ds.near;
    // source at x = 0, y = 0 on the surface z = z_top = 0 at t = 0
    s.x_start = 0.0;
    s.y_line = 0.0;
    s.z_top = 0.0;
    double off[3] = {0.0, 0.0, 0.0}, T = 0.0;
    for (int attempt = 0; attempt < (shell ? 64 : 1); ++attempt) {
      for (int a = 0; a < 3; ++a) {
        const double lo = nr ? ds.near_lo[a] : ds.win_lo[a], hi = nr ? ds.near_hi[a] : ds.win_hi[a];
        off[a] = lo + (hi - lo) * uniform01(ds.seed, 3 + a + 8 * (uint64_t)attempt, i);
      }
      T = scan_field(s, off[0], off[1], -off[2], 0.0);
      if (T >= ds.shell_lo && T <= ds.shell_hi) break;
    }
    raw[q * kSurIn + 0] = (float)off[0];
    raw[q * kSurIn + 1] = (float)off[1];
    raw[q * kSurIn + 2] = (float)off[2];
    raw[q * kSurIn + 3] = (float)s.power;
    raw[q * kSurIn + 4] = (float)s.speed;
    const double yv = (T - ds.t_shift) / ds.t_scale;
    target[q] = (float)(ds.log_out ? log(yv) : yv);
  }
}

// ---------------------------------------------------------------------------
// Frames on the FE node grid: the synthetic field of a scan, and the model.
// Node file coordinates are origin + spacing * index, the field is evaluated
// at file coordinate * length_scale, frame f at field time (f * frame_dt) *
// time_scale (the conventions of amca_set_rosenthal_frames).
// ---------------------------------------------------------------------------
struct FrameJob {
  ScanSource src;
  double origin[3], spacing;
  int nodes[3];
  double length_scale, frame_dt, time_scale;
  int f0, nf;                    // frames f0 .. f0 + nf - 1
  double *ring;                  // frame f goes to slot f % slots
  int slots;
  int64_t nnodes;
  // model frames only
  int box[3];                    // window size in nodes
  double win_lo[3], win_hi[3];   // window around the source (m): along-track, lateral, depth
  float t_liq, band, thresh;     // fallback: |T - t_liq| < band and error estimate > thresh (K)
  unsigned long long *counters;  // [0] nodes evaluated, [1] near the liquidus, [2] fallbacks
};

__device__ __forceinline__ void node_xyz(const FrameJob &j, int64_t I, int64_t J, int64_t K, double &x, double &y,
                                         double &z) {
  x = (j.origin[0] + j.spacing * (double)I) * j.length_scale;
  y = (j.origin[1] + j.spacing * (double)J) * j.length_scale;
  z = (j.origin[2] + j.spacing * (double)K) * j.length_scale;
}

__device__ __forceinline__ double frame_time(const FrameJob &j, int f) { return ((double)f * j.frame_dt) * j.time_scale; }

// the synthetic field of the scan at every node of the frames
__global__ void scan_frames_kernel(FrameJob j) {
  const int64_t total = j.nnodes * j.nf;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total; q += (int64_t)gridDim.x * blockDim.x) {
    const int f = j.f0 + (int)(q / j.nnodes);
    const int64_t n = q % j.nnodes;
    double x, y, z;
    node_xyz(j, n % j.nodes[0], (n / j.nodes[0]) % j.nodes[1], n / ((int64_t)j.nodes[0] * j.nodes[1]), x, y, z);
    j.ring[(int64_t)(f % j.slots) * j.nnodes + n] = scan_field(j.src, x, y, z, frame_time(j, f));
  }
}

// every node of the frames at the ambient temperature (the model's value
// outside its window)
__global__ void fill_frames_kernel(FrameJob j) {
  const int64_t total = j.nnodes * j.nf;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total; q += (int64_t)gridDim.x * blockDim.x) {
    const int f = j.f0 + (int)(q / j.nnodes);
    j.ring[(int64_t)(f % j.slots) * j.nnodes + q % j.nnodes] = j.src.t0;
  }
}

// What the model's queries of one frame share: the frame's time, where the
// source is and which way it moves, and the FE nodes the model answers for:
// the window around the source (job.box nodes from its lower corner) clipped
// to the grid. `first` = queries of the job's frames before this one.
struct FrameBox {
  double t, xl, yl, dir;
  int lo[3], n[3];
  int64_t first;
};

// Frames one launch answers for: their boxes live in shared memory.
constexpr int kJobFrames = 64;

__device__ __forceinline__ void frame_box(const FrameJob &j, int f, FrameBox &b) {
  b.t = frame_time(j, f);
  scan_position(j.src, b.t, b.xl, b.yl, b.dir);
  const double low[3] = {b.dir > 0 ? b.xl + j.win_lo[0] : b.xl - j.win_hi[0], b.yl + j.win_lo[1],
                         j.src.z_top - j.win_hi[2]};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int i0 = (int)floor((low[a] / j.length_scale - j.origin[a]) / j.spacing);
    const int64_t end = min((int64_t)j.nodes[a], (int64_t)i0 + j.box[a]);
    b.lo[a] = max(i0, 0);
    b.n[a] = end > b.lo[a] ? (int)(end - b.lo[a]) : 0;
  }
}

// Boxes of the job's frames into shared memory (every thread of the block);
// returns the job's query count. The callers synchronise afterwards by the
// barrier this ends with.
__device__ int64_t frame_boxes(const FrameJob &j, FrameBox *boxes) {
  if ((int)threadIdx.x < j.nf) frame_box(j, j.f0 + (int)threadIdx.x, boxes[threadIdx.x]);
  __syncthreads();
  int64_t total = 0;
  for (int k = 0; k < j.nf; ++k) {
    if (threadIdx.x == 0) boxes[k].first = total;
    total += (int64_t)boxes[k].n[0] * boxes[k].n[1] * boxes[k].n[2];
  }
  __syncthreads();
  return total;
}

// Query q of the job: the index of its frame's box and its node.
__device__ __forceinline__ int64_t frame_query(const FrameJob &j, const FrameBox *boxes, int64_t q, int &k, int &I,
                                               int &J, int &K) {
  int lo = 0, hi = j.nf - 1;  // the last frame whose first query is at most q (empty frames share theirs)
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (boxes[mid].first <= q) lo = mid; else hi = mid - 1;
  }
  k = lo;
  const FrameBox &b = boxes[k];
  const int64_t l = q - b.first;
  const int64_t row = l / b.n[0], slab = row / b.n[1];
  I = b.lo[0] + (int)(l - row * b.n[0]);
  J = b.lo[1] + (int)(row - slab * b.n[1]);
  K = b.lo[2] + (int)slab;
  return ((int64_t)K * j.nodes[1] + J) * j.nodes[0] + I;
}

// ---------------------------------------------------------------------------
// Fused inference: the whole network on 128-query tiles, persistent.
// Frames: only nodes inside both the source's window and the grid are
// queries (a raster over a 60 x 60 x 40-cell block has 0.5% of its windows'
// nodes inside the grid: with all of them evaluated, 1,484 frames took 250 ms,
// now a few; the whole run of that raster 458 -> 207 ms).
// Shared memory: activations H (128 x 256 bf16, four 64-column blocks of
// 16 KB) and one layer's weights (256 x 256 bf16, four blocks of 64 input
// columns, 32 KB each).
// 16 epilogue warps in four groups (warp w reads TMEM lanes 32 (w % 4), its
// rows; group w / 4 has 64 columns of every layer), a warp that issues the MMAs
// and one that loads weights. A layer's epilogue is bound by instruction issue
// (about nine per element, 1.1 us a tile), its MMAs take as long; they overlap:
//  - the MMAs over the first half of K run as soon as groups 0 and 1 have
//    written it, while groups 2 and 3 still work on the layer before (into the
//    other of two accumulators);
//  - the MMAs over the second half of K finish output columns 0..127 first, so
//    groups 0 and 1 start while columns 128..255 are still being computed;
//  - a weight block is replaced by the next layer's as soon as its MMAs are
//    done, long before it is needed.
//  - the next tile's features are computed in registers while the second and
//    third layers' MMAs run.
// Group 3 also writes a tile's results and fetches the next tile's inputs,
// behind the first layer's MMAs. Each accumulator still adds
// its K steps in order. A tile took 19.5 us with everything one after another;
// now 15.8 (100,003 queries from a cold cache: 117 -> 95 us; a layer's epilogue
// takes 3.5K cycles of the 5.6K, its exposed MMAs 2K).
// ---------------------------------------------------------------------------
constexpr int kInferGroups = 4, kGroupCols = kSurHid / kInferGroups, kIoGroup = 3;
constexpr int kInferEpiWarps = 4 * kInferGroups, kInferThreads = 32 * (kInferEpiWarps + 2);
enum { kSrcArray = 0, kSrcFrames = 1 };

struct InferArgs {
  int64_t nq;
  const float *raw;  // kSrcArray: nq x 5 raw inputs
  float *T, *err;    // kSrcArray: outputs (K)
  FrameJob job;      // kSrcFrames
  int *error;
};

constexpr uint32_t kInferSmem = 64u * 1024u + 128u * 1024u + 1024u;

template <int SRC>
__global__ void __launch_bounds__(kInferThreads, 1)
    mlp_infer_kernel(const __grid_constant__ CUtensorMap tW0, const __grid_constant__ CUtensorMap tW1,
                     const __grid_constant__ CUtensorMap tW2, const __grid_constant__ CUtensorMap tW3, SurModelDev md,
                     InferArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *H = align1024(smem_raw);
  uint8_t *Wsm = H + 64 * 1024;
  // weight block loaded / its MMAs done; half of the layer's input written (8
  // warps); half of the accumulator complete; heads of a tile summed (16
  // warps); inputs of a tile there (4 warps), by tile parity: a warp that is
  // slow to look cannot miss one, the next of the parity waits for its heads
  __shared__ __align__(8) uint64_t wfull[4], wfree[4], hready[2], acc[2], headed, fetched[2], drained;
  __shared__ uint32_t tmem_base;
  __shared__ volatile int s_abort;
  __shared__ __align__(16) float s_bias[kSurLayers][kSurHid];
  __shared__ __align__(16) float s_wh[kSurOut][kSurHid];
  __shared__ float s_bh[kSurOut];
  __shared__ float s_head[2][kInferGroups][128][2];  // by tile parity
  __shared__ float s_in[2][128][kSurIn];             // normalised inputs, by tile parity
  __shared__ __align__(16) float s_fourier[kSurFreq][kFourierPad];
  __shared__ FrameBox s_box[SRC == kSrcFrames ? kJobFrames : 1];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t nq = SRC == kSrcFrames ? frame_boxes(a.job, s_box) : a.nq;
  const int64_t ntiles = (nq + 127) / 128;
  const int64_t tile0 = blockIdx.x, dtile = gridDim.x;
  const SurParamLayout L;

  for (int i = threadIdx.x; i < kSurLayers * kSurHid; i += blockDim.x)
    s_bias[i / kSurHid][i % kSurHid] = md.p[L.b[i / kSurHid] + i % kSurHid];
  for (int i = threadIdx.x; i < kSurOut * kSurHid; i += blockDim.x) s_wh[i / kSurHid][i % kSurHid] = md.p[L.Wh + i];
  if (threadIdx.x < kSurOut) s_bh[threadIdx.x] = md.p[L.bh + threadIdx.x];
  load_fourier(md, s_fourier);
  if (threadIdx.x == 0) {
    for (int k = 0; k < 4; ++k) {
      umma::mbar_init(umma::smem_u32(&wfull[k]), 1);
      umma::mbar_init(umma::smem_u32(&wfree[k]), 1);
    }
    for (int k = 0; k < 2; ++k) {
      umma::mbar_init(umma::smem_u32(&hready[k]), kInferEpiWarps / 2);
      umma::mbar_init(umma::smem_u32(&acc[k]), 1);
      umma::mbar_init(umma::smem_u32(&fetched[k]), 4);
    }
    umma::mbar_init(umma::smem_u32(&headed), kInferEpiWarps);
    umma::mbar_init(umma::smem_u32(&drained), 1);
    umma::mbar_fence_init();
    s_abort = 0;
  }
  if (warp == 0) umma::tmem_alloc(umma::smem_u32(&tmem_base), 512);
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  const uint32_t tmem = tmem_base;
  auto wait = [&](uint64_t &bar, uint32_t parity) {
    return umma::mbar_wait_role(umma::smem_u32(&bar), parity, kWaitNs, &s_abort);
  };
  auto wait_warp = [&](uint64_t &bar, uint32_t parity) {
    return umma::mbar_wait_warp(umma::smem_u32(&bar), parity, kWaitNs, &s_abort);
  };

  if (warp == kInferEpiWarps + 1) {  // ---- weights ----
    if (lane == 0) {
      const CUtensorMap *tW[4] = {&tW0, &tW1, &tW2, &tW3};
      uint32_t uses[4] = {0, 0, 0, 0};
      bool ok = true;
      for (int64_t tile = tile0; tile < ntiles && ok; tile += dtile)
        for (int l = 0; l < kSurLayers && ok; ++l)
          for (int kb = 0; kb < SurParamLayout::in_dim(l) / 64; ++kb) {
            if (uses[kb] && !(ok = wait(wfree[kb], (uses[kb] - 1) & 1))) break;
            const uint32_t bar = umma::smem_u32(&wfull[kb]);
            umma::mbar_expect_tx(bar, 32u * 1024u);
            umma::tma_load_2d(umma::smem_u32(Wsm + kb * 32 * 1024), tW[l], bar, kb * 64, 0);
            ++uses[kb];
          }
      if (!ok)  // let the loads in flight land before the block exits
        for (int kb = 0; kb < 4; ++kb)
          if (uses[kb]) umma::mbar_wait(umma::smem_u32(&wfull[kb]), (uses[kb] - 1) & 1, kWaitNs);
    }
  } else if (warp == kInferEpiWarps) {  // ---- MMAs ----
    if (lane == 0) {
      constexpr uint32_t id_all = umma::idesc_bf16_f32(128, kSurHid), id_half = umma::idesc_bf16_f32(128, kSurHid / 2);
      uint32_t uses[4] = {0, 0, 0, 0}, layers = 0;
      bool ok = true;
      // K block kb of the layer into accumulator columns d.. from weight row n0 on
      auto mma = [&](uint32_t d, int kb, int n0, uint32_t idesc) {
        const uint32_t ha = umma::smem_u32(H + kb * 16 * 1024), wa = umma::smem_u32(Wsm + kb * 32 * 1024 + n0 * 128);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma::mma_bf16(d + n0, umma::sdesc_sw128(ha + 32u * k), umma::sdesc_sw128(wa + 32u * k), idesc,
                         (kb | k) != 0 ? 1u : 0u);
      };
      auto weights = [&](int kb) { return wait(wfull[kb], uses[kb]++ & 1); };
      for (int64_t tile = tile0; tile < ntiles && ok; tile += dtile)
        for (int l = 0; l < kSurLayers; ++l, ++layers) {
          const uint32_t d = tmem + 256u * (l & 1);
          const int first = l == 0 ? 0 : 2;  // K blocks from here on are computed half by half of the columns
          if (!(ok = wait(hready[0], layers & 1))) break;
          for (int kb = 0; kb < first && ok; ++kb) {
            if (!(ok = weights(kb))) break;
            umma::tc_fence_after();
            mma(d, kb, 0, id_all);
            umma::mma_commit(umma::smem_u32(&wfree[kb]));
          }
          if (!ok || !(ok = wait(hready[1], layers & 1) && weights(first) && weights(first + 1))) break;
          umma::tc_fence_after();
          for (int half = 0; half < 2; ++half) {
            mma(d, first, 128 * half, id_half);
            mma(d, first + 1, 128 * half, id_half);
            umma::mma_commit(umma::smem_u32(&acc[half]));
          }
          umma::mma_commit(umma::smem_u32(&wfree[first]));
          umma::mma_commit(umma::smem_u32(&wfree[first + 1]));
        }
      if (!ok) {  // nothing may still write to the tensor memory when it is given back
        umma::mma_commit(umma::smem_u32(&drained));
        umma::mbar_wait(umma::smem_u32(&drained), 0, kWaitNs);
      }
    }
  } else {  // ---- features, epilogues, results ----
    const int q4 = warp & 3, grp = warp >> 2, row = q4 * 32 + lane, half = grp >> 1;
    const uint32_t trow = tmem + ((uint32_t)(q4 * 32) << 16);
    // the io group's row of a tile: whether it is a query, and (frames) its frame's box and node
    struct Row {
      int64_t tile, node;
      int k;
      bool valid;
    };
    auto fetch = [&](int64_t tile, int par) {  // io group: the tile's raw inputs
      Row r{tile, -1, 0, tile * 128 + row < nq};
      const int64_t qi = tile * 128 + row;
      float raw[kSurIn] = {0, 0, 0, 0, 0};
      if (r.valid) {
        if (SRC == kSrcArray) {
#pragma unroll
          for (int i = 0; i < kSurIn; ++i) raw[i] = a.raw[qi * kSurIn + i];
        } else {
          // Along-track offset from the source (positive ahead of it), lateral
          // offset, depth below the top surface (m), power (W), speed (m/s),
          // with the frame's source position at hand: an FP64 instruction holds
          // its scheduler for 64 cycles on GB300, and about 110 of them in
          // every warp (position, window corner and divisions per row) were
          // most of a tile's 13.6 us.
          int I, J, K;
          double x, y, z;
          r.node = frame_query(a.job, s_box, qi, r.k, I, J, K);
          node_xyz(a.job, I, J, K, x, y, z);
          const FrameBox &fb = s_box[r.k];
          raw[0] = (float)((x - fb.xl) * fb.dir);
          raw[1] = (float)(y - fb.yl);
          raw[2] = (float)(a.job.src.z_top - z);
          raw[3] = (float)a.job.src.power;
          raw[4] = (float)a.job.src.speed;
        }
      }
      float u[kSurIn];
      normalise(md, raw, u);
#pragma unroll
      for (int i = 0; i < kSurIn; ++i) s_in[par][row][i] = u[i];
      __syncwarp();
      if (lane == 0) umma::mbar_arrive(umma::smem_u32(&fetched[par]));
      return r;
    };
    auto results = [&](const Row &r, int par) {  // io group (whole warps)
      float m = s_bh[0], s = s_bh[1];
#pragma unroll
      for (int k = 0; k < kInferGroups; ++k) {
        m += s_head[par][k][row][0];
        s += s_head[par][k][row][1];
      }
      s = fminf(fmaxf(s, -12.0f), 4.0f);
      const float T = md.log_out ? md.t_shift + md.t_scale * expf(m) : md.t_shift + md.t_scale * m;
      const float e = md.log_out ? 2.0f * (T - md.t_shift) * expf(s) : 2.0f * md.t_scale * expf(s);
      if (SRC == kSrcArray) {
        if (r.valid) {
          a.T[r.tile * 128 + row] = T;
          a.err[r.tile * 128 + row] = e;
        }
      } else {
        const bool near = r.valid && fabsf(T - a.job.t_liq) < a.job.band;
        const bool fb = near && e > a.job.thresh;
        if (r.valid) {
          double out = (double)T;
          if (fb) {
            double x, y, z;
            const int64_t nx = a.job.nodes[0], ny = a.job.nodes[1];
            node_xyz(a.job, r.node % nx, r.node / nx % ny, r.node / (nx * ny), x, y, z);
            out = scan_field(a.job.src, x, y, z, s_box[r.k].t);
          }
          a.job.ring[(int64_t)((a.job.f0 + r.k) % a.job.slots) * a.job.nnodes + r.node] = out;
        }
        const unsigned nv = __popc(__ballot_sync(0xffffffffu, r.valid));
        const unsigned nn = __popc(__ballot_sync(0xffffffffu, near));
        const unsigned nfb = __popc(__ballot_sync(0xffffffffu, fb));
        if (lane == 0) {
          if (nv) atomicAdd(&a.job.counters[0], (unsigned long long)nv);
          if (nn) atomicAdd(&a.job.counters[1], (unsigned long long)nn);
          if (nfb) atomicAdd(&a.job.counters[2], (unsigned long long)nfb);
        }
      }
    };
    // this warp's part of the layer's input is written (and its TMEM reads are done)
    auto written = [&]() {
      umma::fence_async_smem();
      umma::tc_fence_before();
      __syncwarp();
      if (lane == 0) umma::mbar_arrive(umma::smem_u32(&hready[half]));
    };
    // Fourier features of a tile's row: half h of this group's 16 phases (sines
    // at column j, cosines at 64 + j), held in registers until H is free
    uint4 fs[2], fc[2];
    auto features = [&](int par, int h) {
      float u[kSurIn];
#pragma unroll
      for (int i = 0; i < kSurIn; ++i) u[i] = s_in[par][row][i];
      __align__(16) bf16 sb[8], cb[8];
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        float sv, cv;
        phases(s_fourier[grp * (kSurFreq / kInferGroups) + 8 * h + t], u, sv, cv);
        sb[t] = __float2bfloat16_rn(sv);
        cb[t] = __float2bfloat16_rn(cv);
      }
      fs[h] = *(const uint4 *)sb;
      fc[h] = *(const uint4 *)cb;
    };
    Row cur{}, last{};
    if (grp == kIoGroup && tile0 < ntiles) cur = fetch(tile0, 0);
    uint32_t tiles = 0, layers = 0;
    bool ok = true;
    for (int64_t tile = tile0; tile < ntiles; tile += dtile, ++tiles) {
      const int par = tiles & 1;
      if (tiles == 0) {
        if (!(ok = wait_warp(fetched[0], 0))) break;
        features(0, 0);
        features(0, 1);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int j0 = grp * (kSurFreq / kInferGroups) + 8 * h;
        *(uint4 *)(H + umma::sw128_offset(row, j0, 128)) = fs[h];
        *(uint4 *)(H + umma::sw128_offset(row, kSurFreq + j0, 128)) = fc[h];
      }
      written();
      if (grp == kIoGroup) {
        if (tiles > 0) {
          if (!(ok = wait_warp(headed, par ^ 1))) break;
          results(last, par ^ 1);
        }
        last = cur;
        // (every warp has read the inputs of the tile before: it has its heads)
        if (tile + dtile < ntiles) cur = fetch(tile + dtile, par ^ 1);
      }
      float mu = 0.0f, sl = 0.0f;
      for (int l = 0; l < kSurLayers; ++l, ++layers) {
        const uint32_t dcol = trow + 256u * (l & 1);
        // the next tile's features, while this layer's MMAs run
        if ((l == 1 || l == 2) && tile + dtile < ntiles) {
          if (l == 1 && !(ok = wait_warp(fetched[par ^ 1], (tiles + 1) >> 1 & 1))) break;
          if (l == 1) features(par ^ 1, 0);
          else features(par ^ 1, 1);
        }
        // the first layer's input, which is overwritten below, is read for both halves
        if (!(ok = wait_warp(acc[half], layers & 1) && (l > 0 || wait_warp(acc[half ^ 1], layers & 1)))) break;
        umma::tc_fence_after();
        for (int c0 = grp * kGroupCols; c0 < (grp + 1) * kGroupCols; c0 += 32) {
          float v[32];
          umma::tmem_ld32(dcol + c0, v);
          const float4 *b4 = reinterpret_cast<const float4 *>(&s_bias[l][c0]);
          if (l < kSurLayers - 1) {
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              const float4 ba = b4[j / 4], bb = b4[j / 4 + 1];
              const float b[8] = {ba.x, ba.y, ba.z, ba.w, bb.x, bb.y, bb.z, bb.w};
              __align__(16) bf16 hb[8];
#pragma unroll
              for (int t = 0; t < 8; ++t) hb[t] = __float2bfloat16_rn(silu(v[j + t] + b[t]));
              *(uint4 *)(H + umma::sw128_offset(row, c0 + j, 128)) = *(const uint4 *)hb;
            }
          } else {
            const float4 *w0 = reinterpret_cast<const float4 *>(&s_wh[0][c0]);
            const float4 *w1 = reinterpret_cast<const float4 *>(&s_wh[1][c0]);
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              const float4 bq = b4[j / 4], m0 = w0[j / 4], m1 = w1[j / 4];
              const float b[4] = {bq.x, bq.y, bq.z, bq.w}, x0[4] = {m0.x, m0.y, m0.z, m0.w},
                          x1[4] = {m1.x, m1.y, m1.z, m1.w};
#pragma unroll
              for (int t = 0; t < 4; ++t) {
                const float h = silu(v[j + t] + b[t]);
                mu = fmaf(h, x0[t], mu);
                sl = fmaf(h, x1[t], sl);
              }
            }
          }
        }
        if (l < kSurLayers - 1) written();
      }
      if (!ok) break;
      s_head[par][grp][row][0] = mu;
      s_head[par][grp][row][1] = sl;
      __syncwarp();
      if (lane == 0) umma::mbar_arrive(umma::smem_u32(&headed));
    }
    if (ok && tiles > 0 && grp == kIoGroup && wait_warp(headed, (tiles - 1) & 1)) results(last, (tiles - 1) & 1);
  }
  umma::tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && s_abort) atomicCAS(a.error, 0, kErrWait);
  if (warp == 0) umma::tmem_free(tmem, 512);
}

}  // namespace sur
}  // namespace amca

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
namespace amca {
namespace sur {

#define SCK(call)                                                                                       \
  do {                                                                                                  \
    cudaError_t e_ = (call);                                                                            \
    if (e_ != cudaSuccess) throw std::runtime_error(std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    cudaDriverEntryPointQueryResult q;
    void *p = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
  });
  if (!fn) throw std::runtime_error("cuTensorMapEncodeTiled is not available");
  return fn;
}

// Tensor map of a row-major [rows x cols] bf16 matrix read in boxes of 64
// columns x box_rows rows with the 128-byte swizzle.
CUtensorMap tmap_bf16(const void *base, int64_t rows, int64_t cols, int box_rows) {
  if (cols % 64 != 0 || box_rows > 256 || ((uintptr_t)base & 15) != 0)
    throw std::invalid_argument("tensor map: columns must be a multiple of 64 and the base 16-byte aligned");
  CUtensorMap m;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  const cuuint32_t es[2] = {1, 1};
  const CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box,
                                 es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                 CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw std::runtime_error("cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
  return m;
}

int grid_1d(int64_t n, int threads = 256) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((n + threads - 1) / threads, 152 * 16));
}

// A launch whose blocks may start while the kernel before it in the stream
// still runs (once all of its blocks have let them: launch_dependents); it
// waits by itself (wait_prerequisites) before it needs that kernel's results.
template <typename... P, typename... A>
void launch_early(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  SCK(cudaLaunchKernelEx(&cfg, kernel, P(args)...));
}

uint64_t gcd64(uint64_t a, uint64_t b) {
  while (b) {
    const uint64_t t = a % b;
    a = b;
    b = t;
  }
  return a;
}

}  // namespace sur

// One thermal model on one device: parameters, Adam state, the training set
// and the per-batch buffers of a training step.
struct ThermalModel {
  using bf16 = __nv_bfloat16;
  int device = 0, sms = 0;
  cudaStream_t stream = nullptr;
  SurParamLayout L;
  sur::DataSpec data{};
  float fourier_h[kSurFreq * kSurIn];
  float in_shift[kSurIn], in_scale[kSurIn], t_shift = 0, t_scale = 1;
  // device
  float *fourier = nullptr, *p = nullptr, *m1 = nullptr, *m2 = nullptr, *g = nullptr;
  bf16 *Wb[kSurLayers] = {};
  int *err = nullptr;
  unsigned long long *counters = nullptr;
  float *ds_raw = nullptr, *ds_target = nullptr;
  int64_t ds_n = 0;
  int64_t adam_t = 0;
  int64_t seen = 0;
  // evaluation buffers, kept for calls of up to kEvalRows rows (28 bytes each)
  static constexpr int64_t kEvalRows = 1 << 21;
  int64_t eval_rows = 0;
  float *eval_buf = nullptr;
  CUtensorMap tw[kSurLayers];  // the layers' weights, for the inference kernels
  // batch buffers
  int64_t nb = 0;
  int blocks = 0;                        // of the step kernel
  int pieces = 0, per = 0, width = 256;  // of the weight gradients: pieces, their kWgradRows-row blocks, column slice
  float *braw = nullptr, *by = nullptr, *pred = nullptr, *loss = nullptr, *partial = nullptr;
  sur::ChainArgs chains;
  float2 *dpred = nullptr;
  uint4 *zs = nullptr;
  sur::TrainMaps maps;
  std::vector<void *> allocs, batch_allocs;

  template <typename T>
  T *alloc(size_t n) {
    void *q = nullptr;
    SCK(cudaMalloc(&q, std::max<size_t>(n, 1) * sizeof(T)));
    allocs.push_back(q);
    return (T *)q;
  }
  template <typename T>
  T *balloc(size_t n) {
    void *q = nullptr;
    SCK(cudaMalloc(&q, std::max<size_t>(n, 1) * sizeof(T)));
    batch_allocs.push_back(q);
    return (T *)q;
  }
  ~ThermalModel() {
    if (stream) cudaStreamSynchronize(stream);
    for (void *q : batch_allocs) cudaFree(q);
    for (void *q : allocs) cudaFree(q);
    cudaFree(eval_buf);
    if (stream) cudaStreamDestroy(stream);
  }

  SurModelDev dev() const {
    SurModelDev d{};
    d.fourier = fourier;
    d.p = p;
    for (int l = 0; l < kSurLayers; ++l) d.Wb[l] = Wb[l];
    for (int i = 0; i < kSurIn; ++i) {
      d.in_shift[i] = in_shift[i];
      d.in_scale[i] = in_scale[i];
    }
    d.t_shift = t_shift;
    d.t_scale = t_scale;
    d.log_out = data.log_out;
    return d;
  }
  sur::AdamArgs adam_args() const {
    sur::AdamArgs a{};
    a.p = p;
    a.m = m1;
    a.v = m2;
    a.g = g;
    for (int l = 0; l < kSurLayers; ++l) a.Wb[l] = Wb[l];
    return a;
  }
  void check_error() {
    int e = 0;
    SCK(cudaMemcpyAsync(&e, err, sizeof e, cudaMemcpyDeviceToHost, stream));
    SCK(cudaStreamSynchronize(stream));
    if (e) throw std::runtime_error("thermal model kernel: a bounded wait ran out");
  }
  void refresh_bf16() {
    sur::refresh_bf16_kernel<<<sur::grid_1d(L.total), 256, 0, stream>>>(adam_args());
    SCK(cudaGetLastError());
  }

  ThermalModel(int dev_id, const sur::DataSpec &ds, double fourier_sigma, double fourier_sigma_pv)
      : device(dev_id), data(ds) {
    SCK(cudaSetDevice(device));
    SCK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    // input normalisation: the window's offsets and the power / speed ranges to [-1, 1]
    for (int a = 0; a < 3; ++a) {
      in_shift[a] = (float)(0.5 * (ds.win_lo[a] + ds.win_hi[a]));
      in_scale[a] = (float)(2.0 / (ds.win_hi[a] - ds.win_lo[a]));
    }
    in_shift[3] = (float)(0.5 * (ds.p_lo + ds.p_hi));
    in_scale[3] = (float)(2.0 / (ds.p_hi - ds.p_lo));
    in_shift[4] = (float)(0.5 * (ds.v_lo + ds.v_hi));
    in_scale[4] = (float)(2.0 / (ds.v_hi - ds.v_lo));
    t_shift = ds.t_shift;
    t_scale = ds.t_scale;
    // Fourier matrix: normal draws (Box-Muller on counter-based uniforms) times
    // sigma (offsets) or sigma_pv (power, speed)
    for (int i = 0; i < kSurFreq * kSurIn; ++i) {
      const double u1 = std::max(sur::uniform01(ds.seed, 100, (uint64_t)i), 1e-300);
      const double u2 = sur::uniform01(ds.seed, 101, (uint64_t)i);
      const double sig = (i % kSurIn) < 3 ? fourier_sigma : fourier_sigma_pv;
      fourier_h[i] = (float)(sig * std::sqrt(-2.0 * std::log(u1)) * std::cos(2.0 * M_PI * u2));
    }
    // weights: Xavier-uniform from the seed, biases zero; head small, log-error bias -2
    std::vector<float> ph((size_t)L.total, 0.0f);
    for (int l = 0; l < kSurLayers; ++l) {
      const int K = SurParamLayout::in_dim(l);
      const double bound = std::sqrt(6.0 / (K + kSurHid));
      for (int64_t i = 0; i < (int64_t)kSurHid * K; ++i)
        ph[L.W[l] + i] = (float)(bound * (2.0 * sur::uniform01(ds.seed, 200 + l, (uint64_t)i) - 1.0));
    }
    const double hb = 0.1 * std::sqrt(6.0 / (kSurHid + kSurOut));
    for (int64_t i = 0; i < (int64_t)kSurOut * kSurHid; ++i)
      ph[L.Wh + i] = (float)(hb * (2.0 * sur::uniform01(ds.seed, 300, (uint64_t)i) - 1.0));
    ph[L.bh + 1] = -2.0f;
    fourier = alloc<float>(kSurFreq * kSurIn);
    p = alloc<float>(L.total);
    m1 = alloc<float>(L.total);
    m2 = alloc<float>(L.total);
    g = alloc<float>(L.total);
    for (int l = 0; l < kSurLayers; ++l) {
      const int K = SurParamLayout::in_dim(l);
      Wb[l] = alloc<bf16>((size_t)kSurHid * K);
    }
    for (int l = 0; l < kSurLayers; ++l) tw[l] = sur::tmap_bf16(Wb[l], kSurHid, SurParamLayout::in_dim(l), 256);
    SCK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    SCK(cudaFuncSetAttribute(sur::mlp_infer_kernel<sur::kSrcArray>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sur::kInferSmem));
    SCK(cudaFuncSetAttribute(sur::mlp_infer_kernel<sur::kSrcFrames>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sur::kInferSmem));
    SCK(cudaFuncSetAttribute(sur::mlp_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sur::kTrainSmem));
    SCK(cudaFuncSetAttribute(sur::mlp_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sur::kWgradSmem));
    err = alloc<int>(1);
    counters = alloc<unsigned long long>(4);
    SCK(cudaMemcpyAsync(fourier, fourier_h, sizeof fourier_h, cudaMemcpyHostToDevice, stream));
    set_params(ph.data());
    SCK(cudaMemsetAsync(err, 0, sizeof(int), stream));
    SCK(cudaStreamSynchronize(stream));
  }

  void set_params(const float *host) {
    SCK(cudaMemcpyAsync(p, host, (size_t)L.total * 4, cudaMemcpyHostToDevice, stream));
    SCK(cudaMemsetAsync(m1, 0, (size_t)L.total * 4, stream));
    SCK(cudaMemsetAsync(m2, 0, (size_t)L.total * 4, stream));
    adam_t = 0;
    refresh_bf16();
    SCK(cudaStreamSynchronize(stream));
  }
  void get_params(float *host) {
    SCK(cudaMemcpyAsync(host, p, (size_t)L.total * 4, cudaMemcpyDeviceToHost, stream));
    SCK(cudaStreamSynchronize(stream));
  }

  // Device buffer for an evaluation of n rows (raw inputs, T, error estimate),
  // kept for the calls after it; null for more than kEvalRows rows.
  float *eval_buffer(int64_t n) {
    if (n > kEvalRows) return nullptr;
    if (n > eval_rows) {
      SCK(cudaStreamSynchronize(stream));
      cudaFree(eval_buf);
      eval_buf = nullptr;
      eval_rows = 0;
      const int64_t rows = std::min<int64_t>(kEvalRows, std::max<int64_t>(1024, n + n / 4));
      void *q = nullptr;
      SCK(cudaMalloc(&q, (size_t)rows * (kSurIn + 2) * 4));
      eval_buf = (float *)q;
      eval_rows = rows;
    }
    return eval_buf;
  }

  // Per-batch buffers and tensor maps for batches of n rows (n a multiple of 128).
  void set_batch(int64_t n) {
    if (n == nb) return;
    if (n <= 0 || n % 128) throw std::invalid_argument("batch size must be a positive multiple of 128");
    SCK(cudaStreamSynchronize(stream));
    for (void *q : batch_allocs) cudaFree(q);
    batch_allocs.clear();
    nb = 0;
    const int64_t kblocks = n / 64;
    // pieces of the weight gradients: at most 64, of at least 8 blocks of 64 rows each, all alike
    pieces = 1;
    while (pieces < 64 && kblocks % (pieces * 2) == 0 && kblocks / (pieces * 2) >= 8) pieces *= 2;
    per = (int)(n / sur::kWgradRows / pieces);
    width = kSurHid;
    while (width > 64 && sur::wgrad_items(width) * pieces < sms) width /= 2;
    blocks = (int)std::min<int64_t>(n / 128, sms);
    braw = balloc<float>((size_t)n * kSurIn);
    by = balloc<float>((size_t)n);
    pred = balloc<float>((size_t)n * 2);
    loss = balloc<float>((size_t)n);
    dpred = balloc<float2>((size_t)n);
    partial = balloc<float>((size_t)pieces * sur::kPiece);
    zs = balloc<uint4>((size_t)n / 128 * 3 * (sur::kTrainCols / 8) * sur::kTrainThreads);
    for (int l = 0; l < kSurLayers; ++l) {
      const int K = SurParamLayout::in_dim(l);
      const bf16 *X = balloc<bf16>((size_t)n * K), *dZ = balloc<bf16>((size_t)n * kSurHid);
      chains.dZ[l] = dZ;
      maps.W[l] = sur::tmap_bf16(Wb[l], kSurHid, K, 256);
      maps.X_out[l] = sur::tmap_bf16(X, n, K, 128);
      maps.X_in[l] = sur::tmap_bf16(X, n, K, sur::kWgradRows);
      maps.dZ_out[l] = sur::tmap_bf16(dZ, n, kSurHid, 128);
      maps.dZ_in[l] = sur::tmap_bf16(dZ, n, kSurHid, sur::kWgradRows);
    }
    chains.H = balloc<bf16>((size_t)n * kSurHid);
    maps.X_out[kSurLayers] = sur::tmap_bf16(chains.H, n, kSurHid, 128);
    chains.dpred = dpred;
    chains.n = n;
    chains.chain = balloc<float>((size_t)sur::kChainSets * sur::kChains * kSurHid);
    chains.chainb = balloc<float>((size_t)sur::kChains * kSurOut);
    nb = n;
  }

  // Forward and backward over the nb rows that are samples (start + q) * perm
  // mod nsamples, q = 0.., of raw / target; the gradients' pieces are left for
  // update().
  void forward_backward(const float *raw, const float *target, int64_t nsamples, int64_t start, uint64_t perm) {
    using namespace sur;
    StepArgs a{};
    a.n = nb;
    a.raw = raw;
    a.target = target;
    a.nsamples = (uint64_t)nsamples;
    a.start = (uint64_t)start;
    a.perm = perm;
    a.zs = zs;
    a.pred = pred;
    a.loss = loss;
    a.dpred = dpred;
    a.inv_batch = 1.0f / (float)nb;
    a.lambda_s = 0.1f;
    a.error = err;
    launch_early(mlp_step_kernel, dim3(blocks), kTrainThreads, kTrainSmem, stream, maps, dev(), a);
    mlp_chain_kernel<<<dim3(kChains * (kSurHid / kChainCols) / kChainThreads, kSurLayers + 1), kChainThreads, 0, stream>>>(
        chains);
    SCK(cudaGetLastError());
    launch_early(mlp_wgrad_kernel, dim3(wgrad_items(width), pieces), kWgradThreads, kWgradSmem, stream, maps, width, per,
                 partial, err);
  }

  // The summed gradients into g.
  void gradients() {
    sur::mlp_update_kernel<false><<<sur::kUpdateBlocks, sur::kUpdateThreads, 0, stream>>>(adam_args(), partial, pieces,
                                                                                         chains.chain, chains.chainb);
    SCK(cudaGetLastError());
  }

  void adam(float lr) {
    ++adam_t;
    sur::AdamArgs a = adam_args();
    a.lr = lr;
    a.beta1 = 0.9f;
    a.beta2 = 0.999f;
    a.eps = 1e-8f;
    a.bc1 = (float)(1.0 - std::pow(0.9, (double)adam_t));
    a.bc2 = (float)(1.0 - std::pow(0.999, (double)adam_t));
    sur::mlp_update_kernel<true><<<sur::kUpdateBlocks, sur::kUpdateThreads, 0, stream>>>(a, partial, pieces,
                                                                                        chains.chain, chains.chainb);
    SCK(cudaGetLastError());
  }

  void make_dataset(int64_t n) {
    if (n == ds_n) return;
    if (n <= 0) throw std::invalid_argument("training set size must be positive");
    SCK(cudaStreamSynchronize(stream));
    if (ds_raw) {
      cudaFree(ds_raw);
      cudaFree(ds_target);
      allocs.erase(std::remove(allocs.begin(), allocs.end(), (void *)ds_raw), allocs.end());
      allocs.erase(std::remove(allocs.begin(), allocs.end(), (void *)ds_target), allocs.end());
    }
    ds_raw = alloc<float>((size_t)n * kSurIn);
    ds_target = alloc<float>((size_t)n);
    ds_n = n;
    sur::make_data_kernel<<<sur::grid_1d(n), 256, 0, stream>>>(data, 0, n, ds_raw, ds_target);
    SCK(cudaGetLastError());
  }
};

// FrameJob of a scan: node grid and source from amca_scan.
sur::FrameJob scan_job(const amca_scan &p) {
  sur::FrameJob j{};
  for (int a = 0; a < 3; ++a) {
    j.origin[a] = p.origin[a];
    j.nodes[a] = p.nodes[a];
  }
  j.spacing = p.spacing;
  j.length_scale = p.length_scale;
  j.frame_dt = p.frame_dt;
  j.time_scale = p.time_scale;
  j.nnodes = (int64_t)p.nodes[0] * p.nodes[1] * p.nodes[2];
  ScanSource &s = j.src;
  s.power = p.power;
  s.absorptivity = p.absorptivity;
  s.speed = p.speed;
  s.conductivity = p.conductivity;
  s.diffusivity = p.diffusivity;
  s.t0 = p.t0;
  s.t_cap = p.t_cap;
  s.x_start = p.x_start;
  s.x_turn = p.x_turn;
  s.y_line = p.y_line;
  s.z_top = p.z_top;
  s.hatch = p.hatch;
  s.track_time = p.track_time;
  s.ntracks = p.ntracks;
  return j;
}

void check_scan(const amca_scan &p) {
  for (int a = 0; a < 3; ++a)
    if (p.nodes[a] < 2) throw std::invalid_argument("scan: at least 2 nodes per axis");
  if (p.frames < 2) throw std::invalid_argument("scan: at least two frames");
  if (!(p.spacing > 0) || !(p.length_scale > 0) || !(p.frame_dt > 0) || !(p.time_scale > 0))
    throw std::invalid_argument("scan: spacing, length_scale, frame_dt and time_scale must be positive");
  if (p.ntracks > 1 && !(p.track_time > 0)) throw std::invalid_argument("scan: track_time must be positive");
}

// Frames of job.f0 .. job.f0 + job.nf - 1 into the job's ring: the FE field
// of the scan (model == nullptr) or the model with its fallback.
void produce_frames(ThermalModel *model, sur::FrameJob job, cudaStream_t s) {
  using namespace sur;
  const int64_t total = job.nnodes * job.nf;
  if (!model) {
    scan_frames_kernel<<<grid_1d(total), 256, 0, s>>>(job);
    SCK(cudaGetLastError());
    return;
  }
  fill_frames_kernel<<<grid_1d(total), 256, 0, s>>>(job);
  SCK(cudaGetLastError());
  const double h = job.spacing * job.length_scale;
  for (int a = 0; a < 3; ++a) {
    job.win_lo[a] = model->data.win_lo[a];
    job.win_hi[a] = model->data.win_hi[a];
    job.box[a] = (int)std::ceil((job.win_hi[a] - job.win_lo[a]) / h) + 2;
  }
  if (!job.counters) job.counters = model->counters;
  InferArgs ia{};
  ia.error = model->err;
  const CUtensorMap *tw = model->tw;
  const int sms = model->sms;
  const int f_end = job.f0 + job.nf;
  for (int f = job.f0; f < f_end; f += kJobFrames) {
    ia.job = job;
    ia.job.f0 = f;
    ia.job.nf = std::min(kJobFrames, f_end - f);
    // most queries the frames can have: a window clipped to the grid each
    int64_t most = ia.job.nf;
    for (int a = 0; a < 3; ++a) most *= std::min<int64_t>(job.box[a], job.nodes[a]);
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((most + 127) / 128, sms));
    mlp_infer_kernel<kSrcFrames><<<grid, kInferThreads, kInferSmem, s>>>(tw[0], tw[1], tw[2], tw[3], model->dev(), ia);
    SCK(cudaGetLastError());
  }
}

}  // namespace amca

struct amca_thermal {
  std::string err;
  std::unique_ptr<amca::ThermalModel> m;
};

namespace {

template <typename F>
int tguard(amca_thermal *h, F &&f) {
  try {
    f();
    if (h) h->err.clear();
    return AMCA_OK;
  } catch (const std::invalid_argument &e) {
    if (h) h->err = e.what();
    return AMCA_ERR_ARG;
  } catch (const std::exception &e) {
    if (h) h->err = e.what();
    return AMCA_ERR_CUDA;
  }
}

struct DeviceBuffers {
  std::vector<void *> p;
  void *get(size_t bytes) {
    void *q = nullptr;
    SCK(cudaMalloc(&q, std::max<size_t>(bytes, 1)));
    p.push_back(q);
    return q;
  }
  ~DeviceBuffers() {
    for (void *q : p) cudaFree(q);
  }
};

}  // namespace

namespace amca {

ThermalModel *thermal_model_of(void *handle) { return handle ? ((amca_thermal *)handle)->m.get() : nullptr; }

void fill_scan_frames(const amca_scan *scan, ThermalModel *model, double t_liq, double band, double thresh, int f0,
                      int nf, double *ring, int slots, unsigned long long *counters, cudaStream_t s) {
  sur::FrameJob job = scan_job(*scan);
  job.f0 = f0;
  job.nf = nf;
  job.ring = ring;
  job.slots = slots;
  job.t_liq = (float)t_liq;
  job.band = (float)band;
  job.thresh = (float)thresh;
  job.counters = counters;
  produce_frames(model, job, s);
}

}  // namespace amca

extern "C" {

int amca_thermal_create(int device, const amca_thermal_spec *spec, amca_thermal **out) {
  if (!spec || !out) return AMCA_ERR_ARG;
  *out = nullptr;
  std::unique_ptr<amca_thermal> h(new amca_thermal);
  const int rc = tguard(h.get(), [&] {
    if (!(spec->power_hi > spec->power_lo) || !(spec->speed_hi > spec->speed_lo) || !(spec->t_scale > 0))
      throw std::invalid_argument("amca_thermal_create: empty power or speed range, or t_scale <= 0");
    if (spec->log_output && !(spec->t_shift < spec->t0))
      throw std::invalid_argument("amca_thermal_create: a log output needs t_shift below t0");
    for (int a = 0; a < 3; ++a)
      if (!(spec->window_hi[a] > spec->window_lo[a]) || !(spec->near_hi[a] > spec->near_lo[a]))
        throw std::invalid_argument("amca_thermal_create: empty window or melt-pool box");
    amca::sur::DataSpec ds{};
    ds.seed = spec->seed;
    ds.p_lo = spec->power_lo;
    ds.p_hi = spec->power_hi;
    ds.v_lo = spec->speed_lo;
    ds.v_hi = spec->speed_hi;
    for (int a = 0; a < 3; ++a) {
      ds.win_lo[a] = spec->window_lo[a];
      ds.win_hi[a] = spec->window_hi[a];
      ds.near_lo[a] = spec->near_lo[a];
      ds.near_hi[a] = spec->near_hi[a];
    }
    ds.near = spec->near_fraction;
    ds.shell = spec->shell_fraction;
    ds.shell_lo = spec->shell_lo;
    ds.shell_hi = spec->shell_hi;
    if (!(ds.near >= 0) || !(ds.shell >= 0) || ds.near + ds.shell > 1.0)
      throw std::invalid_argument("amca_thermal_create: near_fraction + shell_fraction must lie in [0, 1]");
    ds.src.absorptivity = spec->absorptivity;
    ds.src.conductivity = spec->conductivity;
    ds.src.diffusivity = spec->diffusivity;
    ds.src.t0 = spec->t0;
    ds.src.t_cap = spec->t_cap;
    ds.src.ntracks = 1;
    ds.t_shift = (float)spec->t_shift;
    ds.t_scale = (float)spec->t_scale;
    ds.log_out = spec->log_output ? 1 : 0;
    h->m.reset(new amca::ThermalModel(device, ds, spec->fourier_sigma, spec->fourier_sigma_pv));
  });
  if (rc == AMCA_OK) *out = h.release();
  return rc;
}

int amca_thermal_train(amca_thermal *h, int64_t samples, int steps, int batch, double lr_max, double lr_min,
                       amca_thermal_train_stats *st) {
  if (!h || steps < 0) return AMCA_ERR_ARG;
  return tguard(h, [&] {
    amca::ThermalModel &m = *h->m;
    SCK(cudaSetDevice(m.device));
    m.make_dataset(samples);
    m.set_batch(batch);
    uint64_t a = 2654435761ull;
    while (amca::sur::gcd64(a, (uint64_t)samples) != 1) a += 2;
    DeviceBuffers tmp;
    double *acc = (double *)tmp.get(2 * sizeof(double));
    SCK(cudaMemsetAsync(acc, 0, 2 * sizeof(double), m.stream));
    SCK(cudaMemsetAsync(m.err, 0, sizeof(int), m.stream));
    const int edge = std::max(1, steps / 20);
    const int warm = std::max(1, steps / 50);
    SCK(cudaStreamSynchronize(m.stream));
    const auto t0 = std::chrono::steady_clock::now();
    for (int s = 0; s < steps; ++s) {
      m.forward_backward(m.ds_raw, m.ds_target, m.ds_n, m.seen % m.ds_n, a);
      m.seen += m.nb;
      const double frac = s < warm ? (double)(s + 1) / warm : (double)(s - warm) / std::max(1, steps - warm);
      const double lr = s < warm ? lr_max * frac : lr_min + 0.5 * (lr_max - lr_min) * (1.0 + std::cos(M_PI * frac));
      m.adam((float)lr);
      if (s < edge || s >= steps - edge)
        amca::sur::accum_loss_kernel<<<64, 256, 0, m.stream>>>(m.loss, m.nb, acc + (s < edge ? 0 : 1));
    }
    SCK(cudaStreamSynchronize(m.stream));
    const auto t1 = std::chrono::steady_clock::now();
    m.check_error();
    double hacc[2] = {0, 0};
    SCK(cudaMemcpy(hacc, acc, sizeof hacc, cudaMemcpyDeviceToHost));
    if (st) {
      st->steps = steps;
      st->samples_seen = m.seen;
      st->first_loss = hacc[0] / ((double)edge * m.nb);
      st->last_loss = hacc[1] / ((double)edge * m.nb);
      st->ms = std::chrono::duration<double, std::milli>(t1 - t0).count();
    }
  });
}

int amca_thermal_eval(amca_thermal *h, const float *raw, int64_t n, float *T, float *err) {
  if (!h || n < 0 || (n > 0 && (!raw || !T || !err))) return AMCA_ERR_ARG;
  return tguard(h, [&] {
    using namespace amca::sur;
    amca::ThermalModel &m = *h->m;
    SCK(cudaSetDevice(m.device));
    if (n == 0) return;
    DeviceBuffers tmp;
    float *d_raw = m.eval_buffer(n);  // allocating and freeing per call cost a 100,000-row call about a third of its time
    if (!d_raw) d_raw = (float *)tmp.get((size_t)n * (amca::kSurIn + 2) * 4);
    float *d_T = d_raw + (size_t)n * amca::kSurIn, *d_e = d_T + n;
    SCK(cudaMemcpyAsync(d_raw, raw, (size_t)n * amca::kSurIn * 4, cudaMemcpyHostToDevice, m.stream));
    SCK(cudaMemsetAsync(m.err, 0, sizeof(int), m.stream));
    InferArgs ia{};
    ia.nq = n;
    ia.raw = d_raw;
    ia.T = d_T;
    ia.err = d_e;
    ia.error = m.err;
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((n + 127) / 128, m.sms));
    mlp_infer_kernel<kSrcArray><<<grid, kInferThreads, kInferSmem, m.stream>>>(m.tw[0], m.tw[1], m.tw[2], m.tw[3],
                                                                               m.dev(), ia);
    SCK(cudaGetLastError());
    SCK(cudaMemcpyAsync(T, d_T, (size_t)n * 4, cudaMemcpyDeviceToHost, m.stream));
    SCK(cudaMemcpyAsync(err, d_e, (size_t)n * 4, cudaMemcpyDeviceToHost, m.stream));
    m.check_error();  // waits for the copies too
  });
}

int amca_thermal_gradients(amca_thermal *h, const float *raw, const float *target, int64_t n, float *grad,
                           float *pred) {
  if (!h || !raw || !target || !grad || n <= 0) return AMCA_ERR_ARG;
  return tguard(h, [&] {
    amca::ThermalModel &m = *h->m;
    SCK(cudaSetDevice(m.device));
    m.set_batch(n);
    SCK(cudaMemcpyAsync(m.braw, raw, (size_t)n * amca::kSurIn * 4, cudaMemcpyHostToDevice, m.stream));
    SCK(cudaMemcpyAsync(m.by, target, (size_t)n * 4, cudaMemcpyHostToDevice, m.stream));
    SCK(cudaMemsetAsync(m.err, 0, sizeof(int), m.stream));
    m.forward_backward(m.braw, m.by, n, 0, 1);
    m.gradients();
    SCK(cudaMemcpyAsync(grad, m.g, (size_t)m.L.total * 4, cudaMemcpyDeviceToHost, m.stream));
    if (pred) SCK(cudaMemcpyAsync(pred, m.pred, (size_t)n * 2 * 4, cudaMemcpyDeviceToHost, m.stream));
    m.check_error();  // waits for the copies too
  });
}

int64_t amca_thermal_param_count(void) { return amca::SurParamLayout().total; }

int amca_thermal_get_params(amca_thermal *h, float *params) {
  if (!h || !params) return AMCA_ERR_ARG;
  return tguard(h, [&] {
    SCK(cudaSetDevice(h->m->device));
    h->m->get_params(params);
  });
}

int amca_thermal_set_params(amca_thermal *h, const float *params) {
  if (!h || !params) return AMCA_ERR_ARG;
  return tguard(h, [&] {
    SCK(cudaSetDevice(h->m->device));
    h->m->set_params(params);
  });
}

int amca_thermal_get_encoding(amca_thermal *h, float *fourier, float *in_shift, float *in_scale, float *t_shift,
                              float *t_scale, int32_t *log_output) {
  if (!h) return AMCA_ERR_ARG;
  const amca::ThermalModel &m = *h->m;
  if (fourier) memcpy(fourier, m.fourier_h, sizeof m.fourier_h);
  if (in_shift) memcpy(in_shift, m.in_shift, sizeof m.in_shift);
  if (in_scale) memcpy(in_scale, m.in_scale, sizeof m.in_scale);
  if (t_shift) *t_shift = m.t_shift;
  if (t_scale) *t_scale = m.t_scale;
  if (log_output) *log_output = m.data.log_out;
  return AMCA_OK;
}

int amca_thermal_frames(amca_thermal *h, const amca_scan *scan, int32_t f0, int32_t nf, double t_liq, double band,
                        double thresh, double *frames, double *fe, int64_t *counts) {
  if (!h || !scan || !frames || f0 < 0 || nf < 1) return AMCA_ERR_ARG;
  return tguard(h, [&] {
    amca::ThermalModel &m = *h->m;
    SCK(cudaSetDevice(m.device));
    amca::check_scan(*scan);
    amca::sur::FrameJob job = amca::scan_job(*scan);
    job.f0 = f0;
    job.nf = nf;
    job.slots = nf;
    job.t_liq = (float)t_liq;
    job.band = (float)band;
    job.thresh = (float)thresh;
    DeviceBuffers tmp;
    double *ring = (double *)tmp.get((size_t)nf * job.nnodes * 8);
    job.ring = ring;
    SCK(cudaMemsetAsync(m.counters, 0, 4 * sizeof(unsigned long long), m.stream));
    SCK(cudaMemsetAsync(m.err, 0, sizeof(int), m.stream));
    amca::produce_frames(&m, job, m.stream);
    // slot of frame f is f % nf: copy back in frame order
    auto fetch = [&](double *dst) {
      for (int k = 0; k < nf; ++k) {
        const int slot = (f0 + k) % nf;
        SCK(cudaMemcpyAsync(dst + (size_t)k * job.nnodes, ring + (size_t)slot * job.nnodes, job.nnodes * 8,
                            cudaMemcpyDeviceToHost, m.stream));
      }
    };
    fetch(frames);
    unsigned long long c[4] = {0, 0, 0, 0};
    SCK(cudaMemcpyAsync(c, m.counters, sizeof c, cudaMemcpyDeviceToHost, m.stream));
    if (fe) {
      amca::produce_frames(nullptr, job, m.stream);
      fetch(fe);
    }
    SCK(cudaStreamSynchronize(m.stream));
    m.check_error();
    if (counts)
      for (int i = 0; i < 3; ++i) counts[i] = (int64_t)c[i];
  });
}

const char *amca_thermal_last_error(const amca_thermal *h) { return h ? h->err.c_str() : "null handle"; }

void amca_thermal_destroy(amca_thermal *h) { delete h; }

}  // extern "C"
