// pbf_learned.cu — the learned lambda warm start: a per-particle MLP
// 8 -> 64 -> 64 -> 1 (SiLU) with BF16 weights and activations and FP32
// accumulation, run and trained with hand-written mma.sync.m16n8k16 kernels.
//
// The reference solves with a fixed number of plain PBF iterations
// (src/simulator/PBF/PBF.ts:417-431) and recomputes lambda from scratch in
// each (pressureConstrain.ts:80-83), so there is no lambda to warm-start in
// the reference itself.  Here the network predicts an effective multiplier
// lambda_hat_i; one projection with it (the ConstrainSolve formula with
// lambda_hat in place of lambda) replaces the first iterations.  Its training
// target is the sum of the multipliers of the plain solver's iterations in
// the same substep: dp is linear in lambda for fixed positions, so one
// projection with the sum reproduces the plain iterations' cumulative
// correction to first order.
//
// Tiles: a warp owns 16 particles (rows).  The D fragment of one layer is the
// A fragment of the next (no shared-memory round trip); weights are staged
// in shared memory, transposed so every B-fragment register is one 32-bit
// load.  Weight gradients (H1^T dZ2, X^T dZ1) are mma.sync products over the
// rows of a 64-row block chunk, read through shared-memory transposes.
#include <cmath>
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/pbf_gb300.h"
#include "pbf_device.cuh"
#include "pbf_kernels.h"
#include "pbf_mlp.cuh"

namespace pbf {
namespace {

using namespace mlp;

constexpr int kInferThreads = 128;

// Inference: lambda_hat for each row (particle) of feat; also starts lam_sum.
// Persistent: the weights are staged once per CTA, each warp then walks
// 16-row tiles.  With xl given, writes xl[r] = (xs[r].xyz, lambda_hat) (the
// packed record the step's delta-p pass gathers) instead of lambda[r].
__global__ void __launch_bounds__(kInferThreads) k_mlp_infer(const float* __restrict__ P, Norm nm,
                                                            const float* __restrict__ feat, uint32_t rows,
                                                            float* __restrict__ lambda, float* __restrict__ lam_sum,
                                                            const float4* __restrict__ xs, float4* __restrict__ xl) {
  __shared__ __align__(16) uint16_t sW1t[kH * kW1S];
  __shared__ __align__(16) uint16_t sW2t[kH * kW2S];
  __shared__ float sB1[kH], sB2[kH], sW3[kH];
  stage_weights(P, sW1t, sW2t, nullptr);
  for (int q = threadIdx.x; q < kH; q += blockDim.x) {
    sB1[q] = P[OFF_B1 + q];
    sB2[q] = P[OFF_B2 + q];
    sW3[q] = P[OFF_W3 + q];
  }
  __syncthreads();
  const float b3 = P[OFF_B3];
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t tile = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); tile * 16 < rows; tile += warps) {
    uint32_t r0 = tile * 16;
    float xg[2], x8[2];
    load_inputs(feat, nm, rows, r0, xg, x8);
    Fwd F;
    forward_tile(xg, x8, sW1t, sW2t, sB1, sB2, sW3, b3, F);
    if (t == 0) {
      uint32_t ra = r0 + g, rb = r0 + g + 8;
      if (ra < rows) {
        float l = F.y0 * nm.lam_scale;
        if (xl) {
          float4 x = xs[ra];
          xl[ra] = make_float4(x.x, x.y, x.z, l);
        } else {
          lambda[ra] = l;
        }
        if (lam_sum) lam_sum[ra] = l;
      }
      if (rb < rows) {
        float l = F.y8 * nm.lam_scale;
        if (xl) {
          float4 x = xs[rb];
          xl[rb] = make_float4(x.x, x.y, x.z, l);
        } else {
          lambda[rb] = l;
        }
        if (lam_sum) lam_sum[rb] = l;
      }
    }
  }
}

constexpr int kTrainWarps = 4;
constexpr int kTrainRows = 16 * kTrainWarps;  // rows per block chunk
constexpr int kTrainSmem = 2 * (kH * kW1S + 3 * kH * kW2S + kTrainRows * kW1S + 3 * kTrainRows * kW2S) +
                           4 * (3 * kH);

// One forward + backward over `rows` training rows: accumulates the loss
// (sum of squared errors) and the gradient of mean((y - t/lam_scale)^2) into
// G (flat layout, FP32, atomically across blocks).
__global__ void __launch_bounds__(32 * kTrainWarps) k_mlp_grad(const float* __restrict__ P, Norm nm,
                                                               const float* __restrict__ feat,
                                                               const float* __restrict__ target, uint32_t rows,
                                                               float inv_batch, float* __restrict__ G,
                                                               float* __restrict__ loss) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint16_t* sW1t = reinterpret_cast<uint16_t*>(smem);
  uint16_t* sW2t = sW1t + kH * kW1S;
  uint16_t* sW2 = sW2t + kH * kW2S;
  uint16_t* sX = sW2 + kH * kW2S;         // [rows][kW1S] normalised inputs (bf16), k 8..15 zero
  uint16_t* sH1 = sX + kTrainRows * kW1S;  // [rows][kW2S]
  uint16_t* sDZ2 = sH1 + kTrainRows * kW2S;
  uint16_t* sDZ1 = sDZ2 + kTrainRows * kW2S;
  float* sB1 = reinterpret_cast<float*>(sDZ1 + kTrainRows * kW2S);
  float* sB2 = sB1 + kH;
  float* sW3 = sB2 + kH;
  stage_weights(P, sW1t, sW2t, sW2);
  for (int q = threadIdx.x; q < kH; q += blockDim.x) {
    sB1[q] = P[OFF_B1 + q];
    sB2[q] = P[OFF_B2 + q];
    sW3[q] = P[OFF_W3 + q];
  }
  for (int q = threadIdx.x; q < kTrainRows * kW1S; q += blockDim.x) sX[q] = 0;
  __syncthreads();
  const float b3 = P[OFF_B3];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;

  // gradient accumulators kept in registers across the block's chunks
  float gW2[8][4];  // output tiles (mt, nt) with (mt*8+nt) % 4 == warp
  float gW1[2][4];  // dW1 n-tiles 2*warp, 2*warp+1
  float gB1[8][2], gB2[8][2], gW3[8][2], gB3 = 0.0f, lsum = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) gW2[i][q] = 0.0f;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) gW1[i][q] = 0.0f;
#pragma unroll
  for (int j = 0; j < 8; ++j) gB1[j][0] = gB1[j][1] = gB2[j][0] = gB2[j][1] = gW3[j][0] = gW3[j][1] = 0.0f;

  for (uint32_t chunk = blockIdx.x; chunk * kTrainRows < rows; chunk += gridDim.x) {
    const uint32_t r0 = chunk * kTrainRows + 16 * warp;
    float xg[2], x8[2];
    load_inputs(feat, nm, rows, r0, xg, x8);
    Fwd F;
    forward_tile(xg, x8, sW1t, sW2t, sB1, sB2, sW3, b3, F);
    const uint32_t ra = r0 + g, rb = r0 + g + 8;
    float tg = (ra < rows) ? target[ra] / nm.lam_scale : 0.0f;
    float t8 = (rb < rows) ? target[rb] / nm.lam_scale : 0.0f;
    float eg = (ra < rows) ? F.y0 - tg : 0.0f;
    float e8 = (rb < rows) ? F.y8 - t8 : 0.0f;
    if (t == 0) lsum += eg * eg + e8 * e8;
    float dyg = 2.0f * eg * inv_batch, dy8 = 2.0f * e8 * inv_batch;
    if (t == 0) gB3 += dyg + dy8;
    // dZ2 = dy w3^T * silu'(z2); dw3 += h2^T dy; db2 += sum dZ2
    float dz2[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float w0 = sW3[8 * j + 2 * t], w1 = sW3[8 * j + 2 * t + 1];
      dz2[j][0] = dyg * w0 * dsilu_f(F.z2[j][0]);
      dz2[j][1] = dyg * w1 * dsilu_f(F.z2[j][1]);
      dz2[j][2] = dy8 * w0 * dsilu_f(F.z2[j][2]);
      dz2[j][3] = dy8 * w1 * dsilu_f(F.z2[j][3]);
      gW3[j][0] += F.h2[j][0] * dyg + F.h2[j][2] * dy8;
      gW3[j][1] += F.h2[j][1] * dyg + F.h2[j][3] * dy8;
      gB2[j][0] += dz2[j][0] + dz2[j][2];
      gB2[j][1] += dz2[j][1] + dz2[j][3];
    }
    // dH1 = dZ2 W2^T (mma; A = dZ2 from the D layout, B from W2 rows)
    uint32_t ad[4][4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      ad[s][0] = pack_bf16(dz2[2 * s][0], dz2[2 * s][1]);
      ad[s][1] = pack_bf16(dz2[2 * s][2], dz2[2 * s][3]);
      ad[s][2] = pack_bf16(dz2[2 * s + 1][0], dz2[2 * s + 1][1]);
      ad[s][3] = pack_bf16(dz2[2 * s + 1][2], dz2[2 * s + 1][3]);
    }
    float dz1[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      int n = 8 * j + g;
      float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        uint32_t b0 = *reinterpret_cast<const uint32_t*>(sW2 + n * kW2S + 16 * s + 2 * t);
        uint32_t b1 = *reinterpret_cast<const uint32_t*>(sW2 + n * kW2S + 16 * s + 8 + 2 * t);
        mma16816(d, ad[s], b0, b1);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) dz1[j][q] = d[q] * dsilu_f(F.z1[j][q]);
      gB1[j][0] += dz1[j][0] + dz1[j][2];
      gB1[j][1] += dz1[j][1] + dz1[j][3];
    }
    // stage X, H1, dZ2, dZ1 of this warp's 16 rows for the weight-gradient products
    __syncthreads();  // previous chunk's readers are done
    {
      const int rl = 16 * warp + g;
      uint16_t* xr = sX + rl * kW1S;
      *reinterpret_cast<uint32_t*>(xr + 2 * t) = pack_bf16(xg[0], xg[1]);
      *reinterpret_cast<uint32_t*>(xr + 8 * kW1S + 2 * t) = pack_bf16(x8[0], x8[1]);
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        *reinterpret_cast<uint32_t*>(sH1 + rl * kW2S + 16 * s + 2 * t) = F.a2[s][0];
        *reinterpret_cast<uint32_t*>(sH1 + (rl + 8) * kW2S + 16 * s + 2 * t) = F.a2[s][1];
        *reinterpret_cast<uint32_t*>(sH1 + rl * kW2S + 16 * s + 8 + 2 * t) = F.a2[s][2];
        *reinterpret_cast<uint32_t*>(sH1 + (rl + 8) * kW2S + 16 * s + 8 + 2 * t) = F.a2[s][3];
        *reinterpret_cast<uint32_t*>(sDZ2 + rl * kW2S + 16 * s + 2 * t) = ad[s][0];
        *reinterpret_cast<uint32_t*>(sDZ2 + (rl + 8) * kW2S + 16 * s + 2 * t) = ad[s][1];
        *reinterpret_cast<uint32_t*>(sDZ2 + rl * kW2S + 16 * s + 8 + 2 * t) = ad[s][2];
        *reinterpret_cast<uint32_t*>(sDZ2 + (rl + 8) * kW2S + 16 * s + 8 + 2 * t) = ad[s][3];
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        *reinterpret_cast<uint32_t*>(sDZ1 + rl * kW2S + 8 * j + 2 * t) = pack_bf16(dz1[j][0], dz1[j][1]);
        *reinterpret_cast<uint32_t*>(sDZ1 + (rl + 8) * kW2S + 8 * j + 2 * t) = pack_bf16(dz1[j][2], dz1[j][3]);
      }
    }
    __syncthreads();
    // dW2 = H1^T dZ2 over the chunk's 64 rows: M = hidden1, N = hidden2, K = rows
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int tile = warp + 4 * i, mt = tile >> 3, nt = tile & 7;
#pragma unroll
      for (int kk = 0; kk < kTrainRows / 16; ++kk) {
        const int rk = 16 * kk + 2 * t, m0 = 16 * mt + g, nn = 8 * nt + g;
        uint32_t a[4];
        a[0] = pack_raw(sH1[rk * kW2S + m0], sH1[(rk + 1) * kW2S + m0]);
        a[1] = pack_raw(sH1[rk * kW2S + m0 + 8], sH1[(rk + 1) * kW2S + m0 + 8]);
        a[2] = pack_raw(sH1[(rk + 8) * kW2S + m0], sH1[(rk + 9) * kW2S + m0]);
        a[3] = pack_raw(sH1[(rk + 8) * kW2S + m0 + 8], sH1[(rk + 9) * kW2S + m0 + 8]);
        uint32_t b0 = pack_raw(sDZ2[rk * kW2S + nn], sDZ2[(rk + 1) * kW2S + nn]);
        uint32_t b1 = pack_raw(sDZ2[(rk + 8) * kW2S + nn], sDZ2[(rk + 9) * kW2S + nn]);
        mma16816(gW2[i], a, b0, b1);
      }
    }
    // dW1 = X^T dZ1: M = inputs (16, rows 8..15 padding), N = hidden1, K = rows
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int nt = 2 * warp + i;
#pragma unroll
      for (int kk = 0; kk < kTrainRows / 16; ++kk) {
        const int rk = 16 * kk + 2 * t, nn = 8 * nt + g;
        uint32_t a[4];
        a[0] = pack_raw(sX[rk * kW1S + g], sX[(rk + 1) * kW1S + g]);
        a[1] = pack_raw(sX[rk * kW1S + g + 8], sX[(rk + 1) * kW1S + g + 8]);
        a[2] = pack_raw(sX[(rk + 8) * kW1S + g], sX[(rk + 9) * kW1S + g]);
        a[3] = pack_raw(sX[(rk + 8) * kW1S + g + 8], sX[(rk + 9) * kW1S + g + 8]);
        uint32_t b0 = pack_raw(sDZ1[rk * kW2S + nn], sDZ1[(rk + 1) * kW2S + nn]);
        uint32_t b1 = pack_raw(sDZ1[(rk + 8) * kW2S + nn], sDZ1[(rk + 9) * kW2S + nn]);
        mma16816(gW1[i], a, b0, b1);
      }
    }
  }
  // flush: weight-gradient tiles (one owner per element), then the
  // per-column sums reduced over the 8 row groups of the warp
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int tile = warp + 4 * i, mt = tile >> 3, nt = tile & 7;
    const int m0 = 16 * mt + g, n0 = 8 * nt + 2 * t;
    atomicAdd(G + OFF_W2 + m0 * kH + n0, gW2[i][0]);
    atomicAdd(G + OFF_W2 + m0 * kH + n0 + 1, gW2[i][1]);
    atomicAdd(G + OFF_W2 + (m0 + 8) * kH + n0, gW2[i][2]);
    atomicAdd(G + OFF_W2 + (m0 + 8) * kH + n0 + 1, gW2[i][3]);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int n0 = 8 * (2 * warp + i) + 2 * t;
    if (g < kIn) {
      atomicAdd(G + OFF_W1 + g * kH + n0, gW1[i][0]);
      atomicAdd(G + OFF_W1 + g * kH + n0 + 1, gW1[i][1]);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      float v1 = gB1[j][c], v2 = gB2[j][c], v3 = gW3[j][c];
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) {
        v1 += __shfl_xor_sync(0xffffffffu, v1, o);
        v2 += __shfl_xor_sync(0xffffffffu, v2, o);
        v3 += __shfl_xor_sync(0xffffffffu, v3, o);
      }
      if (g == 0) {
        atomicAdd(G + OFF_B1 + 8 * j + 2 * t + c, v1);
        atomicAdd(G + OFF_B2 + 8 * j + 2 * t + c, v2);
        atomicAdd(G + OFF_W3 + 8 * j + 2 * t + c, v3);
      }
    }
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    gB3 += __shfl_xor_sync(0xffffffffu, gB3, o);
    lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
  }
  if (lane == 0) {
    atomicAdd(G + OFF_B3, gB3);
    atomicAdd(loss, lsum);
  }
}

// Adam (Kingma & Ba 2015) on the flat FP32 parameters.  Also hands the batch's
// loss over and clears gradient and loss for the next batch (a memset between
// the batches otherwise).
__global__ void k_adam(float* __restrict__ P, float* __restrict__ G, float* __restrict__ M, float* __restrict__ V,
                       int n, float lr, float b1, float b2, float eps, float c1, float c2,
                       float* __restrict__ batch_loss) {
  chain_begin(P, G, M, V);
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == n) {  // the loss follows the gradient
    *batch_loss = G[i];
    G[i] = 0.0f;
  }
  if (i >= n) return;
  float gr = G[i];
  float m = b1 * M[i] + (1.0f - b1) * gr;
  float v = b2 * V[i] + (1.0f - b2) * gr * gr;
  M[i] = m;
  V[i] = v;
  P[i] -= lr * (m / c1) / (sqrtf(v / c2) + eps);
  G[i] = 0.0f;
}

// The draws of a Fisher-Yates shuffle of `rows` entries from the splitmix64
// stream: entry i (from the last down to 1) swaps with draw[i] = value % (i + 1)
// of the stream's value rows - i.  The stream is a hash of a counter, so every
// draw is found by itself; the host only swaps.  At 200,000 rows the 64-bit
// remainders took the host 0.9 ms of a training; here they take 5 us, the swaps
// and the copies both ways about 0.25 ms.
__global__ void k_shuffle_draws(uint64_t seed, uint32_t rows, uint32_t* __restrict__ draw) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows) return;
  uint64_t z = seed + (uint64_t)(rows - i) * 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  z ^= z >> 31;
  draw[i] = (uint32_t)(z % (uint64_t)(i + 1u));
}

// Training rows in their shuffled order: row k of the training is the caller's
// row perm[k].  The inverse first, then each uploaded chunk of the caller's
// rows (starting at row0) goes to its places: 36 bytes read in order and
// written to scattered 32-byte rows, where the host moved them one by one
// through a second copy of the data.
__global__ void k_invert(const uint32_t* __restrict__ perm, uint32_t rows, uint32_t* __restrict__ place) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < rows) place[perm[i]] = i;
}
__global__ void k_place_rows(const float4* __restrict__ feat, const float* __restrict__ target,
                             const uint32_t* __restrict__ place, uint32_t row0, uint32_t rows,
                             float4* __restrict__ feat_out, float* __restrict__ target_out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows) return;
  const size_t k = place[row0 + i];
  feat_out[2 * k] = feat[2 * (size_t)i];
  feat_out[2 * k + 1] = feat[2 * (size_t)i + 1];
  target_out[k] = target[i];
}

Norm norm_of(const pbf_mlp& m) {
  Norm n;
  for (int k = 0; k < kIn; ++k) {
    n.mean[k] = m.feat_mean[k];
    n.inv_std[k] = m.feat_inv_std[k];
  }
  n.lam_scale = m.lam_scale;
  return n;
}

bool grad_kernel_ready = false;
cudaError_t ensure_grad_kernel() {
  if (grad_kernel_ready) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, kTrainSmem);
  if (e == cudaSuccess) grad_kernel_ready = true;
  return e;
}

}  // namespace

// Fallback decision from the last learned iteration's statistics; resets
// them for the next substep.
__global__ void k_fallback_decide(SolveStats* stats, float bound, int* flag, uint32_t* fallbacks, float* last_mean) {
  unsigned cnt = stats->count;
  double mean = cnt ? (double)stats->sum_fx / 1048576.0 / (double)cnt : 0.0;
  int f = mean > (double)bound ? 1 : 0;
  *flag = f;
  if (f) atomicAdd(fallbacks, 1u);
  *last_mean = (float)mean;
  stats->max_bits = 0u;
  stats->count = 0u;
  stats->sum_fx = 0ull;
}

// The adaptive iteration's test: the position update runs (*flag = 1) when
// the mean compression at the iteration's start exceeds the bound; counts[0]
// counts the tests, counts[1] the updates run.  Resets the statistics.
__global__ void k_iterate_decide(SolveStats* stats, float bound, int* flag, uint32_t* counts, float* last_mean) {
  unsigned cnt = stats->count;
  double mean = cnt ? (double)stats->sum_fx / 1048576.0 / (double)cnt : 0.0;
  int f = mean > (double)bound ? 1 : 0;
  *flag = f;
  counts[0] += 1u;
  counts[1] += (uint32_t)f;
  *last_mean = (float)mean;
  stats->max_bits = 0u;
  stats->count = 0u;
  stats->sum_fx = 0ull;
}

// Lagged iteration control: this substep's iterations run (*flag = 1) when
// the previous substep's final mean compression exceeded the threshold;
// counts[0] counts the decisions, counts[1] the substeps that iterated.
__global__ void k_lagged_decide(const float* last_mean, float threshold, int* flag, uint32_t* counts) {
  const int f = *last_mean > threshold ? 1 : 0;
  *flag = f;
  counts[0] += 1u;
  counts[1] += (uint32_t)f;
}

// Records a plain solve's in-solve mean compression (trace capture): running
// max and sum over substeps, then resets the statistics.
__global__ void k_stats_record(SolveStats* stats, float* rec) {
  unsigned cnt = stats->count;
  float mean = cnt ? (float)((double)stats->sum_fx / 1048576.0 / (double)cnt) : 0.0f;
  atomicMax(reinterpret_cast<unsigned int*>(rec), __float_as_uint(mean));
  rec[1] += mean;
  rec[2] += 1.0f;
  stats->max_bits = 0u;
  stats->count = 0u;
  stats->sum_fx = 0ull;
}

__device__ __forceinline__ uint32_t mix_id(uint32_t x) {
  x ^= x >> 16;
  x *= 0x7feb352dU;
  x ^= x >> 15;
  x *= 0x846ca68bU;
  x ^= x >> 16;
  return x;
}

__global__ void k_trace_append(uint32_t n, const uint32_t* __restrict__ ids, const float4* __restrict__ feat,
                               const float* __restrict__ lam_sum, uint32_t stride, uint32_t salt,
                               float* __restrict__ tf, float* __restrict__ tt, uint32_t* count, uint32_t cap) {
  uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  if (mix_id(ids[t] ^ salt) % stride != 0) return;
  uint32_t r = atomicAdd(count, 1u);
  if (r >= cap) return;
  float4 a = feat[2 * t], b = feat[2 * t + 1];
  float* o = tf + 8 * (size_t)r;
  o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w;
  o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
  tt[r] = lam_sum[t];
}

// ---- launch helpers used by the step driver -------------------------------------------
cudaError_t launch_fallback_decide(SolveStats* stats, float bound, int* flag, uint32_t* fallbacks, float* last_mean,
                                   cudaStream_t st) {
  k_fallback_decide<<<1, 1, 0, st>>>(stats, bound, flag, fallbacks, last_mean);
  return cudaGetLastError();
}
cudaError_t launch_iterate_decide(SolveStats* stats, float bound, int* flag, uint32_t* counts, float* last_mean,
                                  cudaStream_t st) {
  k_iterate_decide<<<1, 1, 0, st>>>(stats, bound, flag, counts, last_mean);
  return cudaGetLastError();
}
cudaError_t launch_lagged_decide(const float* last_mean, float threshold, int* flag, uint32_t* counts,
                                 cudaStream_t st) {
  k_lagged_decide<<<1, 1, 0, st>>>(last_mean, threshold, flag, counts);
  return cudaGetLastError();
}
cudaError_t launch_stats_record(SolveStats* stats, float* rec, cudaStream_t st) {
  k_stats_record<<<1, 1, 0, st>>>(stats, rec);
  return cudaGetLastError();
}
cudaError_t launch_trace_append(uint32_t n, const uint32_t* ids, const float4* feat, const float* lam_sum,
                                uint32_t stride, uint32_t salt, float* tf, float* tt, uint32_t* count, uint32_t cap,
                                cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  k_trace_append<<<(n + 255) / 256, 256, 0, st>>>(n, ids, feat, lam_sum, stride, salt, tf, tt, count, cap);
  return cudaGetLastError();
}

cudaError_t launch_mlp_infer(const float* d_params, const pbf_mlp& model, const float* d_feat, uint32_t rows,
                             float* d_lambda, float* d_lam_sum, cudaStream_t st, const float4* d_xs, float4* d_xl) {
  if (rows == 0) return cudaSuccess;
  uint32_t tiles = (rows + 15) / 16;
  uint32_t blocks = (tiles + 3) / 4;
  if (blocks > 152u * 8u) blocks = 152u * 8u;
  k_mlp_infer<<<blocks, kInferThreads, 0, st>>>(d_params, norm_of(model), d_feat, rows, d_lambda, d_lam_sum, d_xs,
                                                d_xl);
  return cudaGetLastError();
}

cudaError_t launch_mlp_grad(const float* d_params, const pbf_mlp& model, const float* d_feat, const float* d_target,
                            uint32_t rows, float* d_grad, float* d_loss, cudaStream_t st) {
  if (rows == 0) return cudaSuccess;
  cudaError_t e = ensure_grad_kernel();
  if (e != cudaSuccess) return e;
  uint32_t chunks = (rows + kTrainRows - 1) / kTrainRows;
  uint32_t blocks = chunks < 152u * 4u ? chunks : 152u * 4u;
  k_mlp_grad<<<blocks, 32 * kTrainWarps, kTrainSmem, st>>>(d_params, norm_of(model), d_feat, d_target, rows,
                                                           1.0f / (float)rows, d_grad, d_loss);
  return cudaGetLastError();
}

cudaError_t launch_adam(float* P, float* G, float* M, float* V, int step, float lr, float* batch_loss,
                        cudaStream_t st) {
  const float b1 = 0.9f, b2 = 0.999f;
  float c1 = 1.0f - std::pow(b1, (float)step), c2 = 1.0f - std::pow(b2, (float)step);
  return launch_chain(true, k_adam, (PBF_MLP_PARAMS + 1 + 255) / 256, 256, 0, st, P, G, M, V, PBF_MLP_PARAMS, lr, b1,
                      b2, 1e-8f, c1, c2, batch_loss);
}

}  // namespace pbf

using namespace pbf;

namespace {
uint64_t splitmix(uint64_t& s) {
  s += 0x9e3779b97f4a7c15ull;
  uint64_t z = s;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
double unif(uint64_t& s) { return (double)(splitmix(s) >> 11) * (1.0 / 9007199254740992.0); }
}  // namespace

extern "C" {

int pbf_mlp_init(pbf_mlp* m, uint64_t seed) {
  if (!m) return PBF_EINVAL;
  std::memset(m, 0, sizeof(*m));
  uint64_t s = seed;
  // Glorot-uniform weights, zero biases, identity normalisation
  double l1 = std::sqrt(6.0 / (kIn + kH)), l2 = std::sqrt(6.0 / (kH + kH)), l3 = std::sqrt(6.0 / (kH + 1));
  for (int i = 0; i < kIn * kH; ++i) m->params[OFF_W1 + i] = (float)((2.0 * unif(s) - 1.0) * l1);
  for (int i = 0; i < kH * kH; ++i) m->params[OFF_W2 + i] = (float)((2.0 * unif(s) - 1.0) * l2);
  for (int i = 0; i < kH; ++i) m->params[OFF_W3 + i] = (float)((2.0 * unif(s) - 1.0) * l3);
  for (int k = 0; k < kIn; ++k) m->feat_inv_std[k] = 1.0f;
  m->lam_scale = 1.0f;
  return PBF_OK;
}

int pbf_mlp_fit_normalization(pbf_mlp* m, const float* feat, const float* target, uint32_t rows) {
  if (!m || !feat || !target || rows == 0) return PBF_EINVAL;
  // two features a vector, each sum in row order
  typedef double pair __attribute__((vector_size(16)));
  pair sum[kIn / 2] = {}, sum2[kIn / 2] = {};
  double tsq = 0;
  for (uint32_t r = 0; r < rows; ++r) {
    const float* f = feat + 8 * (size_t)r;
    for (int k = 0; k < kIn / 2; ++k) {
      const pair v = {(double)f[2 * k], (double)f[2 * k + 1]};
      sum[k] += v;
      sum2[k] += v * v;
    }
    tsq += (double)target[r] * target[r];
  }
  double mean[kIn], sq[kIn];
  for (int k = 0; k < kIn; ++k) {
    mean[k] = sum[k / 2][k % 2];
    sq[k] = sum2[k / 2][k % 2];
  }
  for (int k = 0; k < kIn; ++k) {
    double mu = mean[k] / rows, var = sq[k] / rows - mu * mu;
    m->feat_mean[k] = (float)mu;
    m->feat_inv_std[k] = (float)(var > 1e-20 ? 1.0 / std::sqrt(var) : 1.0);
  }
  double rms = std::sqrt(tsq / rows);
  m->lam_scale = (float)(rms > 0 ? rms : 1.0);
  return PBF_OK;
}

int pbf_mlp_forward_ex(const pbf_mlp* m, const float* feat, uint32_t rows, float* out, uint32_t kernel) {
  if (!m || (!feat && rows) || (!out && rows)) return PBF_EINVAL;
  if (kernel != PBF_MLP_KERNEL_MMA_SYNC && kernel != PBF_MLP_KERNEL_TCGEN05) return PBF_EINVAL;
  if (rows == 0) return PBF_OK;
  float *dP = nullptr, *dF = nullptr, *dO = nullptr;
  uint32_t* dE = nullptr;
  uint32_t herr = 0;
  cudaError_t e = cudaMalloc(&dP, sizeof(m->params));
  if (e == cudaSuccess) e = cudaMalloc(&dF, (size_t)rows * 8 * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&dO, (size_t)rows * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&dE, sizeof(uint32_t));
  if (e == cudaSuccess) e = cudaMemset(dE, 0, sizeof(uint32_t));
  if (e == cudaSuccess) e = cudaMemcpy(dP, m->params, sizeof(m->params), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dF, feat, (size_t)rows * 8 * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    e = kernel == PBF_MLP_KERNEL_TCGEN05 ? launch_mlp_infer_tc(dP, *m, dF, rows, dO, nullptr, 0, nullptr, nullptr, dE)
                                         : launch_mlp_infer(dP, *m, dF, rows, dO, nullptr, 0);
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, dO, (size_t)rows * sizeof(float), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(&herr, dE, sizeof(uint32_t), cudaMemcpyDeviceToHost);
  cudaFree(dP);
  cudaFree(dF);
  cudaFree(dO);
  cudaFree(dE);
  if (e != cudaSuccess) return PBF_ECUDA;
  return herr ? PBF_ETIMEOUT : PBF_OK;
}

int pbf_mlp_forward(const pbf_mlp* m, const float* feat, uint32_t rows, float* out) {
  return pbf_mlp_forward_ex(m, feat, rows, out, PBF_MLP_KERNEL_MMA_SYNC);
}

int pbf_mlp_gradient(const pbf_mlp* m, const float* feat, const float* target, uint32_t rows, float* grad,
                     float* loss) {
  return pbf_mlp_gradient_ex(m, feat, target, rows, grad, loss, PBF_MLP_TRAIN_TCGEN05);
}

int pbf_mlp_gradient_ex(const pbf_mlp* m, const float* feat, const float* target, uint32_t rows, float* grad,
                        float* loss, uint32_t kernel) {
  if (!m || !feat || !target || !grad || rows == 0) return PBF_EINVAL;
  if (kernel != PBF_MLP_TRAIN_TCGEN05 && kernel != PBF_MLP_TRAIN_MMA_SYNC) return PBF_EINVAL;
  float *dP = nullptr, *dF = nullptr, *dT = nullptr, *dG = nullptr;
  cudaError_t e = cudaMalloc(&dP, sizeof(m->params));
  if (e == cudaSuccess) e = cudaMalloc(&dF, (size_t)rows * 8 * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&dT, (size_t)rows * sizeof(float));
  // gradient, loss, then the device error word
  if (e == cudaSuccess) e = cudaMalloc(&dG, (PBF_MLP_PARAMS + 2) * sizeof(float));
  if (e == cudaSuccess) e = cudaMemcpy(dP, m->params, sizeof(m->params), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dF, feat, (size_t)rows * 8 * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dT, target, (size_t)rows * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(dG, 0, (PBF_MLP_PARAMS + 2) * sizeof(float));
  uint32_t* dErr = reinterpret_cast<uint32_t*>(dG + PBF_MLP_PARAMS + 1);
  if (e == cudaSuccess)
    e = kernel == PBF_MLP_TRAIN_TCGEN05 ? launch_mlp_grad_tc(dP, *m, dF, dT, rows, dG, dG + PBF_MLP_PARAMS, dErr, 0)
                                        : launch_mlp_grad(dP, *m, dF, dT, rows, dG, dG + PBF_MLP_PARAMS, 0);
  float l = 0.0f;
  uint32_t herr = 0;
  if (e == cudaSuccess) e = cudaMemcpy(grad, dG, PBF_MLP_PARAMS * sizeof(float), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(&l, dG + PBF_MLP_PARAMS, sizeof(float), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(&herr, dErr, sizeof(uint32_t), cudaMemcpyDeviceToHost);
  if (loss) *loss = l / (float)rows;
  cudaFree(dP);
  cudaFree(dF);
  cudaFree(dT);
  cudaFree(dG);
  if (e != cudaSuccess) return PBF_ECUDA;
  return herr ? PBF_ETIMEOUT : PBF_OK;
}

// Mini-batch Adam on rows (feat, target) held on the host; shuffled once by
// a seeded permutation.  Returns the mean loss of the last epoch.
int pbf_mlp_train(pbf_mlp* m, const float* feat, const float* target, uint32_t rows, const pbf_train_config* tc,
                  float* final_loss) {
  if (!m || !feat || !target || !tc || rows == 0 || tc->batch == 0) return PBF_EINVAL;
  if (tc->kernel != PBF_MLP_TRAIN_TCGEN05 && tc->kernel != PBF_MLP_TRAIN_MMA_SYNC) return PBF_EINVAL;
  std::vector<uint32_t> draw(rows), perm(rows);
  // one allocation: parameters and moments, gradient + loss + error word + the
  // last batch's loss, the shuffled rows, the shuffle and its inverse, and a
  // chunk of the caller's rows on its way to them
  const uint32_t chunk = rows < (1u << 20) ? rows : (1u << 20);
  size_t bytes = 0;
  auto place = [&](size_t count) {
    const size_t at = bytes;
    bytes += (count * sizeof(float) + 255) / 256 * 256;
    return at;
  };
  const size_t oP = place(PBF_MLP_PARAMS), oM = place(PBF_MLP_PARAMS), oV = place(PBF_MLP_PARAMS),
               oG = place(PBF_MLP_PARAMS + 3), cleared = bytes, oF = place((size_t)rows * 8), oT = place(rows),
               oPerm = place(rows), oInv = place(rows), oRawF = place((size_t)chunk * 8), oRawT = place(chunk);
  char* mem = nullptr;
  cudaError_t e = cudaMalloc(&mem, bytes);
  auto at = [&](size_t o) { return reinterpret_cast<float*>(mem + o); };
  float *dP = at(oP), *dF = at(oF), *dT = at(oT), *dG = at(oG), *dM = at(oM), *dV = at(oV);
  float* dLoss = dG + PBF_MLP_PARAMS;
  uint32_t* dErr = reinterpret_cast<uint32_t*>(dG + PBF_MLP_PARAMS + 1);
  float* dBatchLoss = dG + PBF_MLP_PARAMS + 2;
  uint32_t *dPerm = reinterpret_cast<uint32_t*>(at(oPerm)), *dInv = reinterpret_cast<uint32_t*>(at(oInv));
  if (e == cudaSuccess) e = cudaMemsetAsync(mem, 0, cleared, 0);
  if (e == cudaSuccess) e = cudaMemcpyAsync(dP, m->params, sizeof(m->params), cudaMemcpyHostToDevice, 0);
  if (e == cudaSuccess) {
    k_shuffle_draws<<<(rows - 1u) / 256u + 1u, 256, 0, 0>>>(tc->seed ^ 0x5eedull, rows, dPerm);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(draw.data(), dPerm, (size_t)rows * 4, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) {
    for (uint32_t i = 0; i < rows; ++i) perm[i] = i;
    for (uint32_t i = rows - 1; i > 0; --i) std::swap(perm[i], perm[draw[i]]);
    e = cudaMemcpyAsync(dPerm, perm.data(), (size_t)rows * 4, cudaMemcpyHostToDevice, 0);
  }
  if (e == cudaSuccess) {
    k_invert<<<(rows - 1u) / 256u + 1u, 256, 0, 0>>>(dPerm, rows, dInv);
    e = cudaGetLastError();
  }
  for (uint64_t r0 = 0; r0 < rows && e == cudaSuccess; r0 += chunk) {
    const uint32_t c = (uint32_t)(rows - r0 < chunk ? rows - r0 : chunk);
    e = cudaMemcpyAsync(at(oRawF), feat + 8 * r0, (size_t)c * 8 * sizeof(float), cudaMemcpyHostToDevice, 0);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(at(oRawT), target + r0, (size_t)c * sizeof(float), cudaMemcpyHostToDevice, 0);
    if (e == cudaSuccess) {
      k_place_rows<<<(c + 255) / 256, 256, 0, 0>>>((const float4*)at(oRawF), at(oRawT), dInv, (uint32_t)r0, c,
                                                   (float4*)dF, dT);
      e = cudaGetLastError();
    }
  }
  const uint32_t batch = tc->batch < rows ? tc->batch : rows;
  const uint32_t per_epoch = rows / batch;
  double epoch_loss = 0.0;
  int step = 0;
  std::vector<float> lossbuf;
  for (uint32_t ep = 0; ep < tc->epochs && e == cudaSuccess; ++ep) {
    double acc = 0.0;
    for (uint32_t b = 0; b < per_epoch && e == cudaSuccess; ++b) {
      e = tc->kernel == PBF_MLP_TRAIN_TCGEN05
                ? launch_mlp_grad_tc(dP, *m, dF + 8 * (size_t)b * batch, dT + (size_t)b * batch, batch, dG, dLoss,
                                     dErr, 0)
                : launch_mlp_grad(dP, *m, dF + 8 * (size_t)b * batch, dT + (size_t)b * batch, batch, dG, dLoss, 0);
      ++step;
      float lr = tc->learning_rate;
      if (tc->epochs > 1) lr *= (float)(0.5 * (1.0 + std::cos(3.14159265358979 * ep / tc->epochs)));
      if (e == cudaSuccess) e = launch_adam(dP, dG, dM, dV, step, lr, dBatchLoss, 0);
      if (e == cudaSuccess && b + 1 == per_epoch) {
        float l = 0.0f;
        e = cudaMemcpy(&l, dBatchLoss, sizeof(float), cudaMemcpyDeviceToHost);
        acc = l / batch;
      }
    }
    epoch_loss = acc;
  }
  uint32_t herr = 0;
  if (e == cudaSuccess) e = cudaMemcpy(m->params, dP, sizeof(m->params), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(&herr, dErr, sizeof(uint32_t), cudaMemcpyDeviceToHost);
  cudaFree(mem);
  if (final_loss) *final_loss = (float)epoch_loss;
  if (e != cudaSuccess) return PBF_ECUDA;
  return herr ? PBF_ETIMEOUT : PBF_OK;
}

}  // extern "C"
