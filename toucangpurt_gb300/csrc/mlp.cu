// Learned cost model: a 16 -> 64 -> 64 -> 1 FP32 multilayer perceptron (ReLU)
// with hand-written forward, backward and Adam kernels.
//
// It predicts the cost (standardised log of clock64 cycles) of evaluating
// one micro-partition from 16 structural features; the scheduler balances
// warps and blocks on the prediction instead of on gate count.
//
// Parameter layout (floats): W1[64][16], b1[64], W2[64][64], b2[64], W3[64],
// b3[1] -- 5,313 values.  Forward: one warp evaluates one sample, lane l owns
// hidden units l and l + 32 of both layers and the activations move between
// lanes with shuffles.  Gradient: a block takes tiles of 64 samples through
// register-tiled products.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "mlp.h"

namespace tgs {
namespace {

constexpr uint32_t kFull = 0xFFFFFFFFu;
constexpr int kIn = 16, kH = 64;
constexpr int oW1 = 0, oB1 = oW1 + kH * kIn, oW2 = oB1 + kH, oB2 = oW2 + kH * kH, oW3 = oB2 + kH, oB3 = oW3 + kH;
static_assert(oB3 + 1 == kMlpParams, "layout");
// the forward kernel's weights in shared memory: rows of W1 and W2 padded by
// one float, so that 32 lanes reading one column of 32 rows meet 32 banks
// (unpadded, a W2 column met one bank; 200,000 samples 1,450 -> 550 us a call)
constexpr int kW1Row = kIn + 1, kW2Row = kH + 1;
constexpr int gW1 = 0, gB1 = gW1 + kH * kW1Row, gW2 = gB1 + kH, gB2 = gW2 + kH * kW2Row, gW3 = gB2 + kH, gB3 = gW3 + kH,
              kPadded = gB3 + 1;

// padded place of parameter i
__device__ __forceinline__ int paddedAt(int i) {
  if (i < oB1) return gW1 + i / kIn * kW1Row + i % kIn;
  if (i < oW2) return gB1 + (i - oB1);
  if (i < oB2) return gW2 + (i - oW2) / kH * kW2Row + (i - oW2) % kH;
  return gB2 + (i - oB2);  // b2, W3, b3 follow
}

struct Act {
  float h1[2], h2[2], out;
};

// forward of one sample by one warp; w in shared memory (padded)
__device__ __forceinline__ Act forwardWarp(const float *__restrict__ w, const float *__restrict__ x, uint32_t lane) {
  Act a;
  float xv = lane < kIn ? x[lane] : 0.f;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int j = lane + 32 * u;
    float s = w[gB1 + j];
#pragma unroll
    for (int m = 0; m < kIn; ++m) s += w[gW1 + j * kW1Row + m] * __shfl_sync(kFull, xv, m);
    a.h1[u] = fmaxf(s, 0.f);
  }
  float s2[2] = {w[gB2 + lane], w[gB2 + lane + 32]};
#pragma unroll 8
  for (int k = 0; k < kH; ++k) {
    const float hk = __shfl_sync(kFull, a.h1[k >> 5], k & 31);
    s2[0] += w[gW2 + lane * kW2Row + k] * hk;
    s2[1] += w[gW2 + (lane + 32) * kW2Row + k] * hk;
  }
  a.h2[0] = fmaxf(s2[0], 0.f);
  a.h2[1] = fmaxf(s2[1], 0.f);
  float o = w[gW3 + lane] * a.h2[0] + w[gW3 + lane + 32] * a.h2[1];
  for (int off = 16; off > 0; off >>= 1) o += __shfl_xor_sync(kFull, o, off);
  a.out = o + w[gB3];
  return a;
}

__global__ void __launch_bounds__(128) mlpForwardKernel(const float *__restrict__ params, const float *__restrict__ X,
                                                        uint32_t n, float *__restrict__ out) {
  __shared__ float w[kPadded];
  for (int i = threadIdx.x; i < kMlpParams; i += blockDim.x) w[paddedAt(i)] = params[i];
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  for (uint32_t s = blockIdx.x * (blockDim.x >> 5) + warp; s < n; s += gridDim.x * (blockDim.x >> 5)) {
    Act a = forwardWarp(w, X + size_t(s) * kIn, lane);
    if (lane == 0) out[s] = a.out;
  }
}

// ---- gradient of mean squared error over the samples idx[0..n) (idx null: 0..n) ----
// A block of 128 threads takes 64 samples at a time through both layers as
// register-tiled FP32 products out of shared memory (8 samples x 4 units a
// thread: 32 FMAs per three 16-byte shared loads), instead of one sample per
// warp with the activations moving by shuffles and every product read from
// and added to shared memory.  Activations are kept [unit][sample]; the
// weight gradients are dot products over the tile's samples, summed per tile
// and then over the block's tiles in registers, and added to global memory
// once per block.  Bound by FP32 FMA issue and the shared loads beside it.
// tgs_mlp_grad, host arrays in and out: 200,000 samples 2,699 -> 530 us (about
// 430 us of it copies and allocations), 600,000 7,539 -> 1,109 us, 1,024 226 ->
// 218 us; the kernel alone 20,000 samples 244 -> 36 us, 1,024 (a training
// batch) 24 -> 16.5; error against 64 bits unchanged (7e-7).
constexpr uint32_t kTile = 64;     // samples
constexpr int kRow = 68;           // floats of a shared row of 64 (16-byte aligned, rows 4 banks apart)
constexpr int tW1 = 0, tW2t = tW1 + kIn * kRow, tW2 = tW2t + kH * kRow, tB1 = tW2 + kH * kRow, tB2 = tB1 + kH,
              tW3 = tB2 + kH, tX = tW3 + kH, tH = tX + kIn * kRow, tD = tH + kH * kRow, kTileFloats = tD + kH * kRow;

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void st4(float *p, float a, float b, float c, float d) {
  *reinterpret_cast<float4 *>(p) = make_float4(a, b, c, d);
}

// acc[u][i] += sum_k w[k][4 tx + u] * in[k][8 ty + i], k = 0 .. K - 1
template <int K>
__device__ __forceinline__ void tileProduct(const float *__restrict__ w, const float *__restrict__ in, uint32_t tx,
                                            uint32_t ty, float (&acc)[4][8]) {
#pragma unroll 4
  for (int k = 0; k < K; ++k) {
    const float4 wv = ld4(w + k * kRow + 4 * tx), s0 = ld4(in + k * kRow + 8 * ty), s1 = ld4(in + k * kRow + 8 * ty + 4);
    const float a[4] = {wv.x, wv.y, wv.z, wv.w}, s[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[u][i] += a[u] * s[i];
  }
}

// acc[a][b] += sum over the tile's samples of p[rowP + a][s] * q[rowQ + 16 b][s]
template <int A, int B>
__device__ __forceinline__ void tileDot(const float *__restrict__ p, const float *__restrict__ q, float (&acc)[A][B]) {
  float t[A][B] = {};
#pragma unroll 2
  for (int s = 0; s < int(kTile); s += 4) {
    float4 y[B];
#pragma unroll
    for (int b = 0; b < B; ++b) y[b] = ld4(q + 16 * b * kRow + s);
#pragma unroll
    for (int a = 0; a < A; ++a) {
      const float4 x = ld4(p + a * kRow + s);
#pragma unroll
      for (int b = 0; b < B; ++b) t[a][b] += (x.x * y[b].x + x.y * y[b].y) + (x.z * y[b].z + x.w * y[b].w);
    }
  }
#pragma unroll
  for (int a = 0; a < A; ++a)
#pragma unroll
    for (int b = 0; b < B; ++b) acc[a][b] += t[a][b];
}

__global__ void __launch_bounds__(128, 2) mlpGradKernel(const float *__restrict__ params, const float *__restrict__ X,
                                                            const float *__restrict__ y, const uint32_t *__restrict__ idx,
                                                            uint32_t n, float scale, float *__restrict__ grad,
                                                            float *__restrict__ loss) {
  extern __shared__ __align__(16) float sm[];
  const uint32_t tid = threadIdx.x, tx = tid & 15u, ty = tid >> 4;
  for (uint32_t i = tid; i < kH * kIn; i += 128) sm[tW1 + (i % kIn) * kRow + i / kIn] = params[oW1 + i];
  for (uint32_t i = tid; i < kH * kH; i += 128) {
    const float w = params[oW2 + i];
    sm[tW2 + (i / kH) * kRow + i % kH] = w;
    sm[tW2t + (i % kH) * kRow + i / kH] = w;
  }
  if (tid < kH) {
    sm[tB1 + tid] = params[oB1 + tid];
    sm[tB2 + tid] = params[oB2 + tid];
    sm[tW3 + tid] = params[oW3 + tid];
  }
  const float b3 = params[oB3];
  float gw2[8][4] = {}, gw1[2][4] = {}, gb1[4] = {}, gb2[4] = {}, gw3[4] = {}, gb3 = 0.f, lossAcc = 0.f;
  const uint32_t tiles = (n + kTile - 1) / kTile;
  for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const uint32_t s0 = t * kTile;
    __syncthreads();  // the previous tile's rows are no longer read (first tile: the weights are in place)
    for (uint32_t i = tid; i < kTile * kIn / 4; i += 128) {
      const uint32_t s = i % kTile, q = i / kTile;  // four inputs of one sample
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (s0 + s < n) v = ld4(X + size_t(idx ? idx[s0 + s] : s0 + s) * kIn + 4 * q);
      sm[tX + (4 * q) * kRow + s] = v.x;
      sm[tX + (4 * q + 1) * kRow + s] = v.y;
      sm[tX + (4 * q + 2) * kRow + s] = v.z;
      sm[tX + (4 * q + 3) * kRow + s] = v.w;
    }
    __syncthreads();
    // samples from the thread's first one up to the end (the last tile's
    // others keep zero activations: a bias may make theirs infinite where no
    // sample's is, and 0 * infinity would reach the sums)
    const int left = int(min(n - s0, kTile)) - int(8 * ty);
    // layer 1
    float h[4][8];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int i = 0; i < 8; ++i) h[u][i] = sm[tB1 + 4 * tx + u];
    tileProduct<kIn>(sm + tW1, sm + tX, tx, ty, h);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
#pragma unroll
      for (int i = 0; i < 8; ++i) h[u][i] = i < left ? fmaxf(h[u][i], 0.f) : 0.f;
      st4(sm + tH + (4 * tx + u) * kRow + 8 * ty, h[u][0], h[u][1], h[u][2], h[u][3]);
      st4(sm + tH + (4 * tx + u) * kRow + 8 * ty + 4, h[u][4], h[u][5], h[u][6], h[u][7]);
    }
    __syncthreads();
    // layer 2, output, and the error of the thread's 8 samples
    float h2[4][8];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int i = 0; i < 8; ++i) h2[u][i] = sm[tB2 + 4 * tx + u];
    tileProduct<kH>(sm + tW2t, sm + tH, tx, ty, h2);
    float w3[4], dy[8];
#pragma unroll
    for (int u = 0; u < 4; ++u) w3[u] = sm[tW3 + 4 * tx + u];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float o = 0.f;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        h2[u][i] = i < left ? fmaxf(h2[u][i], 0.f) : 0.f;
        o += w3[u] * h2[u][i];
      }
#pragma unroll
      for (int off = 8; off > 0; off >>= 1) o += __shfl_xor_sync(kFull, o, off);
      const uint32_t s = s0 + 8 * ty + i;
      const float d = i < left ? o + b3 - y[idx ? idx[s] : s] : 0.f;
      dy[i] = 2.f * d * scale;
      if (tx == 0) {
        lossAcc += d * d;
        gb3 += dy[i];
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      float g3 = 0.f, g2 = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        g3 += dy[i] * h2[u][i];
        h2[u][i] = h2[u][i] > 0.f ? dy[i] * w3[u] : 0.f;  // d loss / d layer 2
        g2 += h2[u][i];
      }
      gw3[u] += g3;
      gb2[u] += g2;
      st4(sm + tD + (4 * tx + u) * kRow + 8 * ty, h2[u][0], h2[u][1], h2[u][2], h2[u][3]);
      st4(sm + tD + (4 * tx + u) * kRow + 8 * ty + 4, h2[u][4], h2[u][5], h2[u][6], h2[u][7]);
    }
    __syncthreads();
    // dW2[j][k] = sum_s d2[j][s] h1[k][s]; d1[k][s] = sum_j d2[j][s] W2[j][k] where h1 > 0
    tileDot<8, 4>(sm + tD + 8 * ty * kRow, sm + tH + tx * kRow, gw2);
    float d1[4][8] = {};
    tileProduct<kH>(sm + tW2, sm + tD, tx, ty, d1);
    __syncthreads();  // every thread is done with d2
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      float g1 = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        d1[u][i] = h[u][i] > 0.f ? d1[u][i] : 0.f;
        g1 += d1[u][i];
      }
      gb1[u] += g1;
      st4(sm + tD + (4 * tx + u) * kRow + 8 * ty, d1[u][0], d1[u][1], d1[u][2], d1[u][3]);
      st4(sm + tD + (4 * tx + u) * kRow + 8 * ty + 4, d1[u][4], d1[u][5], d1[u][6], d1[u][7]);
    }
    __syncthreads();
    // dW1[k][m] = sum_s d1[k][s] x[m][s]
    tileDot<2, 4>(sm + tX + 2 * ty * kRow, sm + tD + tx * kRow, gw1);
  }
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const uint32_t k = tx + 16 * b;
#pragma unroll
    for (int a = 0; a < 8; ++a) atomicAdd(grad + oW2 + (8 * ty + a) * kH + k, gw2[a][b]);
#pragma unroll
    for (int a = 0; a < 2; ++a) atomicAdd(grad + oW1 + k * kIn + 2 * ty + a, gw1[a][b]);
  }
  // the eight sample groups' sums of the biases, W3 and the loss meet in
  // shared memory, so that each block adds once to a global sum
  __syncthreads();
  float *red = sm + tD;  // [ty][b1 | b2 | W3 | b3, loss]
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    red[ty * 200 + 4 * tx + b] = gb1[b];
    red[ty * 200 + 64 + 4 * tx + b] = gb2[b];
    red[ty * 200 + 128 + 4 * tx + b] = gw3[b];
  }
  if (tx == 0) {
    red[ty * 200 + 192] = gb3;
    red[ty * 200 + 193] = lossAcc;
  }
  __syncthreads();
  for (uint32_t i = tid; i < 194; i += 128) {
    float s = 0.f;
    for (int q = 0; q < 8; ++q) s += red[q * 200 + i];
    if (i < 193)
      atomicAdd(grad + (i < 64 ? oB1 + i : oB2 + (i - 64)), s);  // b2, W3, b3 lie in a row
    else if (loss)
      atomicAdd(loss, s);
  }
}

__global__ void adamKernel(float *__restrict__ p, float *__restrict__ m, float *__restrict__ v,
                           const float *__restrict__ g, uint32_t n, float lr, float b1, float b2, float eps,
                           float c1, float c2) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

}  // namespace

cudaError_t mlpForward(const float *params, const float *X, uint32_t n, float *out, cudaStream_t st) {
  if (!n) return cudaSuccess;
  const uint32_t blocks = std::min<uint32_t>(2048, (n + 3) / 4);
  mlpForwardKernel<<<blocks, 128, 0, st>>>(params, X, n, out);
  return cudaGetLastError();
}

cudaError_t mlpGrad(const float *params, const float *X, const float *y, const uint32_t *idx, uint32_t n, float scale,
                    float *grad, float *loss, cudaStream_t st) {
  if (!n) return cudaSuccess;
  // set on every call: the attribute belongs to the current device's context
  // (another device, or a context re-created after a reset, starts without it)
  const size_t smem = kTileFloats * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(mlpGradKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (e != cudaSuccess) return e;
  const uint32_t blocks = std::min<uint32_t>(304, (n + kTile - 1) / kTile);  // two resident blocks an SM
  mlpGradKernel<<<blocks, 128, smem, st>>>(params, X, y, idx, n, scale, grad, loss);
  return cudaGetLastError();
}

cudaError_t adamStep(float *params, float *m, float *v, const float *grad, uint32_t n, float lr, float b1, float b2,
                     float eps, uint32_t t, cudaStream_t st) {
  float c1 = 1.f, c2 = 1.f;
  for (uint32_t i = 0; i < t; ++i) {
    c1 *= b1;
    c2 *= b2;
  }
  adamKernel<<<(n + 255) / 256, 256, 0, st>>>(params, m, v, grad, n, lr, b1, b2, eps, 1.f - c1, 1.f - c2);
  return cudaGetLastError();
}

}  // namespace tgs
