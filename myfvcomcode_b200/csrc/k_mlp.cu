// k_mlp.cu - the network of the learned vertical closure: an MLP 8 -> 64 -> 64 -> 3 with
// GELU (tanh form) on the two hidden layers, trained in FP32 by the kernels in this file (mean-squared
// error, Adam).  Inference in BF16 on the tensor cores is in k_closure.cu; the FP32
// forward pass here is its reference.
//
// Parameters are one FP32 vector: W1 (64x8, row j = hidden unit j), b1 (64), W2 (64x64),
// b2 (64), W3 (3x64), b3 (3).
//
// Training step over a batch of B samples: k_mlp_fwd_bwd runs blocks of 256 threads over
// tiles of 32 samples, forward and backward as small matrix products from shared memory
// (each thread two samples by four units), and keeps the tile's weight gradients in
// registers (sixteen of W2 and two of W1 per thread); k_mlp_adam sums the blocks' gradients
// in a fixed order and applies Adam.  The gradient is deterministic.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "fvg_model.h"

namespace {

constexpr int MI = 8, MH = 64, MO = 3;
constexpr int OW1 = 0, OB1 = OW1 + MH * MI, OW2 = OB1 + MH, OB2 = OW2 + MH * MH, OW3 = OB2 + MH,
              OB3 = OW3 + MO * MH, NPAR = OB3 + MO;
// GELU in its tanh form, 0.5 z (1 + tanh(u)), u = c (z + 0.044715 z^3), c = sqrt(2/pi), as
// z * s with s = 0.5 (1 + tanh(u)) = 1 / (1 + exp(-2u)), which does not cancel for negative z
// and costs half of tanhf's instructions (the function took nearly half of the forward pass);
// and its derivative s + 2 z s (1 - s) u'.  1 - s is taken as exp(-2u) s, which does not cancel
// (1 - s lost up to 2e-6 of the derivative for z of 4 to 6); the exponential is held finite, so
// that its product with s = 0 is a number.  A batch's gradient against 64 bits, 24 seeds each,
// over tanhf's form: 1 sample 0.93, 33 0.94, 1,000 0.82 of its error (1.08, 1.07 and 0.88 with
// 1 - s); the forward pass 0.97.
constexpr float kGc = 0.79788456080286536f, kGa = 0.044715f;
__device__ __forceinline__ float gelu_e(float z, float z2) {
  return __expf(z * fmaf(-2.0f * kGc * kGa, z2, -2.0f * kGc));
}
__device__ __forceinline__ float gelu(float z) { return z * __fdividef(1.0f, 1.0f + gelu_e(z, z * z)); }
__device__ __forceinline__ float gelu2(float z, float& d) {
  const float z2 = z * z, e = fminf(gelu_e(z, z2), 3.4e38f), s = __fdividef(1.0f, 1.0f + e);
  d = fmaf(2.0f * z * s * (e * s), kGc * fmaf(3.0f * kGa, z2, 1.0f), s);
  return z * s;
}

// Wait for the kernel before and let the one after start its prologue (both no-ops where the
// kernel was not launched as a programmatic dependent).
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// -------------------------------------------------------------------------------------
// Training pass.  A tile is 32 samples.  Activations are sample-major with rows of PD floats
// (16-byte aligned, so that four units are one load, and the rows of a warp's threads fall
// into different banks); W2 is held in both orders, W2[j][k] for the backward product and
// W2T[k][j] for the forward one.  One thread per sample, as before, left 64 blocks of two
// warps per batch of 4,096 with two shared-memory loads per multiply-add: 85 us per batch
// against 10 now (with the update).
// -------------------------------------------------------------------------------------
constexpr int TB = 32;    // samples per tile
constexpr int NT = 256;   // threads per block
constexpr int PD = 68;    // row stride of activations and weights (floats)
constexpr int XD = 12;    // row stride of the inputs
constexpr int kMostBlocks = 296;  // fixed, as the sum over the blocks depends on it
struct TrainShared {
  float w1t[MI][PD];      // W1T[k][j]
  float w2t[MH][PD];      // W2T[k][j]
  float w2[MH][PD];       // W2[j][k]
  float w3[MO][PD];
  float b1[MH], b2[MH], b3[4];
  float x[TB][XD];
  float h1[TB][PD], d1[TB][PD];  // GELU(z1) and its derivative, then dz1
  float h2[TB][PD], d2[TB][PD];  // the same of the second layer
  float dy[TB][4];
};

// acc[2][4] += A(rows r0, r0+1; 64 columns) * B(64 rows; columns c0..c0+3), both with stride PD
__device__ __forceinline__ void gemm24(const float* A, const float* B, int r0, int c0, float acc[2][4]) {
#pragma unroll 4
  for (int k = 0; k < MH; k += 4) {
    const float4 a0 = *reinterpret_cast<const float4*>(A + r0 * PD + k);
    const float4 a1 = *reinterpret_cast<const float4*>(A + (r0 + 1) * PD + k);
    const float av[2][4] = {{a0.x, a0.y, a0.z, a0.w}, {a1.x, a1.y, a1.z, a1.w}};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 b = *reinterpret_cast<const float4*>(B + (k + q) * PD + c0);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        acc[r][0] = fmaf(av[r][q], b.x, acc[r][0]);
        acc[r][1] = fmaf(av[r][q], b.y, acc[r][1]);
        acc[r][2] = fmaf(av[r][q], b.z, acc[r][2]);
        acc[r][3] = fmaf(av[r][q], b.w, acc[r][3]);
      }
    }
  }
}

// x: row-major [n][MI] inputs, y: [n][MO] targets, idx: optional sample order (the
// batch is idx[b0 .. b0+nb-1]).  part: [gridDim.x][NPAR] gradients, lpart: [gridDim.x]
// summed squared errors.  scale = 1/(number of batch samples * MO).
__global__ void __launch_bounds__(NT) k_mlp_fwd_bwd(const float* __restrict__ par, const float* __restrict__ x,
                                                    const float* __restrict__ y, const int* __restrict__ idx,
                                                    int b0, int nb, float scale, float* part, float* lpart) {
  extern __shared__ __align__(16) unsigned char train_sm[];
  TrainShared& S = *reinterpret_cast<TrainShared*>(train_sm);
  __shared__ float e2[TB * MO];
  const int t = threadIdx.x;
  dep_wait();
  dep_launch();
  for (int p = t; p < MH * MI; p += NT) S.w1t[p % MI][p / MI] = par[OW1 + p];
  for (int p = t; p < MH * MH; p += NT) {
    const float w = par[OW2 + p];
    S.w2[p / MH][p % MH] = w;
    S.w2t[p % MH][p / MH] = w;
  }
  for (int p = t; p < MO * MH; p += NT) S.w3[p / MH][p % MH] = par[OW3 + p];
  if (t < MH) {
    S.b1[t] = par[OB1 + t];
    S.b2[t] = par[OB2 + t];
  }
  if (t < MO) S.b3[t] = par[OB3 + t];
  // this thread's part of a product: two samples by four units
  const int c0 = 4 * (t & 15), r0 = 2 * (t >> 4);
  // gradients of the block: W2[j0..j0+3][k0..k0+3], W1[jw][kw, kw+1], and one of the 323 other
  // sums (b1, b2, W3, b3) per thread and a second for the first threads
  const int j0 = 4 * (t >> 4), k0 = 4 * (t & 15), jw = t >> 2, kw = 2 * (t & 3);
  float g2[4][4] = {}, g1[2] = {0.f, 0.f}, gx[2] = {0.f, 0.f}, err = 0.f;
  const int ntile = (nb + TB - 1) / TB;
  for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
    __syncthreads();
    {
      const int s = t >> 3, k = t & 7, r = tile * TB + s;
      float v = 0.f;
      if (r < nb) v = x[(size_t)(idx ? idx[b0 + r] : b0 + r) * MI + k];
      S.x[s][k] = v;
    }
    __syncthreads();
    // layer 1
    {
      float z[2][4];
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) z[r][c] = S.b1[c0 + c];
#pragma unroll
      for (int k = 0; k < MI; ++k) {
        const float4 w = *reinterpret_cast<const float4*>(&S.w1t[k][c0]);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float xv = S.x[r0 + r][k];
          z[r][0] = fmaf(xv, w.x, z[r][0]);
          z[r][1] = fmaf(xv, w.y, z[r][1]);
          z[r][2] = fmaf(xv, w.z, z[r][2]);
          z[r][3] = fmaf(xv, w.w, z[r][3]);
        }
      }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        float4 h, d;
        h.x = gelu2(z[r][0], d.x);
        h.y = gelu2(z[r][1], d.y);
        h.z = gelu2(z[r][2], d.z);
        h.w = gelu2(z[r][3], d.w);
        *reinterpret_cast<float4*>(&S.h1[r0 + r][c0]) = h;
        *reinterpret_cast<float4*>(&S.d1[r0 + r][c0]) = d;
      }
    }
    __syncthreads();
    // layer 2
    {
      float z[2][4];
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) z[r][c] = S.b2[c0 + c];
      gemm24(&S.h1[0][0], &S.w2t[0][0], r0, c0, z);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        float4 h, d;
        h.x = gelu2(z[r][0], d.x);
        h.y = gelu2(z[r][1], d.y);
        h.z = gelu2(z[r][2], d.z);
        h.w = gelu2(z[r][3], d.w);
        *reinterpret_cast<float4*>(&S.h2[r0 + r][c0]) = h;
        *reinterpret_cast<float4*>(&S.d2[r0 + r][c0]) = d;
      }
    }
    __syncthreads();
    // layer 3 and the error: one thread per sample and output
    if (t < TB * MO) {
      const int s = t / MO, o = t % MO, r = tile * TB + s;
      float z = S.b3[o];
#pragma unroll 8
      for (int j = 0; j < MH; ++j) z = fmaf(S.w3[o][j], S.h2[s][j], z);
      float e = 0.f;
      if (r < nb) e = z - y[(size_t)(idx ? idx[b0 + r] : b0 + r) * MO + o];
      err += e * e;
      S.dy[s][o] = 2.f * e * scale;
    }
    __syncthreads();
    // dz2 = (W3' dy) * GELU'(z2)
    {
      const float4 wa = *reinterpret_cast<const float4*>(&S.w3[0][c0]), wb = *reinterpret_cast<const float4*>(&S.w3[1][c0]),
                   wc = *reinterpret_cast<const float4*>(&S.w3[2][c0]);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float y0 = S.dy[r0 + r][0], y1 = S.dy[r0 + r][1], y2 = S.dy[r0 + r][2];
        float4* d = reinterpret_cast<float4*>(&S.d2[r0 + r][c0]);
        float4 v = *d;
        v.x *= fmaf(wc.x, y2, fmaf(wb.x, y1, wa.x * y0));
        v.y *= fmaf(wc.y, y2, fmaf(wb.y, y1, wa.y * y0));
        v.z *= fmaf(wc.z, y2, fmaf(wb.z, y1, wa.z * y0));
        v.w *= fmaf(wc.w, y2, fmaf(wb.w, y1, wa.w * y0));
        *d = v;
      }
    }
    __syncthreads();
    // dz1 = (W2' dz2) * GELU'(z1)
    {
      float d[2][4] = {};
      gemm24(&S.d2[0][0], &S.w2[0][0], r0, c0, d);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        float4* q = reinterpret_cast<float4*>(&S.d1[r0 + r][c0]);
        float4 v = *q;
        v.x *= d[r][0];
        v.y *= d[r][1];
        v.z *= d[r][2];
        v.w *= d[r][3];
        *q = v;
      }
    }
    __syncthreads();
    // weight gradients over the tile's samples, in sample order
#pragma unroll 4
    for (int s = 0; s < TB; ++s) {
      const float4 dj = *reinterpret_cast<const float4*>(&S.d2[s][j0]), hk = *reinterpret_cast<const float4*>(&S.h1[s][k0]);
      const float dv[4] = {dj.x, dj.y, dj.z, dj.w}, hv[4] = {hk.x, hk.y, hk.z, hk.w};
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int k = 0; k < 4; ++k) g2[j][k] = fmaf(dv[j], hv[k], g2[j][k]);
      const float dw = S.d1[s][jw];
      g1[0] = fmaf(dw, S.x[s][kw], g1[0]);
      g1[1] = fmaf(dw, S.x[s][kw + 1], g1[1]);
    }
    for (int q = 0; q < 2; ++q) {
      const int p = t + q * NT;
      float v = gx[q];
      if (p < MH) {
        for (int s = 0; s < TB; ++s) v += S.d1[s][p];
      } else if (p < 2 * MH) {
        for (int s = 0; s < TB; ++s) v += S.d2[s][p - MH];
      } else if (p < 2 * MH + MO * MH) {
        const int o = (p - 2 * MH) / MH, j = (p - 2 * MH) % MH;
        for (int s = 0; s < TB; ++s) v = fmaf(S.dy[s][o], S.h2[s][j], v);
      } else if (p < 2 * MH + MO * MH + MO) {
        for (int s = 0; s < TB; ++s) v += S.dy[s][p - 2 * MH - MO * MH];
      }
      gx[q] = v;
    }
  }
  float* gp = part + (size_t)blockIdx.x * NPAR;
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int k = 0; k < 4; ++k) gp[OW2 + (j0 + j) * MH + k0 + k] = g2[j][k];
  gp[OW1 + jw * MI + kw] = g1[0];
  gp[OW1 + jw * MI + kw + 1] = g1[1];
  for (int q = 0; q < 2; ++q) {
    const int p = t + q * NT;
    if (p < MH) gp[OB1 + p] = gx[q];
    else if (p < 2 * MH) gp[OB2 + p - MH] = gx[q];
    else if (p < 2 * MH + MO * MH) gp[OW3 + p - 2 * MH] = gx[q];
    else if (p < 2 * MH + MO * MH + MO) gp[OB3 + p - 2 * MH - MO * MH] = gx[q];
  }
  // squared error of the block, in sample order
  if (t < TB * MO) e2[t] = err;
  __syncthreads();
  if (t == 0) {
    float s = 0.f;
    for (int u = 0; u < TB * MO; ++u) s += e2[u];
    lpart[blockIdx.x] = s;
  }
}

// Sum of the blocks' gradients and, when step > 0, one Adam update.  Eight threads per
// parameter add every eighth block's gradient in block order; their sums are added in order.
constexpr int AP = 32;  // parameters per block
__global__ void __launch_bounds__(256) k_mlp_adam(float* par, float* m, float* v, const float* part, int nblk,
                                                  float* grad_out, const float* lpart, float* loss_acc, int step,
                                                  float lr) {
  __shared__ float sl[8][AP];
  dep_wait();
  dep_launch();
  const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5, p = blockIdx.x * AP + lane;
  if (blockIdx.x == 0 && slice == 7) {
    float s = 0.f;
    for (int b = lane; b < nblk; b += 32) s += lpart[b];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) *loss_acc += s;
  }
  float g = 0.f;
  if (p < NPAR) {
#pragma unroll 8
    for (int b = slice; b < nblk; b += 8) g += part[(size_t)b * NPAR + p];
  }
  sl[slice][lane] = g;
  __syncthreads();
  if (slice != 0 || p >= NPAR) return;
  for (int q = 1; q < 8; ++q) g += sl[q][lane];
  if (grad_out) grad_out[p] = g;
  if (step <= 0) return;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  float mm = b1 * m[p] + (1.f - b1) * g;
  float vv = b2 * v[p] + (1.f - b2) * g * g;
  m[p] = mm;
  v[p] = vv;
  float mh = mm / (1.f - powf(b1, (float)step));
  float vh = vv / (1.f - powf(b2, (float)step));
  par[p] -= lr * mh / (sqrtf(vh) + eps);
}

// -------------------------------------------------------------------------------------
// FP32 forward pass (the reference of the tensor-core kernel).  A block of 128 threads takes
// tiles of 128 samples; the layers are products from shared memory, eight samples by eight
// units per thread, so that four loads serve 64 multiply-adds.  One thread per sample read
// every weight from L1 for each multiply-add: 698 us for 1,000,003 samples against 367.  Shared
// memory bounds it now (82 % of its wavefronts, more than half of them bank conflicts of the
// stores of h and the loads of W; the FMA pipe at 48 %).
// -------------------------------------------------------------------------------------
constexpr int FR = 128;      // samples per tile, threads per block
constexpr int FD = FR + 4;   // stride of the unit-major activations
struct ForwardShared {
  float w1t[MI][PD], w2t[MH][PD];
  float4 w3[MH];             // {W3[0][j], W3[1][j], W3[2][j], 0}
  float b1[MH], b2[MH], b3[4];
  float x[MI][FD];
  float h[MH][FD];           // GELU(z1), then GELU(z2): [unit][sample]
};
template <int K>
__device__ __forceinline__ void gemm88(const float (*A)[FD], const float (*B)[PD], int r0, int c0, float z[8][8]) {
#pragma unroll 4
  for (int k = 0; k < K; ++k) {
    const float4 a0 = *reinterpret_cast<const float4*>(&A[k][r0]), a1 = *reinterpret_cast<const float4*>(&A[k][r0 + 4]);
    const float4 b0 = *reinterpret_cast<const float4*>(&B[k][c0]), b1 = *reinterpret_cast<const float4*>(&B[k][c0 + 4]);
    const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
    const float bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int c = 0; c < 8; ++c) z[r][c] = fmaf(av[r], bv[c], z[r][c]);
  }
}
__global__ void __launch_bounds__(FR, 3) k_mlp_forward(const float* __restrict__ par, const float* __restrict__ x, int n,
                                                       float* out) {
  extern __shared__ __align__(16) unsigned char fwd_sm[];
  ForwardShared& S = *reinterpret_cast<ForwardShared*>(fwd_sm);
  const int t = threadIdx.x;
  for (int p = t; p < MH * MI; p += FR) S.w1t[p % MI][p / MI] = par[OW1 + p];
  for (int p = t; p < MH * MH; p += FR) S.w2t[p % MH][p / MH] = par[OW2 + p];
  if (t < MH) {
    S.w3[t] = make_float4(par[OW3 + t], par[OW3 + MH + t], par[OW3 + 2 * MH + t], 0.f);
    S.b1[t] = par[OB1 + t];
    S.b2[t] = par[OB2 + t];
  }
  if (t < MO) S.b3[t] = par[OB3 + t];
  const int c0 = 8 * (t & 7), r0 = 8 * (t >> 3);
  const bool wide = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  for (int tile = blockIdx.x; tile < (n + FR - 1) / FR; tile += gridDim.x) {
    const int row = tile * FR + t;
    __syncthreads();
    float xv[MI] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (row < n) {
      const float* xr = x + (size_t)row * MI;
      if (wide) {
        const float4 a = *reinterpret_cast<const float4*>(xr), b = *reinterpret_cast<const float4*>(xr + 4);
        xv[0] = a.x; xv[1] = a.y; xv[2] = a.z; xv[3] = a.w;
        xv[4] = b.x; xv[5] = b.y; xv[6] = b.z; xv[7] = b.w;
      } else {
        for (int k = 0; k < MI; ++k) xv[k] = xr[k];
      }
    }
    for (int k = 0; k < MI; ++k) S.x[k][t] = xv[k];
    __syncthreads();
    float z[8][8];
    auto start = [&](const float* b) {
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = 0; c < 8; ++c) z[r][c] = b[c0 + c];
    };
    auto finish = [&]() {
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        float4 lo, hi;
        lo.x = gelu(z[0][c]); lo.y = gelu(z[1][c]); lo.z = gelu(z[2][c]); lo.w = gelu(z[3][c]);
        hi.x = gelu(z[4][c]); hi.y = gelu(z[5][c]); hi.z = gelu(z[6][c]); hi.w = gelu(z[7][c]);
        *reinterpret_cast<float4*>(&S.h[c0 + c][r0]) = lo;
        *reinterpret_cast<float4*>(&S.h[c0 + c][r0 + 4]) = hi;
      }
    };
    start(S.b1);
    gemm88<MI>(S.x, S.w1t, r0, c0, z);
    finish();
    __syncthreads();
    start(S.b2);
    gemm88<MH>(S.h, S.w2t, r0, c0, z);
    __syncthreads();
    finish();
    __syncthreads();
    if (row < n) {
      float o0 = S.b3[0], o1 = S.b3[1], o2 = S.b3[2];
#pragma unroll 8
      for (int j = 0; j < MH; ++j) {
        const float h = S.h[j][t];
        const float4 w = S.w3[j];
        o0 = fmaf(w.x, h, o0);
        o1 = fmaf(w.y, h, o1);
        o2 = fmaf(w.z, h, o2);
      }
      out[(size_t)row * MO] = o0;
      out[(size_t)row * MO + 1] = o1;
      out[(size_t)row * MO + 2] = o2;
    }
  }
}

// Launch as a programmatic dependent of the kernel before in the stream.
template <typename... KArgs, typename... Args>
void launch_dep(void (*k)(KArgs...), int grid, int block, size_t smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k, args...);
}

}  // namespace

struct fvg_mlp {
  float *par = nullptr, *m = nullptr, *v = nullptr, *part = nullptr, *lpart = nullptr, *grad = nullptr;
  float* loss = nullptr;
  int* idx = nullptr;
  int idx_cap = 0, part_blocks = 0, step = 0, nsm = 148;
  cudaStream_t stream = nullptr;
  std::string err;
};

static int mlp_cuda(fvg_mlp* q, cudaError_t e, const char* what) {
  if (e == cudaSuccess) return FVG_OK;
  q->err = std::string(what) + ": " + cudaGetErrorString(e);
  return FVG_ERR_CUDA;
}
#define MK(call) do { int rc_ = mlp_cuda(q, (call), #call); if (rc_) return rc_; } while (0)

static int mlp_parts(fvg_mlp* q, int nblk) {
  if (nblk <= q->part_blocks) return FVG_OK;
  if (q->part) cudaFree(q->part);
  if (q->lpart) cudaFree(q->lpart);
  q->part = nullptr;
  q->lpart = nullptr;
  q->part_blocks = 0;
  if (cudaMalloc(&q->part, (size_t)nblk * NPAR * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&q->lpart, (size_t)nblk * sizeof(float)) != cudaSuccess) {
    const cudaError_t e = cudaGetLastError();  // reported here, not by the next launch
    return mlp_cuda(q, e, "cudaMalloc (gradients of the blocks)");
  }
  q->part_blocks = nblk;
  return FVG_OK;
}

// One pass of forward/backward over samples b0..b0+nb-1 of the order idx (or the rows
// in order), gradient summed into q->grad; an Adam step when step > 0.
static int mlp_pass(fvg_mlp* q, const float* x, const float* y, const int* idx, int b0, int nb, int step,
                    float lr, float scale) {
  const int nblk = std::min((nb + TB - 1) / TB, kMostBlocks);
  int rc = mlp_parts(q, nblk);
  if (rc) return rc;
  launch_dep(k_mlp_fwd_bwd, nblk, NT, sizeof(TrainShared), q->stream, (const float*)q->par, x, y, idx, b0, nb, scale,
             q->part, q->lpart);
  launch_dep(k_mlp_adam, (NPAR + AP - 1) / AP, 256, 0, q->stream, q->par, q->m, q->v, (const float*)q->part, nblk, q->grad,
             (const float*)q->lpart, q->loss, step, lr);
  MK(cudaGetLastError());
  return FVG_OK;
}

extern "C" {

int fvg_mlp_create(uint64_t seed, fvg_mlp** out) {
  if (!out) return FVG_ERR_ARG;
  *out = nullptr;
  fvg_mlp* q = new fvg_mlp();
  auto fail = [&](int rc) { fvg_mlp_destroy(q); return rc; };
  if (cudaFuncSetAttribute(k_mlp_fwd_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrainShared)) !=
          cudaSuccess ||
      cudaFuncSetAttribute(k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ForwardShared)) !=
          cudaSuccess)
    return fail(FVG_ERR_CUDA);
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&q->nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return fail(FVG_ERR_CUDA);
  if (cudaStreamCreateWithFlags(&q->stream, cudaStreamNonBlocking) != cudaSuccess) return fail(FVG_ERR_CUDA);
  for (float** p : {&q->par, &q->m, &q->v, &q->grad})
    if (cudaMalloc(p, NPAR * sizeof(float)) != cudaSuccess) return fail(FVG_ERR_NOMEM);
  if (cudaMalloc(&q->loss, sizeof(float)) != cudaSuccess) return fail(FVG_ERR_NOMEM);
  // He-style initialisation scaled by fan-in, biases zero.
  std::vector<float> h(NPAR, 0.f);
  std::mt19937_64 rng(seed);
  std::normal_distribution<float> nd(0.f, 1.f);
  for (int p = OW1; p < OB1; ++p) h[p] = nd(rng) * std::sqrt(2.f / MI);
  for (int p = OW2; p < OB2; ++p) h[p] = nd(rng) * std::sqrt(2.f / MH);
  for (int p = OW3; p < OB3; ++p) h[p] = nd(rng) * std::sqrt(1.f / MH);
  if (cudaMemcpy(q->par, h.data(), NPAR * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemsetAsync(q->m, 0, NPAR * sizeof(float), q->stream) != cudaSuccess ||
      cudaMemsetAsync(q->v, 0, NPAR * sizeof(float), q->stream) != cudaSuccess)
    return fail(FVG_ERR_CUDA);
  *out = q;
  return FVG_OK;
}

void fvg_mlp_destroy(fvg_mlp* q) {
  if (!q) return;
  if (q->stream) cudaStreamSynchronize(q->stream);
  for (float* p : {q->par, q->m, q->v, q->part, q->lpart, q->grad, q->loss})
    if (p) cudaFree(p);
  if (q->idx) cudaFree(q->idx);
  if (q->stream) cudaStreamDestroy(q->stream);
  delete q;
}

const char* fvg_mlp_last_error(const fvg_mlp* q) { return q ? q->err.c_str() : "null network"; }

int32_t fvg_mlp_num_params(void) { return NPAR; }

int fvg_mlp_get_params(fvg_mlp* q, float* host, int32_t n) {
  if (!q || !host || n != NPAR) return FVG_ERR_ARG;
  MK(cudaStreamSynchronize(q->stream));
  MK(cudaMemcpy(host, q->par, NPAR * sizeof(float), cudaMemcpyDeviceToHost));
  return FVG_OK;
}

int fvg_mlp_set_params(fvg_mlp* q, const float* host, int32_t n) {
  if (!q || !host || n != NPAR) return FVG_ERR_ARG;
  MK(cudaStreamSynchronize(q->stream));
  MK(cudaMemcpy(q->par, host, NPAR * sizeof(float), cudaMemcpyHostToDevice));
  MK(cudaMemsetAsync(q->m, 0, NPAR * sizeof(float), q->stream));
  MK(cudaMemsetAsync(q->v, 0, NPAR * sizeof(float), q->stream));
  q->step = 0;
  return FVG_OK;
}

int fvg_mlp_loss_grad(fvg_mlp* q, const float* x, const float* y, int32_t n, float* loss, float* grad) {
  if (!q || !x || !y || n < 1 || !loss || !grad) return FVG_ERR_ARG;
  MK(cudaMemsetAsync(q->loss, 0, sizeof(float), q->stream));
  int rc = mlp_pass(q, x, y, nullptr, 0, n, 0, 0.f, 1.f / ((float)n * MO));
  if (rc) return rc;
  MK(cudaMemcpyAsync(grad, q->grad, NPAR * sizeof(float), cudaMemcpyDeviceToHost, q->stream));
  MK(cudaMemcpyAsync(loss, q->loss, sizeof(float), cudaMemcpyDeviceToHost, q->stream));
  MK(cudaStreamSynchronize(q->stream));
  *loss /= (float)n * MO;
  return FVG_OK;
}

int fvg_mlp_train(fvg_mlp* q, const float* x, const float* y, int32_t n, int32_t epochs, int32_t batch,
                  float lr, uint64_t seed, float* epoch_loss) {
  if (!q || !x || !y || n < 1 || epochs < 1 || batch < 1 || batch > n) return FVG_ERR_ARG;
  if (n > q->idx_cap) {
    if (q->idx) cudaFree(q->idx);
    q->idx = nullptr;
    q->idx_cap = 0;
    MK(cudaMalloc(&q->idx, (size_t)n * sizeof(int)));
    q->idx_cap = n;
  }
  std::vector<int> order(n);
  std::mt19937_64 rng(seed);
  for (int e = 0; e < epochs; ++e) {
    for (int i = 0; i < n; ++i) order[i] = i;
    std::shuffle(order.begin(), order.end(), rng);
    MK(cudaStreamSynchronize(q->stream));
    MK(cudaMemcpyAsync(q->idx, order.data(), (size_t)n * sizeof(int), cudaMemcpyHostToDevice, q->stream));
    MK(cudaMemsetAsync(q->loss, 0, sizeof(float), q->stream));
    const int nbat = n / batch;
    for (int b = 0; b < nbat; ++b) {
      q->step += 1;
      int rc = mlp_pass(q, x, y, q->idx, b * batch, batch, q->step, lr, 1.f / ((float)batch * MO));
      if (rc) return rc;
    }
    float l = 0.f;
    MK(cudaMemcpyAsync(&l, q->loss, sizeof(float), cudaMemcpyDeviceToHost, q->stream));
    MK(cudaStreamSynchronize(q->stream));
    if (epoch_loss) epoch_loss[e] = l / ((float)nbat * batch * MO);
  }
  return FVG_OK;
}

int fvg_mlp_forward(fvg_mlp* q, const float* x, int32_t n, float* out) {
  if (!q || !x || !out || n < 1) return FVG_ERR_ARG;
  k_mlp_forward<<<std::min((n + FR - 1) / FR, 3 * q->nsm), FR, sizeof(ForwardShared), q->stream>>>(q->par, x, n, out);
  MK(cudaGetLastError());
  MK(cudaStreamSynchronize(q->stream));
  return FVG_OK;
}

const float* fvg_mlp_device_params(const fvg_mlp* q) { return q ? q->par : nullptr; }

int fvg_mlp_forward_bf16(fvg_mlp* q, const float* x, int32_t n, float* out) {
  if (!q || !x || !out || n < 1) return FVG_ERR_ARG;
  if (fvg::closure_setup_attrs()) { q->err = "cannot configure the tensor-core kernel"; return FVG_ERR_CUDA; }
  std::vector<float> h(NPAR);
  MK(cudaStreamSynchronize(q->stream));
  MK(cudaMemcpy(h.data(), q->par, NPAR * sizeof(float), cudaMemcpyDeviceToHost));
  std::vector<uint8_t> img;
  std::vector<float> bias;
  fvg::closure_weight_image(h.data(), img, bias);
  void* dimg = nullptr;
  float* dbias = nullptr;
  int* derr = nullptr;
  int rc = FVG_OK;
  auto cleanup = [&]() {
    if (dimg) cudaFree(dimg);
    if (dbias) cudaFree(dbias);
    if (derr) cudaFree(derr);
  };
  if (cudaMalloc(&dimg, img.size()) != cudaSuccess || cudaMalloc(&dbias, bias.size() * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&derr, sizeof(int)) != cudaSuccess) {
    cleanup();
    return FVG_ERR_NOMEM;
  }
  cudaMemcpy(dimg, img.data(), img.size(), cudaMemcpyHostToDevice);
  cudaMemcpy(dbias, bias.data(), bias.size() * sizeof(float), cudaMemcpyHostToDevice);
  cudaMemset(derr, 0, sizeof(int));
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int tiles = (n + 127) / 128;
  fvg::launch_mlp_tc_forward(dimg, dbias, x, n, out, derr, tiles < 2 * nsm ? tiles : 2 * nsm, q->stream);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(q->stream);
  int herr = 0;
  if (e == cudaSuccess) cudaMemcpy(&herr, derr, sizeof(int), cudaMemcpyDeviceToHost);
  cleanup();
  if (e != cudaSuccess) { q->err = cudaGetErrorString(e); return FVG_ERR_CUDA; }
  if (herr) { q->err = "a tensor-core wait ran out"; rc = FVG_ERR_TIMEOUT; }
  return rc;
}

}  // extern "C"
