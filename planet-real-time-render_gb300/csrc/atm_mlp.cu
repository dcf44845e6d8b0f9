// atm_mlp.cu - small MLP surrogates: fused FP32 training (forward + backward)
// on CUDA cores, Adam, an FP32 reference forward and a BF16 tensor-core
// forward (mma.sync m16n8k16, FP32 accumulate).
//
// Network: n_in -> [64 SiLU] x n_hidden -> n_out (n_in <= 16, n_out <= 8,
// n_hidden 1..4).  Parameters are one float array: for each layer l, W_l
// (out x in, row-major) then b_l.  The training objective is the mean
// squared error over all outputs of the batch.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "atm_kernels.h"
#include "atm_mlp_tc.cuh"
#include "atm_mlp_tile.cuh"

namespace atm {

namespace {

constexpr int kH = 64;        // hidden width
constexpr int kS = 64;        // samples of a tile
constexpr int kThreads = 256;

// z sigmoid(z), the forward's: the reciprocal is the hardware's with one Newton
// step, within an ulp of the IEEE quotient; 0 for a denominator past 2^126 (z
// below -87.3), the infinite one held at the largest float so that the step
// stays finite.
__device__ __forceinline__ float silu(float z) {
  const float d = fminf(1.0f + expf(-z), FLT_MAX);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  return z * fmaf(fmaf(-d, r, 1.0f), r, r);
}
// The training kernel's sigmoid: the hardware exponential and reciprocal
// (a few ulp; the gradients are checked against the FP64 oracle at 1e-4).
__device__ __forceinline__ float sigmoid_fast(float z) { return __fdividef(1.0f, 1.0f + __expf(-z)); }

// ---- FP32 tiles -----------------------------------------------------------------
// A tile is 64 samples.  Its activations and their gradients lie feature-major
// in shared memory, [feature][sample], weights row-major, [neuron][input], both
// with 4 floats of padding a row, so that a thread's 4 x 4 products read
// nothing but float4s, without bank conflicts, and two FMAs are fed by each
// float read.  Shared memory is still what bounds them (32 floats a cycle
// against 128 FMAs): 4 x 2 products by twice the threads are slower (78 us a
// training step against 65), larger ones do not fit the registers beside the
// weight gradients.
constexpr int kRow = kH + 4;       // row of a 64-wide weight matrix or of 64 samples
constexpr int kInRow = 16 + 4;     // row of the first layer's weights (n_in <= 16)
constexpr int kOutPad = 8;         // output rows (n_out <= 8)

struct Vec4 {
  float v[4];
};
__device__ __forceinline__ Vec4 lds4(const float* p) {
  const float4 f = *reinterpret_cast<const float4*>(p);
  return {f.x, f.y, f.z, f.w};
}
__device__ __forceinline__ void sts4(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
// A warp's threads are 8 sample (or input) groups by 4 neuron groups.
__device__ __forceinline__ int group_wide() { return ((threadIdx.x >> 5) & 1) * 8 + (threadIdx.x & 7); }    // 0..15
__device__ __forceinline__ int group_tall() { return (threadIdx.x >> 6) * 4 + ((threadIdx.x & 31) >> 3); }  // 0..15

// acc[r][c] += sum_k W[j + 16 r][k] in[k][4 s + c], k < 4 quads, in the order of k.
__device__ __forceinline__ void product_forward(const float* __restrict__ W, int w_row, const float* __restrict__ in,
                                                int quads, float (&acc)[4][4]) {
  const int s = group_wide(), j = group_tall();
#pragma unroll 4
  for (int q = 0; q < quads; ++q) {
    Vec4 w[4], a[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) w[r] = lds4(W + (j + 16 * r) * w_row + 4 * q);
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = lds4(in + (4 * q + i) * kRow + 4 * s);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(w[r].v[i], a[i].v[c], acc[r][c]);
  }
}
// acc[r][c] += sum_j W[j][4 k + r] dz[j][4 s + c], j < n.
__device__ __forceinline__ void product_data(const float* __restrict__ W, const float* __restrict__ dz, int n,
                                             float (&acc)[4][4]) {
  const int s = group_wide(), k = group_tall();
#pragma unroll 8
  for (int j = 0; j < n; ++j) {
    const Vec4 w = lds4(W + j * kRow + 4 * k), d = lds4(dz + j * kRow + 4 * s);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(w.v[r], d.v[c], acc[r][c]);
  }
}
// acc[r][c] += sum_s dz[j + 16 r][s] in[k + 16 c][s] over the tile's samples.
__device__ __forceinline__ void product_weights(const float* __restrict__ dz, const float* __restrict__ in,
                                                float (&acc)[4][4]) {
  const int k = group_wide(), j = group_tall();
#pragma unroll 4
  for (int q = 0; q < kS / 4; ++q) {
    Vec4 d[4], a[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) d[r] = lds4(dz + (j + 16 * r) * kRow + 4 * q);
#pragma unroll
    for (int c = 0; c < 4; ++c) a[c] = lds4(in + (k + 16 * c) * kRow + 4 * q);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(d[r].v[i], a[c].v[i], acc[r][c]);
  }
}
__device__ __forceinline__ float sum4(Vec4 a) { return (a.v[0] + a.v[1]) + (a.v[2] + a.v[3]); }
__device__ __forceinline__ float dot4(Vec4 a, Vec4 b, float acc) {
#pragma unroll
  for (int i = 0; i < 4; ++i) acc = fmaf(a.v[i], b.v[i], acc);
  return acc;
}

// Shared-memory layout of a network's FP32 weights (float offsets): rows
// padded, missing inputs and outputs zero.
template <int kHidden>
struct TileWeights {
  static constexpr int kFirst = 0;                                        // [64][kInRow]
  static constexpr int kMiddle = kFirst + kH * kInRow;                    // [kHidden - 1][64][kRow]
  static constexpr int kLast = kMiddle + (kHidden - 1) * kH * kRow;       // [kOutPad][kRow]
  static constexpr int kBias = kLast + kOutPad * kRow;                    // [kHidden][64], [kOutPad]
  static constexpr int kInputs = kBias + kHidden * kH + kOutPad;          // [16][kRow]: the tile's inputs
  static constexpr int kEnd = kInputs + 16 * kRow;
};
template <int kHidden>
__device__ __forceinline__ void load_weights(const MlpShape& m, const float* __restrict__ params, float* sm) {
  using T = TileWeights<kHidden>;
  const int t = threadIdx.x;
  for (int i = t; i < kH * 16; i += kThreads) {
    const int j = i >> 4, k = i & 15;
    sm[T::kFirst + j * kInRow + k] = k < m.n_in ? params[m.off_w[0] + j * m.n_in + k] : 0.0f;
  }
#pragma unroll
  for (int l = 1; l < kHidden; ++l)
    for (int i = t; i < kH * kH; i += kThreads)
      sm[T::kMiddle + (l - 1) * kH * kRow + (i >> 6) * kRow + (i & 63)] = params[m.off_w[l] + i];
  for (int i = t; i < kOutPad * kH; i += kThreads)
    sm[T::kLast + (i >> 6) * kRow + (i & 63)] = (i >> 6) < m.n_out ? params[m.off_w[kHidden] + i] : 0.0f;
#pragma unroll
  for (int l = 0; l < kHidden; ++l)
    if (t < kH) sm[T::kBias + l * kH + t] = params[m.off_b[l] + t];
  if (t < kOutPad) sm[T::kBias + kHidden * kH + t] = t < m.n_out ? params[m.off_b[kHidden] + t] : 0.0f;
  for (int i = t; i < 16 * kRow; i += kThreads) sm[T::kInputs + i] = 0.0f;
}
// The tile's inputs, transposed; rows of samples past n zero.
template <int kHidden>
__device__ __forceinline__ void load_inputs(const MlpShape& m, const float* __restrict__ inputs, long long base,
                                            long long n, float* sm) {
  float* x = sm + TileWeights<kHidden>::kInputs;
  const long long left = (n - base) * m.n_in;
  for (int i = threadIdx.x; i < kS * m.n_in; i += kThreads)
    x[(i % m.n_in) * kRow + i / m.n_in] = i < left ? inputs[base * m.n_in + i] : 0.0f;
}
// Pre-activations of hidden layer l from its inputs, from the bias on.
template <int kHidden>
__device__ __forceinline__ void hidden_layer(const MlpShape& m, const float* sm, int l, const float* in,
                                             float (&acc)[4][4]) {
  using T = TileWeights<kHidden>;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const float b = sm[T::kBias + l * kH + group_tall() + 16 * r];
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = b;
  }
  if (l == 0)
    product_forward(sm + T::kFirst, kInRow, in, (m.n_in + 3) >> 2, acc);
  else
    product_forward(sm + T::kMiddle + (l - 1) * kH * kRow, kRow, in, kH / 4, acc);
}
// Outputs 2 p and 2 p + 1 of sample s = thread & 63, p = thread >> 6.
template <int kHidden>
__device__ __forceinline__ void output_layer(const float* sm, const float* in, float (&y)[2]) {
  using T = TileWeights<kHidden>;
  const int s = threadIdx.x & 63, p = threadIdx.x >> 6;
  const float* w = sm + T::kLast + 2 * p * kRow;
  y[0] = sm[T::kBias + kHidden * kH + 2 * p];
  y[1] = sm[T::kBias + kHidden * kH + 2 * p + 1];
#pragma unroll 4
  for (int q = 0; q < kH / 4; ++q) {
    const Vec4 w0 = lds4(w + 4 * q), w1 = lds4(w + kRow + 4 * q);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float a = in[(4 * q + i) * kRow + s];
      y[0] = fmaf(w0.v[i], a, y[0]);
      y[1] = fmaf(w1.v[i], a, y[1]);
    }
  }
}

template <int kHidden>
constexpr int train_floats() {  // weights and inputs, A and D of each hidden layer, the outputs' gradients
  return TileWeights<kHidden>::kEnd + 2 * kHidden * kH * kRow + kOutPad * kRow;
}

// Fused forward + backward.  Each block stays for the launch: it walks tiles
// of 64 samples with the gradients of all weights in its threads' registers,
// and writes them once (its row of grad_partial, and its squared-error sum).
// A[l] holds layer l's activations, D[l] their derivative and then, in its
// place, the gradient of its pre-activations.  A step of 16,384 samples (11 ->
// 4 x 64 -> 6) takes 65 us with its reduction, 178 us when each 64-sample block
// wrote a gradient row of its own and four launches followed.
template <int kHidden>
__global__ void __launch_bounds__(kThreads, 1) k_mlp_grad(MlpShape m, const float* __restrict__ params,
                                                          const float* __restrict__ inputs,
                                                          const float* __restrict__ targets,
                                                          const float* __restrict__ weights, long long n,
                                                          float inv_count, float* __restrict__ grad_partial,
                                                          float* __restrict__ loss_partial) {
  using T = TileWeights<kHidden>;
  extern __shared__ __align__(16) float sm[];
  __shared__ float s_red[kThreads / 32];
  float* A = sm + T::kEnd;
  float* D = A + kHidden * kH * kRow;
  float* dY = D + kHidden * kH * kRow;
  constexpr int kPlane = kH * kRow;
  const int t = threadIdx.x;
  float gw[kHidden > 1 ? kHidden - 1 : 1][4][4] = {}, gb[kHidden] = {}, g_first[4] = {}, g_last[2] = {}, gb_last = 0.0f;
  float sq = 0.0f;
  load_weights<kHidden>(m, params, sm);
  for (long long base = blockIdx.x * (long long)kS; base < n; base += gridDim.x * (long long)kS) {
    __syncthreads();  // the weights are in; the tile before is done with its inputs
    load_inputs<kHidden>(m, inputs, base, n, sm);
    __syncthreads();
    const int wide = group_wide(), tall = group_tall();
#pragma unroll
    for (int l = 0; l < kHidden; ++l) {
      float acc[4][4];
      hidden_layer<kHidden>(m, sm, l, l == 0 ? sm + T::kInputs : A + (l - 1) * kPlane, acc);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        float a[4], d[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float z = acc[r][c], sg = sigmoid_fast(z);
          a[c] = z * sg;
          d[c] = sg * (1.0f + z * (1.0f - sg));
        }
        sts4(A + l * kPlane + (tall + 16 * r) * kRow + 4 * wide, a);
        sts4(D + l * kPlane + (tall + 16 * r) * kRow + 4 * wide, d);
      }
      __syncthreads();
    }
    // loss and output gradient (mean over batch x outputs)
    {
      float y[2];
      output_layer<kHidden>(sm, A + (kHidden - 1) * kPlane, y);
      const int s = t & 63, o = 2 * (t >> 6);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float g = 0.0f;
        if (base + s < n && o + i < m.n_out) {
          const long long at = (base + s) * m.n_out + o + i;
          const float d = y[i] - targets[at];
          const float w = weights != nullptr ? weights[at] : 1.0f;
          sq += w * d * d;
          g = 2.0f * w * d * inv_count;
        }
        dY[(o + i) * kRow + s] = g;
      }
    }
    __syncthreads();
    // the output layer's weights (row t >> 5, inputs t & 31 and + 32) and biases
    {
      const float* dz = dY + (t >> 5) * kRow;
      const float* a = A + (kHidden - 1) * kPlane + (t & 31) * kRow;
#pragma unroll 4
      for (int q = 0; q < kS / 4; ++q) {
        const Vec4 d = lds4(dz + 4 * q);
        g_last[0] = dot4(d, lds4(a + 4 * q), g_last[0]);
        g_last[1] = dot4(d, lds4(a + 32 * kRow + 4 * q), g_last[1]);
      }
      if (t < 4 * kOutPad)
        for (int q = t & 3; q < kS / 4; q += 4) gb_last += sum4(lds4(dY + (t >> 2) * kRow + 4 * q));
    }
#pragma unroll
    for (int l = kHidden - 1; l >= 0; --l) {
      // gradient of layer l's pre-activations, in place of its derivative
      float acc[4][4] = {};
      if (l == kHidden - 1)
        product_data(sm + T::kLast, dY, m.n_out, acc);
      else
        product_data(sm + T::kMiddle + l * kH * kRow, D + (l + 1) * kPlane, kH, acc);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        float* d = D + l * kPlane + (4 * tall + r) * kRow + 4 * wide;
        const Vec4 v = lds4(d);
        float o[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) o[c] = acc[r][c] * v.v[c];
        sts4(d, o);
      }
      __syncthreads();
      const float* dz = D + l * kPlane;
      if (l > 0) {
        product_weights(dz, A + (l - 1) * kPlane, gw[l - 1]);
      } else {  // inputs (t & 3) + 4 c of neuron t >> 2
        const float* x = sm + T::kInputs + (t & 3) * kRow;
#pragma unroll 4
        for (int q = 0; q < kS / 4; ++q) {
          const Vec4 d = lds4(dz + (t >> 2) * kRow + 4 * q);
#pragma unroll
          for (int c = 0; c < 4; ++c) g_first[c] = dot4(d, lds4(x + 4 * c * kRow + 4 * q), g_first[c]);
        }
      }
      for (int q = t & 3; q < kS / 4; q += 4) gb[l] += sum4(lds4(dz + (t >> 2) * kRow + 4 * q));
    }
  }
  // this block's gradients
  float* gp = grad_partial + static_cast<long long>(blockIdx.x) * m.n_params;
  const int k0 = group_wide(), j0 = group_tall();
#pragma unroll
  for (int l = 1; l < kHidden; ++l)
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) gp[m.off_w[l] + (j0 + 16 * r) * kH + k0 + 16 * c] = gw[l - 1][r][c];
#pragma unroll
  for (int c = 0; c < 4; ++c)
    if ((t & 3) + 4 * c < m.n_in) gp[m.off_w[0] + (t >> 2) * m.n_in + (t & 3) + 4 * c] = g_first[c];
  if ((t >> 5) < m.n_out) {
    gp[m.off_w[kHidden] + (t >> 5) * kH + (t & 31)] = g_last[0];
    gp[m.off_w[kHidden] + (t >> 5) * kH + (t & 31) + 32] = g_last[1];
  }
#pragma unroll
  for (int l = 0; l < kHidden; ++l) {  // four threads a bias
    gb[l] += __shfl_xor_sync(0xffffffffu, gb[l], 1);
    gb[l] += __shfl_xor_sync(0xffffffffu, gb[l], 2);
    if ((t & 3) == 0) gp[m.off_b[l] + (t >> 2)] = gb[l];
  }
  gb_last += __shfl_xor_sync(0xffffffffu, gb_last, 1);
  gb_last += __shfl_xor_sync(0xffffffffu, gb_last, 2);
  if ((t & 3) == 0 && (t >> 2) < m.n_out) gp[m.off_b[kHidden] + (t >> 2)] = gb_last;
  // squared-error sum of the block
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
  if ((t & 31) == 0) s_red[t >> 5] = sq;
  __syncthreads();
  if (t == 0) {
    float total = 0.0f;
    for (int w = 0; w < kThreads / 32; ++w) total += s_red[w];
    loss_partial[blockIdx.x] = total;
  }
}

// Adam's state and rates; params null: the gradient alone.
struct AdamStep {
  float *params, *m1, *m2;
  float lr, b1, b2, eps, c1, c2;
};
// grad[p] = sum of the rows of partial in a fixed order, then Adam's update of
// parameter p; the last block sums the losses (if out).  Eight groups of rows
// by 32 parameters a block: a serial sum over the rows by one thread a
// parameter is a chain of their loads.
constexpr int kReduceGroups = 8;
__global__ void __launch_bounds__(32 * kReduceGroups) k_reduce_adam(const float* __restrict__ partial, int rows,
                                                                    int n_params, float* __restrict__ grad,
                                                                    const float* __restrict__ loss_partial,
                                                                    float* __restrict__ loss, AdamStep S) {
  __shared__ float s_sum[kReduceGroups][32];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  const bool losses = blockIdx.x == gridDim.x - 1;
  const int p = blockIdx.x * 32 + lane;
  float acc = 0.0f;
  if (losses) {
    if (loss != nullptr)
      for (int c = threadIdx.x; c < rows; c += 32 * kReduceGroups) acc += loss_partial[c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  } else if (p < n_params) {
#pragma unroll 4
    for (int c = g; c < rows; c += kReduceGroups) acc += partial[static_cast<long long>(c) * n_params + p];
  }
  s_sum[g][lane] = acc;
  __syncthreads();
  if (g != 0) return;
  acc = 0.0f;
#pragma unroll
  for (int k = 0; k < kReduceGroups; ++k) acc += s_sum[k][lane];
  if (losses) {
    if (loss != nullptr && lane == 0) *loss = acc;
    return;
  }
  if (p >= n_params) return;
  grad[p] = acc;
  if (S.params == nullptr) return;
  const float a = S.b1 * S.m1[p] + (1.0f - S.b1) * acc;
  const float v = S.b2 * S.m2[p] + (1.0f - S.b2) * acc * acc;
  S.m1[p] = a;
  S.m2[p] = v;
  S.params[p] -= S.lr * (a / S.c1) / (sqrtf(v / S.c2) + S.eps);
}

// FP32 forward (reference path of the BF16 kernels): the same tiles, two
// blocks an SM; every output is summed in the order of a sample-by-sample
// forward.  65,536 samples (11 -> 4 x 64 -> 6): 54 us; 64 us with an IEEE
// division in each SiLU, 440 us at one thread a sample with the weights read
// through L1.  8 x 8 products by 64 threads a tile halve the shared-memory
// reads and take 54 us too (20 us instead of 13 for 4,096 samples).
template <int kHidden>
constexpr int forward_floats() {
  return TileWeights<kHidden>::kEnd + 2 * kH * kRow;
}
template <int kHidden>
__global__ void __launch_bounds__(kThreads, 2) k_mlp_forward_f32(MlpShape m, const float* __restrict__ params,
                                                                const float* __restrict__ inputs,
                                                                float* __restrict__ outputs, long long n) {
  using T = TileWeights<kHidden>;
  extern __shared__ __align__(16) float sm[];
  float* A = sm + T::kEnd;
  constexpr int kPlane = kH * kRow;
  load_weights<kHidden>(m, params, sm);
  for (long long base = blockIdx.x * (long long)kS; base < n; base += gridDim.x * (long long)kS) {
    __syncthreads();
    load_inputs<kHidden>(m, inputs, base, n, sm);
    __syncthreads();
#pragma unroll
    for (int l = 0; l < kHidden; ++l) {
      float acc[4][4];
      hidden_layer<kHidden>(m, sm, l, l == 0 ? sm + T::kInputs : A + ((l - 1) & 1) * kPlane, acc);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        float a[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) a[c] = silu(acc[r][c]);
        sts4(A + (l & 1) * kPlane + (group_tall() + 16 * r) * kRow + 4 * group_wide(), a);
      }
      __syncthreads();
    }
    float y[2];
    output_layer<kHidden>(sm, A + ((kHidden - 1) & 1) * kPlane, y);
    const int s = threadIdx.x & 63, o = 2 * (threadIdx.x >> 6);
    if (base + s < n)
      for (int i = 0; i < 2; ++i)
        if (o + i < m.n_out) outputs[(base + s) * m.n_out + o + i] = y[i];
  }
}

}  // namespace

// Byte size of the packed BF16 network.
size_t mlp_bf16_bytes(const MlpShape& m) {
  size_t bytes = 0;
  for (int l = 0; l < m.n_layers; ++l) {
    const int op = mlp_bf16_out_pad(m.out_dim[l]);
    bytes += size_t(op) * mlp_bf16_layer_row(m.in_dim[l]) * 2;
    bytes += size_t(op) * 4;
  }
  return bytes;
}

namespace {

// Hidden layers are stored with W and b halved (exact in BF16), so their
// accumulators hold z / 2 for the packed SiLU of mlp_tile_bf16.
__global__ void k_pack_bf16(MlpShape m, const float* __restrict__ params, unsigned char* __restrict__ packed) {
  size_t off = 0;
  for (int l = 0; l < m.n_layers; ++l) {
    const int in = m.in_dim[l], out = m.out_dim[l];
    const int row = mlp_bf16_layer_row(in), op = mlp_bf16_out_pad(out);
    const float scale = l + 1 < m.n_layers ? 0.5f : 1.0f;
    __nv_bfloat16* W = reinterpret_cast<__nv_bfloat16*>(packed + off);
    for (int i = threadIdx.x; i < op * row; i += blockDim.x) {
      const int j = i / row, k = i % row;
      const float v = (j < out && k < in) ? params[m.off_w[l] + j * in + k] : 0.0f;
      W[i] = __float2bfloat16_rn(v * scale);
    }
    off += size_t(op) * row * 2;
    float* b = reinterpret_cast<float*>(packed + off);
    for (int j = threadIdx.x; j < op; j += blockDim.x) b[j] = j < out ? params[m.off_b[l] + j] * scale : 0.0f;
    off += size_t(op) * 4;
  }
}

// tcgen05 layout of a network (atm_mlp_tc.cuh): weights as K-major core
// matrices, hidden layers halved.
__global__ void k_pack_tc(MlpShape m, const float* __restrict__ params, unsigned char* __restrict__ packed) {
  int off = 0;
  for (int l = 0; l < m.n_layers; ++l) {
    const int in = m.in_dim[l], out = m.out_dim[l];
    const int kp = tc_k_pad(in), np = tc_n_pad(out), bk = tc_bias_k(in);
    const float scale = l + 1 < m.n_layers ? 0.5f : 1.0f;
    for (int i = threadIdx.x; i < kp * np; i += blockDim.x) {
      const int n = i / kp, k = i % kp;
      float v = 0.0f;
      if (n < out && k < in) {
        v = params[m.off_w[l] + n * in + k] * scale;
      } else if (n < out && k >= bk && k < bk + 3) {  // the bias in three BF16 parts
        v = params[m.off_b[l] + n] * scale;
        for (int part = bk; part < k; ++part) v = isinf(v) ? 0.0f : v - __bfloat162float(__float2bfloat16_rn(v));
      }
      *reinterpret_cast<__nv_bfloat16*>(packed + off + tc_w_offset(n, k, np)) = __float2bfloat16_rn(v);
    }
    off += tc_layer_bytes(in, out);
  }
}

// Forward of n samples on the tcgen05 path: one tile of 128 samples per
// block at a time (grid-stride); TMEM: accumulators at column 0, activations
// at column 128 and the bias's ones at 192 of a 256-column allocation.  *error is set when an MMA did
// not complete in time.
template <int kHidden>
__global__ void __launch_bounds__(128) k_mlp_forward_tc(MlpShape m, const unsigned char* __restrict__ packed,
                                                        int packed_bytes, const float* __restrict__ inputs,
                                                        float* __restrict__ outputs, long long n,
                                                        int* __restrict__ error) {
  extern __shared__ __align__(128) unsigned char smw[];
  __shared__ __align__(8) uint64_t s_mbar;
  __shared__ uint32_t s_tmem;
  for (int i = threadIdx.x * 16; i < packed_bytes; i += blockDim.x * 16)
    *reinterpret_cast<uint4*>(smw + i) = *reinterpret_cast<const uint4*>(packed + i);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic writes -> tensor-core reads
  if (threadIdx.x < 32) tc::alloc(&s_tmem, 256);
  if (threadIdx.x == 0) {
    tc::mbar_init(&s_mbar, 1);
    tc::mbar_init_fence();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  TcTile T{s_tmem, s_tmem + 128, s_tmem + 192, &s_mbar, 0u, 0, int(threadIdx.x)};
  store_ones(T.tmem_ones, T.row);
  bool ok = true;
  for (long long base = blockIdx.x * 128LL; base < n; base += gridDim.x * 128LL) {
    const long long r = base + threadIdx.x;
    float x[16] = {}, y[8];
    if (r < n)
      for (int k = 0; k < m.n_in; ++k) x[k] = inputs[r * m.n_in + k];
    uint32_t xp[8];
    pack_inputs(x, m.n_in, xp);
    ok = mlp_tile_tc<kHidden>(smw, m.n_in, T, xp, y);
    if (!ok) break;  // block-uniform (one tile per block); no MMA is issued after it
    if (r < n)
      for (int k = 0; k < m.n_out; ++k) outputs[r * m.n_out + k] = y[k];
  }
  if (!ok && threadIdx.x == 0) atomicExch(error, 1);
  // before the tensor memory is freed, no MMA of this CTA may be in flight:
  // after a timed-out wait, wait once more (bounded) for its one commit
  tc::fence_before_sync();
  if (__syncthreads_or(!ok)) tc::mbar_wait(&s_mbar, T.phase ^ 1u, kTcWaitTries);
  __syncthreads();
  tc::fence_after_sync();
  if (threadIdx.x < 32) tc::dealloc(s_tmem, 256);
}

// The weights (whole 16-byte pieces) are copied once a block: few blocks of
// eight warps, each with several 16-row tiles (65,536 samples: 14 us, 41 us
// with a copy every 64 rows).
constexpr int kBf16Threads = 256;
template <int kHidden>
__global__ void __launch_bounds__(kBf16Threads) k_mlp_forward_bf16(MlpShape m, const unsigned char* __restrict__ packed,
                                                                   int packed_bytes, const float* __restrict__ inputs,
                                                                   float* __restrict__ outputs, long long n) {
  extern __shared__ __align__(128) unsigned char smw[];
  for (int i = threadIdx.x * 16; i < packed_bytes; i += blockDim.x * 16)
    *reinterpret_cast<uint4*>(smw + i) = *reinterpret_cast<const uint4*>(packed + i);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2, q = lane & 3;
  const int in0_row = mlp_bf16_layer_row(m.n_in);
  const long long warps = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  for (long long tile = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); tile * 16 < n; tile += warps) {
    const long long r0 = tile * 16 + g, r1 = r0 + 8;
    auto in = [&](long long r, int k) { return (r < n && k < m.n_in) ? inputs[r * m.n_in + k] : 0.0f; };
    uint32_t x[4];
    x[0] = pack_bf16(in(r0, 2 * q), in(r0, 2 * q + 1));
    x[1] = pack_bf16(in(r1, 2 * q), in(r1, 2 * q + 1));
    x[2] = pack_bf16(in(r0, 8 + 2 * q), in(r0, 8 + 2 * q + 1));
    x[3] = pack_bf16(in(r1, 8 + 2 * q), in(r1, 8 + 2 * q + 1));
    float y[4];
    mlp_tile_bf16<kHidden>(smw, x, in0_row, y);
    for (int i = 0; i < 2; ++i) {
      const int o = 2 * q + i;
      if (o < m.n_out) {
        if (r0 < n) outputs[r0 * m.n_out + o] = y[i];
        if (r1 < n) outputs[r1 * m.n_out + o] = y[2 + i];
      }
    }
  }
}

}  // namespace

MlpShape make_mlp_shape(int n_in, int n_hidden, int n_out) {
  MlpShape m{};
  m.n_in = n_in;
  m.n_out = n_out;
  m.n_layers = n_hidden + 1;
  int off = 0;
  for (int l = 0; l < m.n_layers; ++l) {
    m.in_dim[l] = l == 0 ? n_in : kH;
    m.out_dim[l] = l == n_hidden ? n_out : kH;
    m.off_w[l] = off;
    off += m.in_dim[l] * m.out_dim[l];
    m.off_b[l] = off;
    off += m.out_dim[l];
  }
  m.n_params = off;
  return m;
}

// Blocks of a training launch: one an SM, and no more than there are tiles.
int mlp_train_ctas(long long n, int sm_count) { return int(std::min<long long>((n + kS - 1) / kS, sm_count)); }

namespace {
// Calls f with the network's hidden-layer count as a constant.
template <class F>
cudaError_t with_hidden(const MlpShape& m, F f) {
  switch (m.n_layers - 1) {
    case 1: return f(std::integral_constant<int, 1>{});
    case 2: return f(std::integral_constant<int, 2>{});
    case 3: return f(std::integral_constant<int, 3>{});
    case 4: return f(std::integral_constant<int, 4>{});
    default: return cudaErrorInvalidValue;
  }
}
cudaError_t launch_reduce(const float* partial, int rows, int n_params, float* grad, const float* loss_partial,
                          float* loss, const AdamStep& step, cudaStream_t s) {
  k_reduce_adam<<<(n_params + 31) / 32 + 1, 32 * kReduceGroups, 0, s>>>(partial, rows, n_params, grad, loss_partial,
                                                                       loss, step);
  return cudaGetLastError();
}
}  // namespace

cudaError_t launch_mlp_grad(const MlpShape& m, const float* params, const float* inputs, const float* targets,
                            const float* weights, long long n, float* grad_partial, float* loss_partial, int sm_count,
                            cudaStream_t s) {
  const float inv = 1.0f / float(double(n) * m.n_out);
  return with_hidden(m, [&](auto hidden) {
    constexpr int kBytes = train_floats<hidden.value>() * int(sizeof(float));
    cudaError_t e =
        cudaFuncSetAttribute(k_mlp_grad<hidden.value>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
    if (e != cudaSuccess) return e;
    k_mlp_grad<hidden.value><<<mlp_train_ctas(n, sm_count), kThreads, kBytes, s>>>(
        m, params, inputs, targets, weights, n, inv, grad_partial, loss_partial);
    return cudaGetLastError();
  });
}

cudaError_t launch_mlp_reduce(const MlpShape& m, const float* grad_partial, int rows, float* grad,
                              const float* loss_partial, float* loss, cudaStream_t s) {
  return launch_reduce(grad_partial, rows, m.n_params, grad, loss_partial, loss, AdamStep{}, s);
}

cudaError_t launch_mlp_adam(const MlpShape& m, const float* grad_partial, int rows, float* grad,
                            const float* loss_partial, float* loss, float* params, float* m1, float* m2, float lr,
                            float b1, float b2, float eps, long long step, cudaStream_t s) {
  const float c1 = 1.0f - float(pow(double(b1), double(step)));
  const float c2 = 1.0f - float(pow(double(b2), double(step)));
  return launch_reduce(grad_partial, rows, m.n_params, grad, loss_partial, loss,
                       AdamStep{params, m1, m2, lr, b1, b2, eps, c1, c2}, s);
}

cudaError_t launch_mlp_forward_f32(const MlpShape& m, const float* params, const float* inputs, float* outputs,
                                   long long n, int sm_count, cudaStream_t s) {
  const int blocks = int(std::min<long long>((n + kS - 1) / kS, 2LL * sm_count));
  return with_hidden(m, [&](auto hidden) {
    constexpr int kBytes = forward_floats<hidden.value>() * int(sizeof(float));
    cudaError_t e =
        cudaFuncSetAttribute(k_mlp_forward_f32<hidden.value>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
    if (e != cudaSuccess) return e;
    k_mlp_forward_f32<hidden.value><<<blocks, kThreads, kBytes, s>>>(m, params, inputs, outputs, n);
    return cudaGetLastError();
  });
}

size_t mlp_tc_bytes(const MlpShape& m) {
  size_t b = 0;
  for (int l = 0; l < m.n_layers; ++l) b += size_t(tc_layer_bytes(m.in_dim[l], m.out_dim[l]));
  return b;
}

cudaError_t launch_mlp_pack_tc(const MlpShape& m, const float* params, void* packed, cudaStream_t s) {
  k_pack_tc<<<1, 256, 0, s>>>(m, params, static_cast<unsigned char*>(packed));
  return cudaGetLastError();
}

cudaError_t launch_mlp_forward_tc(const MlpShape& m, const void* packed, const float* inputs, float* outputs,
                                  long long n, int* error, int sm_count, cudaStream_t s) {
  const int bytes = int(mlp_tc_bytes(m));
  const unsigned blocks = unsigned(std::min<long long>((n + 127) / 128, 2LL * sm_count));
  const auto* p = static_cast<const unsigned char*>(packed);
  cudaError_t e = cudaSuccess;
  switch (m.n_layers - 1) {
    case 1: e = cudaFuncSetAttribute(k_mlp_forward_tc<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
      if (e == cudaSuccess) k_mlp_forward_tc<1><<<blocks, 128, bytes, s>>>(m, p, bytes, inputs, outputs, n, error);
      break;
    case 2: e = cudaFuncSetAttribute(k_mlp_forward_tc<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
      if (e == cudaSuccess) k_mlp_forward_tc<2><<<blocks, 128, bytes, s>>>(m, p, bytes, inputs, outputs, n, error);
      break;
    case 3: e = cudaFuncSetAttribute(k_mlp_forward_tc<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
      if (e == cudaSuccess) k_mlp_forward_tc<3><<<blocks, 128, bytes, s>>>(m, p, bytes, inputs, outputs, n, error);
      break;
    case 4: e = cudaFuncSetAttribute(k_mlp_forward_tc<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
      if (e == cudaSuccess) k_mlp_forward_tc<4><<<blocks, 128, bytes, s>>>(m, p, bytes, inputs, outputs, n, error);
      break;
    default: return cudaErrorInvalidValue;
  }
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}

cudaError_t launch_mlp_pack_bf16(const MlpShape& m, const float* params, void* packed, cudaStream_t s) {
  k_pack_bf16<<<1, 256, 0, s>>>(m, params, static_cast<unsigned char*>(packed));
  return cudaGetLastError();
}

cudaError_t launch_mlp_forward_bf16(const MlpShape& m, const void* packed, const float* inputs, float* outputs,
                                    long long n, int sm_count, cudaStream_t s) {
  const int bytes = int(mlp_bf16_bytes(m));
  const unsigned blocks = unsigned(std::min<long long>((n + 127) / 128, 3LL * sm_count));
  const auto* p = static_cast<const unsigned char*>(packed);
  switch (m.n_layers - 1) {
    case 1: k_mlp_forward_bf16<1><<<blocks, kBf16Threads, bytes, s>>>(m, p, bytes, inputs, outputs, n); break;
    case 2: k_mlp_forward_bf16<2><<<blocks, kBf16Threads, bytes, s>>>(m, p, bytes, inputs, outputs, n); break;
    case 3: k_mlp_forward_bf16<3><<<blocks, kBf16Threads, bytes, s>>>(m, p, bytes, inputs, outputs, n); break;
    case 4: k_mlp_forward_bf16<4><<<blocks, kBf16Threads, bytes, s>>>(m, p, bytes, inputs, outputs, n); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace atm
