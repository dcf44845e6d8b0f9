// atm_mlp_tc.cuh - a 64-wide SiLU MLP on 128-row tiles with tcgen05.mma:
// activations in tensor memory (the A operand), weights in shared memory
// (the B operand, read by the tensor core through descriptors), FP32
// accumulators in tensor memory, SiLU epilogue per row by the thread that
// owns the row.  Shared by the batch forward kernel and the surrogate
// composite.
#pragma once

#include <cuda_bf16.h>

#include <cstdint>

#include "atm_kernels.h"
#include "atm_mlp_tile.cuh"
#include "atm_tc.cuh"

namespace atm {

// Packed tcgen05 layout of one network: per layer the weights as K-major core
// matrices (atm_tc.cuh), N padded to 64 (hidden) or 16 (output; the M = 128
// MMA takes N in steps of 16).  The FP32 bias rides along as three more
// inputs that are always 1: its leading, middle and last eight bits, each a
// BF16, whose products add up to it exactly in the FP32 accumulator - the
// tensor pipe is mostly idle, and an addition and a shared-memory load for
// each of 64 accumulators a row and layer are not.  K is padded to 16 with
// them.  Hidden layers hold W / 2 and b / 2 (SiLU of halves).
__host__ __device__ inline int tc_bias_k(int in_dim) {  // the first of the three
  const int pad = (in_dim + 15) / 16 * 16;
  return pad - in_dim >= 3 ? pad - 3 : pad;
}
__host__ __device__ inline int tc_k_pad(int in_dim) { return (tc_bias_k(in_dim) + 3 + 15) / 16 * 16; }
__host__ __device__ inline int tc_n_pad(int out_dim) { return ((out_dim + 15) / 16) * 16; }
__host__ __device__ inline int tc_layer_bytes(int in_dim, int out_dim) {
  return tc_k_pad(in_dim) * tc_n_pad(out_dim) * 2;
}
// Byte offset of element (n, k) inside a layer's weight block.
__host__ __device__ inline int tc_w_offset(int n, int k, int n_pad) {
  const int s = k >> 4, i = (k >> 3) & 1, j = n >> 3, r = n & 7, e = k & 7;
  return (((s * (n_pad >> 3) + j) * 2 + i) << 7) + r * 16 + e * 2;
}

constexpr uint32_t kTcLbo = 128;  // K-adjacent core matrices
constexpr uint32_t kTcSbo = 256;  // N-adjacent core matrices

// Per-tile state of a network run.
struct TcTile {
  uint32_t tmem_d;     // accumulator columns (64), lane 0
  uint32_t tmem_a;     // activation columns (32), lane 0
  uint32_t tmem_ones;  // the bias's inputs (8 columns, store_ones), lane 0
  uint64_t* mbar;      // MMA completion
  uint32_t phase;      // parity of the next completion
  int tile;            // index of the tile in the CTA (named barrier 1 + tile)
  int row;             // this thread's row 0..127
};

// The bias's three inputs of 1 as the 16 inputs of an MMA step of their own,
// for one thread's row; every row of the block's tiles may share them.
__device__ __forceinline__ void store_ones(uint32_t tmem_ones, int row) {
  const uint32_t ones[8] = {0x3f803f80u, 0x00003f80u, 0, 0, 0, 0, 0, 0};
  tc::st8(tmem_ones + (uint32_t(row & ~31) << 16), ones);
  tc::wait_st();
}

// A row's inputs (unused ones zero) as BF16 pairs, the bias's inputs of 1
// beside them where they leave room.
__device__ __forceinline__ void pack_inputs(const float (&x)[16], int n_in, uint32_t (&xp)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) xp[i] = pack_bf16(x[2 * i], x[2 * i + 1]);
  if (tc_bias_k(n_in) == 13) {
    xp[6] = pack_bf16(x[12], 1.0f);
    xp[7] = 0x3f803f80u;
  }
}

// Runs the network (n_in <= 16 inputs, kHidden layers of 64, n_out <= 8) for
// the tile's 128 rows; every thread of the tile calls with its row's packed
// inputs and receives its row's outputs.  w: generic pointer to the packed
// network in shared memory.  Each completion wait polls the mbarrier at most
// wait_tries times.  Returns false, in every thread of the tile, if a layer's
// MMAs did not complete in time: the outputs are then not valid, no further
// MMA was issued, and exactly one commit (parity T.phase ^ 1) may still be
// in flight - the caller waits for it before it frees the tensor memory or
// runs the tile again.  One barrier a layer: it orders the rows' activations
// (and the reads of D) before the issue, and carries whether every thread saw
// the layer before complete.
template <int kHidden>
__device__ __forceinline__ bool mlp_tile_tc(const unsigned char* w, int n_in, TcTile& T, const uint32_t (&xp)[8],
                                            float (&y)[8], int wait_tries = kTcWaitTries) {
  const uint32_t lane_off = uint32_t(T.row & ~31) << 16;  // the warp's quarter of the lanes
  const bool issuer = T.row == 0;
  tc::st8(T.tmem_a + lane_off, xp);  // inputs -> A columns 0..7 (K = 16)
  tc::wait_st();
  const uint32_t w_saddr = tc::smem_addr(w);
  int off = 0;
  int in_dim = n_in;
  bool ok = true;
#pragma unroll
  for (int l = 0; l <= kHidden; ++l) {
    const bool last = l == kHidden;
    const int out_dim = last ? 16 : kMlpH;
    const int kp = tc_k_pad(in_dim), np = tc_n_pad(out_dim), bias_k = tc_bias_k(in_dim);
    // A complete in every lane -> one thread issues this layer's MMAs
    tc::fence_before_sync();
    if (!tc::tile_all(T.tile, ok)) return false;  // tile-uniform: stop issuing, leave tensor memory alone
    if (issuer) {
      tc::fence_after_sync();
      const uint32_t idesc = tc::idesc_bf16(128, np);
      for (int s = 0; s < kp / 16; ++s) {
        const uint64_t bd = tc::smem_desc(w_saddr + off + s * (np / 8) * 256, kTcLbo, kTcSbo);
        tc::mma_ts(T.tmem_d, 16 * s == bias_k ? T.tmem_ones : T.tmem_a + 8 * s, bd, idesc, s > 0 ? 1u : 0u);
      }
      tc::commit(T.mbar);
    }
    __syncwarp();  // the issuer's warp: tensor-memory loads want it converged
    ok = __all_sync(0xffffffffu, tc::mbar_wait(T.mbar, T.phase, wait_tries));
    T.phase ^= 1u;
    if (ok) {  // warp-uniform
      tc::fence_after_sync();
      if (!last) {
        // SiLU epilogue: D (64 FP32 columns) -> A (32 columns of BF16 pairs)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float v[16];
          tc::ld16(T.tmem_d + lane_off + 16 * c, v);
          uint32_t p[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) p[i] = silu_half_pair(v[2 * i], v[2 * i + 1]);
          tc::st8(T.tmem_a + lane_off + 8 * c, p);
        }
        tc::wait_st();
      } else {
        float v[16];
        tc::ld16(T.tmem_d + lane_off, v);
#pragma unroll
        for (int i = 0; i < 8; ++i) y[i] = v[i];
      }
    }
    off += tc_layer_bytes(in_dim, out_dim);
    in_dim = kMlpH;
  }
  // every lane has read D before the next tile's MMAs overwrite it
  tc::fence_before_sync();
  return tc::tile_all(T.tile, ok);
}

}  // namespace atm
