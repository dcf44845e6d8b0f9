// atm_f32.cuh - IEEE float32 vector arithmetic in a written operation order:
// every multiply, add, divide and square root rounds on its own (no FMA
// contraction), so kernels that restate a float32 reference step by step
// produce its bits.  Shared by the terrain raster and the ocean coverage.
#pragma once

#include <cuda_runtime.h>

namespace atm {
namespace f32 {

struct r3 {
  float x, y, z;
};
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float dv(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ float fmx(float a, float b) { return a > b ? a : b; }
__device__ __forceinline__ float fmn(float a, float b) { return a < b ? a : b; }
__device__ __forceinline__ r3 R3(float x, float y, float z) { return {x, y, z}; }
__device__ __forceinline__ r3 radd(r3 a, r3 b) { return {add(a.x, b.x), add(a.y, b.y), add(a.z, b.z)}; }
__device__ __forceinline__ r3 rsub(r3 a, r3 b) { return {sub(a.x, b.x), sub(a.y, b.y), sub(a.z, b.z)}; }
__device__ __forceinline__ r3 rscale(r3 a, float s) { return {mul(a.x, s), mul(a.y, s), mul(a.z, s)}; }
__device__ __forceinline__ float rdot(r3 a, r3 b) { return add(add(mul(a.x, b.x), mul(a.y, b.y)), mul(a.z, b.z)); }
__device__ __forceinline__ r3 rcross(r3 a, r3 b) {
  return {sub(mul(a.y, b.z), mul(a.z, b.y)), sub(mul(a.z, b.x), mul(a.x, b.z)), sub(mul(a.x, b.y), mul(a.y, b.x))};
}
// Taichi's normalized(): (1 / (|v| + 0)) * v
__device__ __forceinline__ r3 rnormalized(r3 v) {
  const float inv = dv(1.0f, add(__fsqrt_rn(rdot(v, v)), 0.0f));
  return {mul(inv, v.x), mul(inv, v.y), mul(inv, v.z)};
}

// Two floats in a 64-bit register: an .f32x2 instruction is the two scalar
// ones, each with its own rounding.  A product is an fma onto zero (its zeros
// are positive): a bloom plane made with mul.rn.f32x2 and add.rn.f32x2 is 3e-7
// off the reference's, whose products are rounded before they are added.
typedef unsigned long long Pair;
__device__ __forceinline__ Pair pair(float a, float b) {
  Pair r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void halves(Pair p, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p));
}
__device__ __forceinline__ Pair mul(Pair a, Pair b) {
  Pair r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(pair(0.0f, 0.0f)));
  return r;
}
__device__ __forceinline__ Pair mul(Pair a, float w) { return mul(a, pair(w, w)); }
__device__ __forceinline__ Pair add(Pair a, Pair b) {
  Pair r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
}  // namespace f32
}  // namespace atm
