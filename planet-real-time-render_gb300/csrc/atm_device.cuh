// atm_device.cuh - device math of the spherical-atmosphere model (sm_103a).
//
// FP32 formulation of the reference's Taichi functions in
// src/planet_renderer/atmosphere/renderer.py (line numbers below).  The
// arithmetic follows the reference expression by expression so results agree
// with it to float rounding; where the reference evaluates the same quantity
// twice with identical inputs (density in extinction and source; horizon and
// sun zenith in disk visibility and representative zenith; a base
// interval's upper boundary and the next one's lower boundary; the
// terminator weight's midpoint visibility and the coarse sample's) it is
// evaluated once here - same inputs, same operations, same value.
//
// LUT storage: float4 texels (rgb + pad), row-major, index y * width + x;
// the aerial volume is [z][y][x].  Reads go through the read-only path.
#pragma once

#include <cmath>
#include <cstdint>

namespace atm {

constexpr float kPiF = 3.14159265358979323846f;  // f32(math.pi), renderer.py:12
constexpr float kLargeF = 1.0e30f;               // _LARGE_DISTANCE, :13

// A 2D LUT's size as its bilinear tap reads it: width and height, 2^23 plus
// the last texel that has a right (lower) neighbour, and the row pitch.  LUTs
// are at least 2 x 2.
struct LutDims {
  float w, h, x_last, y_last;
  int pitch;
};
constexpr float kMagic = 8388608.0f;  // 2^23: adding it leaves floor(x) in the low mantissa bits
__host__ __device__ inline LutDims lut_dims(int w, int h) {
  return {float(w), float(h), kMagic + float(w - 2), kMagic + float(h - 2), w};
}

// Parameters rounded to float exactly where the Taichi trace rounds them
// (Python constants fold in double, then meet f32 values).
struct DevParams {
  float top;                   // top_altitude_m
  float beta_r[3];             // Rayleigh scattering
  float beta_ms[3];            // Mie scattering
  float beta_me[3];            // Mie extinction
  float beta_o[3];             // ozone absorption
  float albedo[3];             // ground albedo
  float h_r, h_m;              // scale heights
  float oz_peak, oz_half;      // ozone tent
  float mie_c1, mie_c2;        // f32(1+g^2), f32(2g)
  float mie_k1, mie_k2;        // f32(3(1-g^2)), f32(8 pi (2+g^2))
  float ray_k;                 // f32(16 pi)
  float exp2_r, exp2_m;        // -log2(e) / scale height: exp(-h / H) = 2^(h exp2)
  float inv_oz_half, inv_top;  // f32 reciprocals of the above
  float ms_half_w;                // half the multi-scattering LUT's width
  LutDims t_lut, ms_lut, sv_lut;  // of the transmittance, multi-scattering and sky-view LUTs
  int t_w, t_h, ms_w, ms_h, sv_w, sv_h, ap_w, ap_h, ap_d;
  int t_steps, ms_dirs, ms_steps, sv_steps, ap_steps, limb_steps, substeps;
};

struct f3 {
  float x, y, z;
};
__device__ __forceinline__ f3 mk(float x, float y, float z) { return {x, y, z}; }
__device__ __forceinline__ f3 splat(float s) { return {s, s, s}; }
__device__ __forceinline__ f3 operator+(f3 a, f3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ f3 operator-(f3 a, f3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ f3 operator-(f3 a) { return {-a.x, -a.y, -a.z}; }
__device__ __forceinline__ f3 operator*(f3 a, f3 b) { return {a.x * b.x, a.y * b.y, a.z * b.z}; }
__device__ __forceinline__ f3 operator*(f3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ f3 operator/(f3 a, float s) { return {a.x / s, a.y / s, a.z / s}; }
__device__ __forceinline__ f3 operator/(f3 a, f3 b) { return {a.x / b.x, a.y / b.y, a.z / b.z}; }
__device__ __forceinline__ float dot(f3 a, f3 b) { return (a.x * b.x + a.y * b.y) + a.z * b.z; }
__device__ __forceinline__ float norm(f3 a) { return sqrtf(dot(a, a)); }
// For a NaN first argument the second one, as a > b ? a : b gives it.
__device__ __forceinline__ float mx(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ float mn(float a, float b) { return fminf(a, b); }
__device__ __forceinline__ float clampf(float x, float lo, float hi) { return mn(mx(x, lo), hi); }
__device__ __forceinline__ f3 vmax(f3 a, float s) { return {mx(a.x, s), mx(a.y, s), mx(a.z, s)}; }
__device__ __forceinline__ f3 vmin(f3 a, float s) { return {mn(a.x, s), mn(a.y, s), mn(a.z, s)}; }
__device__ __forceinline__ f3 vclamp(f3 a, float lo, float hi) { return vmin(vmax(a, lo), hi); }
__device__ __forceinline__ f3 vexp(f3 a) { return {expf(a.x), expf(a.y), expf(a.z)}; }
__device__ __forceinline__ f3 ld3(const float* p) { return {p[0], p[1], p[2]}; }
__device__ __forceinline__ f3 from4(float4 v) { return {v.x, v.y, v.z}; }
__device__ __forceinline__ float4 to4(f3 v) { return make_float4(v.x, v.y, v.z, 0.0f); }
__device__ __forceinline__ f3 arr3(const float (&a)[3]) { return {a[0], a[1], a[2]}; }

// Fast forms used where no Earth-scale cancellation follows: division with
// at most 2 ulp error (div.approx), and the hardware's reciprocal, square
// root and 2^x.  Differences ~1e-7 relative against the reference's IEEE
// operations, far below the 1e-3 parity tolerance.  Subtractions of two
// Earth-scale quantities keep IEEE sqrtf / division (see callers).  The .ftz
// forms flush subnormals, of which these paths have none that matters (the
// smallest, a density, is subnormal past 87 scale heights), and are faster.
__device__ __forceinline__ float fdiv(float a, float b) { return __fdividef(a, b); }
__device__ __forceinline__ float frcp(float b) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
  return r;
}
__device__ __forceinline__ float fsqrt(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float frsqrt(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float fexp2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Adds a per-lane count into a device counter: one atomic per warp.  Every
// lane of the warp must call it (no lane may have exited before).
__device__ __forceinline__ void warp_count(uint32_t n, unsigned long long* counter) {
  __syncwarp();
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  if (counter != nullptr && (threadIdx.x & 31) == 0 && n) atomicAdd(counter, (unsigned long long)n);
}

// Composition of two consecutive ray segments: (L1,T1) then (L2,T2).
struct Seg {
  f3 L, T;
};
__device__ __forceinline__ Seg seg_then(Seg a, Seg b) { return {a.L + a.T * b.L, a.T * b.T}; }

// ---- density and coefficients (:168-209) ----------------------------------
struct Density {
  float r, m, o;
};
// Zero outside the shell: at an infinite altitude the exponentials are 0 and
// the ozone tent has ended.
__device__ __forceinline__ Density density(const DevParams& P, float h) {
  const float a = 0.0f <= h && h <= P.top ? h : INFINITY;
  Density d;
  d.r = fexp2(a * P.exp2_r);
  d.m = fexp2(a * P.exp2_m);
  d.o = mx(1.0f - fabsf(a - P.oz_peak) * P.inv_oz_half, 0.0f);
  return d;
}
// Extinction and scattering of one density share the Rayleigh products.
struct Medium {
  f3 ext, scat;
};
__device__ __forceinline__ Medium medium_of(const DevParams& P, Density d) {
  const f3 r = arr3(P.beta_r) * d.r;
  Medium m;
  m.ext = {fmaf(P.beta_o[0], d.o, fmaf(P.beta_me[0], d.m, r.x)), fmaf(P.beta_o[1], d.o, fmaf(P.beta_me[1], d.m, r.y)),
           fmaf(P.beta_o[2], d.o, fmaf(P.beta_me[2], d.m, r.z))};
  m.scat = {fmaf(P.beta_ms[0], d.m, r.x), fmaf(P.beta_ms[1], d.m, r.y), fmaf(P.beta_ms[2], d.m, r.z)};
  return m;
}
__device__ __forceinline__ f3 extinction_of(const DevParams& P, Density d) {
  return (arr3(P.beta_r) * d.r + arr3(P.beta_me) * d.m) + arr3(P.beta_o) * d.o;
}

// ---- shells and intervals (:211-408) ---------------------------------------
__device__ __forceinline__ void sphere_roots(f3 o, f3 d, float radius, float& nearv, float& farv, bool& hit) {
  float projected = dot(o, d);
  float perpendicular = norm(o - d * projected);
  float clearance = radius - perpendicular;
  hit = clearance >= 0.0f;
  nearv = kLargeF;
  farv = -kLargeF;
  if (hit) {
    float root = sqrtf(mx(mx(clearance, 0.0f) * (radius + perpendicular), 0.0f));
    nearv = -projected - root;
    farv = -projected + root;
  }
}
__device__ __forceinline__ float shell_rho(float h, float bottom) {
  float a = mx(h, 0.0f);
  return fsqrt(a * (2.0f * bottom + a));
}
// Cancellation-free form: the altitude never subtracts two Earth-scale radii.
__device__ __forceinline__ float altitude_on_ray(float h0, float cosv, float t, float bottom) {
  float a = mx(h0, 0.0f);
  float orad = bottom + a;
  float delta = (a * (2.0f * bottom + a) + 2.0f * orad * cosv * t) + t * t;
  float len = fsqrt(mx(bottom * bottom + delta, 0.0f));
  return fdiv(delta, mx(len + bottom, 1.0f));
}
__device__ __forceinline__ void shell_roots(float h0, float cosv, float shell, float bottom, float& nearv,
                                            float& farv, bool& hit) {
  float orad = bottom + h0;
  float hl = orad * cosv;
  float c = (h0 - shell) * ((2.0f * bottom + h0) + shell);
  float disc = hl * hl - c;
  hit = disc >= 0.0f;
  nearv = kLargeF;
  farv = -kLargeF;
  if (hit) {
    float root = sqrtf(mx(disc, 0.0f));
    float sign = hl < 0.0f ? -1.0f : 1.0f;
    float q = -hl - sign * root;
    float r0 = -hl - root;
    float r1 = -hl + root;
    if (fabsf(q) > 1.0e-12f) {
      r0 = q;
      r1 = fdiv(c, q);
    }
    nearv = mn(r0, r1);
    farv = mx(r0, r1);
  }
}
__device__ __forceinline__ void segment_from_altitude(const DevParams& P, float h, float cosv, float bottom,
                                                      float& start, float& end, bool& valid, bool& ground) {
  float on, of;
  bool oh;
  shell_roots(h, cosv, P.top, bottom, on, of, oh);
  start = mx(on, 0.0f);
  end = of;
  valid = oh && end > start;
  ground = false;
  float gn, gf;
  bool gh;
  shell_roots(h, cosv, 0.0f, bottom, gn, gf, gh);
  if (valid && gh) {
    float gd = kLargeF;
    if (gn > start + 1.0e-3f)
      gd = gn;
    else if (gf > start + 1.0e-3f)
      gd = gf;
    if (gd < end) {
      end = gd;
      ground = true;
    }
  }
}
__device__ __forceinline__ void segment_vec(const DevParams& P, f3 o, f3 d, float bottom, float& start, float& end,
                                            bool& valid, bool& ground) {
  float on, of;
  bool oh;
  sphere_roots(o, d, bottom + P.top, on, of, oh);
  start = mx(on, 0.0f);
  end = of;
  valid = oh && end > start;
  ground = false;
  float gn, gf;
  bool gh;
  sphere_roots(o, d, bottom, gn, gf, gh);
  if (valid && gh) {
    float gd = kLargeF;
    float eps = mx(0.001f, bottom * 1.0e-8f);
    if (gn > start + eps)
      gd = gn;
    else if (gf > start + eps)
      gd = gf;
    if (gd < end) {
      end = gd;
      ground = true;
    }
  }
}

// ---- per-ray geometry ---------------------------------------------------------
// a + b = s + err exactly (Knuth's two-sum; no contraction applies to it).
__device__ __forceinline__ float two_sum(float a, float b, float& err) {
  const float s = a + b;
  const float bb = s - a;
  err = (a - (s - bb)) + (b - bb);
  return s;
}
// r(t)^2 - R^2 along a camera ray, t the distance from the camera at
// (0, R + h0, 0), is the quadratic q(u) = (q0 + q1 u) + u^2, u = t - t0.
// Cameras within half a planet radius of the ground use the reference's own
// coefficients about the camera (t0 = 0: _altitude_on_ray :237-262,
// _shell_roots_from_altitude :264-301).  Farther out, every sample is far
// from the camera and those terms, ~r_cam^2, cancel down to r^2 - R^2 ~ R H:
// float keeps no digit of a grazing ray's altitude (a 50 km planet seen from
// 1800 km: 10 m altitude errors against a 300 m Mie scale height, the
// reference's own float result then off by tens of percent).  Such rays
// pivot at the closest approach t_c = -(R + h0) cos v, where q0 = r_c^2 - R^2
// and the shell discriminants are differences of squares formed once per ray
// from the ray's sine in compensated float (r_c = (R + h0) sin v as an
// unevaluated sum hi + lo: Knuth's two-sum and the FMA two-product), which
// keeps r_c^2 - R^2 and (R + top)^2 - r_c^2 to a few float ulps of themselves
// at every grazing angle without FP64 (a small fraction of the FP32 rate on
// this part).
struct RayGeom {
  float h0, cosv;    // camera altitude, view cosine
  float t0, q0, q1;  // pivot and coefficients of q
  float tc;          // closest-approach distance
  float disc_top, disc_ground;  // far: (shell radius)^2 - r_c^2 of the top and the ground
  bool far;          // pivot at t_c (far_camera)
};
// Camera far enough for the closest-approach pivot: above the shell and more
// than half a planet radius up.
__device__ __forceinline__ bool far_camera(const DevParams& P, float bottom, float h0) {
  return h0 > P.top && h0 > 0.5f * bottom;
}
__device__ __forceinline__ RayGeom ray_geom(const DevParams& P, float bottom, float h0, float cosv, float sinv) {
  RayGeom G;
  G.h0 = h0;
  G.cosv = cosv;
  const float a = mx(h0, 0.0f);
  G.far = far_camera(P, bottom, a);
  if (!G.far) {
    const float orad = bottom + a;
    G.t0 = 0.0f;
    G.q0 = a * (2.0f * bottom + a);
    G.q1 = 2.0f * orad * cosv;
    G.tc = -orad * cosv;
    G.disc_top = G.disc_ground = 0.0f;
  } else {
    float o_lo, bt_lo;
    const float o = two_sum(bottom, a, o_lo);         // R + h0 = o + o_lo
    const float rc = o * sinv;                         // r_c = rc + rc_lo
    const float rc_lo = fmaf(o, sinv, -rc) + o_lo * sinv;
    const float bt = two_sum(bottom, P.top, bt_lo);    // R + top = bt + bt_lo
    // R - r_c and (R + top) - r_c: the leading differences are exact where
    // they cancel (Sterbenz), the low parts then carry the digits
    const float dg = (bottom - rc) - rc_lo;
    const float dt = ((bt - rc) + bt_lo) - rc_lo;
    G.disc_ground = dg * (bottom + rc);
    G.disc_top = dt * (bt + rc);
    G.t0 = G.tc = -fmaf(o, cosv, o_lo * cosv);
    G.q0 = -G.disc_ground;
    G.q1 = 0.0f;
  }
  return G;
}
// Altitude at distance t along the ray (the reference's form of :237-262).
__device__ __forceinline__ float altitude_at(const RayGeom& G, float t, float bottom) {
  const float u = t - G.t0;
  const float delta = (G.q0 + G.q1 * u) + u * u;
  const float len = fsqrt(mx(bottom * bottom + delta, 0.0f));
  return fdiv(delta, mx(len + bottom, 1.0f));
}
// Roots of the ray with the sphere of radius bottom + shell.
__device__ __forceinline__ void shell_roots_g(const RayGeom& G, float shell, float bottom, float& nearv, float& farv,
                                              bool& hit) {
  if (!G.far) {
    shell_roots(G.h0, G.cosv, shell, bottom, nearv, farv, hit);
    return;
  }
  const float disc = shell > 0.0f ? G.disc_top : G.disc_ground;  // shell is the top or 0
  hit = disc >= 0.0f;
  nearv = kLargeF;
  farv = -kLargeF;
  if (hit) {
    const float root = sqrtf(disc);
    nearv = G.tc - root;
    farv = G.tc + root;
  }
}
// _atmosphere_segment_from_altitude :303-340 on a ray's geometry.
__device__ __forceinline__ void segment_of(const DevParams& P, const RayGeom& G, float bottom, float& start,
                                           float& end, bool& valid, bool& ground) {
  if (!G.far) {
    segment_from_altitude(P, G.h0, G.cosv, bottom, start, end, valid, ground);
    return;
  }
  float on, of;
  bool oh;
  shell_roots_g(G, P.top, bottom, on, of, oh);
  start = mx(on, 0.0f);
  end = of;
  valid = oh && end > start;
  ground = false;
  float gn, gf;
  bool gh;
  shell_roots_g(G, 0.0f, bottom, gn, gf, gh);
  if (valid && gh) {
    float gd = kLargeF;
    if (gn > start + 1.0e-3f)
      gd = gn;
    else if (gf > start + 1.0e-3f)
      gd = gf;
    if (gd < end) {
      end = gd;
      ground = true;
    }
  }
}
// _aerial_prefix_segment_from_altitude :376-395 on a ray's geometry.
__device__ __forceinline__ void aerial_prefix_of(const DevParams& P, const RayGeom& G, float bottom, float& start,
                                                 float& end, bool& valid) {
  bool v, g;
  segment_of(P, G, bottom, start, end, v, g);
  if (v && !g && G.tc > start && G.tc < end) end = G.tc;
  valid = v && end > start;
}
// ---- LUT parameterisations (:410-568) ---------------------------------------
__device__ __forceinline__ void t_uv_to_ray(const DevParams& P, float u, float v, float bottom, float& h,
                                            float& cosv, float& dist) {
  float sh = shell_rho(P.top, bottom);
  float rho = sh * clampf(v, 0.0f, 1.0f);
  float rl = sqrtf(rho * rho + bottom * bottom);
  h = rho * rho / mx(rl + bottom, 1.0f);
  float radius = bottom + h;
  float dmin = P.top - h;
  float dmax = rho + sh;
  dist = dmin + clampf(u, 0.0f, 1.0f) * (dmax - dmin);
  float c = 1.0f;
  if (dist > 1.0e-6f) c = ((P.top - h) * ((2.0f * bottom + P.top) + h) - dist * dist) / (2.0f * radius * dist);
  cosv = clampf(c, -1.0f, 1.0f);
}
__device__ __forceinline__ float warp_boundary(float closest_raw, float start, float end, float f) {
  float closest = clampf(closest_raw, start, end);
  float eps = mx((end - start) * 1.0e-6f, 1.0e-5f);
  if (closest <= start + eps) return start + (end - start) * f * f;
  if (closest >= end - eps) {
    float inv = 1.0f - f;
    return end - (end - start) * inv * inv;
  }
  if (f < 0.5f) {
    float inv = 1.0f - f * 2.0f;
    return closest - (closest - start) * inv * inv;
  }
  float local = f * 2.0f - 1.0f;
  return closest + (end - closest) * local * local;
}
// Warped interval boundaries of one ray.  Every case of warp_boundary is
// base + len g^2 with g linear in f, and which one holds depends on the ray
// and on the half of the interval alone: it is picked once per half, and a
// boundary costs an FMA, a multiplication and an FMA (the reference's own
// operations: the signs that move into gs and len are exact).
struct RayWarp {
  int mode;  // 0: dense at start, 1: dense at end, 2: dense around the closest point
  float start, end, closest;
};
struct WarpHalf {
  float base, len, gs, go;
};
__device__ __forceinline__ RayWarp make_warp(float closest_raw, float start, float end) {
  RayWarp w;
  w.start = start;
  w.end = end;
  w.closest = clampf(closest_raw, start, end);
  float eps = mx((end - start) * 1.0e-6f, 1.0e-5f);
  w.mode = w.closest <= start + eps ? 0 : (w.closest >= end - eps ? 1 : 2);
  return w;
}
__device__ __forceinline__ WarpHalf warp_half(const RayWarp& w, bool second) {
  if (w.mode == 0) return {w.start, w.end - w.start, 1.0f, 0.0f};
  if (w.mode == 1) return {w.end, w.start - w.end, -1.0f, 1.0f};
  if (second) return {w.closest, w.end - w.closest, 2.0f, -1.0f};
  return {w.closest, w.start - w.closest, -2.0f, 1.0f};
}
__device__ __forceinline__ float warp_at(const WarpHalf& w, float f) {
  const float g = fmaf(f, w.gs, w.go);
  return fmaf(w.len * g, g, w.base);
}
// The boundary i of n, i / n < 1/2 in the first half.
__device__ __forceinline__ bool warp_second(int i, int n) { return 2 * i >= n; }

// Where a march takes the fractions i / n of its boundaries from: a table
// (in shared memory, one load) or the division itself.  Both are the IEEE
// quotient: a boundary's last bit decides on which side of the ground a
// sample next to it lies.
struct TableFraction {
  const float* t;
  __device__ __forceinline__ float operator()(int i) const { return t[i]; }
};
struct DivideFraction {
  float n;
  __device__ __forceinline__ float operator()(int i) const { return float(i) / n; }
};

__device__ __forceinline__ float horizon_cosine(float h, float bottom) {
  float radius = bottom + mx(h, 0.0f);
  return fdiv(-shell_rho(h, bottom), mx(radius, 1.0f));
}
__device__ __forceinline__ float sky_horizon_zenith(float h, float bottom) {
  float a = mx(h, 0.0f);
  float radius = bottom + a;
  float tc = shell_rho(a, bottom) / mx(radius, 1.0f);
  return kPiF - acosf(clampf(tc, 0.0f, 1.0f));
}
__device__ __forceinline__ float sky_v_to_zenith(float v, float hz) {
  if (v < 0.5f) {
    float inv = 1.0f - 2.0f * v;
    return hz * (1.0f - inv * inv);
  }
  float local = 2.0f * v - 1.0f;
  return hz + (kPiF - hz) * local * local;
}
__device__ __forceinline__ float sky_zenith_to_v(float z, float hz) {
  if (z < hz) {
    float n = clampf(z / mx(hz, 1.0e-6f), 0.0f, 1.0f);
    return 0.5f * (1.0f - sqrtf(mx(1.0f - n, 0.0f)));
  }
  float n = clampf((z - hz) / mx(kPiF - hz, 1.0e-6f), 0.0f, 1.0f);
  return 0.5f + 0.5f * sqrtf(n);
}
__device__ __forceinline__ float sun_u_to_cosine(float u, float h, float bottom) {
  float hc = horizon_cosine(h, bottom);
  float c;
  if (u < 0.5f) {
    float inv = 1.0f - 2.0f * u;
    c = hc - (hc + 1.0f) * inv * inv;
  } else {
    float local = 2.0f * u - 1.0f;
    c = hc + (1.0f - hc) * local * local;
  }
  return clampf(c, -1.0f, 1.0f);
}
__device__ __forceinline__ float sun_cosine_to_u(float c, float hc) {
  const float t = c - hc;
  const float side = copysignf(1.0f, t);  // -1 below the horizon
  const float n = __saturatef(fabsf(t) * frcp(mx(fmaf(side, -hc, 1.0f), 1.0e-6f)));
  return fmaf(0.5f * side, fsqrt(n), 0.5f);
}

// ---- LUT sampling -----------------------------------------------------------
// Bilinear tap with the reference's half-texel rule and edge clamp
// (:618-640, :655-683, :1503-1525).  The texel index is formed in float (2^23
// plus an integer below 2^23 is exact), which keeps the conversions off the
// XU pipe and the index arithmetic off the ALU, the two pipes a march is
// short of; past the last texel's centre the last pair's weight saturates at
// its right end, so the four taps are two addresses apart by constants.
__device__ __forceinline__ f3 bilinear_at(const float4* __restrict__ lut, const LutDims& D, float cx, float cy) {
  const float x = mx(cx, 0.0f);
  const float y = mx(cy, 0.0f);
  const float xm = mn(__fadd_rd(x, kMagic), D.x_last);
  const float yf = mn(__fadd_rd(y, kMagic), D.y_last) - kMagic;
  const float fx = __saturatef(x - (xm - kMagic));
  const float fy = __saturatef(y - yf);
  const float4* t = lut + (__float_as_int(fmaf(yf, D.w, xm)) & 0x7fffff);
  const float4* t1 = t + D.pitch;
  const float4 a = __ldg(t), b = __ldg(t + 1), c = __ldg(t1), d = __ldg(t1 + 1);
  const float wd = fx * fy, wc = fy - wd, wb = fx - wd, wa = (1.0f - fx) - wc;
  return {fmaf(d.x, wd, fmaf(c.x, wc, fmaf(b.x, wb, a.x * wa))), fmaf(d.y, wd, fmaf(c.y, wc, fmaf(b.y, wb, a.y * wa))),
          fmaf(d.z, wd, fmaf(c.z, wc, fmaf(b.z, wb, a.z * wa)))};
}

__device__ __forceinline__ f3 bilinear(const float4* __restrict__ lut, const LutDims& D, float u, float v) {
  return bilinear_at(lut, D, fmaf(u, D.w, -0.5f), fmaf(v, D.h, -0.5f));
}

// Per-launch geometry shared by every sample of a kernel, formed on the host
// (a kernel argument: its members are operands from constant memory, not
// registers of every thread).
struct Frame {
  const float4* __restrict__ tlut;
  const float4* __restrict__ mslut;
  float bottom;     // planet radius (f32)
  float shell_top;  // shell_rho(top, bottom)
  float shell2;     // its square, (bottom + top)^2 - bottom^2
  float ar;         // sun angular radius (rad)
  f3 sun;
  f3 E;             // solar irradiance
  float t_rho;           // transmittance LUT rows a metre of rho: its height / shell_top
  float cos_ar, sin_ar;  // of the sun's angular radius: thresholds of the whole-disk tests
  float bottom_sin_ar;
};
inline Frame make_frame(const DevParams& P, const float4* tlut, const float4* mslut, float bottom, float ar, f3 sun,
                        f3 E) {
  Frame F;
  F.tlut = tlut;
  F.mslut = mslut;
  F.bottom = bottom;
  const float top = P.top > 0.0f ? P.top : 0.0f;
  F.shell2 = top * (2.0f * bottom + top);
  F.shell_top = std::sqrt(F.shell2);
  F.ar = ar;
  F.sun = sun;
  F.E = E;
  F.t_rho = P.t_lut.h / (F.shell_top > 1.0e-6f ? F.shell_top : 1.0e-6f);
  F.sin_ar = float(std::sin(double(ar)));
  F.cos_ar = float(std::cos(double(ar)));
  F.bottom_sin_ar = float(bottom * std::sin(double(ar)));
  return F;
}
// Sun of a sky-view LUT: its zenith cosine alone, in the x-y plane.
inline f3 sky_view_sun(float sun_cos) {
  return {std::sqrt(std::fmax(std::fma(-sun_cos, sun_cos, 1.0f), 0.0f)), sun_cos, 0.0f};
}

// _sample_transmittance_unoccluded :609-640 at the point of altitude h inside
// the shell: rho2 = r^2 - R^2 and its root rho, rc = r cos of the direction's
// zenith angle.  The distance to the shell top is then sqrt(rc^2 + shell2 -
// rho2) - rc.
__device__ __forceinline__ f3 sample_t_at(const DevParams& P, const Frame& F, float h, float rho2, float rho, float rc) {
  const float d = fsqrt(mx(fmaf(rc, rc, F.shell2 - rho2), 0.0f)) - rc;  // below 0 only above the shell
  const float dmin = P.top - h;
  const float u = __saturatef((d - dmin) * frcp(mx((rho + F.shell_top) - dmin, 1.0e-6f)));
  return bilinear_at(F.tlut, P.t_lut, fmaf(u, P.t_lut.w, -0.5f), fmaf(rho, F.t_rho, -0.5f));
}
// The same from any altitude, with IEEE operations where the march takes the
// hardware's: once a pixel (camera_t).
__device__ __forceinline__ f3 sample_t(const DevParams& P, const Frame& F, float h, float rc) {
  const float a = clampf(h, 0.0f, P.top);
  const float rho = sqrtf(a * (2.0f * F.bottom + a)), dmin = P.top - a;
  const float d = sqrtf(mx(fmaf(rc, rc, dmin * ((2.0f * F.bottom + P.top) + a)), 0.0f)) - rc;
  const float u = __saturatef((d - dmin) / mx((rho + F.shell_top) - dmin, 1.0e-6f));
  return bilinear_at(F.tlut, P.t_lut, fmaf(u, P.t_lut.w, -0.5f), fmaf(rho, F.t_rho, -0.5f));
}
// _sample_multi_scattering :642-683
__device__ __forceinline__ f3 sample_ms(const DevParams& P, const Frame& F, float h, float sc, float hc) {
  return bilinear(F.mslut, P.ms_lut, sun_cosine_to_u(sc, hc), fsqrt(__saturatef(h * P.inv_top)));
}

// The same at a march's sample: altitude h, radius r, rc = r cos of the sun's
// zenith angle, rho = -r cos of the horizon's.
__device__ __forceinline__ f3 sample_ms_at(const DevParams& P, const Frame& F, float h, float r, float rc, float rho) {
  const float t = rc + rho;
  const float n = __saturatef(fabsf(t) * frcp(mx(fmaf(copysignf(1.0f, t), rho, r), 1.0e-6f)));
  return bilinear_at(F.mslut, P.ms_lut, fmaf(copysignf(P.ms_half_w, t), fsqrt(n), P.ms_half_w - 0.5f),
                     fmaf(fsqrt(__saturatef(h * P.inv_top)), P.ms_lut.h, -0.5f));
}

// Horizon at one sample altitude: cosine hc = -rho/r of the horizon
// zenith, and sin of that zenith, R/r (rho^2 = r^2 - R^2).
struct Horizon {
  float hc;         // horizon cosine
  float sin_hz;     // sine of the horizon zenith
  float rho2, rho;  // r^2 - R^2 and its root, 0 below the ground
};
__device__ __forceinline__ Horizon horizon_of(float rho2, float inv_r, float bottom) {
  Horizon H;
  H.rho2 = rho2;
  H.rho = fsqrt(rho2);
  H.hc = -H.rho * inv_r;
  H.sin_hz = mn(bottom * inv_r, 1.0f);
  return H;
}
__device__ __forceinline__ Horizon horizon_at(float h, float bottom) {
  const float a = mx(h, 0.0f);
  return horizon_of(a * (2.0f * bottom + a), frcp(mx(bottom + a, 1.0f)), bottom);
}
// _solar_disk_visibility :728-754, given horizon and sun zenith angles
__device__ __forceinline__ float disk_visibility(float hz, float sz, float ar) {
  float n = clampf(fdiv(hz - sz, mx(ar, 1.0e-6f)), -1.0f, 1.0f);
  return (acosf(-n) + n * sqrtf(mx(1.0f - n * n, 0.0f))) * (1.0f / kPiF);
}
// _sample_solar_transmittance :756-789 (returns the disk visibility too).
// The reference compares the horizon and sun zenith angles; whole-disk
// cases are decided here in cosine space without acos:
//   disk fully above the horizon  <=> sz <= hz - ar <=> cos sz >= cos(hz - ar)
//   disk fully below the horizon  <=> sz >= hz + ar <=> cos sz <= cos(hz + ar)
// with cos(hz -+ ar) = hc cos ar +- sin hz sin ar.  There the reference's
// visibility is exactly 1 (its representative zenith is then the sun's own,
// whose cosine is sc) or exactly 0; within float rounding of the thresholds
// its visibility differs from 1 or 0 by < 1e-6.  Only the penumbra band
// evaluates the reference's acos formulation.
// The point: altitude h, radius r, sun cosine sc, rc = r sc.
__device__ __forceinline__ f3 sample_solar_t(const DevParams& P, const Frame& F, float h, float r, float sc, float rc,
                                             const Horizon& H, float& vis) {
  const float a = H.hc * F.cos_ar;
  const float b = H.sin_hz * F.sin_ar;
  if (sc >= a + b) {
    vis = 1.0f;
    return sample_t_at(P, F, h, H.rho2, H.rho, rc);
  }
  if (sc <= a - b && H.hc >= -F.cos_ar) {  // hz + ar <= pi
    vis = 0.0f;
    return splat(0.0f);
  }
  const float hz = acosf(clampf(H.hc, -1.0f, 1.0f));
  const float sz = acosf(clampf(sc, -1.0f, 1.0f));
  vis = disk_visibility(hz, sz, F.ar);
  const float rz = mn(sz, hz - F.ar * 0.25f);
  return sample_t_at(P, F, h, H.rho2, H.rho, r * cosf(mx(rz, 0.0f))) * vis;
}
// The same from an altitude (brought into the shell) and a sun cosine.
__device__ __forceinline__ f3 sample_solar_t(const DevParams& P, const Frame& F, float h, float sc, const Horizon& H,
                                             float& vis) {
  const float a = clampf(h, 0.0f, P.top);
  const float r = F.bottom + a;
  const float cs = clampf(sc, -1.0f, 1.0f);
  Horizon I = H;
  I.rho2 = a * (2.0f * F.bottom + a);
  I.rho = fsqrt(I.rho2);
  return sample_solar_t(P, F, a, r, cs, r * cs, I, vis);
}
// _rayleigh_phase / _mie_phase :791-804
__device__ __forceinline__ float rayleigh_phase(const DevParams& P, float c) {
  return 3.0f * (1.0f + c * c) / P.ray_k;
}
__device__ __forceinline__ float mie_phase(const DevParams& P, float c) {
  float den = mx(P.mie_c1 - P.mie_c2 * c, 1.0e-8f);
  return P.mie_k1 * (1.0f + c * c) / (P.mie_k2 * (den * sqrtf(den)));
}
// _segment_integral :806-816: T = exp(-x), x = ext step, and the in-scattering
// weight (1 - T) / ext.  The reference forms 1 - T directly, which cancels in
// f32 when x is small: centimetre segments next to a camera standing on the
// ground give x ~ 1e-7 and a weight with no significant digit left (its own
// f32 result is then percents away from its f64 one).  Up to x = 1 both come
// from phi = (1 - e^-x) / x: weight = step phi, T = 1 - ext weight (step
// itself at ext = 0, as the reference's ext <= 1e-12 branch).  phi is a
// polynomial, near-minimax with phi(0) = 1: degree 4 up to x = 1/4, which
// most segments are within, degree 6 up to 1, both within 3e-9 of phi with
// their float coefficients; a rounding error each in float, 4 and 6 operations
// a channel, against 7 and 2^x for the form e^(-x/2) sinh(x/2) / (x/2).  Larger x take 1 - T, which
// keeps 7 digits.
__device__ __forceinline__ float phi_quarter(float x) {
  return fmaf(x, fmaf(x, fmaf(x, fmaf(x, 0.007530156057327986f, -0.04150012508034706f), 0.1666528880596161f),
                      -0.49999964237213135f), 1.0f);
}
__device__ __forceinline__ float phi_one(float x) {
  const float high = fmaf(x, fmaf(x, 0.00012931223318446428f, -0.0013017107266932726f), 0.008276925422251225f);
  return fmaf(x, fmaf(x, fmaf(x, fmaf(x, high, -0.041647881269454956f), 0.1666637659072876f), -0.49999985098838806f),
              1.0f);
}
__device__ __forceinline__ void segment_any(float ext, float x, float step, float& tr, float& w) {
  w = phi_one(mn(x, 1.0f)) * step;
  tr = fmaf(-w, ext, 1.0f);
  if (x > 1.0f) {
    tr = fexp2(mn(x, 80.0f) * -1.4426950408889634f);
    w = (1.0f - tr) * frcp(ext);
  }
}
__device__ __forceinline__ void segment_integral(f3 ext, float step, f3& tr, f3& w) {
  const f3 x = ext * step;
  if (mx(mx(x.x, x.y), x.z) <= 0.25f) {
    w = mk(phi_quarter(x.x), phi_quarter(x.y), phi_quarter(x.z)) * step;
    tr = {fmaf(-w.x, ext.x, 1.0f), fmaf(-w.y, ext.y, 1.0f), fmaf(-w.z, ext.z, 1.0f)};
  } else {
    segment_any(ext.x, x.x, step, tr.x, w.x);
    segment_any(ext.y, x.y, step, tr.y, w.y);
    segment_any(ext.z, x.z, step, tr.z, w.z);
  }
}
// A segment of extinction ext and source src a metre after what acc holds.
__device__ __forceinline__ void then_segment(Seg& acc, f3 src, f3 ext, float step) {
  const f3 x = ext * step;
  const float thickest = mx(mx(x.x, x.y), x.z);
  if (thickest <= 1.0f) {
    const f3 phi = thickest <= 0.25f ? mk(phi_quarter(x.x), phi_quarter(x.y), phi_quarter(x.z))
                                     : mk(phi_one(x.x), phi_one(x.y), phi_one(x.z));
    const f3 a = acc.T * (phi * step);
    acc.L = {fmaf(a.x, src.x, acc.L.x), fmaf(a.y, src.y, acc.L.y), fmaf(a.z, src.z, acc.L.z)};
    acc.T = {fmaf(-a.x, ext.x, acc.T.x), fmaf(-a.y, ext.y, acc.T.y), fmaf(-a.z, ext.z, acc.T.z)};
  } else {
    f3 t, w;
    segment_integral(ext, step, t, w);
    acc = seg_then(acc, {src * w, t});
  }
}

// Per-ray constants of the constant-source samples (everything of
// _scattering_source :818-856 that does not depend on the sample).
struct RaySource {
  float t0, q0, q1;  // the ray's altitude quadratic (RayGeom)
  float s0;          // (origin + t0 ray) . sun
  float r_sun;       // ray . sun
  f3 ER, EM;         // E * beta_R * phase_R, E * beta_Ms * phase_M
};
__device__ __forceinline__ RaySource make_ray_source(const DevParams& P, const Frame& F, const RayGeom& G, f3 ray) {
  RaySource R;
  R.t0 = G.t0;
  R.q0 = G.q0;
  R.q1 = G.q1;
  R.r_sun = dot(ray, F.sun);
  const float o_y = F.bottom + mx(G.h0, 0.0f);
  if (G.far) {
    // p(t0) . sun with the closest-approach point formed first (one rounding
    // per component, each ~r_c): o_y sun.y + t0 ray . sun cancels ~r_cam
    // down to ~r_c
    const f3 c = mk(G.t0 * ray.x, fmaf(G.t0, ray.y, o_y), G.t0 * ray.z);
    R.s0 = dot(c, F.sun);
  } else {
    R.s0 = o_y * F.sun.y;
  }
  const float cr = clampf(R.r_sun, -1.0f, 1.0f);
  R.ER = F.E * arr3(P.beta_r) * rayleigh_phase(P, cr);
  R.EM = F.E * arr3(P.beta_ms) * mie_phase(P, cr);
  return R;
}

// The medium and the sun at the middle of a segment [start, end] of the ray:
// density, extinction and scattering, the segment's length, finite-disk sun
// transmittance st and disk visibility, altitude h, radius r, rc = r cos of the
// sun's zenith angle, rho = -r cos of the horizon's.  The sample's radius is bottom + h (its altitude on the ray) and
// its sun cosine (p(t0) . sun + (t - t0) ray . sun) / radius; the reference
// forms the point first - same quantities, rounding differs in the last bits.
//
// A march is bound by the instructions it issues, the ALU pipe (compares,
// selects, minima, integers) first.  What a sample shares is formed once:
// delta = r^2 - R^2 gives the altitude, the horizon's rho and the distance to
// the shell top; lengths along the vertical (rc, rho) stand for the cosines,
// which only a partly hidden disk needs.  The altitude keeps the operations
// that decide where the density is cut off (delta's sign).  With the tap and the segment weight
// above, a 1080p composite from 2 km went from 1369 to 758 us (1.48e9 to
// 0.83e9 warp instructions).
struct MarchSample {
  Density d;
  Medium medium;
  f3 st;
  float step, vis, h, r, rc, rho;
};
__device__ __forceinline__ MarchSample march_sample(const DevParams& P, const Frame& F, const RaySource& R,
                                                    float start, float end) {
  MarchSample m;
  m.step = mx(end - start, 0.0f);
  const float u = (start + end) * 0.5f - R.t0;
  const float delta = fmaf(u, u, fmaf(R.q1, u, R.q0));
  m.r = fsqrt(mx(fmaf(F.bottom, F.bottom, delta), 1.0f));
  m.h = delta * frcp(m.r + F.bottom);
  m.d = density(P, m.h);
  m.medium = medium_of(P, m.d);
  m.rc = fmaf(u, R.r_sun, R.s0);
  const float rho2 = mx(delta, 0.0f);
  m.rho = fsqrt(rho2);
  // the disk wholly above the horizon, sample_solar_t's test times r
  if (m.rc >= fmaf(-m.rho, F.cos_ar, F.bottom_sin_ar)) {
    m.vis = 1.0f;
    m.st = sample_t_at(P, F, m.h, rho2, m.rho, m.rc);
  } else {
    const float inv_r = frcp(m.r);
    m.st = sample_solar_t(P, F, m.h, m.r, m.rc * inv_r, m.rc, horizon_of(rho2, inv_r, F.bottom), m.vis);
  }
  return m;
}

// _scattering_source :818-856 at a sample.
__device__ __forceinline__ f3 source_of(const DevParams& P, const Frame& F, const RaySource& R, const MarchSample& m) {
  return m.st * (R.ER * m.d.r + R.EM * m.d.m) + m.medium.scat * sample_ms_at(P, F, m.h, m.r, m.rc, m.rho);
}
// One constant-source segment [start, end] of the ray after what acc holds:
// _scattering_segment :858-899.
__device__ __forceinline__ void then_source_segment(const DevParams& P, const Frame& F, const RaySource& R,
                                                    float start, float end, Seg& acc) {
  const MarchSample m = march_sample(P, F, R, start, end);
  then_segment(acc, source_of(P, F, R, m), m.medium.ext, m.step);
}

// The intervals [i0, i1) of n of a ray's march in ray order: segment(d0, d1).
// The two halves of the warp are two runs of one loop, so that an interval
// costs no look at which half it is in.
template <class Fraction, class Segment>
__device__ __forceinline__ void for_intervals(const RayWarp& w, int i0, int i1, int n, Fraction fraction,
                                              Segment segment) {
  bool second = warp_second(i0, n);
  float d0 = warp_at(warp_half(w, second), fraction(i0));
  int i = i0;
#pragma unroll 1
  for (;;) {
    const WarpHalf half = warp_half(w, second);
    const int stop = second ? i1 : min(i1, (n - 1) / 2);  // boundary i + 1 is in the first half
#pragma unroll 1
    for (; i < stop; ++i) {
      const float d1 = warp_at(half, fraction(i + 1));
      segment(d0, d1);
      d0 = d1;
    }
    if (second || i >= i1) return;
    second = true;
  }
}
// The base intervals without refinement.
template <class Fraction>
__device__ __forceinline__ Seg march(const DevParams& P, const Frame& F, const RaySource& R, const RayWarp& w, int i0,
                                     int i1, int n, Fraction fraction) {
  Seg acc = {splat(0.0f), splat(1.0f)};
  for_intervals(w, i0, i1, n, fraction,
                [&](float d0, float d1) { then_source_segment(P, F, R, d0, d1, acc); });
  return acc;
}

}  // namespace atm
