// atm_lut_warp.cuh - evaluation of sky-view texels and aerial-perspective
// columns (reference atmosphere/renderer.py :1208-1302 and :1304-1420) by
// groups of lanes.  Shared by the single-LUT kernels and the persistent
// batched builder.
//
// A texel's or column's set-up (its ray, the shell intersections, the phases)
// costs as much as one to two march samples and every lane of its group
// repeats it, so a group is as small as the launch allows: one lane where a
// batch fills the machine, more where a single LUT or a small batch would
// leave it idle.  A batch of 512 LUTs takes 2.14 ms at one lane a texel or
// column, 7.8 ms at a warp; a single 192x108 sky-view LUT 11 us at four lanes,
// 26 us at a warp.
#pragma once

#include "atm_device.cuh"

namespace atm {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ f3 shfl_xor3(f3 v, int m) {
  return {__shfl_xor_sync(kFull, v.x, m), __shfl_xor_sync(kFull, v.y, m), __shfl_xor_sync(kFull, v.z, m)};
}
__device__ __forceinline__ f3 shfl_down3(f3 v, int o) {
  return {__shfl_down_sync(kFull, v.x, o), __shfl_down_sync(kFull, v.y, o), __shfl_down_sync(kFull, v.z, o)};
}
__device__ __forceinline__ Seg shfl_down_seg(Seg s, int o) {
  return {{__shfl_down_sync(kFull, s.L.x, o), __shfl_down_sync(kFull, s.L.y, o), __shfl_down_sync(kFull, s.L.z, o)},
          {__shfl_down_sync(kFull, s.T.x, o), __shfl_down_sync(kFull, s.T.y, o), __shfl_down_sync(kFull, s.T.z, o)}};
}
__device__ __forceinline__ Seg shfl_up_seg(Seg s, int o) {
  return {{__shfl_up_sync(kFull, s.L.x, o), __shfl_up_sync(kFull, s.L.y, o), __shfl_up_sync(kFull, s.L.z, o)},
          {__shfl_up_sync(kFull, s.T.x, o), __shfl_up_sync(kFull, s.T.y, o), __shfl_up_sync(kFull, s.T.z, o)}};
}
__device__ __forceinline__ Seg seg_identity() { return {splat(0.0f), splat(1.0f)}; }

// Ordered composition of the segments of each group of kLanes consecutive
// lanes; the group's first lane receives the total.  Every lane must call.
template <int kLanes>
__device__ __forceinline__ Seg group_compose(Seg s) {
#pragma unroll
  for (int o = 1; o < kLanes; o <<= 1) {
    const Seg other = shfl_down_seg(s, o);
    if ((threadIdx.x & (kLanes - 1)) + o < kLanes) s = seg_then(s, other);
  }
  return s;
}
// Ordered inclusive scan within each group of kLanes consecutive lanes: lane i
// receives segment 0 then ... then i.  Every lane must call.
template <int kLanes>
__device__ __forceinline__ Seg group_scan(Seg s) {
  const int lane = threadIdx.x & (kLanes - 1);
#pragma unroll
  for (int o = 1; o < kLanes; o <<= 1) {
    Seg before = shfl_up_seg(s, o);
    if (lane >= o) s = seg_then(before, s);
  }
  return s;
}

// Boundary fractions i / n of a march into t[0..n], by the threads first,
// first + stride, ...
__device__ __forceinline__ void fill_fractions(float* t, int n, int first, int stride) {
  for (int i = first; i <= n; i += stride) t[i] = float(i) / float(n);
}
constexpr int kMaxSkySteps = 256, kMaxAerialSteps = 16;  // atm_create's ranges

// One sky-view texel (x, y) by kLanes consecutive lanes, which split the
// march steps; the (L, T) segments are composed in ray order and the group's
// first lane stores the texel if `store`.  Every lane of the warp must call
// when kLanes > 1.  Returns the radiance samples this lane evaluated.
template <int kLanes>
__device__ __forceinline__ uint32_t sky_view_texel(const DevParams& P, const Frame& F, float cam_alt, int x, int y,
                                                   bool store, TableFraction fraction, float4* __restrict__ out) {
  const int lane = threadIdx.x & (kLanes - 1);
  const float bottom = F.bottom;
  const float sh = mx(cam_alt, 0.0f);
  float az = (float(x) + 0.5f) / float(P.sv_w) * kPiF;
  float vv = (float(y) + 0.5f) / float(P.sv_h);
  float zen = sky_v_to_zenith(vv, sky_horizon_zenith(sh, bottom));
  float vs, vc, saz, caz;
  sincosf(zen, &vs, &vc);
  if (far_camera(P, bottom, sh)) {
    // seen from many planet radii the whole planet spans a few degrees
    // around the nadir: the same mapping in nadir angles keeps the digits
    // that zen itself, near pi, loses.  The horizon's nadir angle
    // pi - hz = acos(rho / r) = asin(R / r): acos of rho / r ~ 1 amplifies one
    // float ulp of its argument to ~2e-6 rad (and 1e-7 rad of direction
    // moves a limb texel's radiance by 0.2%); asin of R / r is well conditioned
    const float nh = asinf(clampf(__fdiv_rn(bottom, bottom + sh), 0.0f, 1.0f));
    float nadir;
    if (vv >= 0.5f) {
      const float local = 2.0f * vv - 1.0f;
      nadir = nh * (1.0f - local * local);  // pi - (hz + (pi - hz) local^2)
    } else {
      const float inv = 1.0f - 2.0f * vv;
      nadir = nh + (kPiF - nh) * (inv * inv);  // pi - hz (1 - inv^2)
    }
    sincosf(nadir, &vs, &vc);
    vc = -vc;
  }
  sincosf(az, &saz, &caz);
  f3 ray = mk(vs * caz, vc, vs * saz);
  const RayGeom G = ray_geom(P, bottom, sh, vc, vs);
  float start, end;
  bool valid, ground;
  segment_of(P, G, bottom, start, end, valid, ground);
  Seg acc = seg_identity();
  uint32_t samples = 0;
  if (valid) {
    const RaySource rs = make_ray_source(P, F, G, ray);
    const int n = P.sv_steps;
    const int per = (n + kLanes - 1) / kLanes;
    const int i0 = lane * per;
    const int i1 = min(i0 + per, n);
    if (i0 < i1) {
      acc = march(P, F, rs, make_warp(G.tc, start, end), i0, i1, n, fraction);
      samples = uint32_t(i1 - i0);
    }
  }
  acc = group_compose<kLanes>(acc);
  if (!store) return 0;
  if (lane == 0) out[y * P.sv_w + x] = to4(vmax(acc.L, 0.0f));
  return samples;
}

// Camera of an aerial-perspective volume; fwd_t = forward / tan(half fov).
struct AerialView {
  float aspect, cam_alt;
  f3 right, up, fwd_t;
};
inline AerialView aerial_view(float aspect, float cam_alt, const float* right, const float* up, const float* fwd,
                              float tanfov) {
  return {aspect, cam_alt, {right[0], right[1], right[2]}, {up[0], up[1], up[2]},
          {fwd[0] / tanfov, fwd[1] / tanfov, fwd[2] / tanfov}};
}

// A froxel column's ray and prefix interval.
struct AerialColumn {
  RaySource rs;
  float start, end, closest;
  bool valid;
};
__device__ __forceinline__ AerialColumn aerial_ray(const DevParams& P, const Frame& F, const AerialView& V, int x,
                                                   int y) {
  float u = (float(x) + 0.5f) / float(P.ap_w);
  float v = (float(y) + 0.5f) / float(P.ap_h);
  float sx = (u * 2.0f - 1.0f) * V.aspect;
  float sy = v * 2.0f - 1.0f;
  f3 rv = (V.right * sx + V.up * sy) + V.fwd_t;
  f3 ray = rv * (1.0f / norm(rv));
  AerialColumn C;
  const RayGeom G = ray_geom(P, F.bottom, V.cam_alt, ray.y, sqrtf(ray.x * ray.x + ray.z * ray.z));
  aerial_prefix_of(P, G, F.bottom, C.start, C.end, C.valid);
  C.rs = make_ray_source(P, F, G, ray);
  C.closest = G.tc;
  return C;
}
// Depth of slice k along the column.
__device__ __forceinline__ float slice_depth(const DevParams& P, const AerialColumn& C, int k) {
  return C.start + (C.end - C.start) * (float(k) / float(P.ap_d - 1));
}
// Segment of a slice between the depths of the slice before it and its own.
__device__ __forceinline__ Seg aerial_slice(const DevParams& P, const Frame& F, const AerialColumn& C, float prev,
                                            float target, TableFraction fraction, uint32_t& samples) {
  if (!C.valid) return seg_identity();
  const float is = mx(prev, C.start);
  const float ie = mn(target, C.end);
  if (!(ie > is)) return seg_identity();
  const int n = P.ap_steps;
  samples += uint32_t(n);
  return march(P, F, C.rs, make_warp(C.closest, is, ie), 0, n, n, fraction);
}

// One froxel column (x, y) by one lane, slice after slice.  Neighbouring
// lanes take neighbouring columns: a slice's stores are contiguous.
__device__ __forceinline__ uint32_t aerial_column_lane(const DevParams& P, const Frame& F, const AerialView& V, int x,
                                                       int y, TableFraction fraction, float4* __restrict__ out) {
  const AerialColumn C = aerial_ray(P, F, V, x, y);
  const size_t plane = size_t(P.ap_w) * P.ap_h;
  float4* o = out + size_t(y) * P.ap_w + x;
  Seg acc = seg_identity();
  uint32_t samples = 0;
  float prev = C.start;
  for (int k = 0; k < P.ap_d; ++k) {
    const float target = slice_depth(P, C, k);
    acc = seg_then(acc, aerial_slice(P, F, C, prev, target, fraction, samples));
    o[k * plane] = to4(vmax(acc.L, 0.0f));
    prev = target;
  }
  return samples;
}

// One froxel column (x, y) by kLanes consecutive lanes, which take runs of
// depth slices; an ordered scan of the runs gives each lane what lies before
// its own.  A run's slices are stored (if `store`) as they are marched and
// completed in place after the scan.  Every lane of the warp must call.
// Returns the samples this lane evaluated.
template <int kLanes>
__device__ __forceinline__ uint32_t aerial_column_group(const DevParams& P, const Frame& F, const AerialView& V, int x,
                                                        int y, bool store, TableFraction fraction,
                                                        float4* __restrict__ out) {
  const int lane = threadIdx.x & (kLanes - 1);
  const AerialColumn C = aerial_ray(P, F, V, x, y);
  const int depth = P.ap_d;
  const int per = (depth + kLanes - 1) / kLanes;
  const int k0 = min(lane * per, depth), k1 = store ? min(k0 + per, depth) : k0;
  const size_t plane = size_t(P.ap_w) * P.ap_h;
  float4* o = out + size_t(y) * P.ap_w + x;
  Seg run = seg_identity();
  uint32_t samples = 0;
  float prev = k0 == 0 ? C.start : slice_depth(P, C, k0 - 1);
  for (int k = k0; k < k1; ++k) {
    const float target = slice_depth(P, C, k);
    run = seg_then(run, aerial_slice(P, F, C, prev, target, fraction, samples));
    if (per > 1) o[k * plane] = to4(run.L);
    prev = target;
  }
  const Seg incl = group_scan<kLanes>(run);
  if (per == 1) {
    if (k0 < k1) o[k0 * plane] = to4(vmax(incl.L, 0.0f));
    return samples;
  }
  Seg before = shfl_up_seg(incl, 1);
  if (lane == 0) before = seg_identity();
  for (int k = k0; k < k1; ++k) o[k * plane] = to4(vmax(before.L + before.T * from4(o[k * plane]), 0.0f));
  return samples;
}

}  // namespace atm
