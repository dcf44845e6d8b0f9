// atm_luts.cu - Transmittance, Multi-scattering, Sky-view and Aerial-perspective
// LUT builds (reference atmosphere/renderer.py :1034-1420) for sm_103a.
//
// Work decomposition (the reference runs one Taichi thread per texel, each
// marching its ray sequentially):
//  - transmittance: 8 lanes per texel split the 40 optical-depth steps and
//    sum with xor shuffles;
//  - multi-scattering: a block per texel, a few lanes per direction which
//    split its march; the directions are summed by shuffles;
//  - sky-view: a few lanes per texel over its march steps; the per-step
//    (radiance, transmittance) segments are composed in ray order by
//    shuffles ((L1,T1) then (L2,T2) = (L1 + T1 L2, T1 T2));
//  - aerial perspective: one warp per froxel column, lanes over depth
//    slices; an ordered inclusive shuffle scan of the slice segments gives
//    each slice's cumulative in-scattering.
// Every LUT is float4 row-major [z][y][x]: stores are 16-byte and coalesced
// along x.
#include <cuda_runtime.h>

#include <algorithm>

#include "atm_device.cuh"
#include "atm_kernels.h"
#include "atm_lut_warp.cuh"

namespace atm {
namespace {

// ---- transmittance (:1034-1063, :570-607) ----------------------------------
constexpr int kTLanes = 8;
constexpr long long kWaveThreads = 152LL * 2048;  // resident threads of the whole chip

constexpr int kTBlock = 64;
__global__ void __launch_bounds__(kTBlock) k_transmittance(DevParams P, float bottom, float4* __restrict__ out) {
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  const int texel = gid / kTLanes;
  const int sub = gid % kTLanes;
  const int n_texels = P.t_w * P.t_h;
  const bool active = texel < n_texels;
  const int t = active ? texel : 0;
  const int x = t % P.t_w, y = t / P.t_w;
  float u = (float(x) + 0.5f) / float(P.t_w);
  float v = (float(y) + 0.5f) / float(P.t_h);
  float h, c, dist;
  t_uv_to_ray(P, u, v, bottom, h, c, dist);
  float s = sqrtf(mx(1.0f - c * c, 0.0f));
  float radius = bottom + h;
  f3 o = mk(0.0f, radius, 0.0f);
  f3 ray = mk(s, c, 0.0f);
  float closest_raw = -dot(o, ray);
  f3 od = splat(0.0f);
  const int n = P.t_steps;
  for (int i = sub; i < n; i += kTLanes) {
    float d0 = warp_boundary(closest_raw, 0.0f, dist, float(i) / float(n));
    float d1 = warp_boundary(closest_raw, 0.0f, dist, float(i + 1) / float(n));
    float step = d1 - d0;
    float mid = (d0 + d1) * 0.5f;
    float alt = norm(o + ray * mid) - bottom;
    od = od + extinction_of(P, density(P, alt)) * step;
  }
#pragma unroll
  for (int m = 1; m < kTLanes; m <<= 1) od = od + shfl_xor3(od, m);
  if (active && sub == 0) out[y * P.t_w + x] = to4(vclamp(vexp(-vmin(od, 80.0f)), 0.0f, 1.0f));
}

// ---- multi-scattering (:1065-1206) ------------------------------------------
constexpr int kMaxDirs = 128, kMaxDirectionSteps = 128;  // atm_create's ranges

// kLanes consecutive lanes share a direction's march; kLanes ms_dirs threads
// (rounded up to whole warps) a texel.  Bound by latency and by the blocks'
// wait for their longest direction: 32x32 texels of 64 directions take 44 us
// at one lane a direction (13 warps an SM), 27 us at four (2.3 waves of
// blocks), 22 us at two, whose 1024 blocks are resident at once at 72
// registers.
template <int kLanes>
__global__ void __maxnreg__(72) k_multi_scattering(DevParams P, Frame F,
                                                                       float4* __restrict__ out,
                                                                       unsigned long long* counter) {
  __shared__ float s_fraction[kMaxDirectionSteps + 1];
  __shared__ f3 s_l[kMaxDirs * kLanes / 32];
  __shared__ f3 s_f[kMaxDirs * kLanes / 32];
  const float bottom = F.bottom;
  fill_fractions(s_fraction, P.ms_steps, threadIdx.x, blockDim.x);
  __syncthreads();
  const int texel = blockIdx.x;
  const int x = texel % P.ms_w, y = texel / P.ms_w;
  const int di = threadIdx.x / kLanes, sub = threadIdx.x % kLanes;
  float u = (float(x) + 0.5f) / float(P.ms_w);
  float v = (float(y) + 0.5f) / float(P.ms_h);
  float h0 = v * v * P.top;
  float radius = bottom + h0;
  float sc = sun_u_to_cosine(u, h0, bottom);
  float ss = sqrtf(mx(1.0f - sc * sc, 0.0f));
  F.sun = mk(ss, sc, 0.0f);
  f3 o = mk(0.0f, radius, 0.0f);
  f3 dL = splat(0.0f), dF = splat(0.0f), pT = splat(1.0f);
  uint32_t samples = 0;
  bool ground = false;
  float end = 0.0f;
  f3 ray = splat(0.0f);
  if (di < P.ms_dirs) {
    const int ndir = P.ms_dirs;
    float si = float(di) + 0.5f;
    float dc = 1.0f - 2.0f * si / float(ndir);
    float ds = sqrtf(mx(1.0f - dc * dc, 0.0f));
    float az = float(di) * 2.39996323f;
    float saz, caz;
    sincosf(az, &saz, &caz);
    ray = mk(ds * caz, dc, ds * saz);
    float start;
    bool valid;
    segment_vec(P, o, ray, bottom, start, end, valid, ground);
    ground = ground && valid;
    if (valid) {
      const float orad = bottom + h0;
      const float closest_raw = -dot(o, ray);
      const RaySource R = make_ray_source(P, F, RayGeom{h0, dc, 0.0f, h0 * (2.0f * bottom + h0), 2.0f * orad * dc}, ray);
      const RayWarp w = make_warp(closest_raw, start, end);
      const int n = P.ms_steps;
      const int per = (n + kLanes - 1) / kLanes;
      const int i0 = min(sub * per, n), i1 = min(i0 + per, n);
      for_intervals(w, i0, i1, n, TableFraction{s_fraction}, [&](float d0, float d1) {
        const MarchSample m = march_sample(P, F, R, d0, d1);
        f3 t, weight;
        segment_integral(m.medium.ext, m.step, t, weight);
        weight = pT * weight;
        dL = dL + weight * (m.st * (R.ER * m.d.r + R.EM * m.d.m));
        dF = dF + weight * m.medium.scat;
        pT = pT * t;
      });
      samples = uint32_t(i1 - i0);
    }
  }
  warp_count(samples, counter);
  // the lanes' parts in ray order: the direction's first lane gets the whole
#pragma unroll
  for (int k = 1; k < kLanes; k <<= 1) {
    const Seg l = shfl_down_seg({dL, pT}, k);
    const f3 f = shfl_down3(dF, k);
    if (sub + k < kLanes) {
      dL = dL + pT * l.L;
      dF = dF + pT * f;
      pT = pT * l.T;
    }
  }
  if (sub != 0) dL = dF = splat(0.0f);
  if (ground && sub == 0) {
    f3 gp = o + ray * end;
    f3 gn = gp * (1.0f / norm(gp));  // Taichi normalized(): v * (1/|v|)
    float gsc = dot(gn, F.sun);
    float vis;
    f3 gT = sample_solar_t(P, F, 0.0f, gsc, horizon_at(0.0f, bottom), vis);
    f3 gL = arr3(P.albedo) * F.E * gT * mx(gsc, 0.0f) / kPiF;
    dL = dL + pT * gL;
  }
  // sum over the directions
#pragma unroll
  for (int k = 16; k >= kLanes; k >>= 1) {
    dL = dL + shfl_xor3(dL, k);
    dF = dF + shfl_xor3(dF, k);
  }
  if ((threadIdx.x & 31) == 0) {
    s_l[threadIdx.x >> 5] = dL;
    s_f[threadIdx.x >> 5] = dF;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < int(blockDim.x >> 5); ++k) {
      dL = dL + s_l[k];
      dF = dF + s_f[k];
    }
    f3 avg_l = dL / float(P.ms_dirs);
    f3 avg_f = vclamp(dF / float(P.ms_dirs), 0.0f, 0.95f);
    out[y * P.ms_w + x] = to4(vmax(avg_l / (splat(1.0f) - avg_f), 0.0f));
  }
}

// ---- sky-view (:1208-1302) and aerial perspective (:1304-1420) -----------------
// A warp a block: 4 lanes of 192x108 texels leave the SMs with 2 or 3
// blocks of 256 (11.9 us) or with 17 or 18 of 32 (11.0 us).
constexpr int kSkyBlock = 32;
template <int kLanes>
__global__ void __launch_bounds__(kSkyBlock) k_sky_view(DevParams P, Frame F, float cam_alt, float4* __restrict__ out,
                                                  unsigned long long* counter) {
  __shared__ float s_fraction[kMaxSkySteps + 1];
  fill_fractions(s_fraction, P.sv_steps, threadIdx.x, blockDim.x);
  __syncthreads();
  const int texels = P.sv_w * P.sv_h;
  const int texel = (blockIdx.x * blockDim.x + threadIdx.x) / kLanes;
  const int t = min(texel, texels - 1);  // every lane takes part in the group's shuffles
  uint32_t samples =
      sky_view_texel<kLanes>(P, F, cam_alt, t % P.sv_w, t / P.sv_w, texel < texels, {s_fraction}, out);
  warp_count(samples, counter);
}

constexpr int kAerialBlock = 128;
__global__ void __launch_bounds__(kAerialBlock) k_aerial(DevParams P, Frame F, AerialView V, float4* __restrict__ out,
                                                unsigned long long* counter) {
  __shared__ float s_fraction[kMaxAerialSteps + 1];
  fill_fractions(s_fraction, P.ap_steps, threadIdx.x, blockDim.x);
  __syncthreads();
  const int warp_id = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (warp_id >= P.ap_w * P.ap_h) return;  // warp-uniform
  uint32_t samples = aerial_column_group<32>(P, F, V, warp_id % P.ap_w, warp_id / P.ap_w, true, {s_fraction}, out);
  warp_count(samples, counter);
}

// Field element i = (x h + y) d + z of a LUT's w x h x d texels, in 32 bits (a
// LUT has at most 2^24 texels).  A read is latency alone, and 64-bit divisions
// were most of that: with launches back to back, 256x64 texels take 1.5 us
// instead of 2.9.
__device__ __forceinline__ unsigned lut_index(unsigned i, unsigned w, unsigned h, unsigned d) {
  const unsigned xy = d == 1 ? i : i / d, z = i - xy * d;
  const unsigned x = xy / h, y = xy - x * h;
  return (z * h + y) * w + x;
}
constexpr int kFieldBlock = 128;
__global__ void __launch_bounds__(kFieldBlock) k_lut_to_fields(const float4* __restrict__ lut, unsigned w, unsigned h,
                                                               unsigned d, float* __restrict__ dst) {
  const unsigned i = blockIdx.x * kFieldBlock + threadIdx.x;
  if (i >= w * h * d) return;
  const float4 v = lut[lut_index(i, w, h, d)];
  dst[i * 3 + 0] = v.x;
  dst[i * 3 + 1] = v.y;
  dst[i * 3 + 2] = v.z;
}
__global__ void __launch_bounds__(kFieldBlock) k_fields_to_lut(const float* __restrict__ src, unsigned w, unsigned h,
                                                               unsigned d, float4* __restrict__ lut) {
  const unsigned i = blockIdx.x * kFieldBlock + threadIdx.x;
  if (i >= w * h * d) return;
  lut[lut_index(i, w, h, d)] = make_float4(src[i * 3 + 0], src[i * 3 + 1], src[i * 3 + 2], 0.0f);
}

inline f3 host3(const float* v) { return {v[0], v[1], v[2]}; }

}  // namespace

cudaError_t launch_transmittance(const DevParams& P, float bottom, float4* out, cudaStream_t s) {
  const int threads = kTBlock;
  const int total = P.t_w * P.t_h * kTLanes;
  k_transmittance<<<(total + threads - 1) / threads, threads, 0, s>>>(P, bottom, out);
  return cudaGetLastError();
}

cudaError_t launch_multi_scattering(const DevParams& P, float bottom, const float E[3], float ar,
                                    const float4* tlut, float4* out, unsigned long long* counter, cudaStream_t s) {
  if (P.ms_dirs > kMaxDirs || P.ms_steps > kMaxDirectionSteps) return cudaErrorInvalidValue;
  // The most lanes a direction that keep the launch within half a wave of the
  // chip's threads, which is what fits at the kernel's registers.
  const long long directions = (long long)P.ms_w * P.ms_h * P.ms_dirs;
  const int lanes = 4 * directions <= kWaveThreads / 2 ? 4 : 2 * directions <= kWaveThreads / 2 ? 2 : 1;
  const int threads = ((lanes * P.ms_dirs + 31) / 32) * 32;
  const int blocks = P.ms_w * P.ms_h;
  const Frame F = make_frame(P, tlut, nullptr, bottom, ar, {0.0f, 1.0f, 0.0f}, host3(E));  // the texel's own sun in it
  if (lanes == 4)
    k_multi_scattering<4><<<blocks, threads, 0, s>>>(P, F, out, counter);
  else if (lanes == 2)
    k_multi_scattering<2><<<blocks, threads, 0, s>>>(P, F, out, counter);
  else
    k_multi_scattering<1><<<blocks, threads, 0, s>>>(P, F, out, counter);
  return cudaGetLastError();
}

cudaError_t launch_sky_view(const DevParams& P, float bottom, float cam_alt, float sun_cos, const float E[3],
                            float ar, const float4* tlut, const float4* mslut, float4* out,
                            unsigned long long* counter, cudaStream_t s) {
  if (P.sv_steps > kMaxSkySteps) return cudaErrorInvalidValue;
  const int threads = kSkyBlock;
  const long long texels = (long long)P.sv_w * P.sv_h;
  const auto go = [&](auto kernel, int lanes) {
    kernel<<<unsigned((lanes * texels + threads - 1) / threads), threads, 0, s>>>(
        P, make_frame(P, tlut, mslut, bottom, ar, sky_view_sun(sun_cos), host3(E)), cam_alt, out, counter);
  };
  // The most lanes a texel that keep the launch within half a resident wave:
  // beyond that the warps only repeat the set-up.
  if (8 * texels <= kWaveThreads / 2)
    go(k_sky_view<8>, 8);
  else if (4 * texels <= kWaveThreads / 2)
    go(k_sky_view<4>, 4);
  else if (2 * texels <= kWaveThreads / 2)
    go(k_sky_view<2>, 2);
  else
    go(k_sky_view<1>, 1);
  return cudaGetLastError();
}

cudaError_t launch_aerial(const DevParams& P, int width, int height, float bottom, float cam_alt, const float sun[3],
                          const float E[3], float ar, const float right[3], const float up[3], const float fwd[3],
                          float tanfov, const float4* tlut, const float4* mslut, float4* out,
                          unsigned long long* counter, cudaStream_t s) {
  if (P.ap_steps > kMaxAerialSteps) return cudaErrorInvalidValue;
  const int threads = kAerialBlock;
  const long long total = 32LL * P.ap_w * P.ap_h;
  const float aspect = float(width) / float(height);
  k_aerial<<<unsigned((total + threads - 1) / threads), threads, 0, s>>>(
      P, make_frame(P, tlut, mslut, bottom, ar, host3(sun), host3(E)),
      aerial_view(aspect, cam_alt, right, up, fwd, tanfov), out, counter);
  return cudaGetLastError();
}

cudaError_t launch_lut_to_fields(const float4* lut, int w, int h, int d, float* dst, cudaStream_t s) {
  k_lut_to_fields<<<(w * h * d - 1) / kFieldBlock + 1, kFieldBlock, 0, s>>>(lut, w, h, d, dst);
  return cudaGetLastError();
}

cudaError_t launch_fields_to_lut(const float* src, int w, int h, int d, float4* lut, cudaStream_t s) {
  k_fields_to_lut<<<(w * h * d - 1) / kFieldBlock + 1, kFieldBlock, 0, s>>>(src, w, h, d, lut);
  return cudaGetLastError();
}

}  // namespace atm
