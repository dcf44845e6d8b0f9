// atm_surrogate.cu - learned surrogates of the sky radiance and of the
// camera-to-surface in-scattering / transmittance.
//
//  * k_gen_samples: training samples produced by the plain integrator itself
//    (the same device functions as the LUT builds and the composite).
//  * k_composite_surrogate + k_surrogate_fallback: the COMPOSITE view with
//    the per-pixel limb integrator (renderer.py :1667-1786) replaced by a
//    BF16 tensor-core MLP and the sky-view lookup (:1474-1525) by a second
//    one.  Pixels where a gate trips (view ray within 0.5 deg of the limb,
//    sun within 0.1 of the local horizon) and a random fraction of the MLP
//    pixels (the error check) go to a queue; the second kernel runs the plain
//    integrator over the queue densely, so a few plain pixels do not stall
//    whole warps of MLP pixels.
//
// Geometry is reparameterised exactly: the atmosphere is spherically
// symmetric, so a segment is described by the altitude of its first point
// inside the shell, the view and sun cosines there, their relative azimuth
// and its length.  Features use the reference's own horizon-concentrating
// coordinates (sky-view v, multi-scattering u) so that the limb and the
// terminator get the same resolution the LUTs give them.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "atm_device.cuh"
#include "atm_frame_paths.cuh"
#include "atm_kernels.h"
#include "atm_mlp_tc.cuh"

namespace atm {

namespace {

constexpr unsigned kAll = 0xffffffffu;

// The features are rounded to BF16, and what they cost is most of what a
// network pixel executes beside its network: the points along the ray and the
// azimuth take the hardware's square root and rsqrt (1-2 ulp) there, and IEEE
// operations in the training samples, whose features are FP32.  The start
// point's altitude and view, a difference of two angles, and the sun cosines
// that gates compare keep IEEE operations in both (a 4K frame of two cameras
// 1.96 ms; 1.94 with hardware functions and a polynomial acos throughout, which
// left the view feature 4.5e-6 off, rms, instead of 1.7e-6; 2.04 ms with IEEE
// operations throughout).

// Sky-view v of a zenith angle whose cosine is mu (sky_zenith_to_v), hz the
// horizon's.
__device__ __forceinline__ float view_feature(float mu, float hz) {
  const float z = acosf(clampf(mu, -1.0f, 1.0f));
  const bool above = z < hz;
  const float n = __saturatef((above ? z : z - hz) / mx(above ? hz : kPiF - hz, 1.0e-6f));
  const float half_root = 0.5f * sqrtf(above ? 1.0f - n : n);
  return above ? 0.5f - half_root : 0.5f + half_root;
}
// Cosine of the azimuth between two horizontal vectors, from their dot
// product and squared lengths; 1 where one is shorter than 1e-6.
__device__ __forceinline__ float azimuth_cosine(float ab, float aa, float bb) {
  return aa > 1.0e-12f && bb > 1.0e-12f ? ab * frsqrt(aa * bb) : 1.0f;
}
// What the features take from the segment's first point alone: up its
// vertical, the sun's cosine and horizontal part there, x[0] and x[2] (altitude
// and sun) and the horizon.  For a camera inside the shell that point is the
// camera and all of it is the frame's: formed once a block.
struct StartPoint {
  f3 up, ts;
  float mu_s, ts2, x0, x2, hz;
};
__device__ __forceinline__ float altitude_feature(const DevParams& P, float h) {
  return 2.0f * sqrtf(__saturatef(h * P.inv_top)) - 1.0f;
}
__device__ __forceinline__ float sun_feature(float bottom, float h, float mu_s) {
  return 2.0f * sun_cosine_to_u(clampf(mu_s, -1.0f, 1.0f), horizon_cosine(h, bottom)) - 1.0f;
}
__device__ __forceinline__ StartPoint start_point(const DevParams& P, const Frame& F, float cam_alt, const RayGeom& G,
                                                  f3 ray, float start) {
  const float o_y = F.bottom + cam_alt;
  const float h = altitude_at(G, start, F.bottom);
  const f3 ps = mk(ray.x * start, o_y + ray.y * start, ray.z * start);
  StartPoint S;
  S.up = ps * (1.0f / mx(norm(ps), 1.0f));
  S.mu_s = dot(F.sun, S.up);
  S.ts = F.sun - S.up * S.mu_s;
  S.ts2 = dot(S.ts, S.ts);
  S.x0 = altitude_feature(P, h);
  S.x2 = sun_feature(F.bottom, h, S.mu_s);
  S.hz = sky_horizon_zenith(h, F.bottom);
  return S;
}

// Sun (multi-scattering u mapping) and altitude features, x[0] and x[1], of
// the point at distance t along a ray leaving (0, o_y, 0) (G: its geometry).
// Where a segment's light comes from depends on where it ends and how low it
// dips as much as on where it starts: with these points given, the sky
// network's held-out error drops by a quarter and the aerial network's on
// camera-to-surface segments to a third.  Returns the point's sun cosine.
// kExactSun, kExactAltitude: IEEE operations (a gate, a training sample).
template <bool kExactSun, bool kExactAltitude>
__device__ __forceinline__ float point_features(const DevParams& P, float bottom, const RayGeom& G, f3 ray, float o_y,
                                                f3 sun, float t, float* x) {
  const f3 pt = mk(ray.x * t, o_y + ray.y * t, ray.z * t);
  const float mu = clampf(kExactSun ? dot(sun, pt) / mx(norm(pt), 1.0f)
                                    : dot(sun, pt) * frsqrt(mx(dot(pt, pt), 1.0f)), -1.0f, 1.0f);
  const float h = altitude_at(G, t, bottom);
  x[0] = 2.0f * sun_cosine_to_u(mu, horizon_cosine(h, bottom)) - 1.0f;
  x[1] = kExactAltitude ? altitude_feature(P, h) : 2.0f * fsqrt(__saturatef(h * P.inv_top)) - 1.0f;
  return mu;
}
// Aerial x[7..10]: the segment's end, then its middle.  Returns the smaller
// |sun cosine| of the two (the twilight gate); `mu_end`, `mu_mid` receive
// the cosines themselves.  kSample: of a training sample.
template <bool kSample>
__device__ __forceinline__ float segment_features(const DevParams& P, float bottom, const RayGeom& G, f3 ray,
                                                  float o_y, f3 sun, float start, float end, float* x,
                                                  float& mu_end, float& mu_mid) {
  mu_end = point_features<true, kSample>(P, bottom, G, ray, o_y, sun, end, x + 7);
  mu_mid = point_features<true, kSample>(P, bottom, G, ray, o_y, sun, 0.5f * (start + end), x + 9);
  return mn(fabsf(mu_end), fabsf(mu_mid));
}
// Sky x[6..9]: the end of the ray's march (the shell top or the ground),
// then its lowest point (the closest approach, clamped to the march).
template <bool kSample>
__device__ __forceinline__ void sky_ray_features(const DevParams& P, float bottom, float h, f3 ray, f3 sun, float* x) {
  const RayGeom G = camera_ray_geom(P, bottom, h, ray);
  float start, end;
  bool valid, ground;
  segment_of(P, G, bottom, start, end, valid, ground);
  if (!valid) start = end = 0.0f;
  const float o_y = bottom + mx(h, 0.0f);
  point_features<kSample, kSample>(P, bottom, G, ray, o_y, sun, end, x + 6);
  point_features<kSample, kSample>(P, bottom, G, ray, o_y, sun, clampf(G.tc, start, end), x + 8);
}

// Counter-based uniform in [0, 1): 64-bit mix of (seed, index, lane).
__device__ __forceinline__ float uniform01(unsigned long long seed, unsigned long long i, unsigned k) {
  unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (i * 16 + k + 1);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return float(z >> 40) * (1.0f / 16777216.0f);
}

// Sky radiance along `ray` from altitude h (the sky-view march, one thread).
__device__ f3 sky_radiance(const DevParams& P, const Frame& F, float h, f3 ray) {
  float start, end;
  bool valid, ground;
  const RayGeom G = camera_ray_geom(P, F.bottom, h, ray);
  segment_of(P, G, F.bottom, start, end, valid, ground);
  if (!valid) return splat(0.0f);
  const RaySource rs = make_ray_source(P, F, G, ray);
  const int n = P.sv_steps;
  return vmax(march(P, F, rs, make_warp(G.tc, start, end), 0, n, n, DivideFraction{float(n)}).L, 0.0f);
}

// Aerial samples may be shaped toward camera-to-surface segments: a share
// starts at the shell top (feature 0 = 1; every segment seen from above the
// shell starts there) and a share ends at a surface altitude, where the ray
// reaches it (the segment's length then follows from the geometry).
__global__ void __launch_bounds__(128) k_gen_samples(const SurrogateSetDev* __restrict__ sets, int n_sets, int kind,
                                                     long long n, unsigned long long seed, SampleShaping shaping,
                                                     float* __restrict__ features, float* __restrict__ targets,
                                                     unsigned long long* __restrict__ counter) {
  const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  uint32_t samples = 0;
  if (i < n) {
    const SurrogateSetDev& S = sets[min(int(uniform01(seed, i, 0) * n_sets), n_sets - 1)];
    const DevParams& P = S.P;
    const float R = S.F.bottom;
    float x[16];
    for (int k = 0; k < 4; ++k) x[k] = 2.0f * uniform01(seed, i, k + 1) - 1.0f;
    if (shaping.x0_lo < shaping.x0_hi) x[0] = shaping.x0_lo + (shaping.x0_hi - shaping.x0_lo) * uniform01(seed, i, 9);
    if (kind == 1 && uniform01(seed, i, 6) < shaping.top_fraction) x[0] = 1.0f;
    // invert the feature maps
    const float h = P.top * 0.25f * (x[0] + 1.0f) * (x[0] + 1.0f);
    const float zen = sky_v_to_zenith(0.5f * (x[1] + 1.0f), sky_horizon_zenith(h, R));
    float sv, mu_v;
    sincosf(zen, &sv, &mu_v);
    // the sun: uniform in the feature, or for a share uniform in zenith angle
    // (the feature's horizon-concentrating map leaves a high sun sparse)
    const float mu_s = uniform01(seed, i, 10) < shaping.sun_angle_fraction
                           ? cosf(shaping.sun_angle_max * uniform01(seed, i, 11))
                           : sun_u_to_cosine(0.5f * (x[2] + 1.0f), h, R);
    const float ss = sqrtf(mx(1.0f - mu_s * mu_s, 0.0f));
    const float cphi = x[3], sphi = sqrtf(mx(1.0f - cphi * cphi, 0.0f));
    const f3 ray = mk(sv, mu_v, 0.0f);
    const f3 sun = mk(ss * cphi, mu_s, ss * sphi);
    // rounding-consistent features
    x[0] = altitude_feature(P, h);
    x[1] = 2.0f * view_feature(mu_v, sky_horizon_zenith(h, R)) - 1.0f;
    x[2] = sun_feature(R, h, mu_s);
    x[3] = clampf(cphi, -1.0f, 1.0f);
    x[4] = S.lhr_n;
    x[5] = S.lhm_n;
    Frame F = S.F;
    F.sun = sun;
    const f3 inv_e = mk(1.0f / F.E.x, 1.0f / F.E.y, 1.0f / F.E.z);
    if (kind == 0) {  // sky: 10 features -> log(L/E + floor)
      const f3 L = sky_radiance(P, F, h, ray) * inv_e;
      samples = uint32_t(P.sv_steps);
      sky_ray_features<true>(P, R, h, ray, sun, x);
      for (int k = 0; k < kSurrogateSkyIn; ++k) features[i * kSurrogateSkyIn + k] = x[k];
      targets[i * 3 + 0] = logf(L.x + kSurrogateFloor);
      targets[i * 3 + 1] = logf(L.y + kSurrogateFloor);
      targets[i * 3 + 2] = logf(L.z + kSurrogateFloor);
    } else {  // aerial: + log length -> log(L/E + floor), optical depth
      const float u = uniform01(seed, i, 5);
      float len = expf(u * logf(kSurrogateMaxLength));
      x[6] = 2.0f * u - 1.0f;
      if (uniform01(seed, i, 7) < shaping.surface_fraction) {
        const float he = shaping.surface_min + (shaping.surface_max - shaping.surface_min) * uniform01(seed, i, 8);
        float nr, fr;
        bool hit;
        shell_roots(h, mu_v, he, R, nr, fr, hit);
        const float t = nr > 0.0f ? nr : fr;
        if (hit && t >= 1.0f && t <= kSurrogateMaxLength) {
          len = t;
          x[6] = 2.0f * logf(len) / logf(kSurrogateMaxLength) - 1.0f;
        }
      }
      f3 L = splat(0.0f), T = splat(1.0f);
      float start, end;
      const RayGeom G = ray_geom(P, R, h, mu_v, sv);
      if (surface_interval(P, G, R, len, start, end)) {
        L = integrate_surface(P, F, G, ray, start, end, divide_fractions(P), samples) * inv_e;
        T = surface_segment_t(P, F, G, start, end);
      } else {
        start = end = 0.0f;
      }
      float mu_end, mu_mid;
      segment_features<true>(P, R, G, ray, R + h, sun, start, end, x, mu_end, mu_mid);
      for (int k = 0; k < kSurrogateApIn; ++k) features[i * kSurrogateApIn + k] = x[k];
      targets[i * 6 + 0] = logf(L.x + kSurrogateFloor);
      targets[i * 6 + 1] = logf(L.y + kSurrogateFloor);
      targets[i * 6 + 2] = logf(L.z + kSurrogateFloor);
      targets[i * 6 + 3] = mn(-logf(mx(T.x, 1.0e-30f)), kSurrogateMaxDepth);
      targets[i * 6 + 4] = mn(-logf(mx(T.y, 1.0e-30f)), kSurrogateMaxDepth);
      targets[i * 6 + 5] = mn(-logf(mx(T.z, 1.0e-30f)), kSurrogateMaxDepth);
    }
  }
  warp_count(samples, counter);
}

__device__ __forceinline__ bool check_pixel(int x, int y, unsigned seed, float fraction) {
  unsigned h = (unsigned(x) * 0x8DA6B343u) ^ (unsigned(y) * 0xD8163841u) ^ (seed * 0x9E3779B1u);
  h ^= h >> 15;
  h *= 0x2C1B3C6Du;
  h ^= h >> 12;
  return float(h >> 8) * (1.0f / 16777216.0f) < fraction;
}

// A pixel's index in storage order (the image's contiguous axis first), the
// order of the calibration scratch image.
__device__ __forceinline__ size_t storage_index(const ImageLayout& L, int x, int y) {
  return L.sy <= L.sx ? size_t(x) * size_t(L.height) + size_t(y) : size_t(y) * size_t(L.width) + size_t(x);
}

// Largest per-channel error of `got` relative to `ref` (floor 1e-6 E).
__device__ __forceinline__ float color_error(f3 got, f3 ref, f3 E) {
  const f3 d = vmax(got - ref, 0.0f) + vmax(ref - got, 0.0f);
  return mx(mx(d.x / mx(ref.x, 1e-6f * E.x), d.y / mx(ref.y, 1e-6f * E.y)), d.z / mx(ref.z, 1e-6f * E.z));
}

// Radiance of a network's log output ln(L / E + floor), per channel.
__device__ __forceinline__ f3 net_radiance(const float (&y)[8], const float* E, f3 floor) {
  return vmax(mk((__expf(y[0]) - floor.x) * E[0], (__expf(y[1]) - floor.y) * E[1], (__expf(y[2]) - floor.z) * E[2]),
              0.0f);
}

enum PixelKind : int { kNone = 0, kSurfMlp, kSurfPlain, kSurfEmpty, kSkyMlp, kSkyLut };

// The network kernels: one block an SM stays for the launch and its kWorkers
// tiles of 128 threads each run 128-pixel tiles of the frame one after
// another, every tile on its own barriers - while one waits for its MMAs the
// others have features and activations to compute.  The weights and the
// tensor memory are taken once a block.  What bounds them is the activations'
// tanh (XU) and the issue of features and outputs around them, at the
// latency of the five serial layers; five tiles are what 512 tensor-memory
// columns hold (64 accumulator and 32 activation columns a tile, the bias's 8
// shared).  A 4K frame takes 0.80 ms; 0.83 ms with the start point's features
// formed by each pixel, 0.99 ms with two tiles a block, three blocks an SM and
// the weights copied by each block.
constexpr int kWorkers = 5;
constexpr uint32_t kWorkerCols = 96, kOnesCol = kWorkers * kWorkerCols, kSurrogateTmemCols = 512;

struct NetBlock {
  uint64_t mbar[kWorkers + 1];  // the tiles' MMA completions, the weights' arrival
  uint32_t tmem;
  float horizon;  // the camera's horizon zenith
  float limb_low, limb_high;  // no ray whose y is outside is within the limb's angle
  StartPoint camera;          // of a camera inside the shell
};
// Whether a ray lies within limb_rad of the limb.  The bounds decide most rays
// without the angle; they are a margin of 1e-5 wider than it, in cosines, so
// that the angle's last bits never matter beyond them.
__device__ __forceinline__ bool near_limb_of(const NetBlock& B, float y, float limb_rad) {
  if (y < B.limb_low || y > B.limb_high) return false;
  return fabsf(acosf(clampf(y, -1.0f, 1.0f)) - B.horizon) < limb_rad;
}
// x[0..3] of a sky ray: the camera's horizontal plane and vertical are y = 0 and y.
__device__ __forceinline__ void sky_start_features(const NetBlock& B, const Frame& F, f3 ray, float* x) {
  x[0] = B.camera.x0;
  x[1] = 2.0f * view_feature(ray.y, B.camera.hz) - 1.0f;
  x[2] = B.camera.x2;
  x[3] = clampf(azimuth_cosine(ray.x * F.sun.x + ray.z * F.sun.z, ray.x * ray.x + ray.z * ray.z,
                               F.sun.x * F.sun.x + F.sun.z * F.sun.z), -1.0f, 1.0f);
}
// Sets a block up (every thread calls): the weights into smem by bulk copies,
// tensor memory, barriers.  Returns this thread's tile; `weights` false if the
// weights did not arrive in time.
__device__ __forceinline__ TcTile net_block_begin(NetBlock& B, unsigned char* smem, const unsigned char* w0, int n0,
                                                  const unsigned char* w1, int n1, const DevParams& P, const Frame& F,
                                                  float cam_alt, float limb_rad, bool& weights) {
  if (threadIdx.x == 0) {
    for (int k = 0; k <= kWorkers; ++k) tc::mbar_init(&B.mbar[k], 1);
    tc::mbar_init_fence();
    tc::mbar_arrive_expect_tx(&B.mbar[kWorkers], uint32_t(n0 + n1));
    if (n0 > 0) tc::bulk_g2s(smem, w0, uint32_t(n0), &B.mbar[kWorkers]);
    if (n1 > 0) tc::bulk_g2s(smem + n0, w1, uint32_t(n1), &B.mbar[kWorkers]);
    B.horizon = sky_horizon_zenith(cam_alt, F.bottom);
    B.limb_low = cosf(mn(B.horizon + limb_rad, kPiF)) - 1.0e-5f;
    B.limb_high = cosf(mx(B.horizon - limb_rad, 0.0f)) + 1.0e-5f;
    const f3 zenith = mk(0.0f, 1.0f, 0.0f);
    B.camera = start_point(P, F, cam_alt, camera_ray_geom(P, F.bottom, cam_alt, zenith), zenith, 0.0f);
  }
  if (threadIdx.x >> 5 == 1) tc::alloc(&B.tmem, kSurrogateTmemCols);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const int tile = threadIdx.x >> 7, row = threadIdx.x & 127;
  if (tile == 0) store_ones(B.tmem + kOnesCol, row);
  // each thread observes the weights' mbarrier before any MMA of its tile reads them
  const bool arrived = tc::mbar_wait(&B.mbar[kWorkers], 0u, kTcWaitTries);
  tc::fence_before_sync();
  weights = __syncthreads_and(arrived);
  tc::fence_after_sync();
  return TcTile{B.tmem + kWorkerCols * tile, B.tmem + kWorkerCols * tile + 64u, B.tmem + kOnesCol, &B.mbar[tile], 0u,
                tile, row};
}
// Frees the tensor memory (every thread calls; no MMA of its tile in flight).
__device__ __forceinline__ void net_block_end(NetBlock& B) {
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (threadIdx.x >> 5 == 1) tc::dealloc(B.tmem, kSurrogateTmemCols);
}
// After a network run that gave up: waits, with the library's full bound
// whatever the frame's own bound was, for the one commit in flight.  False in
// every thread of the tile if that does not come either: no more networks.
__device__ __forceinline__ bool tile_recover(TcTile& T) {
  return tc::tile_all(T.tile, tc::mbar_wait(T.mbar, T.phase ^ 1u, kTcWaitTries));
}

// A frame's 128-pixel tiles: 16 pixels along the image's contiguous axis by 8,
// a warp 16 x 2 of them (whole sectors of every image).
struct PixelTiles {
  int across, count;  // tiles along y (y contiguous) or x, tiles in all
};
__host__ __device__ inline bool y_contiguous(const ImageLayout& L) { return L.sy <= L.sx; }
inline PixelTiles pixel_tiles(const ImageLayout& L) {
  const int fast = y_contiguous(L) ? L.height : L.width, slow = y_contiguous(L) ? L.width : L.height;
  const int across = (fast + 15) / 16;
  return {across, across * ((slow + 7) / 8)};
}
__device__ __forceinline__ bool tile_pixel_of(const ImageLayout& L, const PixelTiles& N, int tile, int row, int& x,
                                              int& y) {
  const int slow = (tile / N.across) * 8 + (row >> 4), fast = (tile % N.across) * 16 + (row & 15);
  x = y_contiguous(L) ? slow : fast;
  y = y_contiguous(L) ? fast : slow;
  return x < L.width && y < L.height;
}

// The fused frame's surface colours (shaded_scene) into hdr, where the
// composite takes them from: shading in the composite itself, on a network
// block's 20 warps an SM, takes 1.61 ms a 4K frame, 1.39 ms so.  Not where hdr
// is also an input (hdr_is_input), which it would overwrite.
__global__ void __launch_bounds__(kRunPixels * kRunRows) k_scene(DevParams P, Frame F, ImageLayout L, CompositeScalars A,
                                                                 ShadeParams S, ShadeImages I,
                                                                 float* __restrict__ hdr) {
  int x, y;
  if (!run_pixel(L, x, y)) return;
  const size_t e = pix_offset(L, x, y);
  const f3 color = shaded_scene(P, F, A, S, L, I, x, y, e, I.surface_id[e]);
  float* out = hdr + e * L.channels;
  out[0] = color.x;
  out[1] = color.y;
  out[2] = color.z;
}

// The surface colour is `scene`'s or, with kShade, the fused frame's own
// (shaded_scene).  hdr may be `scene` or any other image: a pixel is read by
// the thread that then writes it, and by no other.
template <bool kShade>
__global__ void __launch_bounds__(128 * kWorkers, 1) k_composite_surrogate(
    DevParams P, Frame F, ImageLayout L, PixelTiles N, CompositeScalars A, const float* scene,
    const float* __restrict__ space, const int32_t* __restrict__ sid, const float* __restrict__ pos,
    const float4* __restrict__ svlut, SurrogateNets nets, SurrogateQueue Q, float* hdr, ShadeParams S, ShadeImages I) {
  extern __shared__ __align__(128) unsigned char smem[];  // the aerial network, then the sky network
  __shared__ NetBlock B;
  bool nets_ok;  // tile-uniform: the networks may run
  TcTile T = net_block_begin(B, smem, nets.ap, nets.ap_bytes, nets.sky, nets.sky_bytes, P, F, A.cam_alt,
                             nets.limb_rad, nets_ok);
  const int lane = threadIdx.x & 31;
  for (int t = T.tile * gridDim.x + blockIdx.x; t < N.count; t += kWorkers * gridDim.x) {
    int x, y;
    const bool inside = tile_pixel_of(L, N, t, T.row, x, y);
    const int cx = inside ? x : 0, cy = inside ? y : 0;
    const size_t e = pix_offset(L, cx, cy);
    const size_t o = e * L.channels;
    const f3 ray = pixel_ray(L, A, cx, cy).ray;
    const bool near_limb = near_limb_of(B, ray.y, nets.limb_rad);

    int kind = kNone;
    uint32_t xp[8] = {};
    float start = 0.0f, end = 0.0f;
    if (inside) {
      float fx[16] = {};
      if (sid[e] >= 0) {
        const RayGeom G = camera_ray_geom(P, A.bottom, A.cam_alt, ray);
        if (!surface_interval(P, G, A.bottom, norm(ld3(pos + o)), start, end)) {
          kind = kSurfEmpty;
        } else if (nets.ap == nullptr || near_limb) {
          kind = kSurfPlain;
        } else {
          // features at the segment's first point inside the shell
          const float o_y = A.bottom + A.cam_alt;
          const StartPoint sp = start == 0.0f ? B.camera : start_point(P, F, A.cam_alt, G, ray, start);
          const float mu_s = sp.mu_s;
          const float mu_v = dot(ray, sp.up);
          const f3 tv = ray - sp.up * mu_v;
          fx[0] = sp.x0;
          fx[1] = 2.0f * view_feature(mu_v, sp.hz) - 1.0f;
          fx[2] = sp.x2;
          fx[3] = clampf(azimuth_cosine(dot(tv, sp.ts), dot(tv, tv), sp.ts2), -1.0f, 1.0f);
          fx[4] = nets.lhr_n;
          fx[5] = nets.lhm_n;
          fx[6] = 2.0f * __logf(clampf(end - start, 1.0f, kSurrogateMaxLength)) / logf(kSurrogateMaxLength) - 1.0f;
          // twilight gate: the sun cosine small at the start, middle or end, or
          // of different signs there (the segment crosses the terminator)
          float mu_end, mu_mid;
          const float mu_min =
              mn(fabsf(mu_s), segment_features<false>(P, A.bottom, G, ray, o_y, F.sun, start, end, fx, mu_end, mu_mid));
          const bool crosses =
              nets.gate_crossing && ((mu_s > 0.0f) != (mu_end > 0.0f) || (mu_s > 0.0f) != (mu_mid > 0.0f));
          kind = (mu_min < nets.twilight_cos || crosses) ? kSurfPlain : kSurfMlp;
          pack_inputs(fx, kSurrogateApIn, xp);
        }
      } else if (nets.sky != nullptr && A.cam_alt <= P.top && fabsf(F.sun.y) >= nets.sky_twilight_cos && !near_limb) {
        kind = kSkyMlp;
        sky_start_features(B, F, ray, fx);
        fx[4] = nets.lhr_n;
        fx[5] = nets.lhm_n;
        sky_ray_features<false>(P, A.bottom, A.cam_alt, ray, F.sun, fx);
        pack_inputs(fx, kSurrogateSkyIn, xp);
      } else {
        kind = kSkyLut;
      }
    }

    // the networks on the tensor cores, each run by the whole tile when any of
    // its pixels needs it (tile-uniform: every barrier stays convergent).  A
    // tile whose wait timed out issues nothing more and its MLP pixels take
    // the plain path below.
    float yv[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    const bool need_ap = nets.ap != nullptr && tc::tile_any(T.tile, kind == kSurfMlp);
    const bool need_sky = nets.sky != nullptr && tc::tile_any(T.tile, kind == kSkyMlp);
    bool tc_ok = nets_ok;
    if (need_ap && tc_ok) {
      float v[8];
      tc_ok = mlp_tile_tc<kSurrogateApHidden>(smem, kSurrogateApIn, T, xp, v, nets.wait_tries);
      if (kind == kSurfMlp)
        for (int k = 0; k < 8; ++k) yv[k] = v[k];
    }
    if (need_sky && tc_ok) {
      float v[8];
      tc_ok = mlp_tile_tc<kSurrogateSkyHidden>(smem + nets.ap_bytes, kSurrogateSkyIn, T, xp, v, nets.wait_tries);
      if (kind == kSkyMlp)
        for (int k = 0; k < 8; ++k) yv[k] = v[k];
    }
    tc_ok = tc_ok || !(need_ap || need_sky);
    if (!tc_ok) {
      // the networks' outputs are not valid: the plain path for these pixels
      if (kind == kSurfMlp) kind = kSurfPlain;
      if (kind == kSkyMlp) kind = kSkyLut;
      if (T.row == 0) atomicOr(Q.status, 1u);
      if (nets_ok) nets_ok = tile_recover(T);
    }

    bool queued = false;
    uint32_t qkind = kQueueSurface;
    f3 Lnet = mk(-1.0f, 0.0f, 0.0f);  // the network's in-scattering (x < 0: none)
    if (inside && kind != kSurfPlain) {
      f3 color = kShade ? shaded_scene(P, F, A, S, L, I, x, y, e, sid[e]) : ld3(scene + o);
      if (kind == kSurfMlp) {
        // transmittance: the plain path's own two-tap LUT ratio (:1603-1665);
        // in-scattering: the network, ln(L / E + floor + floor_t T)
        const f3 Tm = surface_segment_t(P, F, camera_ray_geom(P, A.bottom, A.cam_alt, ray), start, end);
        const f3 Lm = net_radiance(yv, A.E, splat(nets.floor) + Tm * nets.floor_t);
        color = Lm + color * Tm;
        Lnet = Lm;
        if (check_pixel(x, y, Q.seed, Q.check_fraction)) {
          queued = true;
          qkind = kQueueSurfaceCheck;
        }
      } else if (kind == kSkyMlp) {
        const f3 sky = net_radiance(yv, A.E, splat(nets.sky_floor));
        color = composite_sky_with(P, F, A, sky, ray, color, ld3(space + o), float(L.height));
        if (check_pixel(x, y, Q.seed, Q.check_fraction)) {
          queued = true;
          qkind = kQueueSkyCheck;
        }
      } else if (kind == kSkyLut) {
        color = composite_sky(P, F, A, svlut, ray, color, ld3(space + o), float(L.height));
      }
      color = vmax(color, 0.0f);
      hdr[o + 0] = color.x;
      hdr[o + 1] = color.y;
      hdr[o + 2] = color.z;
    } else if (kind == kSurfPlain) {
      queued = true;
    }
    if (inside && Q.lm != nullptr) {  // the calibration's scratch: every pixel, each frame
      float* lm = Q.lm + 3 * storage_index(L, x, y);
      lm[0] = Lnet.x;
      if (Lnet.x >= 0.0f) {
        lm[1] = Lnet.y;
        lm[2] = Lnet.z;
      }
    }

    // warp-aggregated append to the fallback queue
    const unsigned qm = __ballot_sync(kAll, queued);
    if (qm) {
      const int leader = __ffs(qm) - 1;
      uint32_t base = 0;
      if (lane == leader) base = atomicAdd(Q.count, uint32_t(__popc(qm)));
      base = __shfl_sync(kAll, base, leader);
      if (queued)
        Q.items[base + __popc(qm & ((1u << lane) - 1u))] = (qkind << 30) | uint32_t(cy * L.width + cx);
    }
    if (Q.stats != nullptr) {
      if (!tc_ok && T.row == 0) atomicAdd(Q.stats + 7, 1.0f);  // tiles whose MMA timed out
      const unsigned gs = __ballot_sync(kAll, kind == kSurfPlain), ms = __ballot_sync(kAll, kind == kSurfMlp);
      const unsigned mk_ = __ballot_sync(kAll, kind == kSkyMlp), ls = __ballot_sync(kAll, kind == kSkyLut);
      if (lane == 0) {
        if (gs) atomicAdd(Q.stats + 3, float(__popc(gs)));
        if (ms) atomicAdd(Q.stats + 4, float(__popc(ms)));
        if (mk_) atomicAdd(Q.stats + 5, float(__popc(mk_)));
        if (ls) atomicAdd(Q.stats + 6, float(__popc(ls)));
      }
    }
  }
  net_block_end(B);
}

// Lanes that share a queued pixel's march: a short queue (the checked 1% of a
// frame is about one pixel a resident thread) would run as one or two whole
// marches a thread on part of the warps; a long one would only repeat each
// pixel's set-up.  4K, 1% checked, three blocks an SM: 63 us (4 lanes: 67, 1
// lane: 66; two or four blocks an SM: 73, 66).
constexpr int kQueueLanes = 2, kQueueBlocks = 3;
__device__ __forceinline__ bool split_queue(uint32_t n) { return n <= 8u * gridDim.x * blockDim.x; }

// Sky radiance along `ray` by kLanes consecutive lanes, as sky_radiance; the
// group's first lane receives it.  Every lane of the warp must call.
template <int kLanes>
__device__ __forceinline__ f3 sky_radiance_split(const DevParams& P, const Frame& F, float h, f3 ray, bool active) {
  Seg acc = seg_identity();
  float start, end;
  bool valid, ground;
  const RayGeom G = camera_ray_geom(P, F.bottom, h, ray);
  segment_of(P, G, F.bottom, start, end, valid, ground);
  if (active && valid) {
    const int n = P.sv_steps, per = (n + kLanes - 1) / kLanes;
    const int i0 = min(int(threadIdx.x & (kLanes - 1)) * per, n);
    acc = march(P, F, make_ray_source(P, F, G, ray), make_warp(G.tc, start, end), i0, min(i0 + per, n), n,
                DivideFraction{float(n)});
  }
  return vmax(group_compose<kLanes>(acc).L, 0.0f);
}

// The plain integrator over the queued pixels: gated surface pixels get it
// as their result; checked pixels compare the MLP's color (in hdr) with it,
// then keep the plain result.  Warps take 32 / kLanes entries per ticket.
struct CheckSums {
  uint32_t samples = 0, checked = 0;
  float err_sum = 0.0f, err_max = 0.0f;
};
template <int kLanes, bool kShade>
__device__ __forceinline__ void fallback_queue(const DevParams& P, const Frame& F, const ImageLayout& L,
                                               const CompositeScalars& A, const float* __restrict__ scene,
                                               const float* __restrict__ space, const float* __restrict__ pos,
                                               const SurrogateQueue& Q, float* __restrict__ hdr, const ShadeParams& S,
                                               const ShadeImages& I, uint32_t n, const TableFractions& fractions,
                                               CheckSums& sums) {
  const int lane = threadIdx.x & 31;
  const bool first = (lane & (kLanes - 1)) == 0;
  for (;;) {
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(Q.count + 1, 32u / kLanes);
    base = __shfl_sync(kAll, base, 0);
    if (base >= n) break;
    const uint32_t i = base + uint32_t(lane / kLanes);
    const bool has = i < n;
    const uint32_t entry = has ? Q.items[i] : 0;
    const uint32_t kind = entry >> 30, p = entry & 0x3fffffffu;
    const int x = int(p % uint32_t(L.width)), y = int(p / uint32_t(L.width));
    const size_t e = pix_offset(L, x, y);
    const size_t o = e * L.channels;
    const f3 ray = pixel_ray(L, A, x, y).ray;
    const bool sky_check = has && kind == kQueueSkyCheck;
    f3 color = splat(0.0f);
    if (__any_sync(kAll, sky_check)) {
      const f3 sky = sky_radiance_split<kLanes>(P, F, A.cam_alt, ray, sky_check);
      if (sky_check && first) {
        sums.samples += uint32_t(P.sv_steps);
        color = kShade ? shaded_scene(P, F, A, S, L, I, x, y, e, I.surface_id[e]) : ld3(scene + o);
        color = composite_sky_with(P, F, A, sky, ray, color, ld3(space + o), float(L.height));
      }
    }
    const bool surface = has && !sky_check;
    const RayGeom G = camera_ray_geom(P, A.bottom, A.cam_alt, ray);
    float start = 0.0f, end = 0.0f;
    const bool clipped = surface && surface_interval(P, G, A.bottom, norm(ld3(pos + o)), start, end);
    const f3 Ls = integrate_surface_split<kLanes>(P, F, G, ray, start, end, clipped, fractions, sums.samples);
    if (surface && first) {
      color = kShade ? shaded_scene(P, F, A, S, L, I, x, y, e, I.surface_id[e]) : ld3(scene + o);
      if (clipped) {
        color = Ls + color * surface_segment_t(P, F, G, start, end);
        if (kind == kQueueSurfaceCheck && Q.lm != nullptr) {
          // the calibration: this tile's log ratio of the plain in-scattering
          // to the network's; the pixel itself keeps the plain result
          float* lm = Q.lm + 3 * storage_index(L, x, y);
          const f3 Ln = ld3(lm);
          if (Ln.x >= 0.0f) {
            float* t = Q.tiles + 4 * ((y >> Q.tile_shift) * Q.tiles_x + (x >> Q.tile_shift));
            atomicAdd(t + 0, clampf(__logf(mx(Ls.x, 1e-12f) / mx(Ln.x, 1e-12f)), -kCalibrationClamp,
                                    kCalibrationClamp));
            atomicAdd(t + 1, clampf(__logf(mx(Ls.y, 1e-12f) / mx(Ln.y, 1e-12f)), -kCalibrationClamp,
                                    kCalibrationClamp));
            atomicAdd(t + 2, clampf(__logf(mx(Ls.z, 1e-12f) / mx(Ln.z, 1e-12f)), -kCalibrationClamp,
                                    kCalibrationClamp));
            atomicAdd(t + 3, 1.0f);
          }
          lm[0] = -1.0f;
        }
      }
    }
    if (has && first) {
      color = vmax(color, 0.0f);
      if (kind != kQueueSurface) {
        const float err = color_error(ld3(hdr + o), color, F.E);
        ++sums.checked;
        sums.err_sum += err;
        sums.err_max = mx(sums.err_max, err);
      }
      hdr[o + 0] = color.x;
      hdr[o + 1] = color.y;
      hdr[o + 2] = color.z;
    }
  }
}
template <bool kShade>
__global__ void __launch_bounds__(256, 3) k_surrogate_fallback(
    DevParams P, Frame F, ImageLayout L, CompositeScalars A, const float* __restrict__ scene,
    const float* __restrict__ space, const float* __restrict__ pos, SurrogateQueue Q, float* __restrict__ hdr,
    unsigned long long* counter, ShadeParams S, ShadeImages I) {
  __shared__ float s_fractions[kFractionTable];
  const TableFractions fractions = table_fractions(P, s_fractions);
  const int lane = threadIdx.x & 31;
  const uint32_t n = *Q.count;
  CheckSums sums;
  if (split_queue(n))
    fallback_queue<kQueueLanes, kShade>(P, F, L, A, scene, space, pos, Q, hdr, S, I, n, fractions, sums);
  else
    fallback_queue<1, kShade>(P, F, L, A, scene, space, pos, Q, hdr, S, I, n, fractions, sums);
  warp_count(sums.samples, counter);
  if (Q.stats != nullptr) {
    float c = float(sums.checked);
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) {
      c += __shfl_xor_sync(kAll, c, k);
      sums.err_sum += __shfl_xor_sync(kAll, sums.err_sum, k);
      sums.err_max = mx(sums.err_max, __shfl_xor_sync(kAll, sums.err_max, k));
    }
    if (lane == 0 && c > 0.0f) {
      atomicAdd(Q.stats + 0, c);
      atomicAdd(Q.stats + 1, sums.err_sum);
      atomicMax(reinterpret_cast<int*>(Q.stats + 2), __float_as_int(sums.err_max));  // non-negative floats
    }
  }
}

// The calibration pass: every MLP surface pixel whose tile holds enough
// checked pixels gets its network in-scattering rescaled by the tile's mean
// log ratio, hdr += Lnet (exp(mean) - 1).  Memory-bound: 4K takes 51 us, 56
// with two 64-bit divisions a pixel.
__global__ void __launch_bounds__(kRunPixels * kRunRows) k_surrogate_calibrate(ImageLayout L, SurrogateQueue Q, float* __restrict__ hdr) {
  int x, y;
  if (!run_pixel(L, x, y)) return;
  const float* lm = Q.lm + 3 * storage_index(L, x, y);
  const float lx = lm[0];
  if (lx < 0.0f) return;
  const float4 t = *reinterpret_cast<const float4*>(Q.tiles + 4 * ((y >> Q.tile_shift) * Q.tiles_x + (x >> Q.tile_shift)));
  if (t.w < float(kCalibrationMinChecks)) return;
  const float inv = 1.0f / t.w;
  const size_t o = pix_offset(L, x, y) * L.channels;
  hdr[o + 0] += lx * (__expf(t.x * inv) - 1.0f);
  hdr[o + 1] += lm[1] * (__expf(t.y * inv) - 1.0f);
  hdr[o + 2] += lm[2] * (__expf(t.z * inv) - 1.0f);
}

// Sky radiance of every pixel of a frame, the pixel's own view ray from the
// camera (the learned sky-view workload; the G-buffer is not read):
//  * kSkyPixelsPlain: the plain integrator per pixel - the sky-view march of
//    :1208-1302 (sv_steps warped segments) along the pixel's ray;
//  * kSkyPixelsNet: the sky network on the tensor cores (k_sky_pixels_net);
//    where a gate trips (|sun cosine| at the camera below sky_twilight_cos,
//    the view ray within limb_rad of the limb, the camera above the shell)
//    the plain integrator;
//  * kSkyPixelsLut: the reference's own path, a bilinear tap of the sky-view
//    LUT (:1474-1525).
enum : int { kSkyPixelsPlain = 0, kSkyPixelsNet = 1, kSkyPixelsLut = 2 };
template <int kMode>
__global__ void __launch_bounds__(256, 2) k_sky_pixels(DevParams P, Frame F, ImageLayout L, CompositeScalars A,
                                                       const float4* __restrict__ svlut, float* __restrict__ out,
                                                       unsigned long long* counter) {
  int x, y;
  uint32_t samples = 0;
  if (tile_pixel(L, x, y)) {
    const f3 ray = pixel_ray(L, A, x, y).ray;
    f3 sky;
    if (kMode == kSkyPixelsLut) {
      sky = sample_sky_view(P, svlut, ray, F.sun, A.sky_alt, A.bottom);
    } else {
      sky = sky_radiance(P, F, A.cam_alt, ray);
      samples = uint32_t(P.sv_steps);
    }
    const size_t o = pix_offset(L, x, y) * L.channels;
    out[o + 0] = sky.x;
    out[o + 1] = sky.y;
    out[o + 2] = sky.z;
  }
  warp_count(samples, counter);
}
__global__ void __launch_bounds__(128 * kWorkers, 1) k_sky_pixels_net(DevParams P, Frame F, ImageLayout L, PixelTiles N,
                                                                      CompositeScalars A, SurrogateNets nets,
                                                                      uint32_t* __restrict__ status,
                                                                      float* __restrict__ out,
                                                                      unsigned long long* counter, SurrogateQueue Q) {
  extern __shared__ __align__(128) unsigned char smem[];  // the sky network
  __shared__ NetBlock B;
  bool nets_ok;
  TcTile T = net_block_begin(B, smem, nets.sky, nets.sky_bytes, nullptr, 0, P, F, A.cam_alt, nets.limb_rad, nets_ok);
  const int lane = threadIdx.x & 31;
  uint32_t samples = 0;
  for (int t = T.tile * gridDim.x + blockIdx.x; t < N.count; t += kWorkers * gridDim.x) {
    int x, y;
    const bool inside = tile_pixel_of(L, N, t, T.row, x, y);
    const int cx = inside ? x : 0, cy = inside ? y : 0;
    const f3 ray = pixel_ray(L, A, cx, cy).ray;
    const bool near_limb = near_limb_of(B, ray.y, nets.limb_rad);
    const bool net = inside && A.cam_alt <= P.top && fabsf(F.sun.y) >= nets.sky_twilight_cos && !near_limb;
    bool plain = !net, checked = false;
    uint32_t xp[8] = {};
    if (net) {
      float fx[16] = {};
      sky_start_features(B, F, ray, fx);
      fx[4] = nets.lhr_n;
      fx[5] = nets.lhm_n;
      sky_ray_features<false>(P, A.bottom, A.cam_alt, ray, F.sun, fx);
      pack_inputs(fx, kSurrogateSkyIn, xp);
    }
    const bool need = tc::tile_any(T.tile, net);
    bool tc_ok = nets_ok;
    float yv[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (need && tc_ok) tc_ok = mlp_tile_tc<kSurrogateSkyHidden>(smem, kSurrogateSkyIn, T, xp, yv, nets.wait_tries);
    f3 sky = splat(0.0f);
    if (need && !tc_ok) {
      plain = true;  // the network's outputs are not valid: the plain integrator
      if (T.row == 0) atomicOr(status, 1u);
      if (nets_ok) nets_ok = tile_recover(T);
    } else if (net) {
      sky = net_radiance(yv, A.E, splat(nets.sky_floor));
      checked = Q.net_mask != nullptr && check_pixel(x, y, Q.seed, Q.check_fraction);
    }
    if (inside) {
      if (plain) {
        sky = sky_radiance(P, F, A.cam_alt, ray);
        samples += uint32_t(P.sv_steps);
      }
      const size_t o = pix_offset(L, x, y) * L.channels;
      out[o + 0] = sky.x;
      out[o + 1] = sky.y;
      out[o + 2] = sky.z;
      if (Q.net_mask != nullptr)  // the calibration: which pixels are the network's
        Q.net_mask[storage_index(L, x, y)] = plain ? 0 : 1;
    }
    // checked network pixels to the queue (warp-aggregated)
    const unsigned qm = __ballot_sync(kAll, checked);
    if (qm) {
      const int leader = __ffs(qm) - 1;
      uint32_t base = 0;
      if (lane == leader) base = atomicAdd(Q.count, uint32_t(__popc(qm)));
      base = __shfl_sync(kAll, base, leader);
      if (checked)
        Q.items[base + __popc(qm & ((1u << lane) - 1u))] = (kQueueSkyCheck << 30) | uint32_t(cy * L.width + cx);
    }
  }
  warp_count(samples, counter);
  net_block_end(B);
}

// The sky-pixel calibration pass: every network pixel of a tile holding
// enough checked pixels is scaled by the tile's mean ratio.
__global__ void __launch_bounds__(kRunPixels * kRunRows) k_sky_pixels_calibrate(ImageLayout L, SurrogateQueue Q, float* __restrict__ out) {
  int x, y;
  if (!run_pixel(L, x, y) || Q.net_mask[storage_index(L, x, y)] == 0) return;
  const float4 t = *reinterpret_cast<const float4*>(Q.tiles + 4 * ((y >> Q.tile_shift) * Q.tiles_x + (x >> Q.tile_shift)));
  if (t.w < float(kCalibrationMinChecks)) return;
  const float inv = 1.0f / t.w;
  const size_t o = pix_offset(L, x, y) * L.channels;
  out[o + 0] *= __expf(t.x * inv);
  out[o + 1] *= __expf(t.y * inv);
  out[o + 2] *= __expf(t.z * inv);
}

// The sky-pixel calibration's checks: each queued network pixel gets the
// plain march, adds its tile's log ratio of plain to network radiance, and
// keeps the plain result.  Warps take 32 / kLanes entries per ticket.
template <int kLanes>
__device__ __forceinline__ uint32_t check_queue(const DevParams& P, const Frame& F, const ImageLayout& L,
                                                const CompositeScalars& A, const SurrogateQueue& Q,
                                                float* __restrict__ out, uint32_t n) {
  const int lane = threadIdx.x & 31;
  const bool first = (lane & (kLanes - 1)) == 0;
  uint32_t samples = 0;
  for (;;) {
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(Q.count + 1, 32u / kLanes);
    base = __shfl_sync(kAll, base, 0);
    if (base >= n) break;
    const uint32_t i = base + uint32_t(lane / kLanes);
    const bool has = i < n;
    const uint32_t p = has ? Q.items[i] & 0x3fffffffu : 0;
    const int x = int(p % uint32_t(L.width)), y = int(p / uint32_t(L.width));
    const f3 sky = sky_radiance_split<kLanes>(P, F, A.cam_alt, pixel_ray(L, A, x, y).ray, has);
    if (has && first) {
      samples += uint32_t(P.sv_steps);
      const size_t o = pix_offset(L, x, y) * L.channels;
      const f3 Ln = ld3(out + o);  // the network's radiance
      float* t = Q.tiles + 4 * ((y >> Q.tile_shift) * Q.tiles_x + (x >> Q.tile_shift));
      atomicAdd(t + 0, clampf(__logf(mx(sky.x, 1e-12f) / mx(Ln.x, 1e-12f)), -kCalibrationClamp, kCalibrationClamp));
      atomicAdd(t + 1, clampf(__logf(mx(sky.y, 1e-12f) / mx(Ln.y, 1e-12f)), -kCalibrationClamp, kCalibrationClamp));
      atomicAdd(t + 2, clampf(__logf(mx(sky.z, 1e-12f) / mx(Ln.z, 1e-12f)), -kCalibrationClamp, kCalibrationClamp));
      atomicAdd(t + 3, 1.0f);
      Q.net_mask[storage_index(L, x, y)] = 0;
      out[o + 0] = sky.x;
      out[o + 1] = sky.y;
      out[o + 2] = sky.z;
    }
  }
  return samples;
}
__global__ void __launch_bounds__(256) k_sky_pixels_check(DevParams P, Frame F, ImageLayout L, CompositeScalars A,
                                                          SurrogateQueue Q, float* __restrict__ out,
                                                          unsigned long long* counter) {
  const uint32_t n = *Q.count;
  warp_count(split_queue(n) ? check_queue<kQueueLanes>(P, F, L, A, Q, out, n) : check_queue<1>(P, F, L, A, Q, out, n),
             counter);
}

}  // namespace

cudaError_t launch_sky_pixels(int mode, const DevParams& P, const ImageLayout& L, const CompositeScalars& scalars,
                              const float4* tlut, const float4* mslut, const float4* svlut, const SurrogateNets& nets,
                              uint32_t* status, float* out, unsigned long long* counter, int sm_count, cudaStream_t s,
                              const SurrogateQueue* calibration) {
  const CompositeScalars A = with_image(scalars, L);
  const Frame F = frame_of(P, A, tlut, mslut);
  if (mode != kSkyPixelsNet) {
    const dim3 grid((L.width + 15) / 16, (L.height + 15) / 16);
    if (mode == kSkyPixelsLut)
      k_sky_pixels<kSkyPixelsLut><<<grid, 256, 0, s>>>(P, F, L, A, svlut, out, counter);
    else
      k_sky_pixels<kSkyPixelsPlain><<<grid, 256, 0, s>>>(P, F, L, A, svlut, out, counter);
    return cudaGetLastError();
  }
  SurrogateQueue Q{};
  if (calibration != nullptr && calibration->net_mask != nullptr) Q = *calibration;
  cudaError_t e = cudaFuncSetAttribute(k_sky_pixels_net, cudaFuncAttributeMaxDynamicSharedMemorySize, nets.sky_bytes);
  if (e != cudaSuccess) return e;
  if (Q.net_mask != nullptr) {
    const int tiles_y = (L.height + (1 << Q.tile_shift) - 1) >> Q.tile_shift;
    e = cudaMemsetAsync(Q.count, 0, 2 * sizeof(uint32_t), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(Q.tiles, 0, sizeof(float) * 4 * size_t(Q.tiles_x) * tiles_y, s);
    if (e != cudaSuccess) return e;
  }
  const PixelTiles N = pixel_tiles(L);
  k_sky_pixels_net<<<std::min(sm_count, N.count), 128 * kWorkers, nets.sky_bytes, s>>>(P, F, L, N, A, nets, status, out,
                                                                                     counter, Q);
  e = cudaGetLastError();
  if (e != cudaSuccess || Q.net_mask == nullptr) return e;
  k_sky_pixels_check<<<kQueueBlocks * sm_count, 256, 0, s>>>(P, F, L, A, Q, out, counter);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_sky_pixels_calibrate<<<run_grid(L), run_block(), 0, s>>>(L, Q, out);
  return cudaGetLastError();
}

cudaError_t launch_gen_samples(const SurrogateSetDev* sets, int n_sets, int kind, long long n, unsigned long long seed,
                               const SampleShaping& shaping, float* features, float* targets,
                               unsigned long long* counter, cudaStream_t s) {
  k_gen_samples<<<unsigned((n + 127) / 128), 128, 0, s>>>(sets, n_sets, kind, n, seed, shaping, features, targets,
                                                         counter);
  return cudaGetLastError();
}

namespace {
// Whether hdr shares memory with the stars or with an image of the G-buffer.
bool hdr_is_input(const ImageLayout& L, const float* hdr, const float* space, const ShadeImages& I) {
  const int64_t elements = (L.width - 1) * int64_t(L.sx) + (L.height - 1) * int64_t(L.sy) + 1;
  const auto meets = [&](const void* image, int channels) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(hdr), b = reinterpret_cast<uintptr_t>(image);
    return b != 0 && a < b + uintptr_t(elements) * channels * 4 && b < a + uintptr_t(elements) * L.channels * 4;
  };
  const void* const vectors[] = {space,         I.position,         I.normal,         I.albedo,        I.seabed_albedo,
                                 I.seabed_normal, I.terrain_position, I.terrain_normal, I.terrain_albedo};
  const void* const scalars[] = {I.water_depth, I.slope_variance, I.surface_id, I.terrain_surface_id};
  for (const void* p : vectors)
    if (meets(p, L.channels)) return true;
  for (const void* p : scalars)
    if (meets(p, 1)) return true;
  return false;
}
}  // namespace

size_t surrogate_smem_bytes(const SurrogateNets& nets) { return size_t(nets.ap_bytes) + size_t(nets.sky_bytes); }

cudaError_t launch_composite_surrogate(const DevParams& P, const ImageLayout& L, const CompositeScalars& scalars,
                                       const float* scene, const float* space, const int32_t* sid, const float* pos,
                                       const float4* tlut, const float4* mslut, const float4* svlut,
                                       const SurrogateNets& nets, const SurrogateQueue& Q, float* hdr,
                                       unsigned long long* counter, int sm_count, cudaStream_t s,
                                       const ShadeParams* shade, const ShadeImages* shade_images) {
  cudaError_t e = cudaMemsetAsync(Q.count, 0, 2 * sizeof(uint32_t), s);
  if (e != cudaSuccess) return e;
  const int tiles_y = (L.height + (1 << Q.tile_shift) - 1) >> Q.tile_shift;
  if (Q.lm != nullptr) {
    e = cudaMemsetAsync(Q.tiles, 0, sizeof(float) * 4 * size_t(Q.tiles_x) * tiles_y, s);
    if (e != cudaSuccess) return e;
  }
  const CompositeScalars A = with_image(scalars, L);
  const Frame F = frame_of(P, A, tlut, mslut);
  const int smem = int(surrogate_smem_bytes(nets));
  const PixelTiles N = pixel_tiles(L);
  const int grid = std::min(sm_count, N.count);
  const ShadeParams S = shade ? *shade : ShadeParams{};
  const ShadeImages I = shade_images ? *shade_images : ShadeImages{};
  const bool in_composite = shade && hdr_is_input(L, hdr, space, I);
  if (shade && !in_composite) {
    k_scene<<<run_grid(L), run_block(), 0, s>>>(P, F, L, A, S, I, hdr);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    scene = hdr;
  }
  const auto composite = in_composite ? k_composite_surrogate<true> : k_composite_surrogate<false>;
  e = cudaFuncSetAttribute(composite, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  composite<<<grid, 128 * kWorkers, smem, s>>>(P, F, L, N, A, scene, space, sid, pos, svlut, nets, Q, hdr, S, I);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  // the queued pixels' colours may be overwritten in hdr by then: the fused frame shades them again
  if (shade)
    k_surrogate_fallback<true><<<kQueueBlocks * sm_count, 256, 0, s>>>(P, F, L, A, scene, space, pos, Q, hdr, counter, S,
                                                                      I);
  else
    k_surrogate_fallback<false><<<kQueueBlocks * sm_count, 256, 0, s>>>(P, F, L, A, scene, space, pos, Q, hdr, counter,
                                                                       S, I);
  e = cudaGetLastError();
  if (e != cudaSuccess || Q.lm == nullptr) return e;
  k_surrogate_calibrate<<<run_grid(L), run_block(), 0, s>>>(L, Q, hdr);
  return cudaGetLastError();
}

}  // namespace atm
