// atm_batch.cu - many sky-view and aerial-perspective LUTs in one persistent
// launch (time snapshots x cameras x parameter sets, uneven LUT sizes).
//
// The reference builds one LUT per kernel launch (atmosphere/renderer.py
// :1208, :1304).  Here a job table describes every LUT of a batch; each job is
// split into work items of `per_item` texels (sky-view) or froxel columns
// (aerial).  A grid of blocks_per_sm x SM-count blocks stays resident; each
// warp takes the next work item from an atomic ticket, finds its job by
// binary search over the item prefix sums, copies the job's parameters into
// its shared-memory slot and evaluates the texels or columns, one a lane or,
// in batches of few columns, a column by several.
// Warps never wait on each other (the ticket is a plain atomicAdd), so uneven
// job sizes balance without barriers.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "atm_capi.h"
#include "atm_device.cuh"
#include "atm_kernels.h"
#include "atm_lut_warp.cuh"

namespace atm {

struct BatchJobDev {
  DevParams P;   // the job's parameter set with its own LUT size
  Frame F;       // with the job's sun
  AerialView V;  // sky-view jobs: the camera altitude alone
  float4* out;
  int kind;      // ATM_LUT_SKY_VIEW or ATM_LUT_AERIAL
  int units;     // texels (sky-view) or columns (aerial)
  int per_item;  // units per work item
  int lanes;     // of a warp that share a unit: 1, for columns also 8 or 32
};

namespace {

constexpr int kBatchWarps = 8;  // 256-thread blocks

// The froxel columns [u0, u1) of a job by a warp, kLanes lanes a column.
template <int kLanes>
__device__ __forceinline__ uint32_t aerial_columns(const BatchJobDev& J, int u0, int u1, TableFraction fraction) {
  const int sub = (threadIdx.x & 31) / kLanes;
  uint32_t samples = 0;
  for (int base = u0; base < u1; base += 32 / kLanes) {
    const int c = min(base + sub, u1 - 1);  // every lane takes part in the group's shuffles
    samples += aerial_column_group<kLanes>(J.P, J.F, J.V, c % J.P.ap_w, c / J.P.ap_w, base + sub < u1, fraction, J.out);
  }
  return samples;
}

// kGroups: the jobs' columns are shared by groups of lanes.  A kernel of its
// own: with all forms in one, a batch of 512 LUTs takes 2.18 ms instead of 2.14.
template <bool kGroups>
__global__ void __launch_bounds__(256, 3) k_batch(const BatchJobDev* __restrict__ jobs,
                                               const long long* __restrict__ prefix, int n_jobs, long long n_items,
                                               unsigned long long* __restrict__ ticket,
                                               unsigned long long* __restrict__ samples_counter) {
  __shared__ BatchJobDev s_job[kBatchWarps];
  __shared__ float s_sky[kBatchWarps][kMaxSkySteps + 1];
  __shared__ float s_aerial[kBatchWarps][kMaxAerialSteps + 1];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  uint32_t samples = 0;
  int loaded = -1;
  for (;;) {
    unsigned long long item = 0;
    if (lane == 0) item = atomicAdd(ticket, 1ull);
    item = __shfl_sync(kFull, item, 0);
    if (item >= static_cast<unsigned long long>(n_items)) break;
    // job j: prefix[j] <= item < prefix[j + 1]
    int lo = 0, hi = n_jobs;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (prefix[mid] <= static_cast<long long>(item)) lo = mid;
      else hi = mid;
    }
    const BatchJobDev& J = s_job[warp];
    if (lo != loaded) {  // stage the job in this warp's slot
      __syncwarp();
      const int* src = reinterpret_cast<const int*>(jobs + lo);
      int* dst = reinterpret_cast<int*>(&s_job[warp]);
      for (int k = lane; k < int(sizeof(BatchJobDev) / sizeof(int)); k += 32) dst[k] = src[k];
      __syncwarp();
      if (J.kind == ATM_LUT_SKY_VIEW)
        fill_fractions(s_sky[warp], J.P.sv_steps, lane, 32);
      else
        fill_fractions(s_aerial[warp], J.P.ap_steps, lane, 32);
      __syncwarp();
      loaded = lo;
    }
    const long long local = static_cast<long long>(item) - prefix[lo];
    const int u0 = static_cast<int>(local * J.per_item);
    const int u1 = min(u0 + J.per_item, J.units);
    if (J.kind == ATM_LUT_SKY_VIEW) {
      for (int u = u0 + lane; u < u1; u += 32)
        samples += sky_view_texel<1>(J.P, J.F, J.V.cam_alt, u % J.P.sv_w, u / J.P.sv_w, true, {s_sky[warp]}, J.out);
    } else if (kGroups) {
      samples += J.lanes == 32 ? aerial_columns<32>(J, u0, u1, {s_aerial[warp]})
                               : aerial_columns<8>(J, u0, u1, {s_aerial[warp]});
    } else {
      for (int u = u0 + lane; u < u1; u += 32)
        samples += aerial_column_lane(J.P, J.F, J.V, u % J.P.ap_w, u / J.P.ap_w, {s_aerial[warp]}, J.out);
    }
  }
  warp_count(samples, samples_counter);
}

}  // namespace

// A column is a chain of all its slices, which a batch of few columns waits
// for: lanes share it while the batch's columns are at most a quarter of the
// launch's threads, and a warp takes as many as it holds at a time, whatever
// the tuning's items.  One 16^3, 32^3 or 64^3 volume: 24, 22 and 45 us, 47, 70
// and 118 with a lane a column; 16,384 columns of the three: 43, 57 and 100,
// 52, 76 and 134; 32,768: 66, 90 and 172, 56, 86 and 157.  A volume of fewer
// than 32 slices leaves a whole warp's lanes idle (64 x 16^3: 52 us, 43 on 8
// lanes), a deeper one has work for them (16 x 32^3: 62 us on 8 or 16).
bool batch_groups(long long columns, int sm_count, int blocks_per_sm) {
  return 4 * columns <= 256LL * sm_count * std::min(blocks_per_sm, 3);
}
int batch_column_lanes(bool groups, int depth) { return !groups ? 1 : depth < 32 ? 8 : 32; }

cudaError_t launch_batch(const BatchJobDev* jobs, const long long* prefix, int n_jobs, long long n_items,
                         unsigned long long* ticket, unsigned long long* samples, int blocks, bool groups,
                         cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(ticket, 0, sizeof(unsigned long long), s);
  if (e != cudaSuccess) return e;
  (groups ? k_batch<true> : k_batch<false>)<<<blocks, 256, 0, s>>>(jobs, prefix, n_jobs, n_items, ticket, samples);
  return cudaGetLastError();
}

size_t batch_job_size() { return sizeof(BatchJobDev); }

// Fill one device job descriptor from the ABI job (host side).
void fill_batch_job(BatchJobDev& d, const DevParams& set_params, const AtmBatchJob& j, float4* arena,
                    const float4* tlut, const float4* mslut, double radius, const double E[3], double ar_rad,
                    int per_item, int lanes) {
  std::memset(&d, 0, sizeof(d));
  d.P = set_params;
  d.kind = j.kind;
  d.out = arena + j.output_offset;
  d.per_item = per_item;
  d.lanes = lanes;
  d.units = j.width * j.height;
  f3 sun;
  if (j.kind == ATM_LUT_SKY_VIEW) {
    d.P.sv_w = j.width;
    d.P.sv_h = j.height;
    sun = sky_view_sun(float(j.sun_zenith_cosine));
    d.V.cam_alt = float(j.camera_altitude_m);
  } else {
    d.P.ap_w = j.width;
    d.P.ap_h = j.height;
    d.P.ap_d = j.depth;
    sun = {float(j.sun_local[0]), float(j.sun_local[1]), float(j.sun_local[2])};
    float b[9];
    for (int k = 0; k < 9; ++k) b[k] = float(j.view_basis[k]);
    d.V = aerial_view(float(j.frame_width) / float(j.frame_height), float(j.camera_altitude_m), b, b + 3, b + 6,
                      float(j.tangent_half_fov));
  }
  d.F = make_frame(set_params, tlut, mslut, float(radius), float(ar_rad), sun, {float(E[0]), float(E[1]), float(E[2])});
}

}  // namespace atm
