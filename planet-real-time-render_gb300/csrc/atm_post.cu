// atm_post.cu - the display post-process after the atmosphere stage
// (PostProcessor, src/planet_renderer/postprocess.py:75-207) on sm_103a:
// half-resolution bloom extraction with the soft threshold and bright-pass
// cap, separable 5-tap blur passes, and the resolve (exposure, bilinear
// bloom, ACES fit, sRGB).
//
// Memory-bound work: HDR is read twice (extract, resolve) and the display
// written once; the half-resolution bloom planes (float4, W/2 x H/2) stay in
// L2 between the kernels.  A bloom plane is stored with the image's
// contiguous axis fastest, so the extract's HDR reads and writes and the
// resolve's bloom taps are coalesced in either image layout.  A blur pass (the
// reference's two kernels) streams along the slow axis in registers, two
// passes a kernel.  Edge rules are the reference's clamped indices.
//
// Arithmetic is IEEE float32 in the reference's operation order with no
// contraction (__fmul_rn / __fadd_rn): every result is the reference's
// float32 result, but for the sRGB segment, whose power is formed for the
// smallest error against 64 bits (4K frame 5.2e-8, 8.2e-8 with powf).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>
#include <utility>

#include "atm_f32.cuh"
#include "atm_kernels.h"

namespace atm {

namespace {

using f32::add;
using f32::halves;
using f32::mul;
using f32::pair;
using f32::Pair;
using f32::sub;
__device__ __forceinline__ float fmaxf_(float a, float b) { return a > b ? a : b; }
__device__ __forceinline__ float fminf_(float a, float b) { return a < b ? a : b; }
__device__ __forceinline__ float clampf_(float x, float lo, float hi) { return fminf_(fmaxf_(x, lo), hi); }

__device__ __forceinline__ float4 scale4(float4 v, float s) {
  return make_float4(mul(v.x, s), mul(v.y, s), mul(v.z, s), 0.0f);
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) {
  return make_float4(add(a.x, b.x), add(a.y, b.y), add(a.z, b.z), 0.0f);
}

// Blur weights, postprocess.py:126-129.
constexpr float kW0 = 0.38774f, kW1 = 0.24477f, kW2 = 0.06136f;

__device__ __forceinline__ float4 load_rgb(const float* __restrict__ img, const ImageLayout& L, int x, int y) {
  const float* p = img + (int64_t(x) * L.sx + int64_t(y) * L.sy) * L.channels;
  return make_float4(p[0], p[1], p[2], 0.0f);
}

// _soft_threshold, postprocess.py:88-107.
__device__ __forceinline__ float4 soft_threshold(float4 v, const PostParams& Q) {
  const float brightness = fmaxf_(v.x, fmaxf_(v.y, v.z));
  float soft = clampf_(add(sub(brightness, Q.threshold), Q.knee), 0.0f, Q.two_knee);
  soft = __fdiv_rn(mul(soft, soft), Q.knee_div);
  float contribution = fmaxf_(sub(brightness, Q.threshold), soft);
  contribution = __fdiv_rn(contribution, fmaxf_(brightness, 1.0e-6f));
  float4 r = scale4(v, contribution);
  const float peak = fmaxf_(r.x, fmaxf_(r.y, r.z));
  return scale4(r, fminf_(1.0f, __fdiv_rn(Q.clamp, fmaxf_(peak, 1.0e-6f))));
}

// Storage index of bloom texel (x, y): [y][x] when x is the fast axis, else [x][y].
__device__ __forceinline__ size_t bloom_index(const PostParams& Q, int x, int y) {
  return Q.x_fast ? size_t(y) * Q.hw + x : size_t(x) * Q.hh + y;
}

// Element of a thread of width x height, runs along the image's contiguous axis.
__device__ __forceinline__ bool post_element(const PostParams& Q, int width, int height, int& x, int& y) {
  return Q.x_fast ? run_element(width, height, x, y) : run_element(height, width, y, x);
}

// _extract, postprocess.py:110-119: one thread per half-resolution texel, in
// storage order.
__global__ void __launch_bounds__(kRunPixels * kRunRows) k_post_extract(PostParams Q, ImageLayout L, const float* __restrict__ hdr,
                                                      float scale, float4* __restrict__ bloom) {
  int x, y;
  if (!post_element(Q, Q.hw, Q.hh, x, y)) return;
  float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
  for (int ox = 0; ox < 2; ++ox)
#pragma unroll
    for (int oy = 0; oy < 2; ++oy)
      v = add4(v, load_rgb(hdr, L, min(2 * x + ox, L.width - 1), min(2 * y + oy, L.height - 1)));
  bloom[bloom_index(Q, x, y)] = soft_threshold(scale4(v, scale), Q);
}

// kStages blur passes (_blur_horizontal then _blur_vertical, :121-139) in one
// kernel.  A warp takes a strip of 64 texels of the fast axis, two a lane as
// the halves of a 64-bit register (the .f32x2 instructions: the same roundings,
// two at once), and walks a segment of the slow one: the taps along the
// slow axis are a window of five rows in registers, those along the fast one
// come from the lanes beside by shuffles.  kStages lanes at either side of the
// strip only feed the others.  Bound by issue.  Two passes over 1920x1080
// texels: 41 us when a tile and its halo lay in shared memory (five 16-byte
// reads a tap direction and texel), 38 us with one texel a lane, 21 us so.
struct BlurRow {  // a lane's two texels
  Pair c[3];
};
struct BlurLane {
  int left, right;          // source lanes of the texels before and after
  bool first, last, single;  // the lane has the axis's first texel; its last one; the last as its first half
  bool edge;                // some lane of the warp has an end of the axis
};

// The reference's order of summation: centre, -1, +1, -2, +2.
__device__ __forceinline__ BlurRow taps_slow(const BlurRow (&w)[5]) {
  BlurRow r;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    r.c[k] = add(mul(w[2].c[k], kW0), mul(w[1].c[k], kW1));
    r.c[k] = add(r.c[k], mul(w[3].c[k], kW1));
    r.c[k] = add(r.c[k], mul(w[0].c[k], kW2));
    r.c[k] = add(r.c[k], mul(w[4].c[k], kW2));
  }
  return r;
}
// Past an end of the axis its end texel stands: the lane there reads itself,
// and a last texel that is a first half stands in the second one too.
__device__ __forceinline__ BlurRow taps_fast(const BlurRow& v, const BlurLane& lane) {
  BlurRow r;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float a, b, c0, c1, a1, b1;
    halves(v.c[k], a, b);
    float l0 = __shfl_sync(0xffffffffu, a, lane.left), l1 = __shfl_sync(0xffffffffu, b, lane.left);
    float r0 = __shfl_sync(0xffffffffu, a, lane.right), r1 = __shfl_sync(0xffffffffu, b, lane.right);
    if (lane.edge) {
      l1 = lane.first ? a : l1;
      r0 = lane.last ? b : r0;
    }
    halves(mul(v.c[k], kW0), c0, c1);
    halves(mul(v.c[k], kW1), a1, b1);
    c0 = add(add(c0, mul(l1, kW1)), b1);
    c1 = add(add(c1, a1), mul(r0, kW1));
    r.c[k] = add(add(pair(c0, c1), mul(pair(l0, l1), kW2)), mul(pair(r0, r1), kW2));
    if (lane.edge) {
      halves(r.c[k], a, b);
      r.c[k] = pair(a, lane.single ? a : b);
    }
  }
  return r;
}

// One pass: next() gives its output rows one after another from `row` on,
// pulling the rows of the pass (or the plane) before it as it needs them.
// Rows past either end of the plane are the end row's again.
struct BlurPlane;
template <bool kXFast, class Source>
struct BlurPass {
  Source src;
  BlurLane lane;
  int row, last, rows;  // the next output row, the last row pulled, rows of the plane
  BlurRow w[5];         // rows row - 3 to row + 1, once started
  __device__ __forceinline__ void pull() {
    const BlurRow end = w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] = w[k + 1];
    w[4] = end;
    if (std::is_same_v<Source, BlurPlane> || last < rows - 1) {  // the plane repeats its last row itself
      const BlurRow v = src.next();
      w[4] = kXFast ? taps_fast(v, lane) : v;  // x first, along the fast axis
      ++last;
    }
  }
  __device__ __forceinline__ void start() {
    src.start();
    pull();  // the first row, which stands for rows before the plane's first
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] = w[4];
#pragma unroll 1
    while (last < min(row + 1, rows - 1)) pull();
    if (row + 1 > rows - 1) pull();
  }
  __device__ __forceinline__ BlurRow next() {
    pull();
    ++row;
    const BlurRow v = taps_slow(w);
    return kXFast ? v : taps_fast(v, lane);
  }
};
// The rows of the plane, one read ahead; after the last one, it again.
struct BlurPlane {
  const float4 *p, *q;  // of the lane's texels
  size_t pitch;
  int left;  // rows behind p
  float4 a, b;
  __device__ __forceinline__ void read() {
    a = *p;
    b = *q;
    const size_t step = left > 0 ? pitch : 0;
    --left;
    p += step;
    q += step;
  }
  __device__ __forceinline__ void start() { read(); }
  __device__ __forceinline__ BlurRow next() {
    const BlurRow v = {{pair(a.x, b.x), pair(a.y, b.y), pair(a.z, b.z)}};
    read();
    return v;
  }
};

template <int kStages>
constexpr int kBlurOut = 64 - 4 * kStages;  // texels of a strip that are written
constexpr int kBlurWarps = 4;
constexpr int kBlurSegmentWarps = 152 * 16;

template <bool kXFast, int kStages>
__global__ void __launch_bounds__(32 * kBlurWarps, 4) k_post_blur(PostParams Q, const float4* __restrict__ src,
                                                               float4* __restrict__ dst, int segment) {
  const int nf = kXFast ? Q.hw : Q.hh, ns = kXFast ? Q.hh : Q.hw;  // fast / slow extents
  const int t = threadIdx.x & 31;
  const int begin = (blockIdx.x * kBlurWarps + (threadIdx.x >> 5)) * kBlurOut<kStages>;
  if (begin >= nf) return;  // warp-uniform
  const int f = begin - 2 * kStages + 2 * t;
  const int s0 = blockIdx.y * segment, s1 = min(s0 + segment, ns);
  BlurLane lane;
  lane.first = f == 0;
  lane.single = f == nf - 1;
  lane.last = lane.single || f == nf - 2;
  lane.left = lane.first ? t : max(t - 1, 0);
  lane.right = lane.last ? t : min(t + 1, 31);
  lane.edge = begin == 0 || begin + 64 >= nf;
  // first rows of the passes and of the plane
  const int r1 = kStages == 2 ? max(s0 - 2, 0) : s0, r0 = max(r1 - 2, 0);
  const float4* row = src + size_t(r0) * nf;
  using First = BlurPass<kXFast, BlurPlane>;
  using Last = std::conditional_t<kStages == 2, BlurPass<kXFast, First>, First>;
  First first;
  first.src.p = row + min(max(f, 0), nf - 1);
  first.src.q = row + min(max(f + 1, 0), nf - 1);
  first.src.pitch = size_t(nf);
  first.src.left = ns - 1 - r0;
  first.lane = lane;
  first.row = r1;
  first.last = r0 - 1;
  first.rows = ns;
  Last pass;
  if constexpr (kStages == 2) {
    pass.src = first;
    pass.lane = lane;
    pass.row = s0;
    pass.last = r1 - 1;
    pass.rows = ns;
  } else {
    pass = first;
  }
  pass.start();
  const bool inner = t >= kStages && t < 32 - kStages;
  const bool store0 = inner && f < nf, store1 = inner && f + 1 < nf;
  float4* out = dst + size_t(s0) * nf + f;
  for (int r = s0;;) {
#pragma unroll
    for (int k = 0; k < 5; ++k) {  // five rows: the window's registers come round
      const BlurRow v = pass.next();
      float4 a, b;
      halves(v.c[0], a.x, b.x);
      halves(v.c[1], a.y, b.y);
      halves(v.c[2], a.z, b.z);
      a.w = b.w = 0.0f;
      if (store0) out[0] = a;
      if (store1) out[1] = b;
      out += nf;
      if (++r == s1) return;
    }
  }
}

// Storage [x][y] -> [y][x] (the bloom plane's read-back).
__global__ void __launch_bounds__(256) k_post_transpose(const float4* __restrict__ src, float4* __restrict__ dst,
                                                        int hw, int hh) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= hw * hh) return;
  const int x = i % hw, y = i / hw;
  dst[i] = src[size_t(x) * hh + y];
}

// a / b for positive normal b: the hardware reciprocal's quotient and one
// residual correction of it (Markstein): the IEEE quotient's bits for the ACES
// fit of every float from 1e-9 to 1e6 (of 1.3e9 from 1e-30 to 1e18 two differ)
// and for every (i + 1/2) / n, n <= 16384, compared on the device.
__device__ __forceinline__ float quotient(float a, float b) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
  const float q = a * r;
  return fmaf(fmaf(-q, b, a), r, q);
}
// m^(1/2.4) 1.055 / 1.055f for m in (0.0031, 1], so that 1.055f times it is the
// sRGB segment's 1.055 m^(1/2.4): 2^(log2(m) 5/12) by the hardware functions,
// rounded to 12 bits so that its square is exact, and one Halley-order step of
// p^12 = m^5.  With x = m^5 / p^12 - 1, below 2.93e-3, (1 + x)^(1/12) = 1 + x/12
// - 11 x^2/288 + ...; the next term is below 2^-30.6.  x is formed from the
// difference m^5 - p^12 with the rounding error of p^4 taken out, which counts
// three times in p^12; the others are divided by 12.
__device__ __forceinline__ float srgb_power(float m) {
  float l, p, r;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(m));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(p) : "f"(l * 0.41666666666666667f));
  p = __uint_as_float((__float_as_uint(p) + 0x800u) & 0xfffff000u);
  const float p2 = p * p, p4 = p2 * p2, p8 = p4 * p4, p12 = p8 * p4, m2 = m * m;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(p12));
  const float x = fmaf(p8 * -3.0f, fmaf(p2, p2, -p4), fmaf(m2 * m2, m, -p12)) * r;
  return fmaf(p, fmaf(x, fmaf(x, -0.038194444444444444f, 0.083333333333333333f), 4.971796e-8f), p);
}

// _sample_bloom, postprocess.py:141-153, an axis at a time: pixel i of n
// between two of the plane's m texels.
struct BloomAxis {
  int lo, hi;
  float f, g;  // weights of hi and lo
};
__device__ __forceinline__ BloomAxis bloom_axis(int i, int n, int m) {
  const float p = sub(mul(quotient(add(float(i), 0.5f), float(n)), float(m)), 0.5f);
  const float fp = floorf(p);
  BloomAxis a;
  a.lo = min(max(int(fp), 0), m - 1);
  a.hi = min(a.lo + 1, m - 1);
  a.f = sub(p, fp);  // in 0..1
  a.g = sub(1.0f, a.f);
  return a;
}
template <bool kXFast>
__device__ __forceinline__ float4 sample_bloom(const float4* __restrict__ bloom, int pitch, const BloomAxis& fast,
                                               const BloomAxis& slow) {
  const float4* lo = bloom + size_t(slow.lo) * pitch;
  const float4* hi = bloom + size_t(slow.hi) * pitch;
  const float4 v00 = lo[fast.lo], v01 = lo[fast.hi], v10 = hi[fast.lo], v11 = hi[fast.hi];
  if (kXFast)  // x, then y
    return add4(scale4(add4(scale4(v00, fast.g), scale4(v01, fast.f)), slow.g),
                scale4(add4(scale4(v10, fast.g), scale4(v11, fast.f)), slow.f));
  return add4(scale4(add4(scale4(v00, slow.g), scale4(v10, slow.f)), fast.g),
              scale4(add4(scale4(v01, slow.g), scale4(v11, slow.f)), fast.f));
}

// _display_from_exposed, postprocess.py:56-73: ACES fit, sRGB encoding.
__device__ __forceinline__ float display_channel(float v) {
  v = fmaxf_(v, 0.0f);
  const float num = mul(v, add(mul(2.51f, v), 0.03f));
  const float den = add(mul(v, add(mul(2.43f, v), 0.59f)), 0.14f);
  // past 1e18 the terms near the end of float's range: the IEEE quotient, inf / inf included
  const float mapped = clampf_(v < 1.0e18f ? quotient(num, den) : __fdiv_rn(num, den), 0.0f, 1.0f);
  if (mapped <= 0.0031308f) return mul(mapped, 12.92f);
  return sub(mul(1.055f, srgb_power(mapped)), 0.055f);
}

// _resolve, postprocess.py:155-174: runs along the image's contiguous axis
// (kXFast: x), kRows pixels a thread across it (kResolveRows, in small frames
// 1), which share their place on the fast axis.  The ACES quotients, the power
// and the bloom taps are what it executes; 4K with bloom and tone map took 116
// us with powf, IEEE quotients and a flat 64-bit pixel index, 75 us with a
// pixel a thread, 60 us so and 1.5 more for the nearer power.
constexpr int kResolveRows = 8;
template <bool kXFast, bool kBloom, int kRows>
__global__ void __launch_bounds__(kRunPixels * kRunRows) k_post_resolve(PostParams Q, ImageLayout L, const float* __restrict__ hdr,
                                                      float* __restrict__ display, const float4* __restrict__ bloom,
                                                      float exposure, float strength, int tone_map) {
  const int nf = kXFast ? L.width : L.height, ns = kXFast ? L.height : L.width;
  const int bf = kXFast ? Q.hw : Q.hh, bs = kXFast ? Q.hh : Q.hw;
  int f, group;
  if (!run_element(nf, 0x7fffffff, f, group)) return;
  // the block's rows lie together: thread row t takes t, t + kRunRows, ...
  const unsigned s0 = (unsigned(group) - threadIdx.y) * kRows + threadIdx.y;
  const BloomAxis fast = kBloom ? bloom_axis(f, nf, bf) : BloomAxis();
  const int64_t at = (kXFast ? f * L.sx + int64_t(s0) * L.sy : int64_t(s0) * L.sx + f * L.sy) * L.channels;
  const int64_t step = (kXFast ? L.sy : L.sx) * kRunRows * L.channels;
  const float* in = hdr + at;
  float* out = display + at;
#pragma unroll
  for (int k = 0; k < kRows; ++k) {
    const unsigned sl = s0 + k * kRunRows;
    if (sl >= unsigned(ns)) return;
    float4 v = scale4(make_float4(in[0], in[1], in[2], 0.0f), exposure);
    if (kBloom) v = add4(v, scale4(sample_bloom<kXFast>(bloom, bf, fast, bloom_axis(int(sl), ns, bs)), strength));
    if (tone_map) {
      out[0] = display_channel(v.x);
      out[1] = display_channel(v.y);
      out[2] = display_channel(v.z);
    } else {
      out[0] = clampf_(v.x, 0.0f, 1.0f);
      out[1] = clampf_(v.y, 0.0f, 1.0f);
      out[2] = clampf_(v.z, 0.0f, 1.0f);
    }
    in += step;
    out += step;
  }
}

// centre, -1, +1, -2, +2 in the reference's order of summation
__device__ __forceinline__ float4 taps5(float4 c, float4 m1, float4 p1, float4 m2, float4 p2) {
  float4 r = scale4(c, kW0);
  r = add4(r, scale4(m1, kW1));
  r = add4(r, scale4(p1, kW1));
  r = add4(r, scale4(m2, kW2));
  return add4(r, scale4(p2, kW2));
}
// One blur pass of a small plane: a tile of kTileS slow rows by kTileF fast
// texels a block, its neighbourhood loaded once (clamped, which is the edge
// rule) and both directions' taps taken from shared memory.  A small plane's
// blur is latency: one load here, a dozen rows one after another in a
// streaming warp.
constexpr int kTileF = 32, kTileS = 8, kHalo = 2;
constexpr int kInF = kTileF + 2 * kHalo, kInS = kTileS + 2 * kHalo;
template <bool kXFast>
__global__ void __launch_bounds__(kTileF * kTileS) k_post_blur_tile(PostParams Q, const float4* __restrict__ src,
                                                                    float4* __restrict__ dst) {
  __shared__ float4 s_in[kInS][kInF];
  __shared__ float4 s_mid[kInS][kInF];  // after the x taps
  const int t = threadIdx.x;
  const int nf = kXFast ? Q.hw : Q.hh, ns = kXFast ? Q.hh : Q.hw;  // fast / slow extents
  const int f0 = blockIdx.x * kTileF, s0 = blockIdx.y * kTileS;
  for (int k = t; k < kInS * kInF; k += kTileF * kTileS) {
    const int r = k / kInF, c = k % kInF;
    s_in[r][c] = src[size_t(min(max(s0 - kHalo + r, 0), ns - 1)) * nf + min(max(f0 - kHalo + c, 0), nf - 1)];
  }
  __syncthreads();
  if (kXFast) {  // x along the fast axis, on every slow row
    for (int k = t; k < kInS * kTileF; k += kTileF * kTileS) {
      const int r = k / kTileF, c = k % kTileF + kHalo;
      s_mid[r][c] = taps5(s_in[r][c], s_in[r][c - 1], s_in[r][c + 1], s_in[r][c - 2], s_in[r][c + 2]);
    }
  } else {  // x along the slow axis, on every fast column
    for (int k = t; k < kTileS * kInF; k += kTileF * kTileS) {
      const int r = k / kInF + kHalo, c = k % kInF;
      s_mid[r][c] = taps5(s_in[r][c], s_in[r - 1][c], s_in[r + 1][c], s_in[r - 2][c], s_in[r + 2][c]);
    }
  }
  __syncthreads();
  const int c = t % kTileF + kHalo, r = t / kTileF + kHalo;
  const int f = f0 + c - kHalo, sl = s0 + r - kHalo;
  if (f < nf && sl < ns)
    dst[size_t(sl) * nf + f] =
        kXFast ? taps5(s_mid[r][c], s_mid[r - 1][c], s_mid[r + 1][c], s_mid[r - 2][c], s_mid[r + 2][c])
               : taps5(s_mid[r][c], s_mid[r][c - 1], s_mid[r][c + 1], s_mid[r][c - 2], s_mid[r][c + 2]);
}

// Rows of a blur warp's segment: it first walks 2 kStages rows before and
// after its own, so segments are long, unless the plane is too small to give
// every scheduler of the chip four warps that way (two: 8 us more at 1920x1080).
template <bool kXFast, int kStages>
void blur(const PostParams& Q, const float4* src, float4* dst, cudaStream_t s) {
  const int nf = kXFast ? Q.hw : Q.hh, ns = kXFast ? Q.hh : Q.hw;
  const int strips = (nf - 1) / kBlurOut<kStages> + 1;
  const int wanted = (kBlurSegmentWarps + strips - 1) / strips;  // segments
  const int segment = std::max(std::min(std::max((ns + wanted - 1) / wanted, 8), 64), ns / 65535 + 1);
  const dim3 grid((strips + kBlurWarps - 1) / kBlurWarps, (ns + segment - 1) / segment);
  k_post_blur<kXFast, kStages><<<grid, 32 * kBlurWarps, 0, s>>>(Q, src, dst, segment);
}

template <bool kXFast>
void blur_tiles(const PostParams& Q, const float4* src, float4* dst, cudaStream_t s) {
  const int nf = kXFast ? Q.hw : Q.hh, ns = kXFast ? Q.hh : Q.hw;
  k_post_blur_tile<kXFast><<<dim3((nf - 1) / kTileF + 1, (ns - 1) / kTileS + 1), kTileF * kTileS, 0, s>>>(Q, src, dst);
}
// Planes up to this take the blur by tiles and the resolve a pixel a thread:
// their launches wait for a warp's chain of rows, not for the chip.  Frames of
// 96x54, 640x360 and 960x540 with four passes: 10.9, 14.4 and 19.2 us so, 19.9,
// 22.7 and 23.9 us streaming; 1366x767 27.1 and 28.7, but with its HDR image
// just written the two launches fewer weigh more (a whole frame of that size
// 552 us streaming, 556 so); 1920x1080 45.3 and 41.5.
constexpr long long kSmallPlane = 3LL << 16;

}  // namespace

bool image_x_fast(const ImageLayout& L) {
  const int64_t ax = L.sx < 0 ? -L.sx : L.sx, ay = L.sy < 0 ? -L.sy : L.sy;
  return ax < ay;
}

cudaError_t launch_post(const PostParams& Q, const ImageLayout& L, const float* hdr, float* display, float4* bloom_a,
                        float4* bloom_b, float exposure, float strength, int passes, bool use_bloom, bool tone_map,
                        const float4** bloom_out, cudaStream_t s) {
  const float4* bloom = bloom_a;
  const bool small = (long long)Q.hw * Q.hh <= kSmallPlane;
  if (use_bloom) {
    const int nf = Q.x_fast ? Q.hw : Q.hh, ns = Q.x_fast ? Q.hh : Q.hw;
    k_post_extract<<<run_grid(nf, ns), run_block(), 0, s>>>(Q, L, hdr, 0.25f * exposure, bloom_a);  // exact: a power of two
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    float4* src = bloom_a;
    float4* dst = bloom_b;
    for (int p = 0; p < passes; p += small ? 1 : 2) {
      const bool two = p + 1 < passes;
      if (small)
        Q.x_fast ? blur_tiles<true>(Q, src, dst, s) : blur_tiles<false>(Q, src, dst, s);
      else if (Q.x_fast)
        two ? blur<true, 2>(Q, src, dst, s) : blur<true, 1>(Q, src, dst, s);
      else
        two ? blur<false, 2>(Q, src, dst, s) : blur<false, 1>(Q, src, dst, s);
      e = cudaGetLastError();
      if (e != cudaSuccess) return e;
      std::swap(src, dst);
    }
    bloom = src;
  }
  if (bloom_out != nullptr) *bloom_out = bloom;
  const auto resolve = [&](auto x_fast, auto with_bloom) {
    constexpr bool kXFast = decltype(x_fast)::value, kBloom = decltype(with_bloom)::value;
    const int nf = kXFast ? L.width : L.height, ns = kXFast ? L.height : L.width;
    const auto go = [&](auto kernel, int rows) {
      kernel<<<run_grid(nf, (ns - 1) / rows + 1), run_block(), 0, s>>>(Q, L, hdr, display, bloom, exposure, strength,
                                                                      tone_map ? 1 : 0);
    };
    small ? go(k_post_resolve<kXFast, kBloom, 1>, 1)
          : go(k_post_resolve<kXFast, kBloom, kResolveRows>, kResolveRows);
  };
  if (Q.x_fast)
    use_bloom ? resolve(std::true_type(), std::true_type()) : resolve(std::true_type(), std::false_type());
  else
    use_bloom ? resolve(std::false_type(), std::true_type()) : resolve(std::false_type(), std::false_type());
  return cudaGetLastError();
}

cudaError_t launch_post_read_bloom(const PostParams& Q, const float4* bloom, float4* dst, cudaStream_t s) {
  const size_t n = size_t(Q.hw) * Q.hh;
  if (Q.x_fast) return cudaMemcpyAsync(dst, bloom, n * sizeof(float4), cudaMemcpyDeviceToDevice, s);
  k_post_transpose<<<unsigned((n + 255) / 256), 256, 0, s>>>(bloom, dst, Q.hw, Q.hh);
  return cudaGetLastError();
}

}  // namespace atm
