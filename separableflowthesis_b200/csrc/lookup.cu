// Lookup on the two aggregated 3D cost volumes (the reference's CorrBlock1D, core/corr.py:513-624): a pyramid of
// each volume over its displacement axis (average pooling by 2, core/corr.py:543-548) and, per refinement
// iteration, 2r+1 linearly interpolated samples per pyramid level around the current displacement estimate of every
// image-1 pixel (core/corr.py:576-594, F.grid_sample with align_corners=True and zero padding, one row high).
//
// HBM-bound gathers.  The volumes stay in the layout the rest of the path produces, (B, dim, D, H1, W1): the
// displacement axis of one pixel is strided by the plane size, a warp handles 32 neighbouring pixels, and because
// neighbouring pixels have similar displacements their gathers mostly fall into the same 128-byte lines.  (The
// reference first permutes to (B*H1*W1, dim, 1, D), core/corr.py:531-541.)  Every warp takes one pyramid level of its
// pixels, so that a pixel's levels are gathered side by side and not one after the other.
// Backward: every (b, channel, displacement, pixel) element of a level's gradient is touched by one thread only,
// so the scatter needs no atomics; the levels are then folded into the gradient of the volume in one pass.  A model looks up a dozen
// times on the same two volumes and wants the sum of their gradients: the lookups of a pair of volumes add their windows to one
// accumulator per level (lookup_accumulate_kernel), which is folded once (lookup_gradient_fold_kernel).
#include "kernels.h"
#include "sm100_primitives.cuh"

namespace sfb {

constexpr int LK_THREADS = 128;

template <int VEC> struct LkVec;
template <> struct LkVec<1> { typedef float type; };
template <> struct LkVec<4> { typedef float4 type; };
__device__ __forceinline__ float lk_mean(float a, float b) { return 0.5f * (a + b); }
__device__ __forceinline__ float4 lk_mean(const float4& a, const float4& b) {
  return make_float4(lk_mean(a.x, b.x), lk_mean(a.y, b.y), lk_mean(a.z, b.z), lk_mean(a.w, b.w));
}
__device__ __forceinline__ void lk_fma(float& acc, float w, float v) { acc = fmaf(w, v, acc); }
__device__ __forceinline__ void lk_fma(float4& acc, float w, const float4& v) {
  lk_fma(acc.x, w, v.x); lk_fma(acc.y, w, v.y); lk_fma(acc.z, w, v.z); lk_fma(acc.w, w, v.w);
}

struct LookupLevelsMut {
  float* ptr[LOOKUP_MAX_LEVELS];         // level l: (B, dim, D_l, N1)
  int D[LOOKUP_MAX_LEVELS];
};

// Up to three pyramid levels from the one below them, of one or two volumes, in one launch: entry d of a level is the mean of entries
// 2d and 2d + 1 of the level before.  A thread reads LK_PROWS rows of level `base` and writes the rows of the next levels that they
// make up, VEC neighbouring pixels at a time.  HBM-bound: with a launch per level and volume and 4-byte accesses, 8 x 47 x 156 (both
// volumes, four levels) took 53 us; 15 now.
// grid (ceil(N1 / (LK_THREADS * VEC)), volumes * ceil(largest D / LK_PROWS), planes)
constexpr int LK_PROWS = 8;
struct LookupPyramids { LookupLevelsMut v[2]; };
template <int VEC>
__global__ void __launch_bounds__(LK_THREADS)
lookup_pyramid_kernel(const __grid_constant__ LookupPyramids vols, int base, int levels, int row_blocks, int N1) {
  follow_previous_kernel();
  typedef typename LkVec<VEC>::type V;
  const int p = (blockIdx.x * LK_THREADS + threadIdx.x) * VEC;
  const int vol = blockIdx.y / row_blocks, r0 = (blockIdx.y - vol * row_blocks) * LK_PROWS;
  const LookupLevelsMut& lv = vols.v[vol];
  if (p >= N1 || r0 >= lv.D[base]) return;
  V row[LK_PROWS];
  const float* src = lv.ptr[base] + ((size_t)blockIdx.z * lv.D[base] + r0) * N1 + p;
#pragma unroll
  for (int r = 0; r < LK_PROWS; ++r)
    row[r] = __ldg(reinterpret_cast<const V*>(src + (size_t)min(r, lv.D[base] - 1 - r0) * N1));   // rows past the end are not used
#pragma unroll
  for (int s = 1; s <= 3; ++s) {
    const int l = base + s, n = LK_PROWS >> s;
    if (l >= levels) return;
    float* dst = lv.ptr[l] + ((size_t)blockIdx.z * lv.D[l] + (r0 >> s)) * N1 + p;
#pragma unroll
    for (int r = 0; r < n; ++r) {
      row[r] = lk_mean(row[2 * r], row[2 * r + 1]);
      if ((r0 >> s) + r < lv.D[l]) *reinterpret_cast<V*>(dst + (size_t)r * N1) = row[r];
    }
  }
}

// Sampling position of tap t at level l, exactly as the reference computes it: displacement estimate / 2^l + offset
// (core/corr.py:581-582), optionally clamped to [-1, 1] (core/corr.py:586, the first volume only), then through
// grid_sample's normalisation and back (core/corr.py:553, align_corners=True).
__device__ __forceinline__ float lookup_position(float c, int level, int t, int radius, int clamp_unit, int Dl) {
  float x = (float)(t - radius) + c * (1.f / (float)(1 << level));   // a power of two: the same value as the quotient
  if (clamp_unit) x = fminf(fmaxf(x, -1.f), 1.f);
  const float xn = 2.f * x / (float)(Dl - 1) - 1.f;
  return (xn + 1.f) * 0.5f * (float)(Dl - 1);
}

// One of the (up to two) volumes of a lookup: its levels and displacement component, the output, the reference's clamp.
struct LookupVolume {
  const float* ptr[LOOKUP_MAX_LEVELS];   // level l: (B, dim, D_l, N1)
  int D[LOOKUP_MAX_LEVELS];
  const float* coord;                    // (B, N1), coord_sb elements between samples
  long long coord_sb;
  float* out;
  int clamp_unit;
};
struct LookupVolumes { LookupVolume v[2]; };

// out (B, levels*dim*(2r+1), N1): channel (l*dim + ch)*(2r+1) + t.  A warp takes one level of 32 pixels at a time; a block has
// LK_WARPS warps, min(levels, LK_WARPS) of them for the same pixels (with warps left without a level, one level of
// 4 x 135 x 240 took 24.5 us, 19.2 with one warp for all levels, 16.2 now).
// TAPS = 2r+1 when known at compile time (all loads of a thread in flight together), else 0.  Five blocks per SM: with the
// 140 registers the compiler takes otherwise, three, four levels of 4 x 135 x 240 take 36 us instead of 29.
// The two volumes of a model are looked up in one launch: at 4 x 55 x 128 two launches of 6.8 us each, 9.2 now; at 8 x 47 x 156 10 each, 16.3.
// grid (ceil(N1 / (32 * groups)), B, volumes), block (32, min(levels, LK_WARPS), groups of pixels)
constexpr int LK_WARPS = 4;
template <int TAPS>
__global__ void __launch_bounds__(32 * LK_WARPS, TAPS > 0 ? 5 : 0)
lookup_forward_kernel(const __grid_constant__ LookupVolumes vols, int dim, int N1, int levels, int radius) {
  follow_previous_kernel();
  const int p = (blockIdx.x * blockDim.z + threadIdx.z) * 32 + threadIdx.x, b = blockIdx.y;
  if (p >= N1) return;
  const LookupVolume& lv = vols.v[blockIdx.z];
  const int clamp_unit = lv.clamp_unit;
  const float c = __ldg(lv.coord + (size_t)b * lv.coord_sb + p);
  const int taps = TAPS > 0 ? TAPS : 2 * radius + 1;
  float* o = lv.out + (size_t)b * levels * dim * taps * N1 + p;
  for (int l = threadIdx.y; l < levels; l += blockDim.y) {
    const int Dl = lv.D[l];
    for (int ch = 0; ch < dim; ++ch) {
      const float* v = lv.ptr[l] + ((size_t)(b * dim + ch) * Dl) * N1 + p;
      float* ol = o + (size_t)(l * dim + ch) * taps * N1;
      auto tap = [&](int t) {
        const float ix = lookup_position(c, l, t, radius, clamp_unit, Dl);
        const float fl = floorf(ix);
        const float w1 = ix - fl, w0 = 1.f - w1;
        // a position far outside the volume (or NaN) samples zeros; clamp before the conversion to int
        const int i0 = (int)fminf(fmaxf(fl, -2.f), (float)Dl), i1 = i0 + 1;
        const bool in0 = i0 >= 0 && i0 < Dl && fl == (float)i0, in1 = i1 >= 0 && i1 < Dl && fl == (float)i0;
        float r = 0.f;
        if (in0) r = w0 * __ldg(v + (size_t)i0 * N1);
        if (in1) r = fmaf(w1, __ldg(v + (size_t)i1 * N1), r);
        return r;
      };
      if constexpr (TAPS > 0) {
        float r[TAPS];
#pragma unroll
        for (int t = 0; t < TAPS; ++t) r[t] = tap(t);
#pragma unroll
        for (int t = 0; t < TAPS; ++t) ol[(size_t)t * N1] = r[t];
      } else {
        for (int t = 0; t < taps; ++t) ol[(size_t)t * N1] = tap(t);
      }
    }
  }
}

// Scatter of the output gradients into the (zero-initialised) gradients of the levels.  Same grid.
__global__ void lookup_backward_kernel(const LookupLevelsMut gl, const float* __restrict__ coord, long long coord_sb,
                                       const float* __restrict__ gout, int dim, int N1, int levels, int radius,
                                       int clamp_unit) {
  follow_previous_kernel();
  const int p = blockIdx.x * LK_THREADS + threadIdx.x, b = blockIdx.y;
  if (p >= N1) return;
  const float c = __ldg(coord + (size_t)b * coord_sb + p);
  const int taps = 2 * radius + 1;
  const float* go = gout + (size_t)b * levels * dim * taps * N1 + p;
  for (int l = 0; l < levels; ++l) {
    const int Dl = gl.D[l];
    for (int t = 0; t < taps; ++t) {
      const float ix = lookup_position(c, l, t, radius, clamp_unit, Dl);
      const float fl = floorf(ix);
      const float w1 = ix - fl, w0 = 1.f - w1;
      const int i0 = (int)fminf(fmaxf(fl, -2.f), (float)Dl), i1 = i0 + 1;
      const bool in0 = i0 >= 0 && i0 < Dl && fl == (float)i0, in1 = i1 >= 0 && i1 < Dl && fl == (float)i0;
      for (int ch = 0; ch < dim; ++ch) {
        const float g = __ldg(go + (size_t)((l * dim + ch) * taps + t) * N1);
        float* v = gl.ptr[l] + ((size_t)(b * dim + ch) * Dl) * N1 + p;
        // this thread is the only writer of its pixel's column, and its taps run in program order
        if (in0) v[(size_t)i0 * N1] += w0 * g;
        if (in1) v[(size_t)i1 * N1] += w1 * g;
      }
    }
  }
}

// gcorr[plane][i][p] += sum_{l >= 1} glevel_l[plane][i >> l][p] / 2^l  (the pooling of level l spreads its gradient
// evenly over the 2^l entries it averaged; entries dropped by the floor of an odd size get none).
// grid (ceil(N1/128), D, planes)
__global__ void lookup_fold_kernel(const LookupLevelsMut gl, int N1, int levels) {
  follow_previous_kernel();
  const int p = blockIdx.x * LK_THREADS + threadIdx.x, i = blockIdx.y;
  if (p >= N1) return;
  float acc = 0.f, scale = 1.f;
  int parent_ok = 1;
  for (int l = 1; l < levels; ++l) {
    scale *= 0.5f;
    const int j = i >> l;
    // entry i is inside level l's pooling window only if it was inside every finer level's
    parent_ok = parent_ok && (i >> (l - 1)) < 2 * gl.D[l] && j < gl.D[l];
    if (!parent_ok) break;
    acc = fmaf(scale, gl.ptr[l][((size_t)blockIdx.z * gl.D[l] + j) * N1 + p], acc);
  }
  float* dst = gl.ptr[0] + ((size_t)blockIdx.z * gl.D[0] + i) * N1 + p;
  *dst += acc;
}

// Backward in one pass for radius <= LK_RMAX: per level, the taps of a pixel touch a window of at most 2r+3
// consecutive rows, which one thread accumulates in shared memory (its own column); after a barrier the block's warps
// write the whole displacement columns of its 32 pixels once, eight consecutive rows at a time, folding the levels in as
// they go (a level-l entry spreads evenly over the 2^l level-0 entries it averaged).  No memset, no read-modify-write, no
// pyramid scratch.  What bounds it is the write of the volume gradient, so the column is spread over the block's warps: with
// one thread per pixel doing levels and rows in turn, 58 656 pixels (8 x 47 x 156) were too few threads to cover it.
// grid (ceil(N1/32), B * dim), block 256.
constexpr int LK_RMAX = 4;
constexpr int LK_WIN = 2 * LK_RMAX + 4;
constexpr int LK_BWARPS = 8;
constexpr int LK_ROWS = 8;

template <int TAPS>
__global__ void __launch_bounds__(32 * LK_BWARPS)
lookup_backward_window_kernel(const float* __restrict__ coord, long long coord_sb, const float* __restrict__ gout,
                              float* __restrict__ gcorr, int dim, int D, int N1, int levels, int radius,
                              int clamp_unit) {
  follow_previous_kernel();
  __shared__ float win[LOOKUP_MAX_LEVELS][LK_WIN][32];
  __shared__ int wbase[LOOKUP_MAX_LEVELS][32];
  constexpr int MAX_TAPS = TAPS > 0 ? TAPS : 2 * LK_RMAX + 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int p = blockIdx.x * 32 + lane, b = blockIdx.y / dim, ch = blockIdx.y - b * dim;
  const bool in = p < N1;
  const int taps = TAPS > 0 ? TAPS : 2 * radius + 1;
  const float c = in ? __ldg(coord + (size_t)b * coord_sb + p) : 0.f;
  const float* go = gout + (size_t)b * levels * dim * taps * N1 + (in ? p : 0);
  for (int l = warp; l < levels; l += LK_BWARPS) {
    const int Dl = D >> l;
    for (int s = 0; s < LK_WIN; ++s) win[l][s][lane] = 0.f;
    const float* gl = go + (size_t)(l * dim + ch) * taps * N1;
    float g[MAX_TAPS];
#pragma unroll
    for (int t = 0; t < MAX_TAPS; ++t) g[t] = (in && t < taps) ? __ldg(gl + (size_t)t * N1) : 0.f;
    int base = 0;
#pragma unroll
    for (int t = 0; t < MAX_TAPS; ++t) {
      if (t < taps) {
        const float ix = lookup_position(c, l, t, radius, clamp_unit, Dl);
        const float fl = floorf(ix);
        const float w1 = ix - fl, w0 = 1.f - w1;
        const int i0 = (int)fminf(fmaxf(fl, -2.f), (float)Dl);
        if (t == 0) base = i0;
        const int s0 = i0 - base;   // positions grow with t: 0 <= s0 <= 2r+1 (+1 of rounding slack)
        if (s0 >= 0 && s0 + 1 < LK_WIN) {
          win[l][s0][lane] += w0 * g[t];      // rows outside the volume are dropped when the column is written
          win[l][s0 + 1][lane] += w1 * g[t];
        }
      }
    }
    wbase[l][lane] = base;
  }
  __syncthreads();
  if (!in) return;
  float* dst = gcorr + ((size_t)(b * dim + ch) * D) * N1 + p;
  for (int i0 = warp * LK_ROWS; i0 < D; i0 += LK_BWARPS * LK_ROWS) {
    float acc[LK_ROWS];
#pragma unroll
    for (int r = 0; r < LK_ROWS; ++r) acc[r] = 0.f;
    float scale = 1.f;
    for (int l = 0; l < levels; ++l, scale *= 0.5f) {
      const int wb = wbase[l][lane], Dl = D >> l;
      // rows i0 .. i0+7 meet entries (i0 >> l) .. ((i0 + 7) >> l) of this level
      if ((i0 >> l) - wb >= LK_WIN || ((i0 + LK_ROWS - 1) >> l) < wb) continue;
#pragma unroll
      for (int r = 0; r < LK_ROWS; ++r) {
        const int j = (i0 + r) >> l, s = j - wb;   // j >= Dl: dropped by the floor of an odd size
        if (j < Dl && s >= 0 && s < LK_WIN) acc[r] = fmaf(scale, win[l][s][lane], acc[r]);
      }
    }
#pragma unroll
    for (int r = 0; r < LK_ROWS; ++r)
      if (i0 + r < D) dst[(size_t)(i0 + r) * N1] = acc[r];
  }
}

// ---- gradients of several lookups on the same volumes ------------------------------------------------------
// Accumulator of one volume: per level the rows (B, dim, R_l, N1) that a lookup can touch, all D_l of them, or three where
// the positions are clamped to [-1, 1] (a position of 1 that the normalisation rounds up still lies below 2).
struct LookupAccumulator {
  float* ptr[LOOKUP_MAX_LEVELS];         // level l: (B, dim, R_l, N1)
  int D[LOOKUP_MAX_LEVELS], R[LOOKUP_MAX_LEVELS];
  const float* coord;
  long long coord_sb;
  const float* gout;
  int clamp_unit;
};
struct LookupAccumulators { LookupAccumulator v[2]; };

// Adds the window gradients of one lookup to the accumulators of one or two volumes.  A thread owns one level of one pixel: no
// atomics, a sum in the order of the calls.  A window is at most 2r + 3 rows, so that a call touches some 41 of a column's rows
// over four levels, where the gradient of the volume has D rows and is written whole: 8 x 47 x 156, both volumes, radius 4, four
// levels: 35 us for the two gradients and 17 for adding them to those of the other lookups; 15 now.
// WINDOW: radius <= LK_RMAX; the window is summed in shared memory (a column per thread) on top of the rows as they were, which
// are asked for together with the output gradients.  Else row by row in memory, any radius.
// grid (ceil(N1 / (32 * groups)), B * dim, volumes), block (32, min(levels, LK_WARPS), groups of pixels)
template <bool WINDOW, int TAPS>
__global__ void __launch_bounds__(32 * LK_WARPS)
lookup_accumulate_kernel(const __grid_constant__ LookupAccumulators vols, int dim, int N1, int levels, int radius) {
  follow_previous_kernel();
  __shared__ float win_mem[WINDOW ? LK_WARPS : 1][LK_WIN][32];
  constexpr int MAX_TAPS = TAPS > 0 ? TAPS : 2 * LK_RMAX + 1;
  const int p = (blockIdx.x * blockDim.z + threadIdx.z) * 32 + threadIdx.x;
  if (p >= N1) return;
  const LookupAccumulator& lv = vols.v[blockIdx.z];
  const int b = blockIdx.y / dim, ch = blockIdx.y - b * dim, clamp_unit = lv.clamp_unit;
  const int taps = TAPS > 0 ? TAPS : 2 * radius + 1;
  const float c = __ldg(lv.coord + (size_t)b * lv.coord_sb + p);
  const float* go = lv.gout + (size_t)b * levels * dim * taps * N1 + p;
  for (int l = threadIdx.y; l < levels; l += blockDim.y) {
    const int Dl = lv.D[l], rows = lv.R[l];
    float* acc = lv.ptr[l] + (size_t)blockIdx.y * rows * N1 + p;
    const float* gl = go + (size_t)(l * dim + ch) * taps * N1;
    auto lower = [&](int t, float& w1) {   // row below position t (far outside the volume: -2 or D) and the weight of the one above
      const float ix = lookup_position(c, l, t, radius, clamp_unit, Dl);
      const float fl = floorf(ix);
      w1 = ix - fl;
      return (int)fminf(fmaxf(fl, -2.f), (float)Dl);
    };
    if constexpr (WINDOW) {
      float(*win)[32] = win_mem[threadIdx.z * blockDim.y + threadIdx.y];
      float g[MAX_TAPS], w[MAX_TAPS], old[LK_WIN];
      int i0[MAX_TAPS];
#pragma unroll
      for (int t = 0; t < MAX_TAPS; ++t) g[t] = t < taps ? __ldg(gl + (size_t)t * N1) : 0.f;
#pragma unroll
      for (int t = 0; t < MAX_TAPS; ++t) i0[t] = t < taps ? lower(t, w[t]) : 0;
      const int base = i0[0];
#pragma unroll
      for (int s = 0; s < LK_WIN; ++s) old[s] = base + s >= 0 && base + s < rows ? acc[(ptrdiff_t)(base + s) * N1] : 0.f;
#pragma unroll
      for (int s = 0; s < LK_WIN; ++s) win[s][threadIdx.x] = old[s];
#pragma unroll
      for (int t = 0; t < MAX_TAPS; ++t) {
        const int s0 = i0[t] - base;   // positions grow with t: 0 <= s0 <= 2r+1 (+1 of rounding slack)
        if (t < taps && s0 >= 0 && s0 + 1 < LK_WIN) {
          win[s0][threadIdx.x] += (1.f - w[t]) * g[t];
          win[s0 + 1][threadIdx.x] += w[t] * g[t];
        }
      }
#pragma unroll
      for (int s = 0; s < LK_WIN; ++s) {
        const float v = win[s][threadIdx.x];
        if (base + s >= 0 && base + s < rows && v != old[s]) acc[(ptrdiff_t)(base + s) * N1] = v;
      }
    } else {
      for (int t = 0; t < taps; ++t) {
        float w1;
        const int i = lower(t, w1);
        const float g = __ldg(gl + (size_t)t * N1);
        if (i >= 0 && i < rows) acc[(ptrdiff_t)i * N1] += (1.f - w1) * g;
        if (i + 1 >= 0 && i + 1 < rows) acc[(ptrdiff_t)(i + 1) * N1] += w1 * g;
      }
    }
  }
}

// gcorr[plane][i][p] = sum over levels of accumulator_l[plane][i >> l][p] / 2^l (a level-l entry spreads evenly over the 2^l entries
// it averaged; entries dropped by the floor of an odd size get none).  HBM-bound: a thread writes LK_PROWS rows of VEC neighbouring
// pixels, all loads first.  grid (ceil(N1 / (LK_THREADS * VEC)), ceil(D / LK_PROWS), planes)
template <int VEC>
__global__ void __launch_bounds__(LK_THREADS)
lookup_gradient_fold_kernel(const __grid_constant__ LookupAccumulator lv, float* __restrict__ gcorr, int levels, int N1) {
  follow_previous_kernel();
  typedef typename LkVec<VEC>::type V;
  const int p = (blockIdx.x * LK_THREADS + threadIdx.x) * VEC, r0 = blockIdx.y * LK_PROWS, D = lv.D[0];
  if (p >= N1) return;
  V acc[LK_PROWS];
#pragma unroll
  for (int r = 0; r < LK_PROWS; ++r) acc[r] = V{};
  float scale = 1.f;
  for (int l = 0; l < levels; ++l, scale *= 0.5f) {
    const int rows = min(lv.R[l], lv.D[l]);
    if ((r0 >> l) >= rows) continue;
    const float* src = lv.ptr[l] + (size_t)blockIdx.z * lv.R[l] * N1 + p;
#pragma unroll
    for (int r = 0; r < LK_PROWS; ++r) {
      const int j = (r0 + r) >> l;
      if (j < rows) lk_fma(acc[r], scale, __ldg(reinterpret_cast<const V*>(src + (size_t)j * N1)));
    }
  }
  float* dst = gcorr + ((size_t)blockIdx.z * D + r0) * N1 + p;
#pragma unroll
  for (int r = 0; r < LK_PROWS; ++r)
    if (r0 + r < D) *reinterpret_cast<V*>(dst + (size_t)r * N1) = acc[r];
}

// ---- launchers ---------------------------------------------------------------------------------------
size_t lookup_pyramid_floats(const LookupDims& d) {  // levels 1 .. levels-1
  size_t n = 0;
  int Dl = d.D;
  for (int l = 1; l < d.levels; ++l) { Dl /= 2; n += (size_t)d.B * d.dim * Dl * d.H1 * d.W1; }
  return n;
}

template <class L, class P>
static void fill_levels(L& lv, const LookupDims& d, P* level0, P* pyramid) {
  int Dl = d.D;
  P* next = pyramid;
  for (int l = 0; l < LOOKUP_MAX_LEVELS; ++l) { lv.ptr[l] = nullptr; lv.D[l] = 0; }
  for (int l = 0; l < d.levels; ++l) {
    lv.ptr[l] = l == 0 ? level0 : next;
    lv.D[l] = Dl;
    if (l > 0) next += (size_t)d.B * d.dim * Dl * d.H1 * d.W1;
    Dl /= 2;
  }
}

static bool lk_vec4(int N1, std::initializer_list<const void*> ptrs) {   // whether planes can be read 16 bytes at a time
  uintptr_t all = 0;
  for (const void* p : ptrs) all |= reinterpret_cast<uintptr_t>(p);
  return N1 % 4 == 0 && (all & 15u) == 0;
}

static cudaError_t launch_pyramids(const LookupDims* d, const float* const* corr, float* const* pyramid, int volumes, cudaStream_t st) {
  LookupPyramids vols{};
  const int N1 = d[0].H1 * d[0].W1, levels = d[0].levels;
  for (int v = 0; v < volumes; ++v) fill_levels(vols.v[v], d[v], const_cast<float*>(corr[v]), pyramid[v]);
  const bool vec = lk_vec4(N1, {corr[0], pyramid[0], corr[volumes - 1], pyramid[volumes - 1]});
  const int px = LK_THREADS * (vec ? 4 : 1);
  for (int base = 0; base + 1 < levels; base += 3) {
    int D = 0;
    for (int v = 0; v < volumes; ++v) D = std::max(D, vols.v[v].D[base]);
    const int row_blocks = (D + LK_PROWS - 1) / LK_PROWS;
    const dim3 grid((N1 + px - 1) / px, volumes * row_blocks, d[0].B * d[0].dim);
    launch_next((vec ? lookup_pyramid_kernel<4> : lookup_pyramid_kernel<1>), grid, LK_THREADS, 0, st, vols, base, levels, row_blocks, N1);
  }
  return cudaGetLastError();
}
cudaError_t launch_lookup_pyramid(const LookupDims& d, const float* corr, float* pyramid, cudaStream_t st) {
  return launch_pyramids(&d, &corr, &pyramid, 1, st);
}
cudaError_t launch_lookup_pyramid_pair(const LookupDims (&d)[2], const float* const (&corr)[2], float* const (&pyramid)[2], cudaStream_t st) {
  return launch_pyramids(d, corr, pyramid, 2, st);
}

// Blocks of up to LK_WARPS warps: levels of the same pixels, then further pixels.
static dim3 level_block(int levels) {
  const int warps = levels < LK_WARPS ? levels : LK_WARPS;
  return dim3(32, warps, LK_WARPS / warps);
}
static unsigned pixel_blocks(int N1, const dim3& block) { return (N1 + 32 * block.z - 1) / (32 * block.z); }

static cudaError_t launch_forward(const LookupDims* d, const LookupCall* c, int volumes, cudaStream_t st) {
  LookupVolumes vols{};
  for (int v = 0; v < volumes; ++v) {
    fill_levels(vols.v[v], d[v], c[v].corr, c[v].pyramid);
    vols.v[v].coord = c[v].coord;
    vols.v[v].coord_sb = c[v].coord_sb;
    vols.v[v].out = c[v].out;
    vols.v[v].clamp_unit = c[v].clamp_unit;
  }
  const int N1 = d[0].H1 * d[0].W1;
  const dim3 block = level_block(d[0].levels), grid(pixel_blocks(N1, block), d[0].B, volumes);
  auto kern = d[0].radius == LK_RMAX ? lookup_forward_kernel<2 * LK_RMAX + 1> : lookup_forward_kernel<0>;
  launch_next(kern, grid, block, 0, st, vols, d[0].dim, N1, d[0].levels, d[0].radius);
  return cudaGetLastError();
}
cudaError_t launch_lookup_forward(const LookupDims& d, const LookupCall& c, cudaStream_t st) { return launch_forward(&d, &c, 1, st); }
cudaError_t launch_lookup_forward_pair(const LookupDims (&d)[2], const LookupCall (&c)[2], cudaStream_t st) {
  return launch_forward(d, c, 2, st);
}

static int accumulator_rows(int Dl, int clamp_unit) { return clamp_unit ? std::min(Dl, 3) : Dl; }
static void fill_accumulator(LookupAccumulator& a, const LookupDims& d, float* acc, int clamp_unit) {
  int Dl = d.D;
  a.clamp_unit = clamp_unit;
  for (int l = 0; l < d.levels; ++l, Dl /= 2) {
    a.ptr[l] = acc;
    a.D[l] = Dl;
    a.R[l] = accumulator_rows(Dl, clamp_unit);
    acc += (size_t)d.B * d.dim * a.R[l] * d.H1 * d.W1;
  }
}
size_t lookup_accumulator_floats(const LookupDims& d, int clamp_unit) {
  size_t rows = 0;
  for (int l = 0, Dl = d.D; l < d.levels; ++l, Dl /= 2) rows += accumulator_rows(Dl, clamp_unit);
  return rows * d.B * d.dim * d.H1 * d.W1;
}

cudaError_t launch_lookup_accumulate(const LookupDims* d, const LookupGradient* g, int volumes, cudaStream_t st) {
  LookupAccumulators vols{};
  for (int v = 0; v < volumes; ++v) {
    fill_accumulator(vols.v[v], d[v], g[v].acc, g[v].clamp_unit);
    vols.v[v].coord = g[v].coord;
    vols.v[v].coord_sb = g[v].coord_sb;
    vols.v[v].gout = g[v].gout;
  }
  const int N1 = d[0].H1 * d[0].W1, radius = d[0].radius;
  const dim3 block = level_block(d[0].levels), grid(pixel_blocks(N1, block), d[0].B * d[0].dim, volumes);
  auto kern = radius == LK_RMAX  ? lookup_accumulate_kernel<true, 2 * LK_RMAX + 1>
              : radius < LK_RMAX ? lookup_accumulate_kernel<true, 0>
                                 : lookup_accumulate_kernel<false, 0>;
  launch_next(kern, grid, block, 0, st, vols, d[0].dim, N1, d[0].levels, radius);
  return cudaGetLastError();
}

cudaError_t launch_lookup_gradient_fold(const LookupDims& d, const float* acc, float* gcorr, int clamp_unit, cudaStream_t st) {
  LookupAccumulator a{};
  fill_accumulator(a, d, const_cast<float*>(acc), clamp_unit);
  const int N1 = d.H1 * d.W1;
  const bool vec = lk_vec4(N1, {acc, gcorr});
  const int px = LK_THREADS * (vec ? 4 : 1);
  const dim3 grid((N1 + px - 1) / px, (d.D + LK_PROWS - 1) / LK_PROWS, d.B * d.dim);
  launch_next((vec ? lookup_gradient_fold_kernel<4> : lookup_gradient_fold_kernel<1>), grid, LK_THREADS, 0, st, a, gcorr, d.levels, N1);
  return cudaGetLastError();
}

cudaError_t launch_lookup_backward(const LookupDims& d, const float* gout, const float* coord, long long coord_sb,
                                   float* gcorr, float* gpyramid, int clamp_unit, cudaStream_t st) {
  const int N1 = d.H1 * d.W1;
  if (d.radius <= LK_RMAX) {
    const dim3 wgrid((N1 + 31) / 32, d.B * d.dim);
    auto kern = d.radius == LK_RMAX ? lookup_backward_window_kernel<2 * LK_RMAX + 1> : lookup_backward_window_kernel<0>;
    launch_next(kern, wgrid, 32 * LK_BWARPS, 0, st, coord, coord_sb, gout, gcorr, d.dim, d.D, N1, d.levels, d.radius, clamp_unit);
    return cudaGetLastError();
  }
  LookupLevelsMut gl;
  fill_levels(gl, d, gcorr, gpyramid);
  cudaError_t err = cudaMemsetAsync(gcorr, 0, (size_t)d.B * d.dim * d.D * N1 * sizeof(float), st);
  if (err != cudaSuccess) return err;
  const size_t pyr = lookup_pyramid_floats(d);
  if (pyr > 0) {
    err = cudaMemsetAsync(gpyramid, 0, pyr * sizeof(float), st);
    if (err != cudaSuccess) return err;
  }
  const dim3 grid((N1 + LK_THREADS - 1) / LK_THREADS, d.B);
  launch_next(lookup_backward_kernel, grid, LK_THREADS, 0, st, gl, coord, coord_sb, gout, d.dim, N1, d.levels, d.radius,
                                                     clamp_unit);
  if (d.levels > 1) {
    const dim3 fgrid((N1 + LK_THREADS - 1) / LK_THREADS, d.D, d.B * d.dim);
    launch_next(lookup_fold_kernel, fgrid, LK_THREADS, 0, st, gl, N1, d.levels);
  }
  return cudaGetLastError();
}

}  // namespace sfb
