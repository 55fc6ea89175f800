// Lookup on the 4D correlation volume WITHOUT storing it: the part the reference leaves unimplemented for its
// memory-saving block (core/corr.py:491-510 raises NotImplementedError and then sketches the call it would make,
// alt_cuda_corr.forward(fmap1 (B,H1,W1,C), fmap2_l (B,H2_l,W2_l,C), coords / 2^l, radius) per pyramid level).  The
// result is the dense block's lookup (core/corr.py:192-247): for every image-1 pixel and pyramid level l a
// (2r+1) x (2r+1) window of the level-l volume around coords / 2^l, bilinearly interpolated with zero padding
// (core/utils/utils.py:110-118, F.grid_sample with align_corners=True), divided by sqrt(C) (core/corr.py:286).
// Averaging the volume over 2x2 blocks of image-2 positions (core/corr.py:36-39) equals correlating with the
// average-pooled image-2 features, so level l needs only the pooled features, never the volume.
//
// Work per (pixel, level): the (2r+2)^2 dot products of the pixel's feature row with the image-2 feature rows at
// the integer positions under its window, then (2r+1)^2 bilinear combinations of them.  The image-2 rows (1 KB each at
// C = 256) come through L1/L2, so the kernels share them: a walk serves a block of neighbouring pixels, whose windows
// mostly overlap because neighbouring pixels move alike, visits the bounding box of their windows once, and uses every
// loaded image-2 row for all of them (their feature rows in registers, lanes split the channels).  Partial sums of 32
// (position, pixel) pairs are reduced together with a 31-shuffle transpose.  When the windows lie far apart (a motion
// boundary) the walk is done for fewer pixels at a time.  A CTA covers 8 x 2 pixels and stages its outputs in shared
// memory, so that the (B, levels*(2r+1)^2, H1, W1) result is written in runs of eight pixels (a 32-byte sector).
//
// Backward (features only: the model detaches the coordinates, core/sepflow.py:193): the gradient of a pixel's window is
// spread back onto the integer positions (each takes from at most four window entries); gF1 is the sum over positions of
// that times the image-2 row, gF2 of a position the sum over pixels of the same times the pixel's row.  The channel is a
// free index of both, so a lane owns two channels for all pixels of a 4 x 4 tile, and the box of all their windows is
// walked once: an image-2 row is read, and reduced into L2, once per tile and level.  Tiles whose windows lie too far apart take
// the forward's walks, with one 16-byte vector reduction per lane (red.global.add.v4.f32) and position.
#include <algorithm>
#include <climits>

#include "kernels.h"
#include "sm100_primitives.cuh"

namespace sfb {

constexpr int L4_TW = 8, L4_TH = 2;            // image-1 pixels of a CTA: two-dimensional, so that windows overlap
constexpr int L4_TILE = L4_TW * L4_TH;
constexpr int L4_RMAX = 4;
constexpr int L4_WIN = 2 * L4_RMAX + 1;        // window side
constexpr int L4_SIDE = 2 * L4_RMAX + 2;       // integer positions under a window, per side

struct Lookup4dLevels {
  const float* f2[LOOKUP_MAX_LEVELS];   // level l: (B, H2_l, W2_l, C)
  float* g2[LOOKUP_MAX_LEVELS];         // gradient of the same (backward only)
  int H2[LOOKUP_MAX_LEVELS], W2[LOOKUP_MAX_LEVELS];
};

// A position through grid_sample's normalisation and back (core/utils/utils.py:114-115 and torch's
// grid_sampler_unnormalize for align_corners=True), in the reference's order of float operations.
__device__ __forceinline__ float l4_unnormalise(float x, int size) {
  const float g = 2.f * x / (float)(size - 1) - 1.f;
  return (g + 1.f) * 0.5f * (float)(size - 1);
}

// floor() to an int that later +-radius arithmetic cannot overflow; positions that far out sample only padding.
__device__ __forceinline__ int l4_floor(float x) {
  if (!(x > -1.0e6f)) return -1000000;   // also NaN
  if (x > 1.0e6f) return 1000000;
  return (int)floorf(x);
}

struct L4Pixel {     // geometry of one pixel at one level
  float cx, cy;      // coords / 2^l
  int bx, by;        // integer position under the window centre
};

// Bounding box of the integer positions of several pixels' windows.
struct L4Box {
  int ox, oy, bw, bh;
};

// Four channels as two packed pairs: one fma.rn.f32x2 per pair.
struct L4Quad {
  uint64_t lo, hi;
};
__device__ __forceinline__ L4Quad l4_load(const float* p, bool ok) {
  L4Quad q{0ull, 0ull};
  if (ok) {
    const ulonglong2 t = __ldg(reinterpret_cast<const ulonglong2*>(p));
    q.lo = t.x;
    q.hi = t.y;
  }
  return q;
}

// v[i] summed over each group of N neighbouring lanes; lane i of a group keeps the total of v[i].  N - 1 shuffles for N values.
template <int N>
__device__ __forceinline__ float group_transpose_reduce(float (&v)[N], int lane) {
#pragma unroll
  for (int off = N / 2; off > 0; off /= 2) {
    const bool up = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < off; ++i) {
      const float send = up ? v[i] : v[i + off];
      const float keep = up ? v[i + off] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  return v[0];
}

// Interpolation weight pair of window entry t along one axis: the reference's position of that entry
// (centre / 2^l + t - r, then normalised and back), expressed against the integer position base + t - r.
__device__ __forceinline__ float l4_fraction(float c, int base, int t, int radius, int size) {
  const float pos = l4_unnormalise(c + (float)(t - radius), size);
  return pos - (float)(base + t - radius);
}

__device__ __forceinline__ L4Pixel l4_pixel_geometry(const float* __restrict__ coords, int b, int p, int N1, int level,
                                                     int H2, int W2) {
  L4Pixel g;
  const float inv = 1.f / (float)(1 << level);
  g.cx = __ldg(coords + ((size_t)b * 2 + 0) * N1 + p) * inv;
  g.cy = __ldg(coords + ((size_t)b * 2 + 1) * N1 + p) * inv;
  g.bx = l4_floor(l4_unnormalise(g.cx, W2));
  g.by = l4_floor(l4_unnormalise(g.cy, H2));
  return g;
}

// Box of the pixels in `mask` (lanes hold one pixel each); every lane gets it.  An empty mask gives an empty box.
__device__ __forceinline__ L4Box l4_box(const L4Pixel& g, unsigned mask, int radius, int lane) {
  const bool in = (mask >> lane) & 1u;
  const int xmin = __reduce_min_sync(0xffffffffu, in ? g.bx : INT_MAX), xmax = __reduce_max_sync(0xffffffffu, in ? g.bx : INT_MIN);
  const int ymin = __reduce_min_sync(0xffffffffu, in ? g.by : INT_MAX), ymax = __reduce_max_sync(0xffffffffu, in ? g.by : INT_MIN);
  if (mask == 0) return L4Box{0, 0, 0, 0};
  return L4Box{xmin - radius, ymin - radius, xmax - xmin + 2 * radius + 2, ymax - ymin + 2 * radius + 2};
}
__device__ __forceinline__ bool l4_fits(const L4Box& box, int limit) {  // extents are at most 2e6 + 10: no overflow in 64 bits
  return (long long)box.bw * box.bh <= limit;
}

// Image-2 row of every box position (-1: outside the image, or padding up to a multiple of 32), so that the walk below
// spends one broadcast load per position instead of a division and four comparisons.
__device__ __forceinline__ void l4_fill_rows(int* rows, const L4Box& box, int H2, int W2, int lane) {
  const int nq = box.bw * box.bh;
  for (int q = lane; q < (nq + 31) / 32 * 32; q += 32) {
    const int row = q / box.bw, x = box.ox + q - row * box.bw, y = box.oy + row;
    rows[q] = (q < nq && x >= 0 && x < W2 && y >= 0 && y < H2) ? y * W2 + x : -1;
  }
}

// ---- forward ----------------------------------------------------------------------------------------------
// A CTA owns 8 x 2 pixels at one level, a warp 2 x 2 of them: one walk over the box of their windows with the four
// pixels' feature rows in registers (lanes split the channels).  Bound by instruction issue: the products are packed
// pairs and the positions come from a table.
constexpr int L4_THREADS = 128;
constexpr int L4_WARPS = L4_THREADS / 32;
constexpr int L4_PX = 4;
static_assert(L4_TW == 2 * L4_WARPS && L4_TH == 2, "2 x 2 pixels a warp");
constexpr int L4_BMAX = 224;                   // largest box a four-pixel walk accepts
static_assert(L4_SIDE * L4_SIDE <= L4_BMAX && L4_BMAX % 32 == 0, "one pixel's positions must fit the table");

// Dot products of NPX pixels' feature rows with the image-2 rows of a box, scaled, into S[px0 + px][position]; zero
// outside the image.  LP lanes split the channels, so the warp does 32 / LP positions at a time: up to 256 channels 16 lanes, which
// halves the work of the reductions and keeps the additions of a lane as many as with 32 lanes (two chains).
// FULL: C = NQ * 4 * LP, no lane without channels.
template <int NQ, int NPX, int LP, bool FULL>
__device__ __forceinline__ void l4_box_products(const L4Quad (&f1)[NPX][NQ], const float* __restrict__ F2b, int C,
                                                const int* rows, int nq, float scale, float (*S)[L4_BMAX], int px0,
                                                int lane) {
  constexpr int PB = 32 / LP, STEPS = LP / NPX, HALF = LP == 16 ? (NQ + 1) / 2 : NQ;   // chunks of the first chain
  const int group = lane / LP, at = lane % LP;
  const uint32_t row_bytes = 4 * C;   // (32-bit factors: the product and the sum are one multiply-add)
  const char* const src = reinterpret_cast<const char*>(F2b + at * 4);
  for (int q0 = 0; q0 < nq; q0 += PB * STEPS) {
    float v[LP];
#pragma unroll
    for (int step = 0; step < STEPS; ++step) {
      const int r = rows[q0 + step * PB + group];   // (beyond the image row 0 is read, and not used)
      const float* const row = reinterpret_cast<const float*>(src + (uint64_t)row_bytes * (uint32_t)max(r, 0));
      L4Quad f2[NQ];
#pragma unroll
      for (int ch = 0; ch < NQ; ++ch) f2[ch] = l4_load(row + ch * 4 * LP, FULL || (r >= 0 && (ch * LP + at) * 4 < C));
#pragma unroll
      for (int px = 0; px < NPX; ++px) {
        uint64_t acc = fma2(f1[px][0].hi, f2[0].hi, mul2(f1[px][0].lo, f2[0].lo));
#pragma unroll
        for (int ch = 1; ch < HALF; ++ch) acc = fma2(f1[px][ch].hi, f2[ch].hi, fma2(f1[px][ch].lo, f2[ch].lo, acc));
        if (HALF < NQ) {
          uint64_t acc2 = fma2(f1[px][HALF].hi, f2[HALF].hi, mul2(f1[px][HALF].lo, f2[HALF].lo));
#pragma unroll
          for (int ch = HALF + 1; ch < NQ; ++ch) acc2 = fma2(f1[px][ch].hi, f2[ch].hi, fma2(f1[px][ch].lo, f2[ch].lo, acc2));
          acc = add2(acc, acc2);
        }
        v[step * NPX + px] = sum2(acc);
      }
    }
    const float total = group_transpose_reduce<LP>(v, lane);
    const int q = q0 + at / NPX * PB + group;
    if (q < nq) S[px0 + at % NPX][q] = rows[q] >= 0 ? total * scale : 0.f;
  }
}

// Two packed multiply-adds per 4 channels, pixel and position, and the reductions, bound the forward: 2 x 55 x 128 at C = 256, four
// levels, radius 4 takes 172 us with 32 lanes a position, 148 with 16.  Four CTAs of 8 x 2 pixels per SM instead of two of 8 x 4 wait for less
// at their ends and beginnings: six of them 951 -> 912 us (1 x 60 x 160 664 -> 638; 4 x 4 pixels 936 and 652).
// grid (ceil(W1/8) * ceil(H1/2), levels, B)
template <int NQ, int LP, bool FULL>
__global__ void __launch_bounds__(L4_THREADS, 4)
lookup4d_forward_kernel(const float* __restrict__ F1, Lookup4dLevels lv, const float* __restrict__ coords,
                        float* __restrict__ out, int H1, int W1, int C, int radius, int levels, float scale) {
  follow_previous_kernel();
  __shared__ float s_S[L4_WARPS][L4_PX][L4_BMAX];
  __shared__ float s_out[L4_WIN * L4_WIN][L4_TILE + 1];
  __shared__ int s_rows[L4_WARPS][L4_BMAX];
  __shared__ int2 s_base[L4_WARPS][L4_PX];               // integer positions under the window centres
  __shared__ float s_frac[L4_WARPS][2][L4_PX][L4_WIN];   // l4_fraction of the window entries along x, y

  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int level = blockIdx.y, b = blockIdx.z, N1 = H1 * W1;
  const int H2 = lv.H2[level], W2 = lv.W2[level];
  const float* F2b = lv.f2[level] + (size_t)b * H2 * W2 * C;
  const int tiles_x = (W1 + L4_TW - 1) / L4_TW;
  const int h0 = (int)(blockIdx.x / tiles_x) * L4_TH, w0 = (int)(blockIdx.x % tiles_x) * L4_TW;
  const int win = 2 * radius + 1;
  // warp w: columns 2*w, 2*w + 1 of the tile; its pixel px: column px%2, row px/2
  const int ph = h0, pw = w0 + 2 * w;

  L4Pixel geo{0.f, 0.f, 0, 0};
  const int mh = ph + ((lane >> 1) & 1), mw = pw + (lane & 1);
  const bool mine = lane < L4_PX && mh < H1 && mw < W1;
  if (mine) geo = l4_pixel_geometry(coords, b, mh * W1 + mw, N1, level, H2, W2);
  if (lane < L4_PX) s_base[w][lane] = make_int2(geo.bx, geo.by);
  const unsigned mask = __ballot_sync(0xffffffffu, mine);
  for (int i = lane; i - lane < 2 * L4_PX * win; i += 32) {
    const int axis = i & 1, px = (i >> 1) % L4_PX, t = i / (2 * L4_PX);
    const float cx = __shfl_sync(0xffffffffu, geo.cx, px), cy = __shfl_sync(0xffffffffu, geo.cy, px);
    const int bx = __shfl_sync(0xffffffffu, geo.bx, px), by = __shfl_sync(0xffffffffu, geo.by, px);
    if (t < win) s_frac[w][axis][px][t] = l4_fraction(axis ? cy : cx, axis ? by : bx, t, radius, axis ? H2 : W2);
  }

  if (mask != 0) {
    L4Quad f1[L4_PX][NQ];
#pragma unroll
    for (int px = 0; px < L4_PX; ++px)
#pragma unroll
      for (int ch = 0; ch < NQ; ++ch) {
        const int c = (ch * LP + lane % LP) * 4;
        const size_t p = (size_t)b * N1 + (size_t)(ph + px / 2) * W1 + pw + px % 2;
        const bool ok = ((mask >> px) & 1u) && c < C;
        f1[px][ch] = l4_load(F1 + (ok ? p * C + c : 0), ok);
      }

    L4Box box = l4_box(geo, mask, radius, lane);
    const bool together = l4_fits(box, L4_BMAX);
    if (together) {
      l4_fill_rows(s_rows[w], box, H2, W2, lane);
      __syncwarp();
      l4_box_products<NQ, L4_PX, LP, FULL>(f1, F2b, C, s_rows[w], box.bw * box.bh, scale, s_S[w], 0, lane);
    } else {  // motion boundaries: one pixel at a time
#pragma unroll
      for (int px = 0; px < L4_PX; ++px) {
        if (!((mask >> px) & 1u)) continue;
        L4Quad one[1][NQ];
#pragma unroll
        for (int ch = 0; ch < NQ; ++ch) one[0][ch] = f1[px][ch];
        box = l4_box(geo, 1u << px, radius, lane);
        __syncwarp();
        l4_fill_rows(s_rows[w], box, H2, W2, lane);
        __syncwarp();
        l4_box_products<NQ, 1, LP, FULL>(one, F2b, C, s_rows[w], box.bw * box.bh, scale, s_S[w], px, lane);
      }
    }
    __syncwarp();

    // bilinear combinations
    for (int idx = lane; idx < L4_PX * win * win; idx += 32) {
      const int px = idx / (win * win), o = idx - px * win * win;
      if (!((mask >> px) & 1u)) continue;
      const int a = o / win, bb = o - a * win;
      const int2 g = s_base[w][px];
      const int ox = together ? box.ox : g.x - radius;
      const int oy = together ? box.oy : g.y - radius;
      const int sbw = together ? box.bw : 2 * radius + 2;
      const float fx = s_frac[w][0][px][a], fy = s_frac[w][1][px][bb];
      const float* S = s_S[w][px] + (g.y + bb - radius - oy) * sbw + (g.x + a - radius - ox);
      const float top = S[0] + fx * (S[1] - S[0]);
      const float bot = S[sbw] + fx * (S[sbw + 1] - S[sbw]);
      s_out[o][px / 2 * L4_TW + 2 * w + px % 2] = top + fy * (bot - top);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < win * win * L4_TILE; i += L4_THREADS) {
    const int o = i / L4_TILE, pp = i % L4_TILE, h = h0 + pp / L4_TW, x = w0 + pp % L4_TW;
    if (h < H1 && x < W1) out[(((size_t)b * levels + level) * win * win + o) * N1 + (size_t)h * W1 + x] = s_out[o][pp];
  }
}

// ---- backward ---------------------------------------------------------------------------------------------
constexpr int L4_BT = 4;                        // tile of 4 x 4 pixels
constexpr int L4_BPX = L4_BT * L4_BT;
constexpr int L4_BCH = 256;                      // channels of a CTA, two a lane
constexpr int L4_BBOX = 384;                    // positions of the largest box walked for the whole tile
constexpr int L4_BTHREADS = 128, L4_BWARPS = L4_BTHREADS / 32;
// Largest box of a tile for windows of a radius: what the table holds.  One level of 2 x 55 x 128 pixels at C = 256 takes 0.48 us per position plus
// 40 as whole tiles, 0.9 per position of a 2 x 2 pixels' box plus 34 as four walks of those, so a uniform spread would draw the line at boxes of
// 256 positions (radius 4), 155 (3) and 80 (2).  But a field's tiles differ, and those left apart are a second launch of few long blocks: both lie above
// either alone.  Four levels, smooth motion with objects of another one: all tiles apart 325 us (radius 3) and 226 (2), with limits of 256 and 153
// 380 and 262, with this 219 and 163; noise of 1, 1.5, 2 and 3 pixels, radius 2: 219, 239, 267, 306 apart, 255, 237, 303, 317 with 153,
// 168, 181, 196, 360 with this.  (Blocks of 2 x 3 pixels with motions 4 apart, no two alike, lose: 282 -> 355 and 233 -> 265.)
// Radius 1 and 0 walk 2 x 2 pixels only: whole tiles gain 5 % at C = 256 in a smooth field, and lose 15 at 128.
inline int l4_tile_limit(int radius) { return radius < 2 ? 0 : L4_BBOX; }
static_assert(2 * L4_BTHREADS <= L4_BBOX && L4_BBOX % 4 == 0, "partial sums of warps that share channels; steps of four positions");
static_assert(L4_BCH == L4_BWARPS * 64, "a warp has 64 channels");

__device__ __forceinline__ void red_add_v4(float* addr, uint64_t lo, uint64_t hi) {
  float x, y, z, w;
  unpack2(lo, x, y);
  unpack2(hi, z, w);
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

// One walk of a box for the pixels px0 .. px0+NPX-1: gS[px][position] (already scaled) is in shared memory.
template <int NCH, int NPX>
__device__ __forceinline__ void l4_box_gradients(const L4Quad (&f1)[L4_PX][NCH], L4Quad (&gf1)[L4_PX][NCH],
                                                 const float* __restrict__ F2b, float* __restrict__ G2b, int C,
                                                 const int* rows, int nq, const float (*gS)[L4_BMAX], int px0, int lane) {
  constexpr int J = NCH > 2 ? 1 : 4 / NCH;   // positions per step: their image-2 rows are all requested before any is used
  for (int q0 = 0; q0 < nq; q0 += J) {
    int r[J];
    L4Quad f2[J][NCH];
    int all = -1;
#pragma unroll
    for (int j = 0; j < J; ++j) {
      r[j] = rows[q0 + j];   // -1 past the box
      all &= r[j];
    }
    if (NPX == 1 && all < 0) continue;   // nothing of the window here: beyond the image's edge, or no gradient
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const float* src = F2b + (size_t)(r[j] < 0 ? 0 : r[j]) * C + lane * 4;
#pragma unroll
      for (int ch = 0; ch < NCH; ++ch) f2[j][ch] = l4_load(src + ch * 128, r[j] >= 0 && ch * 128 + lane * 4 < C);
    }
#pragma unroll
    for (int j = 0; j < J; ++j) {
      if (r[j] < 0) continue;
      float g[NPX];
      bool any = false;
#pragma unroll
      for (int k = 0; k < NPX; ++k) {
        g[k] = gS[px0 + k][q0 + j];
        any |= g[k] != 0.f;
      }
      if (!any) continue;   // no pixel of the walk has this position in its window
      uint64_t gg[NPX];
#pragma unroll
      for (int k = 0; k < NPX; ++k) gg[k] = pack2(g[k], g[k]);
      float* dst = G2b + (size_t)r[j] * C + lane * 4;
#pragma unroll
      for (int ch = 0; ch < NCH; ++ch) {
        L4Quad g2{0ull, 0ull};
#pragma unroll
        for (int k = 0; k < NPX; ++k) {
          L4Quad& a = gf1[px0 + k][ch];   // a compile-time index once the caller's loop is unrolled
          a.lo = fma2(gg[k], f2[j][ch].lo, a.lo);
          a.hi = fma2(gg[k], f2[j][ch].hi, a.hi);
          g2.lo = fma2(gg[k], f1[px0 + k][ch].lo, g2.lo);
          g2.hi = fma2(gg[k], f1[px0 + k][ch].hi, g2.hi);
        }
        if (ch * 128 + lane * 4 < C) red_add_v4(dst + ch * 128, g2.lo, g2.hi);
      }
    }
  }
}

// Gradient of one integer position of a pixel's window: position (i, j) of its (2r+2)^2 grid takes from window entries
// a in {i-1, i}, b in {j-1, j} with the weight that entry gives it.  pp: the pixel's column of s_g.
__device__ __forceinline__ float l4_position_gradient(const L4Pixel& g, int i, int j, const float (*s_g)[L4_BPX + 1], int pp,
                                                      int radius, int H2, int W2) {
  const int win = 2 * radius + 1, side = 2 * radius + 2;
  float acc = 0.f;
  if (i >= 0 && i < side && j >= 0 && j < side) {
#pragma unroll
    for (int da = 0; da < 2; ++da) {
      const int a = i - da;
      if (a < 0 || a >= win) continue;
      const float fx = l4_fraction(g.cx, g.bx, a, radius, W2);
      const float wx = da ? fx : 1.f - fx;
#pragma unroll
      for (int db = 0; db < 2; ++db) {
        const int bb = j - db;
        if (bb < 0 || bb >= win) continue;
        const float fy = l4_fraction(g.cy, g.by, bb, radius, H2);
        const float wy = db ? fy : 1.f - fy;
        acc = fmaf(wx * wy, s_g[a * win + bb][pp], acc);
      }
    }
  }
  return acc;
}

// In a walk for one pixel its table of rows lies behind its gradients, with room for the positions that the last step asks for
// past the end.
constexpr int L4_ALONE_ROWS = L4_BMAX / 2, L4_ALONE_PAD = 4;
static_assert(L4_SIDE * L4_SIDE <= L4_ALONE_ROWS && L4_ALONE_ROWS + L4_SIDE * L4_SIDE + L4_ALONE_PAD <= L4_BMAX, "a pixel's positions and rows");

// Geometry of a tile's pixels and the boxes of their windows at all levels, a warp per level; whether every box has at most `limit`
// positions.  All threads; ends with a barrier.
struct L4Tile {
  L4Pixel geo[LOOKUP_MAX_LEVELS][L4_BPX];
  L4Box box[LOOKUP_MAX_LEVELS];
};
__device__ __forceinline__ bool l4_tile(L4Tile& t, const float* __restrict__ coords, const Lookup4dLevels& lv, int levels, int b, int h0, int w0,
                                        int H1, int W1, int radius, int limit) {
  const int lane = threadIdx.x & 31, h = h0 + lane / L4_BT, x = w0 + lane % L4_BT;
  const bool in = lane < L4_BPX && h < H1 && x < W1;
  for (int level = threadIdx.x >> 5; level < levels; level += blockDim.x >> 5) {
    L4Pixel geo{0.f, 0.f, 0, 0};
    if (in) geo = l4_pixel_geometry(coords, b, h * W1 + x, H1 * W1, level, lv.H2[level], lv.W2[level]);
    const L4Box box = l4_box(geo, __ballot_sync(0xffffffffu, in), radius, lane);
    if (lane < L4_BPX) t.geo[level][lane] = geo;
    if (lane == 0) t.box[level] = box;
  }
  __syncthreads();
  bool fits = true;
  for (int level = 0; level < levels; ++level) fits &= l4_fits(t.box[level], limit);
  return fits;
}

constexpr int L4_TROW = L4_WIN + 2;             // window rows with a zero before and behind

// A step of four positions where a feature is infinite or NaN: it reaches only what has it under its window.
template <class Load, class Add>
__device__ __forceinline__ void l4_nonfinite(const float (*gS)[L4_BPX], const int* rows, int q0, const float (&f1)[L4_BPX], float (&gf1)[L4_BPX],
                                             Load&& f2_at, Add&& add_at) {
#pragma unroll 1
  for (int q = q0; q < q0 + 4; ++q) {
    const float f = f2_at(rows[q]);
    float total = 0.f;
#pragma unroll
    for (int px = 0; px < L4_BPX; ++px) {
      const float g = gS[q][px];
      if (g != 0.f) {
        gf1[px] = fmaf(g, f, gf1[px]);
        total = fmaf(g, f1[px], total);
      }
    }
    add_at(rows[q], total);
  }
}

// The levels of a tile are done by two CTAs, the pairs 0 and 3, 1 and 2 (and so on) about alike in length.
__host__ __device__ constexpr int l4_parts(int levels) { return levels > 1 ? 2 : 1; }
__device__ __forceinline__ int l4_part(int level) { return (level + 1) >> 1 & 1; }

// A lane's CH consecutive channels.
template <int CH> struct L4Channels { float f[CH]; };
template <int CH>
__device__ __forceinline__ L4Channels<CH> l4_load_channels(const float* p) {
  L4Channels<CH> v;
  if constexpr (CH == 2) {
    const float2 t = __ldg(reinterpret_cast<const float2*>(p));
    v.f[0] = t.x;
    v.f[1] = t.y;
  } else {
    v.f[0] = __ldg(p);
  }
  return v;
}
template <int CH>
__device__ __forceinline__ void l4_add_channels(float* p, const float (&v)[CH]) {
  if constexpr (CH == 2) asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(v[0]), "f"(v[1]) : "memory");
  else atomicAdd(p, v[0]);
}

// A CTA walks half the levels of its tile; gF1 is cleared and the two sums added to it (either order gives the same bits; one level: stored).
// Warp w owns channels 32 CH (w % groups) .. of the CTA's 256; warps beyond the channels share out the positions.  Bound by FP32 issue: 32
// multiply-adds per channel and position at 1.3 cycles or so (packed pairs with three different operands take 3 cycles, no gain over two
// scalar ones).  CH: a gradient's 16 bytes come back to 32 lanes at 128 bytes a cycle and SM, so with one channel a lane shared memory
// took 16 cycles of a position where the multiply-adds take 11; with two they serve twice the products (one where there are no more than 32
// channels).  Three CTAs: 128 registers for four spill (2 x 55 x 128 pixels at C = 256, four levels, radius 4: 315 us).
// Two CTAs a tile: tiles alone, as in the last wave, left an SM with four warps (1 x 60 x 160: 1429 -> 1369 us for four
// iterations forward and backward, with one channel and 8 warps a tile 1385).
// With a walk per 2 x 2 pixels, lanes splitting the channels, each walk reduced its own 140 positions of 1 KB into L2: the first size took
// 416 us; 280 with one channel a lane, 252 now.
// grid (ceil(W1/4) * ceil(H1/4), ceil(C/256) * l4_parts, B)
template <int CH>
__global__ void __launch_bounds__(L4_BTHREADS, 3)
lookup4d_backward_kernel(const float* __restrict__ F1, Lookup4dLevels lv, const float* __restrict__ coords,
                         const float* __restrict__ gout, float* __restrict__ gF1, int H1, int W1, int C, int radius,
                         int levels, int limit, float scale) {
  follow_previous_kernel();
  __shared__ L4Tile s_tile;
  __shared__ __align__(16) float s_gS[L4_BBOX + 4][L4_BPX];     // gradient of (position, pixel), scaled; positions without any are left out
  __shared__ __align__(16) int s_rows[L4_BBOX + 4];             // their image-2 rows
  __shared__ float s_t[L4_BPX][L4_SIDE][L4_TROW];               // gradients of a pixel's window, spread along x
  __shared__ float s_fx[L4_BPX][L4_WIN];                        // l4_fraction of a pixel's window entries
  __shared__ float s_wy[L4_BPX][L4_SIDE][2];                    // what a position takes along y from the window row above it and its own
  __shared__ __align__(16) int s_bx[L4_BPX], s_by[L4_BPX];      // of this level, next to one another: four a load
  __shared__ int s_count[L4_BWARPS];
  float(*const s_g)[L4_BPX + 1] = reinterpret_cast<float(*)[L4_BPX + 1]>(s_gS);   // output gradients; dead before s_gS is written
  static_assert(L4_WIN * L4_WIN * (L4_BPX + 1) <= L4_BBOX * L4_BPX, "both uses of s_gS");

  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int b = blockIdx.z, N1 = H1 * W1, win = 2 * radius + 1, side = 2 * radius + 2;
  const int tiles_x = (W1 + L4_BT - 1) / L4_BT;
  const int h0 = (int)(blockIdx.x / tiles_x) * L4_BT, w0 = (int)(blockIdx.x % tiles_x) * L4_BT;
  const bool in = lane < L4_BPX && h0 + lane / L4_BT < H1 && w0 + lane % L4_BT < W1;
  const unsigned mask = __ballot_sync(0xffffffffu, in);
  const size_t tile = ((size_t)b * N1 + (size_t)h0 * W1 + w0) * C;
  constexpr int WARP_CH = 32 * CH;
  const int parts = l4_parts(levels), part = (int)blockIdx.y % parts;
  const int c0 = (int)blockIdx.y / parts * L4_BCH, groups = min(L4_BWARPS, (C - c0 + WARP_CH - 1) / WARP_CH), sharers = L4_BWARPS / groups;
  const int c = c0 + w % groups * WARP_CH + lane * CH, share = w / groups;
  const bool mine = c < C && share < sharers;
  float f1[CH][L4_BPX], gf1[CH][L4_BPX];
  bool finite1 = true;
#pragma unroll
  for (int px = 0; px < L4_BPX; ++px) {
    const bool ok = mine && h0 + px / L4_BT < H1 && w0 + px % L4_BT < W1;
    L4Channels<CH> v{};
    if (ok) v = l4_load_channels<CH>(F1 + tile + ((size_t)(px / L4_BT) * W1 + px % L4_BT) * C + c);
#pragma unroll
    for (int k = 0; k < CH; ++k) {
      f1[k][px] = v.f[k];
      finite1 &= isfinite(v.f[k]);
      gf1[k][px] = 0.f;
    }
  }
  if (!l4_tile(s_tile, coords, lv, levels, b, h0, w0, H1, W1, radius, limit)) return;   // lookup4d_backward_apart_kernel does it
  for (int level = 0; level < levels; ++level) {
    if (parts > 1 && l4_part(level) != part) continue;
    const int H2 = lv.H2[level], W2 = lv.W2[level];
    const L4Box box = s_tile.box[level];
    const int nq = box.bw * box.bh;

    constexpr int PER = (L4_WIN * L4_WIN * L4_BPX + L4_BTHREADS - 1) / L4_BTHREADS;
    float g[PER];
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int i = k * L4_BTHREADS + threadIdx.x, o = i / L4_BPX, h = h0 + i % L4_BPX / L4_BT, x = w0 + i % L4_BT;
      const bool ok = o < win * win && h < H1 && x < W1;
      g[k] = ok ? __ldg(gout + (((size_t)b * levels + level) * win * win + o) * N1 + (size_t)h * W1 + x) * scale : 0.f;
    }
    __syncthreads();   // the previous level's tables are no longer read
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int i = k * L4_BTHREADS + threadIdx.x;
      if (i < win * win * L4_BPX) s_g[i / L4_BPX][i % L4_BPX] = g[k];
    }
    if (lane < L4_BPX) {   // warp w: window entries w, w + 8, ...
      const L4Pixel geo = s_tile.geo[level][lane];
      for (int t = w; t < win; t += L4_BWARPS) {
        s_fx[lane][t] = l4_fraction(geo.cx, geo.bx, t, radius, W2);
        const float fy = l4_fraction(geo.cy, geo.by, t, radius, H2);
        s_wy[lane][t][1] = 1.f - fy;
        s_wy[lane][t + 1][0] = fy;
      }
      if (w == 0) {
        s_bx[lane] = geo.bx;
        s_by[lane] = geo.by;
        s_wy[lane][0][0] = s_wy[lane][win][1] = 0.f;
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < L4_BPX * side * (win + 2); i += L4_BTHREADS) {
      const int px = i % L4_BPX, r = i / L4_BPX, bb = r % (win + 2) - 1, at = r / (win + 2);   // window row, column of positions
      float t = 0.f;
      if (bb >= 0 && bb < win) {
        if (at < win) t = (1.f - s_fx[px][at]) * s_g[at * win + bb][px];
        if (at > 0) t = fmaf(s_fx[px][at - 1], s_g[(at - 1) * win + bb][px], t);
      }
      s_t[px][at][bb + 1] = t;
    }
    __syncthreads();
    int count = 0;   // positions with a gradient
    for (int q0 = 0; q0 < nq; q0 += L4_BTHREADS) {
      const int q = q0 + threadIdx.x, row = q / box.bw, x = box.ox + q - row * box.bw, y = box.oy + row;
      float v[L4_BPX];
      bool any = false;
      if (q < nq && x >= 0 && x < W2 && y >= 0 && y < H2) {
#pragma unroll
        for (int px = 0; px < L4_BPX; ++px) {
          const int i = x - (s_bx[px] - radius), j = y - (s_by[px] - radius);
          v[px] = 0.f;
          if (((mask >> px) & 1u) && (unsigned)i < (unsigned)side && (unsigned)j < (unsigned)side)
            v[px] = fmaf(s_wy[px][j][0], s_t[px][i][j], s_wy[px][j][1] * s_t[px][i][j + 1]);
          any |= v[px] != 0.f;
        }
      }
      const unsigned with = __ballot_sync(0xffffffffu, any);
      if (lane == 0) s_count[w] = __popc(with);
      __syncthreads();
      int at = count + __popc(with & ((1u << lane) - 1));
#pragma unroll
      for (int k = 0; k < L4_BWARPS; ++k) {
        at += k < w ? s_count[k] : 0;
        count += s_count[k];
      }
      if (any) {
        s_rows[at] = y * W2 + x;
#pragma unroll
        for (int p4 = 0; p4 < L4_BPX; p4 += 4) *reinterpret_cast<float4*>(&s_gS[at][p4]) = make_float4(v[p4], v[p4 + 1], v[p4 + 2], v[p4 + 3]);
      }
      __syncthreads();
    }
    if (count == 0) continue;
    // up to a multiple of four: the last position again, with no gradient
    const int padded = (count + 3) & ~3;
    if (threadIdx.x < (padded - count) * L4_BPX) s_gS[count + threadIdx.x / L4_BPX][threadIdx.x % L4_BPX] = 0.f;
    if (threadIdx.x < padded - count) s_rows[count + threadIdx.x] = s_rows[count - 1];
    __syncthreads();
    if (!mine) continue;

    // (32-bit factors: the product and the sum are one multiply-add)
    const char* const F2c = reinterpret_cast<const char*>(lv.f2[level] + (size_t)b * H2 * W2 * C + c);
    char* const G2c = reinterpret_cast<char*>(lv.g2[level] + (size_t)b * H2 * W2 * C + c);
    const uint32_t row_bytes = 4 * C;
    const auto f2_row = [&](int r) { return reinterpret_cast<const float*>(F2c + (uint64_t)row_bytes * (uint32_t)r); };
    const auto g2_row = [&](int r) { return reinterpret_cast<float*>(G2c + (uint64_t)row_bytes * (uint32_t)r); };
    // four positions a step; the next step's rows are requested before this one's are used
    int next_r[4];
    L4Channels<CH> next_f[4];
    const auto fetch = [&](int q0) {
      if (q0 >= padded) return;
      *reinterpret_cast<int4*>(next_r) = *reinterpret_cast<const int4*>(&s_rows[q0]);
#pragma unroll
      for (int k = 0; k < 4; ++k) next_f[k] = l4_load_channels<CH>(f2_row(next_r[k]));
    };
    fetch(share * 4);
#pragma unroll 2
    for (int q0 = share * 4; q0 < padded; q0 += sharers * 4) {
      int r[4];
      L4Channels<CH> f[4];
      float magnitude = 0.f;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        r[k] = next_r[k];
        f[k] = next_f[k];
#pragma unroll
        for (int i = 0; i < CH; ++i) magnitude += fabsf(f[k].f[i]);
      }
      fetch(q0 + sharers * 4);
      if (!finite1 || !isfinite(magnitude)) {
#pragma unroll
        for (int i = 0; i < CH; ++i)
          l4_nonfinite(s_gS, s_rows, q0, f1[i], gf1[i], [&](int at) { return __ldg(f2_row(at) + i); },
                       [&](int at, float v) { atomicAdd(g2_row(at) + i, v); });
        continue;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float g2[CH][4], total[CH];
#pragma unroll
        for (int p4 = 0; p4 < L4_BPX; p4 += 4) {
          const float4 t = *reinterpret_cast<const float4*>(&s_gS[q0 + k][p4]);
          const float g[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
          for (int j = 0; j < CH; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              gf1[j][p4 + i] = fmaf(g[i], f[k].f[j], gf1[j][p4 + i]);
              g2[j][i] = p4 == 0 ? g[i] * f1[j][i] : fmaf(g[i], f1[j][p4 + i], g2[j][i]);
            }
        }
#pragma unroll
        for (int j = 0; j < CH; ++j) total[j] = (g2[j][0] + g2[j][1]) + (g2[j][2] + g2[j][3]);
        l4_add_channels<CH>(g2_row(r[k]), total);
      }
    }
  }
  if (sharers > 1) {   // sum over the warps of the same channels, in their order
    __syncthreads();
    if (mine && share > 0) {
#pragma unroll
      for (int j = 0; j < CH; ++j)
#pragma unroll
        for (int px = 0; px < L4_BPX; ++px) s_gS[threadIdx.x + j * L4_BTHREADS][px] = gf1[j][px];
    }
    __syncthreads();
    if (mine && share == 0) {
      for (int k = 1; k < sharers; ++k)
#pragma unroll
        for (int j = 0; j < CH; ++j)
#pragma unroll
          for (int px = 0; px < L4_BPX; ++px) gf1[j][px] += s_gS[threadIdx.x + k * groups * 32 + j * L4_BTHREADS][px];
    }
  }
  if (mine && share == 0) {
#pragma unroll
    for (int px = 0; px < L4_BPX; ++px)
      if (h0 + px / L4_BT < H1 && w0 + px % L4_BT < W1) {
        float* const dst = gF1 + tile + ((size_t)(px / L4_BT) * W1 + px % L4_BT) * C + c;
        float sum[CH];
#pragma unroll
        for (int j = 0; j < CH; ++j) sum[j] = gf1[j][px];
        if (parts > 1) {
          l4_add_channels<CH>(dst, sum);
        } else {
#pragma unroll
          for (int j = 0; j < CH; ++j) dst[j] = sum[j];
        }
      }
  }
}

// The tiles that the kernel above leaves out: four warps with 2 x 2 pixels each, together at the levels where the box of their windows has at
// most L4_BMAX positions, else one pixel at a time.  Same grid.
constexpr int L4_APART = 128, L4_APART_WARPS = L4_APART / 32;
static_assert(L4_APART_WARPS * L4_PX == L4_BPX, "2 x 2 pixels a warp");

template <int NCH>
__global__ void __launch_bounds__(L4_APART, 4)
lookup4d_backward_apart_kernel(const float* __restrict__ F1, Lookup4dLevels lv, const float* __restrict__ coords,
                               const float* __restrict__ gout, float* __restrict__ gF1, int H1, int W1, int C, int radius,
                               int levels, int limit, float scale) {
  follow_previous_kernel();
  __shared__ L4Tile s_tile;
  __shared__ float s_gS[L4_APART_WARPS][L4_PX][L4_BMAX];
  __shared__ float s_g[L4_WIN * L4_WIN][L4_BPX + 1];
  __shared__ int s_rows[L4_APART_WARPS][L4_BMAX];

  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int b = blockIdx.z, N1 = H1 * W1, win = 2 * radius + 1;
  const int tiles_x = (W1 + L4_BT - 1) / L4_BT;
  const int h0 = (int)(blockIdx.x / tiles_x) * L4_BT, w0 = (int)(blockIdx.x % tiles_x) * L4_BT;
  if (l4_tile(s_tile, coords, lv, levels, b, h0, w0, H1, W1, radius, limit)) return;
  const int ph = h0 + 2 * (w >> 1), pw = w0 + 2 * (w & 1);
  const int mh = ph + ((lane >> 1) & 1), mw = pw + (lane & 1);
  const bool mine = lane < L4_PX && mh < H1 && mw < W1;
  const unsigned mask = __ballot_sync(0xffffffffu, mine);
  const int px0 = 2 * (w >> 1) * L4_BT + 2 * (w & 1);   // this warp's first pixel of the tile; pixel px: + px/2 rows, + px%2

  L4Quad f1[L4_PX][NCH], gf1[L4_PX][NCH];
#pragma unroll
  for (int px = 0; px < L4_PX; ++px)
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) {
      const int c = ch * 128 + lane * 4;
      const size_t p = (size_t)b * N1 + (size_t)(ph + px / 2) * W1 + pw + px % 2;
      const bool ok = ((mask >> px) & 1u) && c < C;
      f1[px][ch] = l4_load(F1 + (ok ? p * C + c : 0), ok);
      gf1[px][ch] = L4Quad{0ull, 0ull};
    }

  for (int level = 0; level < levels; ++level) {
    const int H2 = lv.H2[level], W2 = lv.W2[level];
    const float* F2b = lv.f2[level] + (size_t)b * H2 * W2 * C;
    float* G2b = lv.g2[level] + (size_t)b * H2 * W2 * C;

    __syncthreads();   // the previous level's s_g is no longer read
    for (int i = threadIdx.x; i < win * win * L4_BPX; i += L4_APART) {
      const int o = i / L4_BPX, pp = i % L4_BPX, h = h0 + pp / L4_BT, x = w0 + pp % L4_BT;
      s_g[o][pp] = (h < H1 && x < W1)
                       ? __ldg(gout + (((size_t)b * levels + level) * win * win + o) * N1 + (size_t)h * W1 + x)
                       : 0.f;
    }
    const L4Pixel geo = s_tile.geo[level][px0 + lane / 2 % 2 * L4_BT + lane % 2];
    __syncthreads();
    if (mask == 0) continue;

    const L4Box box = l4_box(geo, mask, radius, lane);
    if (l4_fits(box, L4_BMAX)) {
      l4_fill_rows(s_rows[w], box, H2, W2, lane);
      const int nq = box.bw * box.bh;
      for (int px = 0; px < L4_PX; ++px) {
        const L4Pixel g = s_tile.geo[level][px0 + px / 2 * L4_BT + px % 2];
        const bool live = (mask >> px) & 1u;
        for (int q = lane; q < nq; q += 32) {
          const int row = q / box.bw, i = box.ox + q - row * box.bw - (g.bx - radius), j = box.oy + row - (g.by - radius);
          s_gS[w][px][q] = live ? l4_position_gradient(g, i, j, s_g, px0 + px / 2 * L4_BT + px % 2, radius, H2, W2) * scale : 0.f;
        }
      }
      __syncwarp();
      l4_box_gradients<NCH, L4_PX>(f1, gf1, F2b, G2b, C, s_rows[w], nq, s_gS[w], 0, lane);
    } else {
      // motion boundaries: one pixel at a time, each over its own window.  All four pixels' positions are prepared together (a
      // pixel alone leaves lanes idle and waits on its own), a pixel's rows behind its gradients.  Windows scattered over
      // 2 x 55 x 128 at C = 256, radius 4, four levels: 1121 us with a preparation per pixel, 857 with this
      // one, 1058 against 1117 at uniformly scattered windows with tiles sorted out first.
      const int side = 2 * radius + 2, nq = side * side;
      for (int idx = lane; idx < L4_PX * nq; idx += 32) {
        const int px = idx / nq, q = idx - px * nq, j = q / side, i = q - j * side;
        const L4Pixel g = s_tile.geo[level][px0 + px / 2 * L4_BT + px % 2];
        const int x = g.bx - radius + i, y = g.by - radius + j;
        const bool live = (mask >> px) & 1u;
        const float v = live ? l4_position_gradient(g, i, j, s_g, px0 + px / 2 * L4_BT + px % 2, radius, H2, W2) * scale : 0.f;
        s_gS[w][px][q] = v;
        s_gS[w][px][L4_ALONE_ROWS + q] = __int_as_float(x >= 0 && x < W2 && y >= 0 && y < H2 && v != 0.f ? y * W2 + x : -1);
      }
      if (lane < L4_PX * L4_ALONE_PAD)   // a walk asks for up to L4_ALONE_PAD positions past the last
        s_gS[w][lane / L4_ALONE_PAD][L4_ALONE_ROWS + nq + lane % L4_ALONE_PAD] = __int_as_float(-1);
      __syncwarp();
#pragma unroll
      for (int px = 0; px < L4_PX; ++px)
        if ((mask >> px) & 1u)
          l4_box_gradients<NCH, 1>(f1, gf1, F2b, G2b, C, reinterpret_cast<const int*>(&s_gS[w][px][L4_ALONE_ROWS]), nq, s_gS[w], px,
                                   lane);
    }
    __syncwarp();
  }

#pragma unroll
  for (int px = 0; px < L4_PX; ++px)
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) {
      const int c = ch * 128 + lane * 4;
      if (((mask >> px) & 1u) && c < C) {
        const size_t p = (size_t)b * N1 + (size_t)(ph + px / 2) * W1 + pw + px % 2;
        *reinterpret_cast<ulonglong2*>(gF1 + p * C + c) = make_ulonglong2(gf1[px][ch].lo, gf1[px][ch].hi);
      }
    }
}

// Zeros for the reductions, all arrays in one launch (C is a multiple of 4 and the pointers are 16-byte aligned).
struct L4Clear {
  float* p[LOOKUP_MAX_LEVELS + 1];
  size_t quads[LOOKUP_MAX_LEVELS + 1];
};
__global__ void __launch_bounds__(256) lookup4d_clear_kernel(L4Clear clear) {
  follow_previous_kernel();
  float4* const p = reinterpret_cast<float4*>(clear.p[blockIdx.y]);
  const size_t n = clear.quads[blockIdx.y];
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (size_t)gridDim.x * 256) p[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

static Lookup4dLevels make_levels(const Lookup4dDims& d, const float* const* F2, float* const* gF2) {
  Lookup4dLevels lv{};
  for (int l = 0; l < d.levels; ++l) {
    lv.f2[l] = F2[l];
    lv.g2[l] = gF2 ? gF2[l] : nullptr;
    lv.H2[l] = d.H2[l];
    lv.W2[l] = d.W2[l];
  }
  return lv;
}

static unsigned l4_tiles(const Lookup4dDims& d) {
  return (unsigned)((d.W1 + L4_TW - 1) / L4_TW) * (unsigned)((d.H1 + L4_TH - 1) / L4_TH);
}

cudaError_t launch_lookup4d_forward(const Lookup4dDims& d, const float* F1, const float* const* F2,
                                    const float* coords, float* out, float scale, cudaStream_t stream) {
  const Lookup4dLevels lv = make_levels(d, F2, nullptr);
  const dim3 grid(l4_tiles(d), d.levels, d.B);
#define SFB_L4_FWD(NQ, LP)                                                                                                             \
  launch_next((d.C == NQ * 4 * LP ? lookup4d_forward_kernel<NQ, LP, true> : lookup4d_forward_kernel<NQ, LP, false>), grid, L4_THREADS, 0, stream, \
      F1, lv, coords, out, d.H1, d.W1, d.C, d.radius, d.levels, scale)
  switch ((d.C + 63) / 64) {
    case 1: SFB_L4_FWD(1, 16); break;
    case 2: SFB_L4_FWD(2, 16); break;
    case 3: SFB_L4_FWD(3, 16); break;
    case 4: SFB_L4_FWD(4, 16); break;
    case 5: case 6: SFB_L4_FWD(3, 32); break;
    case 7: case 8: SFB_L4_FWD(4, 32); break;
    default: return cudaErrorInvalidValue;
  }
#undef SFB_L4_FWD
  return cudaGetLastError();
}

int lookup4d_backward_launches(const Lookup4dDims& d) { return l4_tile_limit(d.radius) > 0 ? 3 : 2; }

cudaError_t launch_lookup4d_backward(const Lookup4dDims& d, const float* F1, const float* const* F2,
                                     const float* coords, const float* gout, float* gF1, float* const* gF2,
                                     float scale, cudaStream_t stream) {
  const Lookup4dLevels lv = make_levels(d, F2, gF2);
  const int limit = l4_tile_limit(d.radius), parts = l4_parts(d.levels);
  L4Clear clear{};
  int arrays = 0;
  size_t largest = 0;
  const auto add = [&](float* p, size_t quads) {
    clear.p[arrays] = p;
    clear.quads[arrays++] = quads;
    largest = std::max(largest, quads);
  };
  for (int l = 0; l < d.levels; ++l) add(gF2[l], (size_t)d.B * d.H2[l] * d.W2[l] * (d.C / 4));
  if (limit > 0 && parts > 1) add(gF1, (size_t)d.B * d.H1 * d.W1 * (d.C / 4));
  launch_next(lookup4d_clear_kernel, dim3((unsigned)std::min<size_t>((largest + 1023) / 1024, 148 * 8), arrays), 256, 0, stream, clear);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return err;
  const dim3 grid((unsigned)((d.W1 + L4_BT - 1) / L4_BT) * (unsigned)((d.H1 + L4_BT - 1) / L4_BT), 1, d.B);   // per tile
  if (limit > 0) {
    const dim3 whole(grid.x, (unsigned)((d.C + L4_BCH - 1) / L4_BCH * parts), d.B);
    launch_next(d.C > 32 ? lookup4d_backward_kernel<2> : lookup4d_backward_kernel<1>, whole, L4_BTHREADS, 0, stream, F1, lv, coords, gout, gF1, d.H1, d.W1, d.C, d.radius, d.levels, limit, scale);
    err = cudaGetLastError();
    if (err != cudaSuccess) return err;
  }
  // launch_after: 1 x 30 x 40 pixels, windows scattered, 257 us; launched early, blocks lie two to an SM and take 319
#define SFB_L4_BWD(NCH)                                                                                                                 \
  launch_after(lookup4d_backward_apart_kernel<NCH>, grid, L4_APART, 0, stream, F1, lv, coords, gout, gF1, d.H1, d.W1, d.C, d.radius, d.levels, \
              limit, scale)
  switch ((d.C + 127) / 128) {
    case 1: SFB_L4_BWD(1); break;
    case 2: SFB_L4_BWD(2); break;
    case 3: SFB_L4_BWD(3); break;
    case 4: SFB_L4_BWD(4); break;
    default: return cudaErrorInvalidValue;
  }
#undef SFB_L4_BWD
  return cudaGetLastError();
}

}  // namespace sfb
