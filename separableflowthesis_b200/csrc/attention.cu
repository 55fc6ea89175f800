// Attention weights of the separation (stencil kernels on the FP32 pipes, no tensor cores):
//   A = softmax_over_d( Conv3d(2 -> Kc, 3x3x3, padding 1)(X) )       core/corr.py:437-442, core/sepflow.py:59-60
// on the channels-first tensors X (B, 2, D, H1, W1) -> A (B, Kc, D, H1, W1), and its backward.
//
// The stencil kernels give one thread one image-1 pixel (h, w) and let it walk the displacement axis d, or a piece of it, so
// that a warp reads 32 neighbouring pixels of a (channel, d) plane per load.  The 3x3x3 stencil is applied in "scatter" form:
// the 3x3 neighbourhood of the plane that was just loaded is added into the three outputs (d-1, d, d+1) it belongs to, which
// are kept in registers.  The softmax over d and its backward are kernels of their own that share a pixel's column among
// warps (short columns: the softmax ends the walk).
//
// Two things decide the speed of such a walk, and both are handled explicitly:
//  * latency: a thread needs plane e+1 only after it is done with plane e, so planes are fetched a few ahead: the tiled form
//    (calls with a status word) into a ring of tiles that a block shares, see PlaneFeed; the gather form, every thread its
//    own neighbourhoods with cp.async, see PlaneRing.
//  * operand bandwidth: all threads multiply by the same 54*Kc filter weights.  Reading them from shared memory
//    costs a 32-lane register write per weight, more than the FMA they feed; instead the weights of the (up to
//    four) channels being processed are staged in __constant__ memory, where an FMA reads them as an operand.
//
// A launch works through a list of jobs: the two modules of a level, or those of all levels of a pyramid.  A module is a compile-time
// index into the constant memory, so every walk is there once per module.
//
//   forward     : logits -> A (the stencil kernel parks the raw logits in A, where they are normalised in place)
//   logit grads : gL = A * (gA - sum_d gA*A), in place over gA; per-block sums of gL for the bias gradient
//   input grads : gX = transposed stencil of gL (+ an optional addend: the direct gradient of the max/avg channels)
//   weight grads: gW[k,c,tap] = sum X(shifted by tap) * gL, per-block partial sums, reduced in a fixed order by
//                 a second kernel (bit-reproducible; no floating-point atomics)
#include <climits>
#include <cmath>
#include <mutex>
#include <type_traits>

#include "kernels.h"
#include "sm100_primitives.cuh"

namespace sfb {

constexpr int AT_THREADS = 128;
constexpr int AT_TAPS = 27;
constexpr int AT_KC = 4;  // channels per launch of the forward / logit-gradient kernels and per constant-memory stage

// Filter weights of the channels the running kernel works on, of both modules, in the order in which the kernel reads them, so that
// weights which are used together lie in one 16-byte word (stage_weights_kernel).  n = 3 * th + tw is the neighbour a value comes
// from: of the forward's tap (th, tw), of the input gradients' tap (2 - th, 2 - tw).
constexpr int AT_WEIGHTS = 3 * AT_KC * 20;
__constant__ float4 c_att_weights[2 * AT_WEIGHTS / 4];
__host__ __device__ constexpr int forward_weight(int k, int c, int td, int n) { return ((td * 2 + c) * 9 + n) * AT_KC + k; }
__host__ __device__ constexpr int input_grad_weight(int k, int c, int td, int n) { return (td * AT_KC + k) * 20 + n * 2 + c; }
static_assert(forward_weight(AT_KC - 1, 1, 2, 8) < AT_WEIGHTS && input_grad_weight(AT_KC - 1, 1, 2, 8) < AT_WEIGHTS, "weights staged");
template <int MODULE>
__device__ __forceinline__ float att_weight(int i) { return reinterpret_cast<const float*>(c_att_weights)[MODULE * AT_WEIGHTS + i]; }

struct StageWeights {
  const float* weight[2];   // (k, c, td, th, tw), `channels` of them; null where no job uses the module
  int channels;
  bool input_grad;
};
__device__ float g_att_weights[2 * AT_WEIGHTS];   // on their way into constant memory
__global__ void __launch_bounds__(AT_KC * 2 * AT_TAPS) stage_weights_kernel(const __grid_constant__ StageWeights s) {
  follow_previous_kernel();
  const int m = blockIdx.x, i = threadIdx.x, k = i / (2 * AT_TAPS), c = i / AT_TAPS & 1, tap = i % AT_TAPS, td = tap / 9, n = tap % 9;
  if (s.weight[m] == nullptr || k >= s.channels) return;
  g_att_weights[m * AT_WEIGHTS + (s.input_grad ? input_grad_weight(k, c, td, 8 - n) : forward_weight(k, c, td, n))] = __ldg(s.weight[m] + i);
}

// Jobs of a launch: blocks first[j] .. first[j+1]-1 belong to job j.
struct JobBlocks {
  int first[MAX_ATTENTION_JOBS + 1];
};
__device__ __forceinline__ int job_of(const JobBlocks& jb, int block) {
  int job = 0;
#pragma unroll
  for (int j = 1; j < MAX_ATTENTION_JOBS; ++j) job = block >= jb.first[j] ? j : job;
  return job;
}
// f(integral constant) with the job's module
template <class F>
__device__ __forceinline__ void by_module(int module, F&& f) {
  if (module == 0) f(std::integral_constant<int, 0>{});
  else f(std::integral_constant<int, 1>{});
}

// Offsets of the 3x3 neighbourhood of pixel (h, w) inside a plane, and which of them exist.
struct Neighbourhood {
  int off[9];
  unsigned valid;  // bit (3*th + tw)
  __device__ Neighbourhood(int h, int w, int H1, int W1) {
    valid = 0;
#pragma unroll
    for (int th = 0; th < 3; ++th)
#pragma unroll
      for (int tw = 0; tw < 3; ++tw) {
        const int hh = h + th - 1, ww = w + tw - 1;
        off[3 * th + tw] = (th - 1) * W1 + (tw - 1);
        if (hh >= 0 && hh < H1 && ww >= 0 && ww < W1) valid |= 1u << (3 * th + tw);
      }
  }
  __device__ bool has(int nb) const { return (valid >> nb) & 1u; }
};

// ---- per-thread prefetch ring -------------------------------------------------------------------------
// ring[stage][value][thread]: a thread copies the NV values it will need for plane e into stage e % STAGES with
// 4-byte cp.async (zero fill for values that do not exist) and reads them back itself STAGES-1 planes later.
__device__ __forceinline__ void cp_async4(float* smem_dst, const float* src, bool valid) {
  const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem_dst);
  const int bytes = valid ? 4 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int NV, int STAGES>
struct PlaneRing {
  float* base;  // this thread's column: value v of stage s at base[(s * NV + v) * AT_THREADS]
  __device__ PlaneRing(float* smem) : base(smem + threadIdx.x) {}
  __device__ float* slot(int stage, int v) const { return base + (stage * NV + v) * AT_THREADS; }
  static constexpr size_t bytes() { return (size_t)STAGES * NV * AT_THREADS * sizeof(float); }
};

// ---- forward: logits --------------------------------------------------------------------------------------
// The walk along d is cut into pieces of `dc` displacements, one block each (a piece re-reads one plane on either
// side): a walk is a serial chain, and a single 55 x 128 image has 56 pixel tiles for 148 SMs.  A logit is the same
// sum in the same order whatever the cut.  The softmax has a kernel of its own (attention_softmax_kernel), which
// keeps the online maximum, its branch and its exponential out of this issue-bound loop; only a column of at most
// AT_SOFT_MAX displacements walked in one piece is normalised at its end (SOFT, softmax_column): there the launch and the
// idle warps of the other kernel cost more than the exponentials (8 x 47 x 156, four channels, D = 5, 8 and 16: 30, 36 and 44 us
// with it, 21, 26 and 37 without).
// Gather form: grid of ceil(N1/128) * B * pieces blocks per job, block 128.  Channels k0 .. k0+KC-1 of Kc, weights in c_att_weights.
constexpr int FW_STAGES = 4;
constexpr int AT_SOFT_MAX = 16;

// Softmax of a pixel's column of D <= AT_SOFT_MAX logits, which the same thread has stored, in place.  The sum is formed as
// attention_softmax_kernel forms it (SM_GROUPS partial sums of every SM_GROUPS-th value, then those in order), so that a
// pixel's weights are the same whichever of the two its launch takes.
constexpr int SM_GROUPS = 8;
__device__ __forceinline__ void softmax_column(float* col, int D, size_t plane) {
  float v[AT_SOFT_MAX], m = -INFINITY, l = 0.f;
#pragma unroll
  for (int d = 0; d < AT_SOFT_MAX; ++d) v[d] = d < D ? col[d * plane] : -INFINITY;
#pragma unroll
  for (int d = 0; d < AT_SOFT_MAX; ++d) m = fmaxf(m, v[d]);
#pragma unroll
  for (int g = 0; g < SM_GROUPS; ++g) {
    float s = 0.f;
#pragma unroll
    for (int d = g; d < AT_SOFT_MAX; d += SM_GROUPS) {
      if (d < D) {
        v[d] = __expf(v[d] - m);
        s += v[d];
      }
    }
    l += s;
  }
  const float inv = 1.f / l;
#pragma unroll
  for (int d = 0; d < AT_SOFT_MAX; ++d)
    if (d < D) col[d * plane] = v[d] * inv;
}

struct LogitsJobs {
  JobBlocks blocks;
  struct Job {
    const float* x;
    long long x_sb;
    const float* bias;
    float* a;
    int D, dc, module;
  } j[MAX_ATTENTION_JOBS];
};

template <int KC, int MODULE>
__device__ __forceinline__ void logits_walk_gather(const LogitsJobs::Job& job, float* ring_mem, int Kc, int k0, int b, int d0, int p,
                                                   int H1, int W1) {
  const int N1 = H1 * W1, D = job.D, dc = job.dc;
  const int d1 = min(d0 + dc, D);                              // this block's logits: d0 <= d < d1
  const int e0 = max(d0 - 1, 0), e1 = min(d1 + 1, D);          // the planes they need
  const int h = p / W1, w = p - h * W1;
  const Neighbourhood nb(h, w, H1, W1);
  const PlaneRing<18, FW_STAGES> ring(ring_mem);
  const size_t plane = (size_t)N1;
  const float* x0 = job.x + (size_t)b * job.x_sb + p;       // channel 0, plane 0
  const float* x1 = x0 + (size_t)D * plane;         // channel 1
  float* out = job.a + ((size_t)b * Kc + k0) * D * plane + p;

  auto issue = [&](int e) {  // neighbourhoods of plane e (both channels) -> stage e % FW_STAGES
    if (e < e1) {
      const int s = e % FW_STAGES;
      const float* q0 = x0 + (size_t)e * plane;
      const float* q1 = x1 + (size_t)e * plane;
#pragma unroll
      for (int n = 0; n < 9; ++n) {
        cp_async4(ring.slot(s, n), nb.has(n) ? q0 + nb.off[n] : q0, nb.has(n));
        cp_async4(ring.slot(s, 9 + n), nb.has(n) ? q1 + nb.off[n] : q1, nb.has(n));
      }
    }
    cp_async_commit();
  };

  float bk[KC], acc[3][KC];
#pragma unroll
  for (int k = 0; k < KC; ++k) {
    bk[k] = __ldg(job.bias + k0 + k);
    acc[0][k] = acc[1][k] = acc[2][k] = bk[k];
  }
  auto emit = [&](int d) {  // logit d is complete in acc[0]
#pragma unroll
    for (int k = 0; k < KC; ++k) out[((size_t)k * D + d) * plane] = acc[0][k];
  };
#pragma unroll
  for (int s = 0; s < FW_STAGES - 1; ++s) issue(e0 + s);
  for (int e = e0; e < e1; ++e) {  // plane e feeds logits e+1 (tap td=0), e (td=1), e-1 (td=2)
    issue(e + FW_STAGES - 1);
    cp_async_wait<FW_STAGES - 1>();
    const int s = e % FW_STAGES;
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int n = 0; n < 9; ++n) {
        const float xv = *ring.slot(s, c * 9 + n);
#pragma unroll
        for (int k = 0; k < KC; ++k) {
          acc[2][k] = fmaf(xv, att_weight<MODULE>(forward_weight(k, c, 0, n)), acc[2][k]);
          acc[1][k] = fmaf(xv, att_weight<MODULE>(forward_weight(k, c, 1, n)), acc[1][k]);
          acc[0][k] = fmaf(xv, att_weight<MODULE>(forward_weight(k, c, 2, n)), acc[0][k]);
        }
      }
    if (e > d0) emit(e - 1);
#pragma unroll
    for (int k = 0; k < KC; ++k) { acc[0][k] = acc[1][k]; acc[1][k] = acc[2][k]; acc[2][k] = bk[k]; }
  }
  if (d1 == D) emit(D - 1);
}

// SOFT: the walks end with the softmax of their columns.
template <int KC>
__device__ __forceinline__ void softmax_columns(const LogitsJobs::Job& job, int Kc, int k0, int b, int p, size_t plane) {
  float* const out = job.a + ((size_t)b * Kc + k0) * job.D * plane + p;
#pragma unroll 1
  for (int k = 0; k < KC; ++k) softmax_column(out + (size_t)k * job.D * plane, job.D, plane);
}

template <int KC, bool SOFT>
__global__ void __launch_bounds__(AT_THREADS)
attention_logits_kernel(const __grid_constant__ LogitsJobs jobs, int Kc, int k0, int B, int H1, int W1) {
  follow_previous_kernel();
  __shared__ float ring_mem[FW_STAGES * 18 * AT_THREADS];
  const int ji = job_of(jobs.blocks, blockIdx.x);
  const LogitsJobs::Job& job = jobs.j[ji];
  const int N1 = H1 * W1, pb = (N1 + AT_THREADS - 1) / AT_THREADS;
  const int r = blockIdx.x - jobs.blocks.first[ji], z = r / pb;
  const int p = (r - z * pb) * AT_THREADS + threadIdx.x, b = z % B, d0 = (z / B) * job.dc;
  if (p >= N1) return;
  by_module(job.module, [&](auto m) { logits_walk_gather<KC, decltype(m)::value>(job, ring_mem, Kc, k0, b, d0, p, H1, W1); });
  if (SOFT) softmax_columns<KC>(job, Kc, k0, b, p, (size_t)N1);
}

// ---- logits, pixel tiles in shared memory -------------------------------------------------------------------
// A block owns a tile of AT_TW x AT_TILE_ROWS image-1 pixels; a thread does AT_ROWS pixels of a column, one below the other.  The tile of both input
// channels with its one-pixel halo comes in plane by plane through a ring of stages (PlaneFeed), a few planes ahead, and the threads read
// their neighbours from shared memory at constant offsets.  Pixels outside the image are zeros = the convolution's padding.
// A plane e adds to the outputs e - 1, e and e + 1: `older` (e - 1, complete after this plane), `newer` (e), and e + 1, which starts from the
// bias.  Each takes over from the one before it in its first multiply-add, so nothing is moved from plane to plane.
// Bound: FP32 issue.  Every pixel takes 54 multiply-adds per channel and plane with weights that are the same for all: they are operands from
// constant memory (uniform registers), which a multiply-add takes at full rate, where one with three registers takes 1.2 to 1.6 cycles and a
// packed one needs its weights moved to registers first (measured; 173 us instead of 118 for the logits below).  With one pixel to a thread
// multiply-adds were 40 % of the instructions; four share a loaded weight, 18 of 36 neighbours, addresses and barrier: 75 %.  Two or three
// pixels are within 5 % of it, with two channels slower (88 and 81 us instead of 69).  Logits of four levels: 1 x 55 x 128, four channels
// 51 -> 33 us, 4 x 55 x 128 168 -> 103, 1 x 135 x 240 427 -> 238, 3 x 47 x 155 (three channels, copies) 121 -> 85; 8 x 47 x 156, one level,
// two channels 96 -> 69.  The loop is 17 KB of instructions at four channels; what is left above the multiply-adds is fetching them, and barriers.
// grid of ceil(W1/32) * ceil(H1/16) * B * pieces blocks per job, block 128.
enum Feed : int { FEED_COPIES = 0, FEED_TMA = 1 };
constexpr int AT_TW = 32, AT_WARPS = AT_THREADS / 32;
constexpr int AT_BOX_W = AT_TW + 8;   // both forms: pixel w0 lies at column 4
constexpr int AT_ROWS = 4, AT_TILE_ROWS = AT_WARPS * AT_ROWS;   // of a thread, of a tile
constexpr int AT_STAGE_BYTES = 46 * 1024, AT_MAX_STAGES = 6;   // ring of a block

// A TMA destination in shared memory must be 128-byte aligned, so every stage is padded to a multiple of 128.
template <int NCH>
struct alignas(128) AttentionTileStage {
  float v[NCH][AT_TILE_ROWS + 2][AT_BOX_W];
};
constexpr int at_stages(size_t stage_bytes) {
  return AT_STAGE_BYTES / (int)stage_bytes < AT_MAX_STAGES ? AT_STAGE_BYTES / (int)stage_bytes : AT_MAX_STAGES;
}
template <int NCH>
struct AttentionTileSmem {
  static constexpr int STAGES = at_stages(sizeof(AttentionTileStage<NCH>));
  AttentionTileStage<NCH> x[STAGES];
  uint64_t full[STAGES];
  WaitCtl ctl;
};
static_assert(AttentionTileSmem<AT_KC>::STAGES >= 3, "planes in flight");

// A block of a job: its pixel tile, sample and piece of the walk.
struct TileBlock {
  int w0, h0, b, piece;
};
template <int ROWS>
__device__ __forceinline__ TileBlock tile_block(int r, int B, int H1, int W1) {
  const int tx = (W1 + AT_TW - 1) / AT_TW, tiles = tx * ((H1 + ROWS - 1) / ROWS);
  const int z = r / tiles, t = r - z * tiles, ty = t / tx;
  return TileBlock{(t - ty * tx) * AT_TW, ty * ROWS, z % B, z / B};
}
struct TileMaps {
  CUtensorMap m[MAX_ATTENTION_JOBS];
};

// Copies by all WARPS warps of a block of a plane's tile of NCH channels (`src`: channel 0; channels `channel_stride` apart, of which
// `channels` exist) with a halo of HALO pixels, a row per instruction.  Pixels and channels that do not exist become zeros.
template <int NCH, int ROWS, int WIDTH, int HALO, int WARPS>
__device__ __forceinline__ void copy_tile(float (&dst)[NCH][ROWS][WIDTH], const float* src, size_t channel_stride, int channels, int h0,
                                          int w0, int H1, int W1) {
  constexpr int COL0 = HALO != 0 ? 4 : 0;   // column of pixel w0
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, h = h0 - HALO + warp, w = w0 + lane;
  const float* const at = src + (ptrdiff_t)h * W1 + w;   // dereferenced where the pixel exists
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const bool column = c < channels && w < W1;
    const float* row = at + c * channel_stride;
#pragma unroll
    for (int r = 0; r < ROWS; r += WARPS, row += WARPS * W1) {
      if (ROWS % WARPS != 0 && r + WARPS > ROWS && r + warp >= ROWS) break;
      const bool ok = column && (unsigned)(h + r) < (unsigned)H1;
      cp_async4(&dst[c][r + warp][COL0 + lane], ok ? row : src, ok);
    }
  }
  if (HALO == 0) return;
  for (int i = threadIdx.x; i < NCH * ROWS * 2; i += WARPS * 32) {   // the columns on either side
    const int c = i / (ROWS * 2), r = (i >> 1) % ROWS, hh = h0 - HALO + r, ww = (i & 1) != 0 ? w0 + AT_TW : w0 - 1;
    const bool ok = c < channels && (unsigned)hh < (unsigned)H1 && (unsigned)ww < (unsigned)W1;
    cp_async4(&dst[c][r][(i & 1) != 0 ? COL0 + AT_TW : COL0 - 1], ok ? src + c * channel_stride + hh * W1 + ww : src, ok);
  }
}

// The planes e0 .. e0 + n_planes - 1 of a tile, channels channel0 .. channel0 + NCH - 1 of each, to all threads of a block.  Where W1 is a
// multiple of 4 and the tensor 16-byte aligned (TMA strides and addresses), a plane is ONE tiled TMA load, whose box starts 4 pixels
// to the left so that its x coordinate is a multiple of 16 bytes; else 4-byte cp.async copies by all threads.  One barrier per plane: it
// says that the plane is there for all, and that the stage of the one before has been read.  (With a warp of its own as the producer, and
// stages handed back through mbarriers, a fifth of the instructions were polls and a plane's copies took that warp longer than the others its
// arithmetic: 1 x 135 x 240 275 us instead of 250, 3 x 47 x 155 127 instead of 119, its weight gradients 290 instead of 151.)
template <int NCH, int FEED>
struct PlaneFeed {
  static constexpr int STAGES = AttentionTileSmem<NCH>::STAGES;
  AttentionTileSmem<NCH>& sm;
  const CUtensorMap* tm;
  const float* src;   // copies: first channel of the sample, plane e0; channels `channel_stride` apart, `channels` of them
  size_t channel_stride;
  int channels, e0, n_planes, channel0, H1, W1;
  TileBlock t;
  int* status;

  __device__ __forceinline__ void fetch(int i) {
    if constexpr (FEED == FEED_TMA) {
      if (threadIdx.x == 0 && i < n_planes) {
        const int s = i % STAGES;
        mbar_expect_tx(&sm.full[s], sizeof(sm.x[s].v));
        tma_load_5d(sm.x[s].v, tm, &sm.full[s], t.w0 - 4, t.h0 - 1, e0 + i, channel0, t.b);
      }
    } else {
      if (i < n_planes)
        copy_tile<NCH, AT_TILE_ROWS + 2, AT_BOX_W, 1, AT_WARPS>(sm.x[i % STAGES].v, src + (size_t)i * H1 * W1, channel_stride, channels,
                                                                   t.h0, t.w0, H1, W1);
      cp_async_commit();   // a group per plane, also where there is none
    }
  }
  __device__ __forceinline__ void start() {
    for (int i = 0; i < STAGES - 1; ++i) fetch(i);
  }
  // Plane i, or null in all threads when a wait ran out.
  __device__ __forceinline__ const AttentionTileStage<NCH>* plane(int i) {
    if constexpr (FEED == FEED_TMA) {
      const bool ok = mbar_wait(&sm.full[i % STAGES], (i / STAGES) & 1u, &sm.ctl, status, DEV_TIMEOUT_EPILOGUE);
      fence_proxy_async_smem();   // this thread's reads of the stage that is filled again are over
      if (!__syncthreads_and(ok)) return nullptr;
    } else {
      cp_async_wait<STAGES - 2>();
      __syncthreads();
    }
    fetch(i + STAGES - 1);
    return &sm.x[i % STAGES];
  }
};

template <int KC, int MODULE, int FEED>   // false: a wait ran out
__device__ __forceinline__ bool logits_walk_tiled(PlaneFeed<2, FEED>& feed, const LogitsJobs::Job& job, int Kc, int k0, int d0, int d1) {
  constexpr int R = AT_ROWS;
  const int D = job.D, H1 = feed.H1, W1 = feed.W1, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = feed.t.h0 + warp * R, w = feed.t.w0 + lane;
  const int rows = w < W1 ? min(R, H1 - h) : 0;   // of this thread; may be <= 0
  const bool warp_has_rows = h < H1;
  const size_t plane = (size_t)H1 * W1;
  float* const out = job.a + ((size_t)feed.t.b * Kc + k0) * D * plane;   // the same for the whole block
  const uint32_t p = rows > 0 ? (uint32_t)(h * W1 + w) : 0u;

  float bk[KC], older[KC][R], newer[KC][R];
#pragma unroll
  for (int k = 0; k < KC; ++k) {
    bk[k] = __ldg(job.bias + k0 + k);
#pragma unroll
    for (int r = 0; r < R; ++r) older[k][r] = newer[k][r] = bk[k];
  }
  auto emit = [&](int d) {
#pragma unroll
    for (int k = 0; k < KC; ++k)
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (r < rows) (out + ((size_t)k * D + d) * plane + r * W1)[p] = older[k][r];
  };
  for (int i = 0; i < feed.n_planes; ++i) {
    const int e = feed.e0 + i;
    const auto* stage = feed.plane(i);
    if (stage == nullptr) return false;
    if (!warp_has_rows) continue;
    float x[2][R + 2][3];
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int r = 0; r < R + 2; ++r)
#pragma unroll
        for (int j = 0; j < 3; ++j) x[c][r][j] = stage->v[c][warp * R + r][lane + 3 + j];
    auto taps = [&](auto td, float (&a)[KC][R], auto&& from) {   // a = from + taps
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int n = 0; n < 9; ++n)
#pragma unroll
          for (int k = 0; k < KC; ++k) {
            const float wt = att_weight<MODULE>(forward_weight(k, c, decltype(td)::value, n));
#pragma unroll
            for (int r = 0; r < R; ++r) a[k][r] = fmaf(x[c][r + n / 3][n % 3], wt, c == 0 && n == 0 ? from(k, r) : a[k][r]);
          }
    };
    if (e > d0) {
      taps(std::integral_constant<int, 2>{}, older, [&](int k, int r) { return older[k][r]; });
      emit(e - 1);
    }
    if (e >= d0 && e < d1) taps(std::integral_constant<int, 1>{}, older, [&](int k, int r) { return newer[k][r]; });
    if (e + 1 < d1) taps(std::integral_constant<int, 0>{}, newer, [&](int k, int) { return bk[k]; });
  }
  if (d1 == D && warp_has_rows) emit(D - 1);
  return true;
}

template <int KC, bool SOFT, int FEED>
__global__ void __launch_bounds__(AT_THREADS)
attention_logits_tiled_kernel(const __grid_constant__ TileMaps maps, const __grid_constant__ LogitsJobs jobs, int Kc, int k0, int B,
                              int H1, int W1, int* status) {
  if (!cta_has_work(status)) return;
  __shared__ __align__(128) AttentionTileSmem<2> sm;
  const int ji = job_of(jobs.blocks, blockIdx.x);
  const LogitsJobs::Job& job = jobs.j[ji];
  const TileBlock t = tile_block<AT_TILE_ROWS>(blockIdx.x - jobs.blocks.first[ji], B, H1, W1);
  const int d0 = t.piece * job.dc, d1 = min(d0 + job.dc, job.D);
  const int e0 = max(d0 - 1, 0), n_planes = min(d1 + 1, job.D) - e0;
  const size_t plane = (size_t)H1 * W1;
  PlaneFeed<2, FEED> feed{sm, &maps.m[ji], job.x + (size_t)t.b * job.x_sb + e0 * plane, job.D * plane, 2, e0, n_planes, 0, H1, W1, t, status};
  if (threadIdx.x == 0) {
    if (FEED == FEED_TMA) {
      for (int s = 0; s < feed.STAGES; ++s) mbar_init(&sm.full[s], 1);
      prefetch_tensormap(feed.tm);
    }
    wait_ctl_init(&sm.ctl, 0);
    fence_barrier_init();
  }
  __syncthreads();
  feed.start();
  bool ok = true;
  by_module(job.module, [&](auto m) { ok = logits_walk_tiled<KC, decltype(m)::value>(feed, job, Kc, k0, d0, d1); });
  if (SOFT && ok) {
    const int warp = threadIdx.x >> 5, w = t.w0 + (threadIdx.x & 31);
    if (w < W1)
      for (int h = t.h0 + warp * AT_ROWS; h < min(t.h0 + (warp + 1) * AT_ROWS, H1); ++h) softmax_columns<KC>(job, Kc, k0, t.b, h * W1 + w, plane);
  }
  __syncthreads();
  if (wait_ctl_aborted(&sm.ctl)) {
    let_copies_land();
  }
}

// ---- softmax over d, in place -------------------------------------------------------------------------------
// A block owns 32 * VEC consecutive pixels of one (sample, channel); warp g takes displacements g, g + 8, ... and keeps its
// V = ceil(D / 8) values of VEC pixels in registers, so that every logit is read once and every weight written once (HBM-bound, all
// loads of a thread in flight together).  V = 0: any D, the values are read again in each of the three walks.  The
// order of the sums depends on D only.  grid of ceil(N1/(32*VEC)) * planes (= B * Kc) blocks per job, block 256.
// VEC: neighbouring pixels of a lane, moved by one access (planes of a multiple of VEC pixels, 16-byte aligned): with one, the
// accesses' addresses and the two exchanges between warps cost as much as the data.  Inference at four levels, both
// modules: 4 x 55 x 128 689 -> 678 us, 1 x 135 x 240 2384 -> 2357 (four pixels only up to V = 8: 682 and 2364).
constexpr int SM_THREADS = SM_GROUPS * 32;
struct SoftmaxJobs {
  JobBlocks blocks;
  float* a[MAX_ATTENTION_JOBS];
  int D[MAX_ATTENTION_JOBS];
};
template <int VEC> struct SoftmaxVec { float f[VEC]; };
template <int VEC>
__device__ __forceinline__ SoftmaxVec<VEC> load_pixels(const float* p) {
  SoftmaxVec<VEC> v;
  if constexpr (VEC == 4) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v.f[0] = t.x; v.f[1] = t.y; v.f[2] = t.z; v.f[3] = t.w;
  } else if constexpr (VEC == 2) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    v.f[0] = t.x; v.f[1] = t.y;
  } else {
    v.f[0] = *p;
  }
  return v;
}
template <int VEC>
__device__ __forceinline__ void store_pixels(float* p, const SoftmaxVec<VEC>& v) {
  if constexpr (VEC == 4) *reinterpret_cast<float4*>(p) = make_float4(v.f[0], v.f[1], v.f[2], v.f[3]);
  else if constexpr (VEC == 2) *reinterpret_cast<float2*>(p) = make_float2(v.f[0], v.f[1]);
  else *p = v.f[0];
}

template <int V, int VEC>
__global__ void __launch_bounds__(SM_THREADS, V == 0 ? 8 : (V * VEC <= 8 ? 6 : (V * VEC <= 20 ? 3 : 2)))
attention_softmax_kernel(const __grid_constant__ SoftmaxJobs jobs, int N1, unsigned pixel_blocks) {
  follow_previous_kernel();
  __shared__ SoftmaxVec<VEC> red[2][SM_GROUPS][32];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int ji = job_of(jobs.blocks, blockIdx.x), D = jobs.D[ji];
  const unsigned block = blockIdx.x - jobs.blocks.first[ji], row = block / pixel_blocks;
  const int p = ((int)(block - row * pixel_blocks) * 32 + lane) * VEC;
  const bool in = p < N1;
  float* base = jobs.a[ji] + (size_t)row * D * N1 + (in ? p : 0);
  constexpr int NV = V > 0 ? V : 1;
  SoftmaxVec<VEC> v[NV], m, l;
#pragma unroll
  for (int j = 0; j < VEC; ++j) m.f[j] = -INFINITY;
  if constexpr (V > 0) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int d = g + i * SM_GROUPS;
      if (in && d < D) {
        v[i] = load_pixels<VEC>(base + (size_t)d * N1);
      } else {
#pragma unroll
        for (int j = 0; j < VEC; ++j) v[i].f[j] = -INFINITY;
      }
    }
#pragma unroll
    for (int i = 0; i < V; ++i)
#pragma unroll
      for (int j = 0; j < VEC; ++j) m.f[j] = fmaxf(m.f[j], v[i].f[j]);
  } else {
    for (int d = g; d < D; d += SM_GROUPS) m.f[0] = fmaxf(m.f[0], in ? base[(size_t)d * N1] : 0.f);
  }
  red[0][g][lane] = m;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < SM_GROUPS; ++i) {
    const SoftmaxVec<VEC> other = red[0][i][lane];
#pragma unroll
    for (int j = 0; j < VEC; ++j) m.f[j] = fmaxf(m.f[j], other.f[j]);
  }
#pragma unroll
  for (int j = 0; j < VEC; ++j) l.f[j] = 0.f;
  if constexpr (V > 0) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      if (g + i * SM_GROUPS < D) {
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
          v[i].f[j] = __expf(v[i].f[j] - m.f[j]);
          l.f[j] += v[i].f[j];
        }
      }
    }
  } else {
    for (int d = g; d < D; d += SM_GROUPS) l.f[0] += __expf((in ? base[(size_t)d * N1] : 0.f) - m.f[0]);
  }
  red[1][g][lane] = l;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < VEC; ++j) l.f[j] = 0.f;
#pragma unroll
  for (int i = 0; i < SM_GROUPS; ++i) {
    const SoftmaxVec<VEC> other = red[1][i][lane];
#pragma unroll
    for (int j = 0; j < VEC; ++j) l.f[j] += other.f[j];
  }
  SoftmaxVec<VEC> inv;
#pragma unroll
  for (int j = 0; j < VEC; ++j) inv.f[j] = 1.f / l.f[j];
  if (!in) return;
  if constexpr (V > 0) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int d = g + i * SM_GROUPS;
      if (d < D) {
#pragma unroll
        for (int j = 0; j < VEC; ++j) v[i].f[j] *= inv.f[j];
        store_pixels<VEC>(base + (size_t)d * N1, v[i]);
      }
    }
  } else {
    for (int d = g; d < D; d += SM_GROUPS) base[(size_t)d * N1] = __expf(base[(size_t)d * N1] - m.f[0]) * inv.f[0];
  }
}

// Tensor map over a channels-first tensor (B, nch, D, H1, W1) whose samples are `sb` elements apart; the box is one
// plane's pixel tile of `box_ch` channels, with the stencil's halo or without.
static cudaError_t tile_map(CUtensorMap* tm, const float* x, long long sb, int nch, int box_ch, const AttentionDims& d, int rows,
                            bool halo) {
  const uint64_t N1 = (uint64_t)d.H1 * d.W1;
  const uint64_t dims[5] = {(uint64_t)d.W1, (uint64_t)d.H1, (uint64_t)d.D, (uint64_t)nch, (uint64_t)d.B};
  const uint64_t strides[4] = {(uint64_t)d.W1 * 4, N1 * 4, (uint64_t)d.D * N1 * 4, (uint64_t)sb * 4};
  const uint32_t box[5] = {(uint32_t)(halo ? AT_BOX_W : AT_TW), (uint32_t)(rows + (halo ? 2 : 0)), 1, (uint32_t)box_ch, 1};
  return encode_plain_map(tm, x, 5, dims, strides, box);
}
static bool tileable(const AttentionDims& d, const void* x, long long sb) {
  return d.W1 % 4 == 0 && sb % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
}

// ---- logit gradients (softmax backward), in place -------------------------------------------------------
// gL = A * (gA - sum_d gA*A).  A column is shared by G warps: warp g of them takes displacements g, g + G, ... and keeps its
// V = ceil(D / G) values of both arrays in registers, so that each is read once and all loads of a thread are in flight
// together (HBM-bound).  A block is max(G, 8) warps, so short columns give it 8 / G groups of 32 pixels of one (sample,
// channel).  V = 0: any D, both arrays read twice.  The order of the sums depends on D only.  Eight warps for every D
// took 66 us for the attention backward of 2 x 135 x 240 and four channels at D = 5 and, spilling at V = 32, 635 us at
// D = 135; 55 and 554 now.
// A block's sum of gL goes to its module's bias partials (Kc, rows).  grid of pixel_blocks * B * Kc blocks per job, block
// 32 * max(G, 8).
struct LogitGradJobs {
  JobBlocks blocks;
  struct Job {
    const float* a;
    float* g;
    float* partial;   // of the module
    int D, row0, rows;
  } j[MAX_ATTENTION_JOBS];
};
__host__ __device__ constexpr int lg_warps(int G) { return G > 8 ? G : 8; }
__host__ __device__ constexpr int lg_pixels(int G) { return lg_warps(G) / G * 32; }
template <int G, int V, int MIN_BLOCKS>
__global__ void __launch_bounds__(32 * lg_warps(G), MIN_BLOCKS)
attention_logit_grad_kernel(const __grid_constant__ LogitGradJobs jobs, int Kc, int N1, unsigned pixel_blocks) {
  follow_previous_kernel();
  const int ji = job_of(jobs.blocks, blockIdx.x);
  const LogitGradJobs::Job& job = jobs.j[ji];
  const float* __restrict__ const a = job.a;
  float* __restrict__ const g = job.g;
  const int D = job.D;
  const unsigned block = blockIdx.x - jobs.blocks.first[ji];
  constexpr int WARPS = lg_warps(G);
  __shared__ float red[WARPS][32];
  __shared__ float bred[WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, grp = warp % G;
  const unsigned row = block / pixel_blocks;   // sample * Kc + channel
  const unsigned pb = block - row * pixel_blocks;
  const int p = (int)pb * lg_pixels(G) + warp / G * 32 + lane;
  const bool in = p < N1;
  const size_t base = (size_t)row * D * N1 + (in ? p : 0);
  constexpr int NV = V > 0 ? V : 1;
  float gv[NV], av[NV];
  float s = 0.f;
  if constexpr (V > 0) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int d = grp + i * G;
      const bool ok = in && d < D;
      gv[i] = ok ? g[base + (size_t)d * N1] : 0.f;
      av[i] = ok ? __ldg(a + base + (size_t)d * N1) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < V; ++i) s = fmaf(gv[i], av[i], s);
  } else if (in) {
    for (int d = grp; d < D; d += G) s = fmaf(g[base + (size_t)d * N1], __ldg(a + base + (size_t)d * N1), s);
  }
  if constexpr (G > 1) {
    red[warp][lane] = s;
    __syncthreads();
    s = 0.f;
#pragma unroll
    for (int i = 0; i < G; ++i) s += red[warp - grp + i][lane];
  }
  float bsum = 0.f;
  if constexpr (V > 0) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int d = grp + i * G;
      if (in && d < D) {
        const float gl = av[i] * (gv[i] - s);
        g[base + (size_t)d * N1] = gl;
        bsum += gl;
      }
    }
  } else if (in) {
    for (int d = grp; d < D; d += G) {
      const float gl = __ldg(a + base + (size_t)d * N1) * (g[base + (size_t)d * N1] - s);
      g[base + (size_t)d * N1] = gl;
      bsum += gl;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) bsum += __shfl_xor_sync(0xffffffffu, bsum, o);
  if (lane == 0) bred[warp] = bsum;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < WARPS; ++i) t += bred[i];
    const unsigned k = row % Kc, b = row / Kc;
    job.partial[(size_t)k * job.rows + job.row0 + (size_t)b * pixel_blocks + pb] = t;
  }
}

// ---- input gradients -----------------------------------------------------------------------------------
// gX[c, d, h, w] = add[c, d, h, w] + sum_{k, td, th, tw} W[k, c, td, th, tw] * gL[k, d - td + 1, h - th + 1, w - tw + 1]
// Channels k0 .. k0+KC-1 (weights in c_att_weights); a later chunk adds to what the earlier ones stored.
// The walk is cut into pieces of `dc` displacements like the forward's.
// grid of ceil(N1/128) * B * pieces blocks per job, block 128, dynamic shared memory PlaneRing<9*KC, IG_STAGES>::bytes().
constexpr int IG_STAGES = 3;
struct InputGradJobs {
  JobBlocks blocks;
  struct Job {
    const float *gl, *add;
    long long add_sb;
    float* gx;
    int D, dc, module;
  } j[MAX_ATTENTION_JOBS];
};

template <int KC, int MODULE>
__device__ __forceinline__ void input_grad_walk_gather(const InputGradJobs::Job& job, float* ring_dyn, int accumulate, int Kc, int k0, int b,
                                                       int d0, int p, int H1, int W1) {
  const float* __restrict__ const gl = job.gl;
  const float* __restrict__ const add = k0 == 0 ? job.add : nullptr;
  const long long add_sb = job.add_sb;
  float* __restrict__ const gx = job.gx;
  const int N1 = H1 * W1, D = job.D, dc = job.dc;
  const int d1 = min(d0 + dc, D), e0 = max(d0 - 1, 0), e1 = min(d1 + 1, D);
  const int h = p / W1, w = p - h * W1;
  const Neighbourhood nb(h, w, H1, W1);
  const PlaneRing<9 * KC, IG_STAGES> ring(ring_dyn);
  const size_t plane = (size_t)N1;
  const float* g0 = gl + ((size_t)b * Kc + k0) * D * plane + p;
  float* o0 = gx + (size_t)b * 2 * D * plane + p;
  const float* ad = add != nullptr ? add + (size_t)b * add_sb + p : nullptr;

  auto issue = [&](int e) {
    if (e < e1) {
      const int s = e % IG_STAGES;
#pragma unroll
      for (int k = 0; k < KC; ++k) {
        const float* q = g0 + ((size_t)k * D + e) * plane;
#pragma unroll
        for (int n = 0; n < 9; ++n) cp_async4(ring.slot(s, k * 9 + n), nb.has(n) ? q + nb.off[n] : q, nb.has(n));
      }
    }
    cp_async_commit();
  };
  float acc[2][3];  // [c][output d = e-1, e, e+1]
#pragma unroll
  for (int c = 0; c < 2; ++c) acc[c][0] = acc[c][1] = acc[c][2] = 0.f;
  auto emit = [&](int d) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const size_t i = ((size_t)c * D + d) * plane;
      float v = acc[c][0];
      if (ad != nullptr) v += __ldg(ad + i);
      if (accumulate) v += o0[i];
      o0[i] = v;
    }
  };
#pragma unroll
  for (int s = 0; s < IG_STAGES - 1; ++s) issue(e0 + s);
  for (int e = e0; e < e1; ++e) {  // plane e of gL feeds gX planes e-1 (td=0), e (td=1), e+1 (td=2)
    issue(e + IG_STAGES - 1);
    cp_async_wait<IG_STAGES - 1>();
    const int s = e % IG_STAGES;
#pragma unroll
    for (int k = 0; k < KC; ++k)
#pragma unroll
      for (int n = 0; n < 9; ++n) {
        const float v = *ring.slot(s, k * 9 + n);
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int td = 0; td < 3; ++td)
            acc[c][td] = fmaf(v, att_weight<MODULE>(input_grad_weight(k, c, td, n)), acc[c][td]);
      }
    if (e > d0) emit(e - 1);
#pragma unroll
    for (int c = 0; c < 2; ++c) { acc[c][0] = acc[c][1]; acc[c][1] = acc[c][2]; acc[c][2] = 0.f; }
  }
  if (d1 == D) emit(D - 1);
}

template <int KC>
__global__ void __launch_bounds__(AT_THREADS)
attention_input_grad_kernel(const __grid_constant__ InputGradJobs jobs, int accumulate, int Kc, int k0, int B, int H1, int W1) {
  follow_previous_kernel();
  extern __shared__ float ring_dyn[];
  const int ji = job_of(jobs.blocks, blockIdx.x);
  const InputGradJobs::Job& job = jobs.j[ji];
  const int N1 = H1 * W1, pb = (N1 + AT_THREADS - 1) / AT_THREADS;
  const int r = blockIdx.x - jobs.blocks.first[ji], z = r / pb;
  const int p = (r - z * pb) * AT_THREADS + threadIdx.x, b = z % B, d0 = (z / B) * job.dc;
  if (p >= N1) return;
  by_module(job.module, [&](auto m) { input_grad_walk_gather<KC, decltype(m)::value>(job, ring_dyn, accumulate, Kc, k0, b, d0, p, H1, W1); });
}

// ---- weight gradients ----------------------------------------------------------------------------------
// gW[k, c, td, th, tw] = sum_{b, d, h, w} gL[k, d, h, w] * X[c, d + td - 1, h + th - 1, w + tw - 1]
// grid (ceil(N1/128) * B * pieces blocks per job, 2 * ceil(Kc/KW)), block 128: a thread owns input channel c and KW output channels;
// its KW*27 sums live in registers, every X value it reads feeds 3*KW of them.  A piece is `dc` planes of X.
// partial: of the module, (Kc * 2 * 27, rows), one column per block, so that the reduction reads consecutive values.
constexpr int WG_STAGES = 4;
struct WeightGradJobs {
  JobBlocks blocks;
  struct Job {
    const float* x;
    long long x_sb;
    const float* gl;
    float* partial;
    int D, dc, row0, rows;
  } j[MAX_ATTENTION_JOBS];
};

template <int KW>
__global__ void __launch_bounds__(AT_THREADS)
attention_weight_grad_kernel(const __grid_constant__ WeightGradJobs jobs, int Kc, int B, int H1, int W1) {
  follow_previous_kernel();
  const int ji = job_of(jobs.blocks, blockIdx.x);
  const WeightGradJobs::Job& job = jobs.j[ji];
  const float* __restrict__ const x = job.x;
  const float* __restrict__ const gl = job.gl;
  const long long x_sb = job.x_sb;
  const int D = job.D, dc = job.dc;
  constexpr int NV = 9 + KW;
  __shared__ float ring_mem[WG_STAGES * NV * AT_THREADS];
  __shared__ float red[(AT_THREADS / 32) * KW * AT_TAPS];
  const int N1 = H1 * W1, pb = (N1 + AT_THREADS - 1) / AT_THREADS;
  const int r = blockIdx.x - jobs.blocks.first[ji], z = r / pb;
  const int b = z % B, c = blockIdx.y & 1, k0 = (blockIdx.y >> 1) * KW;
  const int e0 = (z / B) * dc, e1 = min(e0 + dc, D);
  const size_t plane = (size_t)N1;
  const int p = (r - z * pb) * AT_THREADS + threadIdx.x;
  float acc[KW * AT_TAPS];  // [k][td][neighbour]
#pragma unroll
  for (int i = 0; i < KW * AT_TAPS; ++i) acc[i] = 0.f;
  if (p < N1) {
    const int h = p / W1, w = p - h * W1;
    const Neighbourhood nb(h, w, H1, W1);
    const PlaneRing<NV, WG_STAGES> ring(ring_mem);
    const float* xc = x + (size_t)b * x_sb + (size_t)c * D * plane + p;
    const float* g = gl + ((size_t)b * Kc + k0) * D * plane + p;
    auto issue = [&](int e) {  // X neighbourhood of plane e and gL of plane e+1
      if (e < e1) {
        const int s = e % WG_STAGES;
        const float* q = xc + (size_t)e * plane;
#pragma unroll
        for (int n = 0; n < 9; ++n) cp_async4(ring.slot(s, n), nb.has(n) ? q + nb.off[n] : q, nb.has(n));
#pragma unroll
        for (int k = 0; k < KW; ++k) {
          const bool ok = e + 1 < D && k0 + k < Kc;
          cp_async4(ring.slot(s, 9 + k), ok ? g + ((size_t)k * D + e + 1) * plane : g, ok);
        }
      }
      cp_async_commit();
    };
    float g_prev[KW], g_cur[KW], g_next[KW];
#pragma unroll
    for (int k = 0; k < KW; ++k) {
      g_prev[k] = (e0 > 0 && k0 + k < Kc) ? __ldg(g + ((size_t)k * D + e0 - 1) * plane) : 0.f;
      g_cur[k] = k0 + k < Kc ? __ldg(g + ((size_t)k * D + e0) * plane) : 0.f;
    }
#pragma unroll
    for (int s = 0; s < WG_STAGES - 1; ++s) issue(e0 + s);
    for (int e = e0; e < e1; ++e) {  // plane e of X meets gL at d = e+1 (td=0), e (td=1), e-1 (td=2)
      issue(e + WG_STAGES - 1);
      cp_async_wait<WG_STAGES - 1>();
      const int s = e % WG_STAGES;
      float v[9];
#pragma unroll
      for (int n = 0; n < 9; ++n) v[n] = *ring.slot(s, n);
#pragma unroll
      for (int k = 0; k < KW; ++k) g_next[k] = *ring.slot(s, 9 + k);
#pragma unroll
      for (int k = 0; k < KW; ++k)
#pragma unroll
        for (int n = 0; n < 9; ++n) {
          acc[k * AT_TAPS + n] = fmaf(g_next[k], v[n], acc[k * AT_TAPS + n]);
          acc[k * AT_TAPS + 9 + n] = fmaf(g_cur[k], v[n], acc[k * AT_TAPS + 9 + n]);
          acc[k * AT_TAPS + 18 + n] = fmaf(g_prev[k], v[n], acc[k * AT_TAPS + 18 + n]);
        }
#pragma unroll
      for (int k = 0; k < KW; ++k) { g_prev[k] = g_cur[k]; g_cur[k] = g_next[k]; }
    }
  }
  // reduce over the block; thread i < KW*27 then holds column (k, td, n) and stores it at [k0 + k][c][td*9 + n]
#pragma unroll
  for (int i = 0; i < KW * AT_TAPS; ++i) {
    float s = acc[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    acc[i] = s;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
#pragma unroll
    for (int i = 0; i < KW * AT_TAPS; ++i) red[warp * KW * AT_TAPS + i] = acc[i];
  }
  __syncthreads();
  const size_t rows = job.rows;
  float* dst = job.partial + job.row0 + r;
  for (int i = threadIdx.x; i < KW * AT_TAPS; i += AT_THREADS) {
    const int k = i / AT_TAPS, t = i - k * AT_TAPS;
    if (k0 + k >= Kc) continue;
    float s = 0.f;
#pragma unroll
    for (int wv = 0; wv < AT_THREADS / 32; ++wv) s += red[wv * KW * AT_TAPS + i];
    dst[(((size_t)(k0 + k) * 2 + c) * AT_TAPS + t) * rows] = s;
  }
}

// out[i] = sum over rows of partial[i][row], for the weight and bias gradients of both modules in one launch.  One block per column:
// thread t adds rows t, t + 256, ... in order, then the 256 partial sums are combined in a fixed tree, so the result does not depend on
// scheduling (bit-reproducible).
constexpr int RP_THREADS = 256, RP_SUMS = 4;
struct PartialSums {
  const float* partial[RP_SUMS];
  float* out[RP_SUMS];
  int rows[RP_SUMS], first[RP_SUMS + 1];   // blocks first[i] .. first[i+1]-1
};
__global__ void __launch_bounds__(RP_THREADS)
attention_reduce_partials_kernel(const __grid_constant__ PartialSums sums) {
  follow_previous_kernel();
  __shared__ float red[RP_THREADS];
  int j = 0;
#pragma unroll
  for (int i = 1; i < RP_SUMS; ++i) j = (int)blockIdx.x >= sums.first[i] ? i : j;
  const int rows = sums.rows[j], i = blockIdx.x - sums.first[j];
  const float* __restrict__ const partial = sums.partial[j];
  float s = 0.f;
  for (int r = threadIdx.x; r < rows; r += RP_THREADS) s += __ldg(partial + (size_t)i * rows + r);
  red[threadIdx.x] = s;
  __syncthreads();
#pragma unroll
  for (int o = RP_THREADS / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) sums.out[j][i] = red[0];
}

// ---- input and weight gradients, pixel tiles in shared memory ---------------------------------------------
// Same arithmetic as the two gather kernels above with the tile scheme of attention_logits_tiled_kernel.
// Input gradients: the stage holds the tile (with halo) of the KC logit-gradient channels of one plane.  Bound like the logits.
// 8 x 47 x 156, two channels, one level: 122 -> 82 us; 3 x 47 x 155, three channels, four levels (copies) 157 -> 98; 8 x 135 x 240, four
// channels 1.76 -> 1.42 ms; 2 x 48 x 64, two channels, four levels 19 -> 13.
template <int KC, int MODULE, int FEED>
__device__ __forceinline__ void input_grad_walk_tiled(PlaneFeed<KC, FEED>& feed, const InputGradJobs::Job& job, int accumulate, int k0,
                                                      int d0, int d1) {
  constexpr int R = AT_ROWS;
  const int D = job.D, H1 = feed.H1, W1 = feed.W1, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = feed.t.h0 + warp * R, w = feed.t.w0 + lane;
  const int rows = w < W1 ? min(R, H1 - h) : 0;   // of this thread; may be <= 0
  const bool warp_has_rows = h < H1;
  const size_t plane = (size_t)H1 * W1;
  const uint32_t p = rows > 0 ? (uint32_t)(h * W1 + w) : 0u;
  float* const o0 = job.gx + (size_t)feed.t.b * 2 * D * plane;   // the same for the whole block
  // what the sums are added to: the given addend, for a later chunk of channels the earlier ones' sums
  const float* const before = accumulate ? o0 : (job.add != nullptr ? job.add + (size_t)feed.t.b * job.add_sb : nullptr);
  float older[2][R], newer[2][R], addend[2][R];
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int r = 0; r < R; ++r) older[c][r] = newer[c][r] = 0.f;
  auto fetch = [&](int d) {   // asked for a plane's arithmetic before it is needed
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int r = 0; r < R; ++r)
        addend[c][r] = before != nullptr && r < rows ? (before + ((size_t)c * D + d) * plane + r * W1)[p] : 0.f;
  };
  auto emit = [&](int d) {
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (r < rows) (o0 + ((size_t)c * D + d) * plane + r * W1)[p] = older[c][r] + addend[c][r];
  };
  for (int i = 0; i < feed.n_planes; ++i) {  // plane e of gL feeds gX planes e-1 (td=0), e (td=1), e+1 (td=2)
    const int e = feed.e0 + i;
    if (e > d0) fetch(e - 1);
    const auto* stage = feed.plane(i);
    if (stage == nullptr) return;
    if (!warp_has_rows) continue;
    float v[KC][R + 2][3];
#pragma unroll
    for (int k = 0; k < KC; ++k)
#pragma unroll
      for (int r = 0; r < R + 2; ++r)
#pragma unroll
        for (int j = 0; j < 3; ++j) v[k][r][j] = stage->v[k][warp * R + r][lane + 3 + j];
    auto taps = [&](auto td, float (&a)[2][R], auto&& from) {   // a = from + taps
#pragma unroll
      for (int k = 0; k < KC; ++k)
#pragma unroll
        for (int n = 0; n < 9; ++n)
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const float wt = att_weight<MODULE>(input_grad_weight(k, c, decltype(td)::value, n));
#pragma unroll
            for (int r = 0; r < R; ++r) a[c][r] = fmaf(v[k][r + n / 3][n % 3], wt, k == 0 && n == 0 ? from(c, r) : a[c][r]);
          }
    };
    if (e > d0) {
      taps(std::integral_constant<int, 0>{}, older, [&](int c, int r) { return older[c][r]; });
      emit(e - 1);
    }
    if (e >= d0 && e < d1) taps(std::integral_constant<int, 1>{}, older, [&](int c, int r) { return newer[c][r]; });
    if (e + 1 < d1) taps(std::integral_constant<int, 2>{}, newer, [&](int, int) { return 0.f; });
  }
  if (d1 == D) {
    fetch(D - 1);
    emit(D - 1);
  }
}

template <int KC, int FEED>
__global__ void __launch_bounds__(AT_THREADS)
attention_input_grad_tiled_kernel(const __grid_constant__ TileMaps maps, const __grid_constant__ InputGradJobs jobs, int accumulate, int Kc,
                                  int k0, int B, int H1, int W1, int* status) {
  if (!cta_has_work(status)) return;
  __shared__ __align__(128) AttentionTileSmem<KC> sm;
  const int ji = job_of(jobs.blocks, blockIdx.x);
  const InputGradJobs::Job& job = jobs.j[ji];
  const TileBlock t = tile_block<AT_TILE_ROWS>(blockIdx.x - jobs.blocks.first[ji], B, H1, W1);
  const int d0 = t.piece * job.dc, d1 = min(d0 + job.dc, job.D);
  const int e0 = max(d0 - 1, 0), n_planes = min(d1 + 1, job.D) - e0;
  const size_t plane = (size_t)H1 * W1;
  PlaneFeed<KC, FEED> feed{sm, &maps.m[ji], job.gl + (((size_t)t.b * Kc + k0) * job.D + e0) * plane, job.D * plane, Kc - k0, e0, n_planes, k0,
                              H1, W1, t, status};
  if (threadIdx.x == 0) {
    if (FEED == FEED_TMA) {
      for (int s = 0; s < feed.STAGES; ++s) mbar_init(&sm.full[s], 1);
      prefetch_tensormap(feed.tm);
    }
    wait_ctl_init(&sm.ctl, 0);
    fence_barrier_init();
  }
  __syncthreads();
  feed.start();
  by_module(job.module, [&](auto m) { input_grad_walk_tiled<KC, decltype(m)::value>(feed, job, accumulate, k0, d0, d1); });
  __syncthreads();
  if (wait_ctl_aborted(&sm.ctl)) {
    let_copies_land();
  }
}

// Weight gradients: half of the warps own input channel 0, the others input channel 1, each thread KW output channels of its WG_ROWS
// pixels; the stage holds the tile (with halo) of plane e of both X channels and the tile (without halo) of plane e+1 of
// the KW logit-gradient channels, which the two halves share.  The sums of two output channels are one packed pair
// (fma.rn.f32x2 with the X value in both halves), which halves the multiply-add instructions.  Several pixels to a thread share the X
// values they read; with two channels to a thread the sums leave registers for three blocks on an SM (with four there was one, of eight warps).
// 8 x 47 x 156, two channels, one level: 151 -> 73 us; 3 x 47 x 155, three channels, four levels (copies) 193 -> 151; 8 x 135 x 240, four
// channels 1.67 -> 1.34 ms; 2 x 48 x 64, two channels, four levels 32 -> 15.  Bound: the FMA pipe (2.25 cycles for a packed multiply-add with
// an operand kept) and issue beside it.  Logit gradients of three planes are
// held, in registers whose roles rotate over three planes of the loop.  A piece is `dc` planes of X.
// TMA loads are issued by a warp of their own; copies by all warps, which then meet at a barrier per plane as in PlaneFeed.
// grid (ceil(W1/32) * ceil(H1/8) * B * pieces blocks per job, chunks of KW channels), block wg_threads(FEED); partial: of the module,
// (Kc * 2 * 27, rows).
constexpr int WG_PER_SM = 3;   // blocks on an SM, by the launch bounds; the number by which walks are cut, whose partial sums size the workspace
constexpr int WG_GROUPS = 2, WG_WARPS = 2 * WG_GROUPS, WG_ROWS = 4, WG_TILE_ROWS = WG_GROUPS * WG_ROWS, WG_MAX_CHANNELS = 2;
constexpr int wg_channels(int Kc) { return Kc < WG_MAX_CHANNELS ? Kc : WG_MAX_CHANNELS; }   // of a thread
template <int KW>
struct WeightGradTileSmem {
  struct alignas(128) Stage {   // both parts are TMA destinations: 128-byte aligned
    alignas(128) float x[2][WG_TILE_ROWS + 2][AT_BOX_W];
    alignas(128) float g[KW][WG_TILE_ROWS][AT_TW];
  };
  static constexpr int STAGES = at_stages(sizeof(Stage));
  Stage st[STAGES];
  uint64_t full[STAGES];
  uint64_t empty[STAGES];
  WaitCtl ctl;
  float red[WG_WARPS * KW * AT_TAPS];
};

__host__ __device__ constexpr int wg_threads(int feed) { return WG_WARPS * 32 + (feed == FEED_TMA ? 32 : 0); }
template <int KW, int FEED>
__global__ void __launch_bounds__(wg_threads(FEED), WG_PER_SM)
attention_weight_grad_tiled_kernel(const __grid_constant__ TileMaps maps_x, const __grid_constant__ TileMaps maps_gl,
                                   const __grid_constant__ WeightGradJobs jobs, int Kc, int B, int H1, int W1, int* status) {
  if (!cta_has_work(status)) return;
  __shared__ __align__(128) WeightGradTileSmem<KW> sm;
  constexpr int R = WG_ROWS, STAGES = WeightGradTileSmem<KW>::STAGES;
  const int ji = job_of(jobs.blocks, blockIdx.x), r = blockIdx.x - jobs.blocks.first[ji];
  const WeightGradJobs::Job& job = jobs.j[ji];
  const TileBlock tb = tile_block<WG_TILE_ROWS>(r, B, H1, W1);
  const int w0 = tb.w0, h0 = tb.h0, b = tb.b, k0 = blockIdx.y * KW, D = job.D;
  const float* __restrict__ const gl = job.gl;
  const CUtensorMap *const tm_x = &maps_x.m[ji], *const tm_gl = &maps_gl.m[ji];
  const int e0 = tb.piece * job.dc, n_planes = min(job.dc, D - e0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t plane = (size_t)H1 * W1;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&sm.full[s], 1); mbar_init(&sm.empty[s], WG_WARPS); }
    wait_ctl_init(&sm.ctl, 0);
    fence_barrier_init();
    if (FEED == FEED_TMA) {
      prefetch_tensormap(tm_x);
      prefetch_tensormap(tm_gl);
    }
  }
  __syncthreads();
  auto copy_plane = [&](int i) {
    if (i < n_planes) {
      auto& st = sm.st[i % STAGES];
      copy_tile<2, WG_TILE_ROWS + 2, AT_BOX_W, 1, WG_WARPS>(st.x, job.x + (size_t)b * job.x_sb + (size_t)(e0 + i) * plane, D * plane, 2, h0, w0, H1,
                                                            W1);
      const bool has_next = e0 + i + 1 < D;
      copy_tile<KW, WG_TILE_ROWS, AT_TW, 0, WG_WARPS>(st.g, gl + (((size_t)b * Kc + k0) * D + (has_next ? e0 + i + 1 : 0)) * plane, D * plane,
                                                      has_next ? Kc - k0 : 0, h0, w0, H1, W1);
    }
    cp_async_commit();   // a group per plane, also where there is none
  };
  if constexpr (FEED == FEED_COPIES) {
    for (int i = 0; i < STAGES - 1; ++i) copy_plane(i);
  } else if (warp == WG_WARPS) {  // producer
    if (lane != 0) return;
    for (int i = 0; i < n_planes; ++i) {
      const uint32_t s = i % STAGES, ph = (i / STAGES) & 1u;
      if (!mbar_wait(&sm.empty[s], ph ^ 1u, &sm.ctl, status, DEV_TIMEOUT_PRODUCER)) { let_copies_land(); break; }
      mbar_expect_tx(&sm.full[s], sizeof(sm.st[s].x) + sizeof(sm.st[s].g));
      tma_load_5d(sm.st[s].x, tm_x, &sm.full[s], w0 - 4, h0 - 1, e0 + i, 0, b);
      tma_load_5d(sm.st[s].g, tm_gl, &sm.full[s], w0, h0, e0 + i + 1, k0, b);  // plane D, channels >= Kc read as zero
    }
    return;
  }
  const int q = warp % WG_GROUPS, c = warp / WG_GROUPS;
  const int h = h0 + q * R, w = w0 + lane, rows = w < W1 ? min(R, H1 - h) : 0;
  using Value = std::conditional_t<KW == 2, uint64_t, float>;   // a value of all channels of the thread
  auto mul_add = [](Value g, float v, Value a) -> Value {
    if constexpr (KW == 2) return fma2(pack2(v, v), g, a);
    else return fmaf(v, g, a);
  };
  Value acc[AT_TAPS];   // [td * 9 + neighbour]
#pragma unroll
  for (int i = 0; i < AT_TAPS; ++i) acc[i] = Value(0);
  Value g[3][R];        // gL of plane d in g[(d - e0 + 3) % 3]
#pragma unroll
  for (int rr = 0; rr < R; ++rr) {
    float before[2], here[2];
#pragma unroll
    for (int k = 0; k < KW; ++k) {
      const bool ok = rr < rows && k0 + k < Kc;
      const float* gp = gl + (((size_t)b * Kc + (ok ? k0 + k : 0)) * D + e0) * plane + (ok ? (size_t)(h + rr) * W1 + w : 0);
      before[k] = (ok && e0 > 0) ? __ldg(gp - plane) : 0.f;
      here[k] = ok ? __ldg(gp) : 0.f;
    }
    if constexpr (KW == 2) {
      g[2][rr] = pack2(before[0], before[1]);
      g[0][rr] = pack2(here[0], here[1]);
    } else {
      g[2][rr] = before[0];
      g[0][rr] = here[0];
    }
  }
  bool alive = true;
  auto plane_sums = [&](int i, auto phase) -> bool {   // plane e0 + i of X meets gL at d = e+1 (td=0), e (td=1), e-1 (td=2); i % 3 == phase
    constexpr int P = decltype(phase)::value;
    const uint32_t s = i % STAGES, ph = (i / STAGES) & 1u;
    if constexpr (FEED == FEED_TMA) {
      if (!mbar_wait_warp(&sm.full[s], ph, &sm.ctl, status, DEV_TIMEOUT_EPILOGUE)) { let_copies_land(); return false; }
    } else {
      cp_async_wait<STAGES - 2>();
      named_bar_sync(1, WG_WARPS * 32);   // the plane is there for all, and the one before has been read
      copy_plane(i + STAGES - 1);
    }
#pragma unroll
    for (int rr = 0; rr < R; ++rr) {
      if constexpr (KW == 2) g[(P + 1) % 3][rr] = pack2(sm.st[s].g[0][q * R + rr][lane], sm.st[s].g[1][q * R + rr][lane]);
      else g[(P + 1) % 3][rr] = sm.st[s].g[0][q * R + rr][lane];
    }
#pragma unroll
    for (int y = 0; y < R + 2; ++y)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const float v = sm.st[s].x[c][q * R + y][lane + 3 + j];
#pragma unroll
        for (int th = 0; th < 3; ++th) {   // the pixel in row y - th sees the value as its neighbour (th, j)
          if (y - th < 0 || y - th >= R) continue;
#pragma unroll
          for (int td = 0; td < 3; ++td) {
            Value& a = acc[td * 9 + th * 3 + j];
            a = mul_add(g[(P + 4 - td) % 3][y - th], v, a);
          }
        }
      }
    if constexpr (FEED == FEED_TMA) hand_back_stage(&sm.empty[s], lane);
    return true;
  };
  for (int i = 0; i < n_planes && alive; i += 3) {
    alive = plane_sums(i, std::integral_constant<int, 0>{});
    if (alive && i + 1 < n_planes) alive = plane_sums(i + 1, std::integral_constant<int, 1>{});
    if (alive && i + 2 < n_planes) alive = plane_sums(i + 2, std::integral_constant<int, 2>{});
  }
  // reduce over the threads of each input channel (named barrier 1: the producer warp has left);
  // column (k, c, td, n) goes to row (k0 + k) * 54 + c * 27 + td * 9 + n of the partial sums
  auto put = [&](int i, float sum) {
    if (!alive) sum = 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) sm.red[warp * KW * AT_TAPS + i] = sum;
  };
#pragma unroll
  for (int t = 0; t < AT_TAPS; ++t) {
    if constexpr (KW == 2) {
      float lo, hi;
      unpack2(acc[t], lo, hi);
      put(t, lo);
      put(AT_TAPS + t, hi);
    } else {
      put(t, acc[t]);
    }
  }
  named_bar_sync(1, WG_WARPS * 32);
  const size_t n_rows = job.rows;
  float* dst = job.partial + job.row0 + r;
  for (int i = threadIdx.x; i < 2 * KW * AT_TAPS; i += WG_WARPS * 32) {
    const int cc = i / (KW * AT_TAPS), j = i - cc * KW * AT_TAPS, k = j / AT_TAPS, t = j - k * AT_TAPS;
    if (k0 + k >= Kc) continue;
    float sum = 0.f;
#pragma unroll
    for (int wv = 0; wv < WG_GROUPS; ++wv) sum += sm.red[(cc * WG_GROUPS + wv) * KW * AT_TAPS + j];
    dst[(((size_t)(k0 + k) * 2 + cc) * AT_TAPS + t) * n_rows] = sum;
  }
}

// ---- staging of the filter weights in constant memory ---------------------------------------------------
// c_att_weights is one array per device.  Work on one stream is ordered anyway; a call on another stream first
// waits for the event the previous user recorded after its last kernel, so the copy below never overtakes a
// kernel that still reads the old weights.  The lock is held from the copy to that record.
namespace {
constexpr int AT_MAX_DEVICES = 64;
struct WeightStage {
  std::mutex mu;
  cudaEvent_t done[AT_MAX_DEVICES] = {nullptr};
  cudaStream_t last[AT_MAX_DEVICES] = {nullptr};
  bool used[AT_MAX_DEVICES] = {false};
  void* constant[AT_MAX_DEVICES] = {nullptr};   // addresses of c_att_weights and g_att_weights
  void* ordered[AT_MAX_DEVICES] = {nullptr};
} g_stage;

class StagedWeights {
 public:
  explicit StagedWeights(cudaStream_t st) : lock_(g_stage.mu), st_(st) {
    err_ = cudaGetDevice(&dev_);
    if (err_ == cudaSuccess && (dev_ < 0 || dev_ >= AT_MAX_DEVICES)) err_ = cudaErrorInvalidDevice;
    if (err_ != cudaSuccess) return;
    if (g_stage.done[dev_] == nullptr) err_ = cudaEventCreateWithFlags(&g_stage.done[dev_], cudaEventDisableTiming);
    if (err_ == cudaSuccess && g_stage.ordered[dev_] == nullptr) {
      err_ = cudaGetSymbolAddress(&g_stage.constant[dev_], c_att_weights);
      if (err_ == cudaSuccess) err_ = cudaGetSymbolAddress(&g_stage.ordered[dev_], g_att_weights);
    }
    if (err_ == cudaSuccess && g_stage.used[dev_] && g_stage.last[dev_] != st_)
      err_ = cudaStreamWaitEvent(st_, g_stage.done[dev_], 0);
  }
  // Weights of channels k0 .. k0 + channels - 1 (at most AT_KC) of both modules.
  cudaError_t put(const AttentionModules& modules, int k0, int channels, bool input_grad) {
    if (err_ != cudaSuccess) return err_;
    StageWeights s{{nullptr, nullptr}, channels, input_grad};
    for (int m = 0; m < 2; ++m)
      if (modules.weight[m] != nullptr) s.weight[m] = modules.weight[m] + (size_t)k0 * 2 * AT_TAPS;
    launch_next(stage_weights_kernel, 2, AT_KC * 2 * AT_TAPS, 0, st_, s);
    err_ = cudaGetLastError();
    if (err_ == cudaSuccess) err_ = cudaMemcpyAsync(g_stage.constant[dev_], g_stage.ordered[dev_], sizeof(c_att_weights), cudaMemcpyDeviceToDevice, st_);
    return err_;
  }
  ~StagedWeights() {
    if (err_ != cudaSuccess) return;
    if (cudaEventRecord(g_stage.done[dev_], st_) == cudaSuccess) {
      g_stage.last[dev_] = st_;
      g_stage.used[dev_] = true;
    }
  }

 private:
  std::lock_guard<std::mutex> lock_;
  cudaStream_t st_;
  int dev_ = 0;
  cudaError_t err_ = cudaSuccess;
};
}  // namespace

// ---- launchers ---------------------------------------------------------------------------------------
static dim3 pixel_grid(const AttentionDims& d) { return dim3((d.H1 * d.W1 + AT_THREADS - 1) / AT_THREADS, d.B); }

static size_t tile_count(const AttentionDims& d, int rows) { return (size_t)((d.W1 + AT_TW - 1) / AT_TW) * ((d.H1 + rows - 1) / rows); }
// Blocks of a job whose walks are not cut, in the tiled form and in the gather form (callers without a status word).
static size_t form_blocks(const AttentionDims& d, bool tiled) { return (tiled ? tile_count(d, AT_TILE_ROWS) : (size_t)pixel_grid(d).x) * d.B; }
// Displacements per block of a walk of the gather form: enough blocks (AT_BLOCKS_TARGET) to fill the 148 SMs several times over,
// but at least AT_MIN_WALK displacements, because every block also reads a plane on either side of its own.
// The weight gradients pay for a reduction over the block at the end of a walk as well and keep one or two blocks on an
// SM, hence fewer and longer pieces.
constexpr int AT_BLOCKS_TARGET = 148 * 8, AT_MIN_WALK = 8;
constexpr int WG_BLOCKS_TARGET = 148 * 3, WG_MIN_WALK = 16;
static int even_walk(int D, int dc) {   // the walks of a column of D, cut into pieces of at most dc
  const int pieces = (D + dc - 1) / dc;
  return (D + pieces - 1) / pieces;
}
static int gather_walk(size_t blocks, int D, int total, int target = AT_BLOCKS_TARGET, int min_walk = AT_MIN_WALK) {
  const int pieces = (int)((target + blocks - 1) / blocks);   // of all jobs
  return even_walk(D, std::max((total + pieces - 1) / pieces, min_walk));
}
// Longest piece of the tiled walks, for all jobs of a launch (same blocks, columns of D[0 .. n-1]), on `slots` blocks at a time.  Pieces are cut
// so that all of them make one round of the slots, or two, ...: with k rounds a launch takes between the work of a slot and k times its longest
// piece.  A piece costs `extra` planes beside its own: the planes on either side of it, whose values it needs in part, its start and end.
static int tiled_walk(size_t blocks, const int* D, int n, int slots, double extra) {
  int most = 1, total = 0;
  for (int i = 0; i < n; ++i) {
    most = std::max(most, D[i]);
    total += D[i];
  }
  auto pieces = [&](int dc) {
    double count = 0;
    for (int i = 0; i < n; ++i) count += (D[i] + dc - 1) / dc;
    return count * blocks;
  };
  double best = 0;
  int walk = most;
  for (int rounds = 1; rounds <= 8; ++rounds) {
    const double room = (double)rounds * slots;
    int dc = std::max(1, (int)((double)blocks * total / room));
    while (dc < most && pieces(dc) > room) dc += 1 + dc / 16;
    dc = even_walk(most, std::min(dc, most));
    const double count = pieces(dc), work = ((double)blocks * total + count * extra) / slots;
    const double cost = 0.5 * (work + std::max(work, std::ceil(count / slots) * (dc + extra)));
    if (best == 0 || cost < 0.98 * best) {
      best = cost;
      walk = dc;
    }
  }
  return walk;
}
// What a piece costs beside its planes.
constexpr double AT_PIECE_EXTRA = 3.0, WG_PIECE_EXTRA = 8.0;
// Displacements per block of the weight gradients' walks, and the blocks of a job (partial sums of a weight).
struct WeightWalks {
  int dc[MAX_ATTENTION_JOBS];
  size_t rows[MAX_ATTENTION_JOBS];
};
static WeightWalks weight_walks(const AttentionDims* d, int count, bool tiled) {
  WeightWalks r{};
  int D[MAX_ATTENTION_JOBS], total = 0;
  for (int i = 0; i < count; ++i) total += D[i] = d[i].D;
  const size_t blocks = tiled ? tile_count(d[0], WG_TILE_ROWS) * d[0].B : form_blocks(d[0], false);
  const int chunks = (d[0].Kc + wg_channels(d[0].Kc) - 1) / wg_channels(d[0].Kc);
  const int walk = tiled ? tiled_walk(blocks * chunks, D, count, WG_PER_SM * SM_COUNT, WG_PIECE_EXTRA) : 0;
  for (int i = 0; i < count; ++i) {
    r.dc[i] = tiled ? even_walk(D[i], walk) : gather_walk(2 * blocks, D[i], total, WG_BLOCKS_TARGET, WG_MIN_WALK);
    r.rows[i] = blocks * ((D[i] + r.dc[i] - 1) / r.dc[i]);
  }
  return r;
}
// The softmax backward: pixels of a block by the length of the column (attention_logit_grad_kernel).
static int logit_grad_pixels(int D) { return D <= 8 ? lg_pixels(1) : D <= 16 ? lg_pixels(2) : D <= 32 ? lg_pixels(4) : 32; }
static size_t bias_rows(const AttentionDims& d) { return (size_t)d.B * ((d.H1 * d.W1 + logit_grad_pixels(d.D) - 1) / logit_grad_pixels(d.D)); }

// Bias partials per block of the softmax backward, weight partials per block of the weight gradients, whichever form they take.
size_t attention_partial_floats(const AttentionDims* d, int count) {
  size_t floats = 0;
  const WeightWalks tiled = weight_walks(d, count, true), gather = weight_walks(d, count, false);
  for (int i = 0; i < count; ++i) floats += d[i].Kc * (bias_rows(d[i]) + 2 * AT_TAPS * std::max(tiled.rows[i], gather.rows[i]));
  return floats;
}

// Columns of a class of lengths are done by one launch.
template <int V, int VEC>
static cudaError_t launch_softmax_jobs(const AttentionJob* job, int count, int above, int upto, cudaStream_t st) {
  SoftmaxJobs jobs{};
  const AttentionDims& d = job[0].d;
  const unsigned pb = (unsigned)((d.H1 * d.W1 + 32 * VEC - 1) / (32 * VEC));
  unsigned long long blocks = 0;
  int n = 0;
  for (int i = 0; i < count; ++i) {
    const int v = (job[i].d.D + SM_GROUPS - 1) / SM_GROUPS;
    if (v <= above || v > upto) continue;
    jobs.a[n] = job[i].a;
    jobs.D[n] = job[i].d.D;
    jobs.blocks.first[n++] = (int)blocks;
    blocks += (unsigned long long)pb * d.B * d.Kc;
    if (blocks > 0x7fffffffull) return cudaErrorInvalidConfiguration;
  }
  if (n == 0) return cudaSuccess;
  for (; n <= MAX_ATTENTION_JOBS; ++n) jobs.blocks.first[n] = (int)blocks;
  launch_next(attention_softmax_kernel<V, VEC>, (unsigned)blocks, SM_THREADS, 0, st, jobs, d.H1 * d.W1, pb);
  return cudaGetLastError();
}
// Pixels of a lane: as many as the values of a thread leave registers for (128 of them, two blocks per SM), in launches that
// have a block for every SM all the same.  Two at V <= 32 spill and gained nothing over one.
template <int V>
static cudaError_t launch_softmax_class(const AttentionJob* job, int count, int above, int upto, cudaStream_t st) {
  constexpr int VEC = V == 0 || V > 24 ? 1 : (V <= 16 ? 4 : 2);
  if constexpr (VEC > 1) {
    const AttentionDims& d = job[0].d;
    const long long N1 = (long long)d.H1 * d.W1;
    bool wide = N1 % VEC == 0 && N1 / (32 * VEC) * d.B * d.Kc >= SM_COUNT;
    for (int i = 0; i < count; ++i) wide = wide && (reinterpret_cast<uintptr_t>(job[i].a) & 15u) == 0;
    if (wide) return launch_softmax_jobs<V, VEC>(job, count, above, upto, st);
  }
  return launch_softmax_jobs<V, 1>(job, count, above, upto, st);
}
static int softmax_class(int D) {   // largest values per warp of a class; 0: any
  const int v = (D + SM_GROUPS - 1) / SM_GROUPS;
  for (const int c : {4, 8, 16, 20, 24, 32})
    if (v <= c) return c;
  return 0;
}
static cudaError_t launch_softmax(const AttentionJob* job, int count, cudaStream_t st) {
  cudaError_t err;
  if ((err = launch_softmax_class<4>(job, count, 0, 4, st)) != cudaSuccess) return err;
  if ((err = launch_softmax_class<8>(job, count, 4, 8, st)) != cudaSuccess) return err;
  if ((err = launch_softmax_class<16>(job, count, 8, 16, st)) != cudaSuccess) return err;
  if ((err = launch_softmax_class<20>(job, count, 16, 20, st)) != cudaSuccess) return err;
  if ((err = launch_softmax_class<24>(job, count, 20, 24, st)) != cudaSuccess) return err;
  if ((err = launch_softmax_class<32>(job, count, 24, 32, st)) != cudaSuccess) return err;
  return launch_softmax_class<0>(job, count, 32, INT_MAX, st);
}

// Displacements per block of the walks of a launch (logits or input gradients).  A column short enough for the walks to end with its softmax is
// not cut by launches that have two blocks per SM without it.
struct Walks {
  int dc[MAX_ATTENTION_JOBS];
  bool soft;   // all columns end with their softmax
};
template <class Job>
static Walks stencil_walks(const Job* job, int count, bool tiled, int blocks_per_sm, bool with_softmax) {
  Walks r{};
  int D[MAX_ATTENTION_JOBS], total = 0;
  for (int i = 0; i < count; ++i) total += D[i] = job[i].d.D;
  const size_t blocks = form_blocks(job[0].d, tiled);
  const int walk = tiled ? tiled_walk(blocks, D, count, blocks_per_sm * SM_COUNT, AT_PIECE_EXTRA) : 0;
  r.soft = with_softmax;
  for (int i = 0; i < count; ++i) {
    const bool whole = with_softmax && D[i] <= AT_SOFT_MAX && blocks * count >= 2 * SM_COUNT;
    r.dc[i] = whole ? D[i] : (tiled ? even_walk(D[i], walk) : gather_walk(blocks, D[i], total));
    r.soft = r.soft && D[i] <= AT_SOFT_MAX && r.dc[i] == D[i];
  }
  return r;
}
// f(integral constant) of a number of channels
template <class F>
static void by_channels(int kc, F&& f) {
  if (kc == 1) f(std::integral_constant<int, 1>{});
  else if (kc == 2) f(std::integral_constant<int, 2>{});
  else if (kc == 3) f(std::integral_constant<int, 3>{});
  else f(std::integral_constant<int, 4>{});
}

// Blocks on an SM of a tiled kernel (AT_THREADS threads, static shared memory), as it was compiled: 3 to 5 of the forms that copy, 3 to 8 of those by
// TMA.  Written down as 4 or 6 (logits, three channels and more, or fewer) and 3 or 5 (input gradients) for both forms, where a round of the
// slots was none: logits 1 x 135 x 241, one level, four channels (3 on an SM) 205 -> 163 us, 1 x 55 x 127, two channels (4) 17.0 -> 14.3; input
// gradients 4 x 55 x 128, four levels, three channels (4) 129 -> 95.  104 sizes, one and four levels, one to four channels: 2.7 % less for
// either kernel; up to a tenth more where rounds of fewer blocks happened to fit (4 x 55 x 128, one level, three channels: logits 49 -> 54).
// Asked once per kernel and device.
template <auto KERNEL>
static int blocks_per_sm() {
  static std::atomic<int> known[AT_MAX_DEVICES];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= AT_MAX_DEVICES) return 1;
  int n = known[dev].load(std::memory_order_relaxed);
  if (n == 0 && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, KERNEL, AT_THREADS, 0) == cudaSuccess)
    known[dev].store(n, std::memory_order_relaxed);
  return std::max(n, 1);
}
// The order of a launch's jobs: the longest pieces first, so that the short ones fill the end.
static void by_length(const Walks& walks, int count, int* order) {
  for (int i = 0; i < count; ++i) {
    int at = i;
    for (; at > 0 && walks.dc[order[at - 1]] < walks.dc[i]; --at) order[at] = order[at - 1];
    order[at] = i;
  }
}
static bool logits_by_tma(const AttentionJob* job, int count) {
  bool tma = true;
  for (int i = 0; i < count; ++i) tma = tma && tileable(job[i].d, job[i].x, job[i].x_sb);
  return tma;
}
static Walks logits_walks(const AttentionJob* job, int count, bool tiled, bool tma) {
  int per_sm = 0;
  if (tiled)
    by_channels(std::min(job[0].d.Kc, AT_KC), [&](auto c) {
      constexpr int KC = decltype(c)::value;
      per_sm = tma ? blocks_per_sm<attention_logits_tiled_kernel<KC, false, FEED_TMA>>()
                   : blocks_per_sm<attention_logits_tiled_kernel<KC, false, FEED_COPIES>>();
    });
  return stencil_walks(job, count, tiled, per_sm, true);
}
static Walks input_grad_walks(const AttentionGradJob* job, int count, bool tiled, bool tma) {
  int per_sm = 0;
  if (tiled)
    by_channels(std::min(job[0].d.Kc, AT_KC), [&](auto c) {
      constexpr int KC = decltype(c)::value;
      per_sm = tma ? blocks_per_sm<attention_input_grad_tiled_kernel<KC, FEED_TMA>>() : blocks_per_sm<attention_input_grad_tiled_kernel<KC, FEED_COPIES>>();
    });
  return stencil_walks(job, count, tiled, per_sm, false);
}

int attention_forward_launches(const AttentionJob* job, int count, const int* status) {
  int n = 2 * ((job[0].d.Kc + AT_KC - 1) / AT_KC);   // the weights' staging and the walks per chunk of channels
  if (logits_walks(job, count, status != nullptr, status != nullptr && logits_by_tma(job, count)).soft) return n;
  for (int i = 0; i < count; ++i) {
    bool first = true;   // of its class of lengths
    for (int k = 0; k < i; ++k) first = first && softmax_class(job[k].d.D) != softmax_class(job[i].d.D);
    n += first ? 1 : 0;
  }
  return n;
}

cudaError_t launch_attention_forward(const AttentionJob* job, int count, const AttentionModules& modules, cudaStream_t st, int* status) {
  if (count < 1 || count > MAX_ATTENTION_JOBS) return cudaErrorInvalidValue;
  const AttentionDims& d = job[0].d;
  const bool tiled = status != nullptr, tma = tiled && logits_by_tma(job, count);
  const Walks walks = logits_walks(job, count, tiled, tma);
  const bool soft = walks.soft;
  int order[MAX_ATTENTION_JOBS];
  by_length(walks, count, order);
  TileMaps maps;
  LogitsJobs jobs{};
  unsigned long long blocks = 0;
  for (int i = 0; i < MAX_ATTENTION_JOBS; ++i) {
    jobs.blocks.first[i] = (int)blocks;
    if (i >= count) continue;
    const AttentionJob& j = job[order[i]];
    if (tma) {
      cudaError_t err = tile_map(&maps.m[i], j.x, j.x_sb, 2, 2, j.d, AT_TILE_ROWS, true);
      if (err != cudaSuccess) return err;
    }
    const int dc = walks.dc[order[i]];
    jobs.j[i] = LogitsJobs::Job{j.x, j.x_sb, modules.bias[j.module], j.a, j.d.D, dc, j.module};
    blocks += (unsigned long long)form_blocks(d, tiled) * ((j.d.D + dc - 1) / dc);
    if (blocks > 0x7fffffffull) return cudaErrorInvalidConfiguration;
  }
  jobs.blocks.first[MAX_ATTENTION_JOBS] = (int)blocks;
  {
    StagedWeights staged(st);
    for (int k0 = 0; k0 < d.Kc; k0 += AT_KC) {
      const int kc = d.Kc - k0 < AT_KC ? d.Kc - k0 : AT_KC;
      cudaError_t err = staged.put(modules, k0, kc, false);
      if (err != cudaSuccess) return err;
      by_channels(kc, [&](auto c) {
        constexpr int KC = decltype(c)::value;
        if (!tiled) {
          launch_next(soft ? attention_logits_kernel<KC, true> : attention_logits_kernel<KC, false>, (unsigned)blocks, AT_THREADS, 0, st, jobs,
                      d.Kc, k0, d.B, d.H1, d.W1);
          return;
        }
        auto kernel = tma ? (soft ? attention_logits_tiled_kernel<KC, true, FEED_TMA> : attention_logits_tiled_kernel<KC, false, FEED_TMA>)
                          : (soft ? attention_logits_tiled_kernel<KC, true, FEED_COPIES> : attention_logits_tiled_kernel<KC, false, FEED_COPIES>);
        launch_next(kernel, (unsigned)blocks, AT_THREADS, 0, st, maps, jobs, d.Kc, k0, d.B, d.H1, d.W1, status);
      });
      if ((err = cudaGetLastError()) != cudaSuccess) return err;
    }
  }
  return soft ? cudaSuccess : launch_softmax(job, count, st);
}

template <int KC>
static cudaError_t launch_input_grad(unsigned blocks, const InputGradJobs& jobs, int accumulate, const AttentionDims& d, int k0,
                                     cudaStream_t st) {
  constexpr size_t smem = PlaneRing<9 * KC, IG_STAGES>::bytes();
  static DeviceOnce configured;
  if (smem > 48 * 1024) {
    cudaError_t err = configured.run(
        [&] { return cudaFuncSetAttribute(attention_input_grad_kernel<KC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); });
    if (err != cudaSuccess) return err;
  }
  launch_next(attention_input_grad_kernel<KC>, blocks, AT_THREADS, smem, st, jobs, accumulate, d.Kc, k0, d.B, d.H1, d.W1);
  return cudaGetLastError();
}

// A job's place among the partial sums of its module.
struct PartialPlace {
  float *bias, *weight;   // of the module
  int bias_row0, bias_rows, weight_row0, weight_rows;
};

// Softmax backward of the jobs with above < D <= upto, by one launch.
template <int G, int V, int MIN_BLOCKS>
static cudaError_t launch_logit_grad_class(const AttentionGradJob* job, const PartialPlace* place, int count, int above, int upto,
                                           cudaStream_t st) {
  LogitGradJobs jobs{};
  const AttentionDims& d = job[0].d;
  const unsigned pb = (unsigned)((d.H1 * d.W1 + lg_pixels(G) - 1) / lg_pixels(G));
  unsigned long long blocks = 0;
  int n = 0;
  for (int i = 0; i < count; ++i) {
    if (job[i].d.D <= above || job[i].d.D > upto) continue;
    jobs.j[n] = LogitGradJobs::Job{job[i].a, job[i].g, place[i].bias, job[i].d.D, place[i].bias_row0, place[i].bias_rows};
    jobs.blocks.first[n++] = (int)blocks;
    blocks += (unsigned long long)pb * d.B * d.Kc;
    if (blocks > 0x7fffffffull) return cudaErrorInvalidConfiguration;
  }
  if (n == 0) return cudaSuccess;
  for (; n <= MAX_ATTENTION_JOBS; ++n) jobs.blocks.first[n] = (int)blocks;
  launch_next(attention_logit_grad_kernel<G, V, MIN_BLOCKS>, (unsigned)blocks, 32 * lg_warps(G), 0, st, jobs, d.Kc, d.H1 * d.W1, pb);
  return cudaGetLastError();
}
static int logit_grad_class(int D) {
  for (const int c : {8, 16, 32, 64, 128, 160, 256})
    if (D <= c) return c;
  return 0;
}
static cudaError_t launch_logit_grad(const AttentionGradJob* job, const PartialPlace* place, int count, cudaStream_t st) {
  cudaError_t err;
  if ((err = launch_logit_grad_class<1, 8, 5>(job, place, count, 0, 8, st)) != cudaSuccess) return err;
  if ((err = launch_logit_grad_class<2, 8, 6>(job, place, count, 8, 16, st)) != cudaSuccess) return err;
  if ((err = launch_logit_grad_class<4, 8, 6>(job, place, count, 16, 32, st)) != cudaSuccess) return err;
  if ((err = launch_logit_grad_class<8, 8, 6>(job, place, count, 32, 64, st)) != cudaSuccess) return err;
  if ((err = launch_logit_grad_class<8, 16, 3>(job, place, count, 64, 128, st)) != cudaSuccess) return err;
  if ((err = launch_logit_grad_class<16, 10, 2>(job, place, count, 128, 160, st)) != cudaSuccess) return err;
  if ((err = launch_logit_grad_class<16, 16, 2>(job, place, count, 160, 256, st)) != cudaSuccess) return err;
  return launch_logit_grad_class<8, 0, 6>(job, place, count, 256, INT_MAX, st);
}

int attention_backward_launches(const AttentionGradJob* job, int count) {
  int n = 2 * ((job[0].d.Kc + AT_KC - 1) / AT_KC) + 2;   // staging and input gradients per chunk of channels, weight gradients, the reduction
  for (int i = 0; i < count; ++i) {
    bool first = true;   // of its class of lengths
    for (int k = 0; k < i; ++k) first = first && logit_grad_class(job[k].d.D) != logit_grad_class(job[i].d.D);
    n += first ? 1 : 0;
  }
  return n;
}

cudaError_t launch_attention_backward(const AttentionGradJob* job, int count, const AttentionModules& modules,
                                      const AttentionGradients& grads, float* partial, cudaStream_t st, int* status) {
  if (count < 1 || count > MAX_ATTENTION_JOBS) return cudaErrorInvalidValue;
  const AttentionDims& d = job[0].d;
  const int N1 = d.H1 * d.W1;
  auto g_sb = [&](const AttentionGradJob& j) { return (long long)d.Kc * j.d.D * N1; };
  const bool tiled = status != nullptr;
  bool tma = tiled;
  for (int i = 0; i < count; ++i) tma = tma && tileable(job[i].d, job[i].x, job[i].x_sb) && tileable(job[i].d, job[i].g, g_sb(job[i]));
  AttentionDims dims[MAX_ATTENTION_JOBS];
  for (int i = 0; i < count; ++i) dims[i] = job[i].d;
  const WeightWalks weights = weight_walks(dims, count, tiled);

  // partial sums: per module the bias partials (Kc, rows), then the weight partials (Kc * 54, rows)
  PartialPlace place[MAX_ATTENTION_JOBS];
  PartialSums sums{};
  int columns = 0;
  for (int m = 0; m < 2; ++m) {
    int brows = 0, wrows = 0;
    for (int i = 0; i < count; ++i) {
      if (job[i].module != m) continue;
      place[i].bias_row0 = brows;
      place[i].weight_row0 = wrows;
      brows += (int)bias_rows(job[i].d);
      wrows += (int)weights.rows[i];
    }
    float *const bias = partial, *const weight = bias + (size_t)brows * d.Kc;
    partial = weight + (size_t)wrows * d.Kc * 2 * AT_TAPS;
    for (int i = 0; i < count; ++i) {
      if (job[i].module != m) continue;
      place[i].bias = bias;
      place[i].weight = weight;
      place[i].bias_rows = brows;
      place[i].weight_rows = wrows;
    }
    const bool used = brows > 0;
    sums.partial[2 * m] = weight; sums.out[2 * m] = grads.weight[m]; sums.rows[2 * m] = wrows; sums.first[2 * m] = columns;
    columns += used ? d.Kc * 2 * AT_TAPS : 0;
    sums.partial[2 * m + 1] = bias; sums.out[2 * m + 1] = grads.bias[m]; sums.rows[2 * m + 1] = brows; sums.first[2 * m + 1] = columns;
    columns += used ? d.Kc : 0;
  }
  sums.first[RP_SUMS] = columns;

  cudaError_t err = launch_logit_grad(job, place, count, st);
  if (err != cudaSuccess) return err;
  {
    const Walks walks = input_grad_walks(job, count, tiled, tma);
    int order[MAX_ATTENTION_JOBS];
    by_length(walks, count, order);
    InputGradJobs jobs{};
    unsigned long long blocks = 0;
    for (int i = 0; i <= MAX_ATTENTION_JOBS; ++i) {
      jobs.blocks.first[i] = (int)blocks;
      if (i >= count) continue;
      const AttentionGradJob& j = job[order[i]];
      const int dc = walks.dc[order[i]];
      jobs.j[i] = InputGradJobs::Job{j.g, j.add, j.add_sb, j.gx, j.d.D, dc, j.module};
      blocks += (unsigned long long)form_blocks(d, tiled) * ((j.d.D + dc - 1) / dc);
      if (blocks > 0x7fffffffull) return cudaErrorInvalidConfiguration;
    }
    StagedWeights staged(st);
    for (int k0 = 0; k0 < d.Kc; k0 += AT_KC) {
      const int kc = d.Kc - k0 < AT_KC ? d.Kc - k0 : AT_KC, accumulate = k0 == 0 ? 0 : 1;
      if ((err = staged.put(modules, k0, kc, true)) != cudaSuccess) return err;
      TileMaps maps;
      if (tma) {
        for (int i = 0; i < count; ++i) {
          const AttentionGradJob& j = job[order[i]];
          err = tile_map(&maps.m[i], j.g, g_sb(j), d.Kc, kc, j.d, AT_TILE_ROWS, true);
          if (err != cudaSuccess) return err;
        }
      }
      by_channels(kc, [&](auto c) {
        constexpr int KC = decltype(c)::value;
        if (!tiled) {
          err = launch_input_grad<KC>((unsigned)blocks, jobs, accumulate, d, k0, st);
          return;
        }
        launch_next(tma ? attention_input_grad_tiled_kernel<KC, FEED_TMA> : attention_input_grad_tiled_kernel<KC, FEED_COPIES>, (unsigned)blocks,
                    AT_THREADS, 0, st, maps, jobs, accumulate, d.Kc, k0, d.B, d.H1, d.W1, status);
        err = cudaGetLastError();
      });
      if (err != cudaSuccess) return err;
    }
  }
  const int kw = tiled ? wg_channels(d.Kc) : std::min(d.Kc, 4), chunks = (d.Kc + kw - 1) / kw;
  WeightGradJobs jobs{};
  unsigned long long blocks = 0;
  TileMaps maps_x, maps_gl;
  for (int i = 0; i <= MAX_ATTENTION_JOBS; ++i) {
    jobs.blocks.first[i] = (int)blocks;
    if (i >= count) continue;
    jobs.j[i] = WeightGradJobs::Job{job[i].x, job[i].x_sb, job[i].g, place[i].weight, job[i].d.D, weights.dc[i],
                                    place[i].weight_row0, place[i].weight_rows};
    blocks += weights.rows[i];
    if (blocks > 0x7fffffffull) return cudaErrorInvalidConfiguration;
    if (tma) {
      err = tile_map(&maps_x.m[i], job[i].x, job[i].x_sb, 2, 2, job[i].d, WG_TILE_ROWS, true);
      if (err == cudaSuccess) err = tile_map(&maps_gl.m[i], job[i].g, g_sb(job[i]), d.Kc, kw, job[i].d, WG_TILE_ROWS, false);
      if (err != cudaSuccess) return err;
    }
  }
  by_channels(kw, [&](auto c) {
    constexpr int KW = decltype(c)::value;
    if (!tiled) {
      launch_next(attention_weight_grad_kernel<KW>, dim3((unsigned)blocks, 2 * chunks), AT_THREADS, 0, st, jobs, d.Kc, d.B, d.H1, d.W1);
    } else if constexpr (KW <= WG_MAX_CHANNELS) {
      launch_next(tma ? attention_weight_grad_tiled_kernel<KW, FEED_TMA> : attention_weight_grad_tiled_kernel<KW, FEED_COPIES>,
                  dim3((unsigned)blocks, chunks), wg_threads(tma ? FEED_TMA : FEED_COPIES), 0, st, maps_x, maps_gl, jobs, d.Kc, d.B, d.H1, d.W1,
                  status);
    }
  });
  if ((err = cudaGetLastError()) != cudaSuccess) return err;
  launch_next(attention_reduce_partials_kernel, columns, RP_THREADS, 0, st, sums);
  return cudaGetLastError();
}

}  // namespace sfb
