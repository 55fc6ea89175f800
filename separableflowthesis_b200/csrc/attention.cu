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
//  * latency: a thread needs plane e+1 only after it is done with plane e, so on its own it has one plane of
//    loads in flight.  Each thread therefore prefetches its neighbourhoods a few planes ahead with cp.async into
//    a ring of shared-memory slots that only it reads (no block barrier), see PlaneRing.
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
#include <mutex>
#include <type_traits>

#include "kernels.h"
#include "sm100_primitives.cuh"

namespace sfb {

constexpr int AT_THREADS = 128;
constexpr int AT_TAPS = 27;
constexpr int AT_KC = 4;  // channels per launch of the forward / logit-gradient kernels and per constant-memory stage

// Filter weights (k, c, td, th, tw) of the channels the running kernel works on, of both modules.
constexpr int AT_WEIGHTS = AT_KC * 2 * AT_TAPS;
__constant__ float c_att_weights[2 * AT_WEIGHTS];

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
          acc[2][k] = fmaf(xv, c_att_weights[MODULE * AT_WEIGHTS + (k * 2 + c) * AT_TAPS + n], acc[2][k]);
          acc[1][k] = fmaf(xv, c_att_weights[MODULE * AT_WEIGHTS + (k * 2 + c) * AT_TAPS + 9 + n], acc[1][k]);
          acc[0][k] = fmaf(xv, c_att_weights[MODULE * AT_WEIGHTS + (k * 2 + c) * AT_TAPS + 18 + n], acc[0][k]);
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

// ---- logits, pixel tiles fetched by TMA -----------------------------------------------------------------
// A block owns a tile of AT_TW x AT_TH image-1 pixels.  A producer warp fetches, plane by plane, the tile of both
// input channels with its one-pixel halo as ONE tiled TMA load into a ring of stages (the box starts 4 pixels to the
// left so that its x coordinate is a multiple of 16 bytes; pixels outside the image arrive as zeros, which is the
// convolution's zero padding), and the 128 pixel threads read their 18 neighbours from shared memory at constant
// offsets.  Against the gather above this removes the 18 per-thread copies per plane and their address arithmetic,
// which were a third of the instructions of an issue-bound kernel.  Needs W1 % 4 == 0 (TMA strides are multiples of
// 16 bytes).  grid of ceil(W1/32) * ceil(H1/4) * B * pieces blocks per job, block 128 + 32.
constexpr int AT_TW = 32, AT_TH = 4;
constexpr int AT_BOX_W = AT_TW + 8, AT_BOX_H = AT_TH + 2;
constexpr int AT_TSTAGES = 6;

// A TMA destination in shared memory must be 128-byte aligned; one channel's tile is 960 bytes, so every stage is
// padded to a multiple of 128.
constexpr uint32_t AT_TILE_BYTES = AT_BOX_H * AT_BOX_W * sizeof(float);
template <int NCH>
struct alignas(128) AttentionTileStage {
  float v[NCH][AT_BOX_H][AT_BOX_W];
};
template <int NCH>
struct AttentionTileSmem {
  AttentionTileStage<NCH> x[AT_TSTAGES];
  uint64_t full[AT_TSTAGES];
  uint64_t empty[AT_TSTAGES];
  WaitCtl ctl;
};

// A block of a job: its pixel tile, sample and piece of the walk.
struct TileBlock {
  int w0, h0, b, piece;
};
__device__ __forceinline__ TileBlock tile_block(int r, int B, int H1, int W1) {
  const int tx = (W1 + AT_TW - 1) / AT_TW, tiles = tx * ((H1 + AT_TH - 1) / AT_TH);
  const int z = r / tiles, t = r - z * tiles, ty = t / tx;
  return TileBlock{(t - ty * tx) * AT_TW, ty * AT_TH, z % B, z / B};
}
struct TileMaps {
  CUtensorMap m[MAX_ATTENTION_JOBS];
};

// The planes e0 .. e0 + n_planes - 1 of a tile, one box of `channel0` .. per plane.
template <int NCH, class Smem>
__device__ __forceinline__ void tile_producer(Smem& sm, const CUtensorMap* tm, const TileBlock& t, int e0, int n_planes, int channel0,
                                              int* status) {
  for (int i = 0; i < n_planes; ++i) {
    const uint32_t s = i % AT_TSTAGES, ph = (i / AT_TSTAGES) & 1u;
    if (!mbar_wait(&sm.empty[s], ph ^ 1u, &sm.ctl, status, DEV_TIMEOUT_PRODUCER)) return;
    mbar_expect_tx(&sm.full[s], NCH * AT_TILE_BYTES);
    tma_load_5d(sm.x[s].v, tm, &sm.full[s], t.w0 - 4, t.h0 - 1, e0 + i, channel0, t.b);
  }
}

template <int KC, int MODULE>   // false: a wait ran out
__device__ __forceinline__ bool logits_walk_tiled(AttentionTileSmem<2>& sm, const LogitsJobs::Job& job, const TileBlock& t, int Kc, int k0,
                                                  int d0, int d1, int e0, int n_planes, int ty, int tx, int H1, int W1, int* status) {
  const int D = job.D, h = t.h0 + ty, w = t.w0 + tx;
  const bool valid = h < H1 && w < W1;
  const size_t plane = (size_t)H1 * W1;
  float* out = job.a + ((size_t)t.b * Kc + k0) * D * plane + (size_t)(valid ? h * W1 + w : 0);

  float bk[KC], acc[3][KC];
#pragma unroll
  for (int k = 0; k < KC; ++k) {
    bk[k] = __ldg(job.bias + k0 + k);
    acc[0][k] = acc[1][k] = acc[2][k] = bk[k];
  }
  auto emit = [&](int d) {  // logit d is complete in acc[0]
#pragma unroll
    for (int k = 0; k < KC; ++k)
      if (valid) out[((size_t)k * D + d) * plane] = acc[0][k];
  };
  for (int i = 0; i < n_planes; ++i) {  // plane e feeds logits e+1 (tap td=0), e (td=1), e-1 (td=2)
    const int e = e0 + i;
    const uint32_t s = i % AT_TSTAGES, ph = (i / AT_TSTAGES) & 1u;
    if (!mbar_wait_warp(&sm.full[s], ph, &sm.ctl, status, DEV_TIMEOUT_EPILOGUE)) return false;
    float xv[2][9];
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int n = 0; n < 9; ++n) xv[c][n] = sm.x[s].v[c][ty + n / 3][tx + 3 + n % 3];
    hand_back_stage(&sm.empty[s], tx);   // the neighbourhoods are in registers
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int n = 0; n < 9; ++n) {
#pragma unroll
        for (int k = 0; k < KC; ++k) {
          acc[2][k] = fmaf(xv[c][n], c_att_weights[MODULE * AT_WEIGHTS + (k * 2 + c) * AT_TAPS + n], acc[2][k]);
          acc[1][k] = fmaf(xv[c][n], c_att_weights[MODULE * AT_WEIGHTS + (k * 2 + c) * AT_TAPS + 9 + n], acc[1][k]);
          acc[0][k] = fmaf(xv[c][n], c_att_weights[MODULE * AT_WEIGHTS + (k * 2 + c) * AT_TAPS + 18 + n], acc[0][k]);
        }
      }
    if (e > d0) emit(e - 1);
#pragma unroll
    for (int k = 0; k < KC; ++k) { acc[0][k] = acc[1][k]; acc[1][k] = acc[2][k]; acc[2][k] = bk[k]; }
  }
  if (d1 == D) emit(D - 1);
  return true;
}

template <int KC, bool SOFT>
__global__ void __launch_bounds__(AT_THREADS + 32)
attention_logits_tiled_kernel(const __grid_constant__ TileMaps maps, const __grid_constant__ LogitsJobs jobs, int Kc, int k0, int B,
                              int H1, int W1, int* status) {
  if (!cta_has_work(status)) return;
  __shared__ __align__(128) AttentionTileSmem<2> sm;
  const int ji = job_of(jobs.blocks, blockIdx.x);
  const LogitsJobs::Job& job = jobs.j[ji];
  const TileBlock t = tile_block(blockIdx.x - jobs.blocks.first[ji], B, H1, W1);
  const int d0 = t.piece * job.dc, d1 = min(d0 + job.dc, job.D);
  const int e0 = max(d0 - 1, 0), n_planes = min(d1 + 1, job.D) - e0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < AT_TSTAGES; ++s) { mbar_init(&sm.full[s], 1); mbar_init(&sm.empty[s], AT_THREADS / 32); }
    wait_ctl_init(&sm.ctl, 0);
    fence_barrier_init();
    prefetch_tensormap(&maps.m[ji]);
  }
  __syncthreads();
  if (warp == AT_THREADS / 32) {
    if (lane == 0) tile_producer<2>(sm, &maps.m[ji], t, e0, n_planes, 0, status);
    __syncwarp();
  } else {
    bool ok = true;
    by_module(job.module, [&](auto m) {
      ok = logits_walk_tiled<KC, decltype(m)::value>(sm, job, t, Kc, k0, d0, d1, e0, n_planes, warp, lane, H1, W1, status);
    });
    const int h = t.h0 + warp, w = t.w0 + lane;
    if (SOFT && ok && h < H1 && w < W1) softmax_columns<KC>(job, Kc, k0, t.b, h * W1 + w, (size_t)H1 * W1);
  }
  __syncthreads();
  if (wait_ctl_aborted(&sm.ctl)) {
    let_copies_land();
  }
}

// ---- softmax over d, in place -------------------------------------------------------------------------------
// A block owns 32 consecutive pixels of one (sample, channel); warp g takes displacements g, g + 8, ... and keeps its
// V = ceil(D / 8) values in registers, so that every logit is read once and every weight written once (HBM-bound, all
// loads of a thread in flight together).  V = 0: any D, the values are read again in each of the three walks.  The
// order of the sums depends on D only.  grid of ceil(N1/32) * planes (= B * Kc) blocks per job, block 256.
constexpr int SM_THREADS = SM_GROUPS * 32;
struct SoftmaxJobs {
  JobBlocks blocks;
  float* a[MAX_ATTENTION_JOBS];
  int D[MAX_ATTENTION_JOBS];
};

template <int V>
__global__ void __launch_bounds__(SM_THREADS, V == 0 ? 8 : (V <= 8 ? 6 : (V <= 20 ? 3 : 2)))
attention_softmax_kernel(const __grid_constant__ SoftmaxJobs jobs, int N1, unsigned pixel_blocks) {
  __shared__ float red[2][SM_GROUPS][32];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int ji = job_of(jobs.blocks, blockIdx.x), D = jobs.D[ji];
  const unsigned block = blockIdx.x - jobs.blocks.first[ji], row = block / pixel_blocks;
  const int p = (int)(block - row * pixel_blocks) * 32 + lane;
  const bool in = p < N1;
  float* base = jobs.a[ji] + (size_t)row * D * N1 + (in ? p : 0);
  constexpr int NV = V > 0 ? V : 1;
  float v[NV];
  float m = -INFINITY;
  if constexpr (V > 0) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int d = g + i * SM_GROUPS;
      v[i] = in && d < D ? base[(size_t)d * N1] : -INFINITY;
    }
#pragma unroll
    for (int i = 0; i < V; ++i) m = fmaxf(m, v[i]);
  } else {
    for (int d = g; d < D; d += SM_GROUPS) m = fmaxf(m, in ? base[(size_t)d * N1] : 0.f);
  }
  red[0][g][lane] = m;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < SM_GROUPS; ++i) m = fmaxf(m, red[0][i][lane]);
  float l = 0.f;
  if constexpr (V > 0) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      if (g + i * SM_GROUPS < D) {
        v[i] = __expf(v[i] - m);
        l += v[i];
      }
    }
  } else {
    for (int d = g; d < D; d += SM_GROUPS) l += __expf((in ? base[(size_t)d * N1] : 0.f) - m);
  }
  red[1][g][lane] = l;
  __syncthreads();
  l = 0.f;
#pragma unroll
  for (int i = 0; i < SM_GROUPS; ++i) l += red[1][i][lane];
  const float inv = 1.f / l;
  if (!in) return;
  if constexpr (V > 0) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int d = g + i * SM_GROUPS;
      if (d < D) base[(size_t)d * N1] = v[i] * inv;
    }
  } else {
    for (int d = g; d < D; d += SM_GROUPS) base[(size_t)d * N1] = __expf(base[(size_t)d * N1] - m) * inv;
  }
}

// Tensor map over a channels-first tensor (B, nch, D, H1, W1) whose samples are `sb` elements apart; the box is one
// plane's pixel tile of `box_ch` channels, with the stencil's halo or without.
static cudaError_t tile_map(CUtensorMap* tm, const float* x, long long sb, int nch, int box_ch, const AttentionDims& d,
                            bool halo) {
  const uint64_t N1 = (uint64_t)d.H1 * d.W1;
  const uint64_t dims[5] = {(uint64_t)d.W1, (uint64_t)d.H1, (uint64_t)d.D, (uint64_t)nch, (uint64_t)d.B};
  const uint64_t strides[4] = {(uint64_t)d.W1 * 4, N1 * 4, (uint64_t)d.D * N1 * 4, (uint64_t)sb * 4};
  const uint32_t box[5] = {(uint32_t)(halo ? AT_BOX_W : AT_TW), (uint32_t)(halo ? AT_BOX_H : AT_TH), 1, (uint32_t)box_ch, 1};
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
        // neighbour n = (nh, nw) holds gL at (h + nh - 1, w + nw - 1), which meets tap th = 2 - nh, tw = 2 - nw
        const int t = (2 - n / 3) * 3 + (2 - n % 3);
        const float v = *ring.slot(s, k * 9 + n);
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int td = 0; td < 3; ++td)
            acc[c][td] = fmaf(v, c_att_weights[MODULE * AT_WEIGHTS + (k * 2 + c) * AT_TAPS + td * 9 + t], acc[c][td]);
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

// ---- input and weight gradients, pixel tiles fetched by TMA -------------------------------------------------
// Same arithmetic as the two gather kernels above with the tile scheme of attention_logits_tiled_kernel.
// Input gradients: the stage holds the tile (with halo) of the KC logit-gradient channels of one plane.
template <int KC, int MODULE>
__device__ __forceinline__ void input_grad_walk_tiled(AttentionTileSmem<KC>& sm, const InputGradJobs::Job& job, const TileBlock& t,
                                                      int accumulate, int k0, int d0, int d1, int e0, int n_planes, int ty, int tx, int H1,
                                                      int W1, int* status) {
  const int D = job.D, h = t.h0 + ty, w = t.w0 + tx;
  const bool valid = h < H1 && w < W1;
  const size_t plane = (size_t)H1 * W1, p = valid ? (size_t)h * W1 + w : 0;
  float* o0 = job.gx + (size_t)t.b * 2 * D * plane + p;
  const float* ad = job.add != nullptr && k0 == 0 ? job.add + (size_t)t.b * job.add_sb + p : nullptr;
  float acc[2][3];  // [c][output d = e-1, e, e+1]
#pragma unroll
  for (int c = 0; c < 2; ++c) acc[c][0] = acc[c][1] = acc[c][2] = 0.f;
  auto emit = [&](int d) {
    if (!valid) return;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const size_t i = ((size_t)c * D + d) * plane;
      float v = acc[c][0];
      if (ad != nullptr) v += __ldg(ad + i);
      if (accumulate) v += o0[i];
      o0[i] = v;
    }
  };
  for (int i = 0; i < n_planes; ++i) {  // plane e of gL feeds gX planes e-1 (td=0), e (td=1), e+1 (td=2)
    const int e = e0 + i;
    const uint32_t s = i % AT_TSTAGES, ph = (i / AT_TSTAGES) & 1u;
    if (!mbar_wait_warp(&sm.full[s], ph, &sm.ctl, status, DEV_TIMEOUT_EPILOGUE)) return;
    float v[KC][9];
#pragma unroll
    for (int k = 0; k < KC; ++k)
#pragma unroll
      for (int n = 0; n < 9; ++n) v[k][n] = sm.x[s].v[k][ty + n / 3][tx + 3 + n % 3];
    hand_back_stage(&sm.empty[s], tx);
#pragma unroll
    for (int k = 0; k < KC; ++k)
#pragma unroll
      for (int n = 0; n < 9; ++n) {
        // neighbour n = (nh, nw) holds gL at (h + nh - 1, w + nw - 1), which meets tap th = 2 - nh, tw = 2 - nw
        const int tap = (2 - n / 3) * 3 + (2 - n % 3);
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int td = 0; td < 3; ++td)
            acc[c][td] = fmaf(v[k][n], c_att_weights[MODULE * AT_WEIGHTS + (k * 2 + c) * AT_TAPS + td * 9 + tap], acc[c][td]);
      }
    if (e > d0) emit(e - 1);
#pragma unroll
    for (int c = 0; c < 2; ++c) { acc[c][0] = acc[c][1]; acc[c][1] = acc[c][2]; acc[c][2] = 0.f; }
  }
  if (d1 == D) emit(D - 1);
}

template <int KC>
__global__ void __launch_bounds__(AT_THREADS + 32)
attention_input_grad_tiled_kernel(const __grid_constant__ TileMaps maps, const __grid_constant__ InputGradJobs jobs, int accumulate, int k0,
                                  int B, int H1, int W1, int* status) {
  if (!cta_has_work(status)) return;
  __shared__ __align__(128) AttentionTileSmem<KC> sm;
  const int ji = job_of(jobs.blocks, blockIdx.x);
  const InputGradJobs::Job& job = jobs.j[ji];
  const TileBlock t = tile_block(blockIdx.x - jobs.blocks.first[ji], B, H1, W1);
  const int d0 = t.piece * job.dc, d1 = min(d0 + job.dc, job.D);
  const int e0 = max(d0 - 1, 0), n_planes = min(d1 + 1, job.D) - e0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < AT_TSTAGES; ++s) { mbar_init(&sm.full[s], 1); mbar_init(&sm.empty[s], AT_THREADS / 32); }
    wait_ctl_init(&sm.ctl, 0);
    fence_barrier_init();
    prefetch_tensormap(&maps.m[ji]);
  }
  __syncthreads();
  if (warp == AT_THREADS / 32) {
    if (lane == 0) tile_producer<KC>(sm, &maps.m[ji], t, e0, n_planes, k0, status);
    __syncwarp();
  } else {
    by_module(job.module, [&](auto m) {
      input_grad_walk_tiled<KC, decltype(m)::value>(sm, job, t, accumulate, k0, d0, d1, e0, n_planes, warp, lane, H1, W1, status);
    });
  }
  __syncthreads();
  if (wait_ctl_aborted(&sm.ctl)) {
    let_copies_land();
  }
}

// Weight gradients: warps 0-3 own input channel 0, warps 4-7 input channel 1, each thread KW output channels of its
// pixel; the stage holds the tile (with halo) of plane e of both X channels and the tile (without halo) of plane e+1 of
// the KW logit-gradient channels, which the two halves share.  The sums of two output channels are one packed pair
// (fma.rn.f32x2 with the X value in both halves), which halves the multiply-add instructions; KW odd leaves one
// channel on scalar ones.  A piece is `dc` planes of X.
// grid (ceil(W1/32) * ceil(H1/4) * B * pieces blocks per job, chunks of KW channels); partial: of the module, (Kc * 2 * 27, rows).
constexpr int WG_WARPS = 8;
template <int KW>
struct WeightGradTileSmem {
  struct alignas(128) Stage {   // both parts are TMA destinations: 128-byte aligned
    alignas(128) float x[2][AT_BOX_H][AT_BOX_W];
    alignas(128) float g[KW][AT_TH][AT_TW];
  } st[AT_TSTAGES];
  uint64_t full[AT_TSTAGES];
  uint64_t empty[AT_TSTAGES];
  WaitCtl ctl;
  float red[WG_WARPS * KW * AT_TAPS];
};

template <int KW>
__global__ void __launch_bounds__(WG_WARPS * 32 + 32, 1)
attention_weight_grad_tiled_kernel(const __grid_constant__ TileMaps maps_x, const __grid_constant__ TileMaps maps_gl,
                                   const __grid_constant__ WeightGradJobs jobs, int Kc, int B, int H1, int W1, int* status) {
  if (!cta_has_work(status)) return;
  __shared__ __align__(128) WeightGradTileSmem<KW> sm;
  constexpr int KP = KW / 2;   // packed channel pairs
  const int ji = job_of(jobs.blocks, blockIdx.x), r = blockIdx.x - jobs.blocks.first[ji];
  const WeightGradJobs::Job& job = jobs.j[ji];
  const TileBlock tb = tile_block(r, B, H1, W1);
  const int w0 = tb.w0, h0 = tb.h0, b = tb.b, k0 = blockIdx.y * KW, D = job.D;
  const float* __restrict__ const gl = job.gl;
  const CUtensorMap *const tm_x = &maps_x.m[ji], *const tm_gl = &maps_gl.m[ji];
  const int e0 = tb.piece * job.dc, n_planes = min(job.dc, D - e0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < AT_TSTAGES; ++s) { mbar_init(&sm.full[s], 1); mbar_init(&sm.empty[s], WG_WARPS); }
    wait_ctl_init(&sm.ctl, 0);
    fence_barrier_init();
    prefetch_tensormap(tm_x);
    prefetch_tensormap(tm_gl);
  }
  __syncthreads();
  if (warp == WG_WARPS) {  // producer
    if (lane == 0) {
      for (int i = 0; i < n_planes; ++i) {
        const uint32_t s = i % AT_TSTAGES, ph = (i / AT_TSTAGES) & 1u;
        if (!mbar_wait(&sm.empty[s], ph ^ 1u, &sm.ctl, status, DEV_TIMEOUT_PRODUCER)) { let_copies_land(); break; }
        mbar_expect_tx(&sm.full[s], 2 * AT_TILE_BYTES + KW * AT_TH * AT_TW * (uint32_t)sizeof(float));
        tma_load_5d(sm.st[s].x, tm_x, &sm.full[s], w0 - 4, h0 - 1, e0 + i, 0, b);
        tma_load_5d(sm.st[s].g, tm_gl, &sm.full[s], w0, h0, e0 + i + 1, k0, b);  // plane D, channels >= Kc read as zero
      }
    }
    return;
  }
  const int tx = lane, ty = warp & 3, c = warp >> 2;
  const int h = h0 + ty, w = w0 + tx;
  const bool valid = h < H1 && w < W1;
  const size_t plane = (size_t)H1 * W1;
  uint64_t acc2[KP > 0 ? KP * AT_TAPS : 1];         // [pair][td][neighbour]
  float acc1[(KW & 1) != 0 ? AT_TAPS : 1];          // the odd channel
#pragma unroll
  for (int i = 0; i < KP * AT_TAPS; ++i) acc2[i] = 0ull;
  if constexpr ((KW & 1) != 0) {
#pragma unroll
    for (int i = 0; i < AT_TAPS; ++i) acc1[i] = 0.f;
  }
  float g_prev[KW], g_cur[KW], g_next[KW];
#pragma unroll
  for (int k = 0; k < KW; ++k) {
    const bool ok = valid && k0 + k < Kc;
    const float* gp = gl + (((size_t)b * Kc + (ok ? k0 + k : 0)) * D + e0) * plane + (ok ? (size_t)h * W1 + w : 0);
    g_prev[k] = (ok && e0 > 0) ? __ldg(gp - plane) : 0.f;
    g_cur[k] = ok ? __ldg(gp) : 0.f;
  }
  bool alive = true;
  for (int i = 0; i < n_planes; ++i) {  // plane e of X meets gL at d = e+1 (td=0), e (td=1), e-1 (td=2)
    const uint32_t s = i % AT_TSTAGES, ph = (i / AT_TSTAGES) & 1u;
    const bool ok = mbar_wait(&sm.full[s], ph, &sm.ctl, status, DEV_TIMEOUT_EPILOGUE);
    if (!__all_sync(0xffffffffu, ok)) { let_copies_land(); alive = false; break; }
    float v[9];
#pragma unroll
    for (int n = 0; n < 9; ++n) v[n] = sm.st[s].x[c][ty + n / 3][tx + 3 + n % 3];
#pragma unroll
    for (int k = 0; k < KW; ++k) g_next[k] = sm.st[s].g[k][ty][tx];
    hand_back_stage(&sm.empty[s], lane);
#pragma unroll
    for (int q = 0; q < KP; ++q) {
      const uint64_t gn = pack2(g_next[2 * q], g_next[2 * q + 1]), gc = pack2(g_cur[2 * q], g_cur[2 * q + 1]),
                     gp = pack2(g_prev[2 * q], g_prev[2 * q + 1]);
#pragma unroll
      for (int n = 0; n < 9; ++n) {
        const uint64_t vv = pack2(v[n], v[n]);
        acc2[q * AT_TAPS + n] = fma2(gn, vv, acc2[q * AT_TAPS + n]);
        acc2[q * AT_TAPS + 9 + n] = fma2(gc, vv, acc2[q * AT_TAPS + 9 + n]);
        acc2[q * AT_TAPS + 18 + n] = fma2(gp, vv, acc2[q * AT_TAPS + 18 + n]);
      }
    }
    if constexpr ((KW & 1) != 0) {
#pragma unroll
      for (int n = 0; n < 9; ++n) {
        acc1[n] = fmaf(g_next[KW - 1], v[n], acc1[n]);
        acc1[9 + n] = fmaf(g_cur[KW - 1], v[n], acc1[9 + n]);
        acc1[18 + n] = fmaf(g_prev[KW - 1], v[n], acc1[18 + n]);
      }
    }
#pragma unroll
    for (int k = 0; k < KW; ++k) { g_prev[k] = g_cur[k]; g_cur[k] = g_next[k]; }
  }
  // reduce over the 128 pixel threads of each input channel (named barrier 1: the producer warp has left);
  // column (k, c, td, n) goes to row (k0 + k) * 54 + c * 27 + td * 9 + n of the partial sums
  auto put = [&](int i, float sum) {
    if (!alive) sum = 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) sm.red[warp * KW * AT_TAPS + i] = sum;
  };
#pragma unroll
  for (int q = 0; q < KP; ++q)
#pragma unroll
    for (int t = 0; t < AT_TAPS; ++t) {
      float lo, hi;
      unpack2(acc2[q * AT_TAPS + t], lo, hi);
      put(2 * q * AT_TAPS + t, lo);
      put((2 * q + 1) * AT_TAPS + t, hi);
    }
  if constexpr ((KW & 1) != 0) {
#pragma unroll
    for (int t = 0; t < AT_TAPS; ++t) put((KW - 1) * AT_TAPS + t, acc1[t]);
  }
  named_bar_sync(1, WG_WARPS * 32);
  const size_t rows = job.rows;
  float* dst = job.partial + job.row0 + r;
  for (int i = threadIdx.x; i < 2 * KW * AT_TAPS; i += WG_WARPS * 32) {
    const int cc = i / (KW * AT_TAPS), j = i - cc * KW * AT_TAPS, k = j / AT_TAPS, t = j - k * AT_TAPS;
    if (k0 + k >= Kc) continue;
    float sum = 0.f;
#pragma unroll
    for (int wv = 0; wv < 4; ++wv) sum += sm.red[(cc * 4 + wv) * KW * AT_TAPS + j];
    dst[(((size_t)(k0 + k) * 2 + cc) * AT_TAPS + t) * rows] = sum;
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
  void* address[AT_MAX_DEVICES] = {nullptr};   // of c_att_weights
} g_stage;

class StagedWeights {
 public:
  explicit StagedWeights(cudaStream_t st) : lock_(g_stage.mu), st_(st) {
    err_ = cudaGetDevice(&dev_);
    if (err_ == cudaSuccess && (dev_ < 0 || dev_ >= AT_MAX_DEVICES)) err_ = cudaErrorInvalidDevice;
    if (err_ != cudaSuccess) return;
    if (g_stage.done[dev_] == nullptr) err_ = cudaEventCreateWithFlags(&g_stage.done[dev_], cudaEventDisableTiming);
    if (err_ == cudaSuccess && g_stage.address[dev_] == nullptr) err_ = cudaGetSymbolAddress(&g_stage.address[dev_], c_att_weights);
    if (err_ == cudaSuccess && g_stage.used[dev_] && g_stage.last[dev_] != st_)
      err_ = cudaStreamWaitEvent(st_, g_stage.done[dev_], 0);
  }
  cudaError_t put(const float* device_weights, int channels, int module = 0) {  // weights of `channels` <= AT_KC channels
    if (err_ != cudaSuccess) return err_;
    err_ = cudaMemcpyAsync(static_cast<float*>(g_stage.address[dev_]) + module * AT_WEIGHTS, device_weights,
                           (size_t)channels * 2 * AT_TAPS * sizeof(float), cudaMemcpyDeviceToDevice, st_);
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

static size_t tile_count(const AttentionDims& d) {
  return (size_t)((d.W1 + AT_TW - 1) / AT_TW) * ((d.H1 + AT_TH - 1) / AT_TH);
}
// Displacements per block of a stencil walk: enough blocks (AT_BLOCKS_TARGET) to fill the 148 SMs several times over,
// but at least AT_MIN_WALK displacements, because every block also reads a plane on either side of its own.
// The weight gradients pay for a reduction over the block at the end of a walk as well and keep one or two blocks on an
// SM, hence fewer and longer pieces.
constexpr int AT_BLOCKS_TARGET = 148 * 8, AT_MIN_WALK = 8;
constexpr int WG_BLOCKS_TARGET = 148 * 3, WG_MIN_WALK = 16;
// The jobs of a launch fill the SMs together, with walks of about the same length: `total` is the sum of their D.  (Every job with as
// many pieces as if it were the only one of its size, 1 x 55 x 128 with four levels and channels spent the last half of its logits on a few
// long walks: 56 us, 50 now.)
static int walk_length(size_t blocks, int D, int total, int target = AT_BLOCKS_TARGET, int min_walk = AT_MIN_WALK) {
  const int pieces = (int)((target + blocks - 1) / blocks);   // of all jobs
  const int dc = std::max((total + pieces - 1) / pieces, min_walk), own = (D + dc - 1) / dc;
  return (D + own - 1) / own;
}
// Displacements per block of the weight gradients' walk, and the blocks of a job (partial sums of a weight).
static int weight_walk(const AttentionDims& d, int total, bool tiled) {
  return walk_length((tiled ? tile_count(d) : 2 * (size_t)pixel_grid(d).x) * d.B, d.D, total, WG_BLOCKS_TARGET, WG_MIN_WALK);
}
static size_t weight_rows(const AttentionDims& d, int total, bool tiled) {
  const int dc = weight_walk(d, total, tiled);
  return (tiled ? tile_count(d) : (size_t)pixel_grid(d).x) * d.B * ((d.D + dc - 1) / dc);
}
// The softmax backward: pixels of a block by the length of the column (attention_logit_grad_kernel).
static int logit_grad_pixels(int D) { return D <= 8 ? lg_pixels(1) : D <= 16 ? lg_pixels(2) : D <= 32 ? lg_pixels(4) : 32; }
static size_t bias_rows(const AttentionDims& d) { return (size_t)d.B * ((d.H1 * d.W1 + logit_grad_pixels(d.D) - 1) / logit_grad_pixels(d.D)); }

// Bias partials per block of the softmax backward, weight partials per block of the weight gradients, whichever form they take.
size_t attention_partial_floats(const AttentionDims* d, int count) {
  size_t floats = 0;
  int total = 0;
  for (int i = 0; i < count; ++i) total += d[i].D;
  for (int i = 0; i < count; ++i)
    floats += d[i].Kc * (bias_rows(d[i]) + 2 * AT_TAPS * std::max(weight_rows(d[i], total, true), weight_rows(d[i], total, false)));
  return floats;
}

// Columns of a class of lengths are done by one launch.
template <int V>
static cudaError_t launch_softmax_class(const AttentionJob* job, int count, int above, int upto, cudaStream_t st) {
  SoftmaxJobs jobs{};
  const AttentionDims& d = job[0].d;
  const unsigned pb = (unsigned)((d.H1 * d.W1 + 31) / 32);
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
  attention_softmax_kernel<V><<<(unsigned)blocks, SM_THREADS, 0, st>>>(jobs, d.H1 * d.W1, pb);
  return cudaGetLastError();
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

template <class Job>
static int total_D(const Job* job, int count) {
  int total = 0;
  for (int i = 0; i < count; ++i) total += job[i].d.D;
  return total;
}
// Displacements per block of the forward's walk, and whether the walks of a launch end with the softmax of their columns.  A column
// short enough for that is not cut by launches that have two blocks per SM without it.
static int forward_walk(const AttentionDims& d, int jobs, int total, bool tiled) {
  const size_t blocks = (tiled ? tile_count(d) : (size_t)pixel_grid(d).x) * d.B;
  return d.D <= AT_SOFT_MAX && blocks * jobs >= 2 * SM_COUNT ? d.D : walk_length(blocks, d.D, total);
}
static bool softmax_in_walk(const AttentionJob* job, int count, bool tiled) {
  const int total = total_D(job, count);
  for (int i = 0; i < count; ++i)
    if (job[i].d.D > AT_SOFT_MAX || forward_walk(job[i].d, count, total, tiled) < job[i].d.D) return false;
  return true;
}
static bool all_tileable(const AttentionJob* job, int count, const int* status) {
  bool ok = status != nullptr;
  for (int i = 0; i < count; ++i) ok = ok && tileable(job[i].d, job[i].x, job[i].x_sb);
  return ok;
}

int attention_forward_launches(const AttentionJob* job, int count, const int* status) {
  const bool tiled = all_tileable(job, count, status);
  int n = (job[0].d.Kc + AT_KC - 1) / AT_KC;
  if (softmax_in_walk(job, count, tiled)) return n;
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
  const bool tiled = all_tileable(job, count, status);
  const bool soft = softmax_in_walk(job, count, tiled);
  TileMaps maps;
  LogitsJobs jobs{};
  unsigned long long blocks = 0;
  for (int i = 0; i < MAX_ATTENTION_JOBS; ++i) {
    jobs.blocks.first[i] = (int)blocks;
    if (i >= count) continue;
    const AttentionJob& j = job[i];
    if (tiled) {
      cudaError_t err = tile_map(&maps.m[i], j.x, j.x_sb, 2, 2, j.d, true);
      if (err != cudaSuccess) return err;
    }
    const int dc = forward_walk(j.d, count, total_D(job, count), tiled);
    jobs.j[i] = LogitsJobs::Job{j.x, j.x_sb, modules.bias[j.module], j.a, j.d.D, dc, j.module};
    blocks += (unsigned long long)(tiled ? tile_count(d) : (size_t)pixel_grid(d).x) * d.B * ((j.d.D + dc - 1) / dc);
    if (blocks > 0x7fffffffull) return cudaErrorInvalidConfiguration;
  }
  jobs.blocks.first[MAX_ATTENTION_JOBS] = (int)blocks;
  {
    StagedWeights staged(st);
    for (int k0 = 0; k0 < d.Kc; k0 += AT_KC) {
      const int kc = d.Kc - k0 < AT_KC ? d.Kc - k0 : AT_KC;
      for (int m = 0; m < 2; ++m) {
        if (modules.weight[m] == nullptr) continue;
        cudaError_t err = staged.put(modules.weight[m] + (size_t)k0 * 2 * AT_TAPS, kc, m);
        if (err != cudaSuccess) return err;
      }
      if (tiled) {
#define SFB_AT_FWD_T(KC) (soft ? attention_logits_tiled_kernel<KC, true> : attention_logits_tiled_kernel<KC, false>)<<<(unsigned)blocks, AT_THREADS + 32, 0, st>>>(maps, jobs, d.Kc, k0, d.B, d.H1, d.W1, status)
        if (kc == 1) SFB_AT_FWD_T(1); else if (kc == 2) SFB_AT_FWD_T(2); else if (kc == 3) SFB_AT_FWD_T(3); else SFB_AT_FWD_T(4);
#undef SFB_AT_FWD_T
        continue;
      }
#define SFB_AT_FWD(KC) (soft ? attention_logits_kernel<KC, true> : attention_logits_kernel<KC, false>)<<<(unsigned)blocks, AT_THREADS, 0, st>>>(jobs, d.Kc, k0, d.B, d.H1, d.W1)
      if (kc == 1) SFB_AT_FWD(1); else if (kc == 2) SFB_AT_FWD(2); else if (kc == 3) SFB_AT_FWD(3); else SFB_AT_FWD(4);
#undef SFB_AT_FWD
    }
  }
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess || soft) return err;
  return launch_softmax(job, count, st);
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
  attention_input_grad_kernel<KC><<<blocks, AT_THREADS, smem, st>>>(jobs, accumulate, d.Kc, k0, d.B, d.H1, d.W1);
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
  attention_logit_grad_kernel<G, V, MIN_BLOCKS><<<(unsigned)blocks, 32 * lg_warps(G), 0, st>>>(jobs, d.Kc, d.H1 * d.W1, pb);
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
  int n = (job[0].d.Kc + AT_KC - 1) / AT_KC + 2;   // input gradients per chunk of channels, weight gradients, the reduction
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
  const int N1 = d.H1 * d.W1, total = total_D(job, count);
  auto g_sb = [&](const AttentionGradJob& j) { return (long long)d.Kc * j.d.D * N1; };
  bool tiled = status != nullptr;
  for (int i = 0; i < count; ++i) tiled = tiled && tileable(job[i].d, job[i].x, job[i].x_sb) && tileable(job[i].d, job[i].g, g_sb(job[i]));

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
      wrows += (int)weight_rows(job[i].d, total, tiled);
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
    InputGradJobs jobs{};
    unsigned long long blocks = 0;
    for (int i = 0; i <= MAX_ATTENTION_JOBS; ++i) {
      jobs.blocks.first[i] = (int)blocks;
      if (i >= count) continue;
      const size_t tiles = (tiled ? tile_count(d) : (size_t)pixel_grid(d).x) * d.B;
      const int dc = walk_length(tiles, job[i].d.D, total);
      jobs.j[i] = InputGradJobs::Job{job[i].g, job[i].add, job[i].add_sb, job[i].gx, job[i].d.D, dc, job[i].module};
      blocks += (unsigned long long)tiles * ((job[i].d.D + dc - 1) / dc);
      if (blocks > 0x7fffffffull) return cudaErrorInvalidConfiguration;
    }
    StagedWeights staged(st);
    for (int k0 = 0; k0 < d.Kc; k0 += AT_KC) {
      const int kc = d.Kc - k0 < AT_KC ? d.Kc - k0 : AT_KC, accumulate = k0 == 0 ? 0 : 1;
      for (int m = 0; m < 2; ++m) {
        if (modules.weight[m] == nullptr) continue;
        err = staged.put(modules.weight[m] + (size_t)k0 * 2 * AT_TAPS, kc, m);
        if (err != cudaSuccess) return err;
      }
      if (tiled) {
        TileMaps maps;
        for (int i = 0; i < count; ++i) {
          err = tile_map(&maps.m[i], job[i].g, g_sb(job[i]), d.Kc, kc, job[i].d, true);
          if (err != cudaSuccess) return err;
        }
#define SFB_AT_IG_T(KC) attention_input_grad_tiled_kernel<KC><<<(unsigned)blocks, AT_THREADS + 32, 0, st>>>(maps, jobs, accumulate, k0, d.B, d.H1, d.W1, status)
        if (kc == 1) SFB_AT_IG_T(1); else if (kc == 2) SFB_AT_IG_T(2); else if (kc == 3) SFB_AT_IG_T(3); else SFB_AT_IG_T(4);
#undef SFB_AT_IG_T
        continue;
      }
      if (kc == 1) err = launch_input_grad<1>((unsigned)blocks, jobs, accumulate, d, k0, st);
      else if (kc == 2) err = launch_input_grad<2>((unsigned)blocks, jobs, accumulate, d, k0, st);
      else if (kc == 3) err = launch_input_grad<3>((unsigned)blocks, jobs, accumulate, d, k0, st);
      else err = launch_input_grad<4>((unsigned)blocks, jobs, accumulate, d, k0, st);
      if (err != cudaSuccess) return err;
    }
  }
  const int kw = d.Kc >= 4 ? 4 : d.Kc, chunks = (d.Kc + kw - 1) / kw;
  WeightGradJobs jobs{};
  unsigned long long blocks = 0;
  TileMaps maps_x, maps_gl;
  for (int i = 0; i <= MAX_ATTENTION_JOBS; ++i) {
    jobs.blocks.first[i] = (int)blocks;
    if (i >= count) continue;
    jobs.j[i] = WeightGradJobs::Job{job[i].x, job[i].x_sb, job[i].g, place[i].weight, job[i].d.D, weight_walk(job[i].d, total, tiled),
                                    place[i].weight_row0, place[i].weight_rows};
    blocks += weight_rows(job[i].d, total, tiled);
    if (blocks > 0x7fffffffull) return cudaErrorInvalidConfiguration;
    if (tiled) {
      err = tile_map(&maps_x.m[i], job[i].x, job[i].x_sb, 2, 2, job[i].d, true);
      if (err == cudaSuccess) err = tile_map(&maps_gl.m[i], job[i].g, g_sb(job[i]), d.Kc, kw, job[i].d, false);
      if (err != cudaSuccess) return err;
    }
  }
  if (tiled) {
#define SFB_AT_WG_T(KW) attention_weight_grad_tiled_kernel<KW><<<dim3((unsigned)blocks, chunks), WG_WARPS * 32 + 32, 0, st>>>(maps_x, maps_gl, jobs, d.Kc, d.B, d.H1, d.W1, status)
    if (kw == 1) SFB_AT_WG_T(1); else if (kw == 2) SFB_AT_WG_T(2); else if (kw == 3) SFB_AT_WG_T(3); else SFB_AT_WG_T(4);
#undef SFB_AT_WG_T
  } else {
#define SFB_AT_WG(KW) attention_weight_grad_kernel<KW><<<dim3((unsigned)blocks, 2 * chunks), AT_THREADS, 0, st>>>(jobs, d.Kc, d.B, d.H1, d.W1)
    if (kw == 1) SFB_AT_WG(1); else if (kw == 2) SFB_AT_WG(2); else if (kw == 3) SFB_AT_WG(3); else SFB_AT_WG(4);
#undef SFB_AT_WG
  }
  if ((err = cudaGetLastError()) != cudaSuccess) return err;
  attention_reduce_partials_kernel<<<columns, RP_THREADS, 0, st>>>(sums);
  return cudaGetLastError();
}

}  // namespace sfb
