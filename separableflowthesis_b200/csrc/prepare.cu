// Operand preparation (HBM-bound, a few percent of an op's time):
//  * copies of F1 and F2 rounded to TF32 with round-to-nearest.  tcgen05.mma kind::tf32 ignores the
//    low 13 mantissa bits of its fp32 operands, i.e. truncates; truncation shrinks every product by
//    ~2^-10 and would put a bias of that relative size on every S value, rounding does not.
//  * the "aux" rows of F2 used for the mean channels: row u of aux = mean over v of F2[u,v,:],
//    row H2+v = mean over u of F2[u,v,:]  (mean_v S[p,u,v] = F1[p] . mean_v F2[u,v], the same sum the
//    reference accumulates cell by cell, MemorySaver_kernel_forward.cu:286-290).
//  * 16-bit operand copies (BF16, or FP16 for the operand type with TF32's mantissa at twice its tensor-core rate).
//    FP16 has a narrow exponent range, so every tensor that becomes an FP16 operand is first multiplied by a power
//    of two that brings its largest magnitude next to 1 (exact, undone when results are stored): absmax_kernel
//    finds the magnitudes and its last block turns them into the multipliers, all on the device.
// The FP32 copies are made for TF32 operands only; with 16-bit operands every reader takes the 16-bit copies or the
// caller's features themselves.
#include <algorithm>
#include <climits>

#include <cuda_bf16.h>

#include "kernels.h"
#include "sm100_primitives.cuh"

namespace sfb {

// The power of two that brings a largest magnitude (float bits in `amax_bits`) into [target, 2*target); 1 when the
// magnitude is zero, not finite or subnormal, and never beyond 2^+-40, so that products of three scales stay finite
// (tensors whose largest magnitude lies outside about 1e-12 .. 1e12 are not brought all the way into FP16's range;
// TF32 operands are the choice for such data).
__device__ __forceinline__ float pow2_scale(unsigned amax_bits, int target_log2) {
  const int e = (int)(amax_bits >> 23) & 0xff;
  if (e == 0 || e == 255) return 1.f;
  int shift = target_log2 - (e - 127);
  shift = max(-40, min(40, shift));
  return __uint_as_float((unsigned)(127 + shift) << 23);
}

// scales[] (SCALE_* in kernels.h): feature scales from the two magnitudes found by absmax_kernel (image 1's: amax1).
__device__ void feature_scales(float* scales, const float* amax1) {
  const float s1 = pow2_scale(__float_as_uint(__ldcg(amax1)), 0);
  const float s2 = pow2_scale(__float_as_uint(__ldcg(scales + SCALE_AMAX_F2)), 0);
  scales[SCALE_F1] = s1;
  scales[SCALE_F2] = s2;
  scales[SCALE_INV_F1F2] = 1.f / (s1 * s2);
}
// Gradient-operand scales (after the feature scales of the same call): G is generated as (sg * sa) * G.
__device__ void grad_scales(float* scales) {
  const float sg = pow2_scale(__float_as_uint(__ldcg(scales + SCALE_AMAX_G)), 7);   // largest gradient value -> [128, 256)
  const float sa = pow2_scale(__float_as_uint(__ldcg(scales + SCALE_AMAX_A)), 0);   // largest weight -> [1, 2)
  scales[SCALE_GA] = sg * sa;
  scales[SCALE_G] = sg;
  scales[SCALE_A] = sa;
  scales[SCALE_INV_GF1] = 1.f / (sg * sa * scales[SCALE_F2]);   // gF1 = G * F2
  scales[SCALE_INV_GF2] = 1.f / (sg * sa * scales[SCALE_F1]);   // gF2 = G^T * F1
}

// Largest |x| * premul of up to ABSMAX_MAX arrays, each as the bits of a non-negative float combined into its slot of
// scales[] with atomicMax (integer order = float order for non-negative values; NaNs are ignored), one atomic per
// block; the block that finishes last (SCALE_TICKET counts them, and is left at zero) turns the magnitudes of every level into the
// multipliers.  One launch in place of one per array and one for the multipliers.  Every array has blocks for its own size: with those of
// the largest for all, the coarse levels of a pyramid had as many that found nothing, and each took a ticket (five maps of 1 x 55 x 128,
// C = 256: 9.8 us, 7.8 now; of 4 x 55 x 128 19.9 and 16.6).  grid of the blocks of every sample of every array, block 256.
constexpr int AM_THREADS = 256, AM_UNROLL = 4;
struct AbsmaxJobs {
  AbsmaxSource src[ABSMAX_MAX];
  int first[ABSMAX_MAX];    // blocks; sources that do not exist start past the end of the grid
  int blocks[ABSMAX_MAX];   // of a sample
};
__global__ void __launch_bounds__(AM_THREADS)
absmax_kernel(const __grid_constant__ AbsmaxJobs jobs, float* scales, int levels, int gradients) {
  follow_previous_kernel();
  __shared__ float red[AM_THREADS / 32];
  int job = 0;
#pragma unroll
  for (int j = 1; j < ABSMAX_MAX; ++j) job = (int)blockIdx.x >= jobs.first[j] ? j : job;
  const AbsmaxSource& src = jobs.src[job];
  const int blocks = jobs.blocks[job], r = blockIdx.x - jobs.first[job], sample = r / blocks, block = r - sample * blocks;
  const float* x = src.p + (size_t)sample * src.sb;
  // a sample's channels may start off a 16-byte boundary: up to three values before the first vector, up to three behind the last
  const size_t n = src.n, head = min((size_t)((16u - (reinterpret_cast<uintptr_t>(x) & 15u)) & 15u) / 4, n);
  const size_t n4 = (n - head) / 4, stride = (size_t)blocks * AM_THREADS;
  const float4* x4 = reinterpret_cast<const float4*>(x + head);
  float m = 0.f;
  for (size_t i = (size_t)block * AM_THREADS + threadIdx.x; i < n4; i += AM_UNROLL * stride) {
    float4 v[AM_UNROLL];
#pragma unroll
    for (int j = 0; j < AM_UNROLL; ++j) v[j] = i + j * stride < n4 ? __ldg(x4 + i + j * stride) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < AM_UNROLL; ++j)
      m = fmaxf(m, fmaxf(fmaxf(fabsf(v[j].x), fabsf(v[j].y)), fmaxf(fabsf(v[j].z), fabsf(v[j].w))));
  }
  if (block == 0 && threadIdx.x < head) m = fmaxf(m, fabsf(__ldg(x + threadIdx.x)));
  if (block == 0 && threadIdx.x < n - head - 4 * n4) m = fmaxf(m, fabsf(__ldg(x + head + 4 * n4 + threadIdx.x)));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x != 0) return;
#pragma unroll
  for (int i = 1; i < AM_THREADS / 32; ++i) m = fmaxf(m, red[i]);
  if (m > 0.f) atomicMax(reinterpret_cast<unsigned*>(scales) + src.slot, __float_as_uint(m * fabsf(src.premul)));
  __threadfence();
  unsigned* ticket = reinterpret_cast<unsigned*>(scales) + SCALE_TICKET;
  if (atomicAdd(ticket, 1u) != gridDim.x - 1) return;
  __threadfence();
  for (int l = 0; l < levels; ++l) {
    if (gradients) grad_scales(scales + l * SCALE_LEVEL);
    else feature_scales(scales + l * SCALE_LEVEL, scales + SCALE_AMAX_F1);
  }
  *ticket = 0;
}

// The coarser levels of image 2, each the 2 x 2 average of the one before (core/corr.py:377-382, in avg_pool2d's order of additions), and
// with FP16 operands the magnitudes of all levels and of image 1 and the multipliers that follow, in one launch: one walk over both images
// in place of a launch per level and one over all of them.  A thread makes what 8 x 8 pixels of a plane contribute, so that no level
// is read back.  HBM-bound.  1 x 55 x 128, C = 256, three levels from one: 23 us in four launches (averages and magnitudes), 9 now.
// grid: blocks of 256 of the planes' 8 x 8 regions, then those of image 1; block 256.
struct PoolJob {
  const float* in;              // (planes, H, W)
  float* out[MAX_FUSED_LEVELS - 1];
  int planes, H, W, levels;     // levels made here
  const float* image1;
  size_t n1;
  float premul1;
  int blocks2;                  // blocks of image 2
};
static_assert(MAX_FUSED_LEVELS == 4, "8 x 8 pixels are one of the coarsest level");
template <bool VEC, bool MAGNITUDES>
__global__ void __launch_bounds__(AM_THREADS)
pool_levels_kernel(const __grid_constant__ PoolJob job, float* scales) {
  follow_previous_kernel();
  constexpr int SLOTS = MAX_FUSED_LEVELS + 1;   // magnitudes of the levels of image 2, of image 1
  float m[SLOTS];
#pragma unroll
  for (int i = 0; i < SLOTS; ++i) m[i] = 0.f;
  if ((int)blockIdx.x < job.blocks2) {
    const int H = job.H, W = job.W, rw = (W + 7) / 8, rh = (H + 7) / 8;
    const long long i = (long long)blockIdx.x * AM_THREADS + threadIdx.x;
    const int plane = (int)(i / (rw * rh)), r = (int)(i - (long long)plane * (rw * rh)), ry = r / rw, rx = r - ry * rw;
    if (plane < job.planes) {
      const float* in = job.in + (size_t)plane * H * W + rx * 8;
      float fine[2][8], mid[2][4], top[2][2];   // rows of level 0, 1 and 2 that make a row of the next
      // one row of a level from two of the one before; stored where it exists
      auto next = [&](int l, int y, const float* upper, const float* lower, float* out, int n, float& most) {
        const int h = H >> l, w = W >> l, x0 = rx * n;
        float* dst = l <= job.levels ? job.out[l - 1] + ((size_t)plane * h + y) * w + x0 : nullptr;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (j >= n) break;
          out[j] = (((upper[2 * j] + upper[2 * j + 1]) + lower[2 * j]) + lower[2 * j + 1]) * 0.25f;
          if (dst != nullptr && y < h && x0 + j < w) {
            dst[j] = out[j];
            if (MAGNITUDES) most = fmaxf(most, fabsf(out[j]));
          }
        }
      };
#pragma unroll
      for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int y = ry * 8 + 2 * q + k;
          const float* row = in + (size_t)y * W;
          if constexpr (VEC) {
#pragma unroll
            for (int c = 0; c < 8; c += 4) {
              const float4 v = y < H && rx * 8 + c < W ? __ldg(reinterpret_cast<const float4*>(row + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
              fine[k][c] = v.x; fine[k][c + 1] = v.y; fine[k][c + 2] = v.z; fine[k][c + 3] = v.w;
            }
          } else {
#pragma unroll
            for (int c = 0; c < 8; ++c) fine[k][c] = y < H && rx * 8 + c < W ? __ldg(row + c) : 0.f;
          }
          if (MAGNITUDES) {
#pragma unroll
            for (int c = 0; c < 8; ++c) m[0] = fmaxf(m[0], fabsf(fine[k][c]));
          }
        }
        next(1, ry * 4 + q, fine[0], fine[1], mid[q & 1], 4, m[1]);
        if (q & 1) next(2, ry * 2 + q / 2, mid[0], mid[1], top[q / 2], 2, m[2]);
      }
      float last[1];
      next(3, ry, top[0], top[1], last, 1, m[3]);
    }
  } else if (MAGNITUDES) {
    const float4* x4 = reinterpret_cast<const float4*>(job.image1);   // 16-byte aligned
    const size_t n4 = job.n1 / 4, stride = (size_t)(gridDim.x - job.blocks2) * AM_THREADS;
    const size_t at = (size_t)(blockIdx.x - job.blocks2) * AM_THREADS + threadIdx.x;
    for (size_t i = at; i < n4; i += AM_UNROLL * stride) {
      float4 v[AM_UNROLL];
#pragma unroll
      for (int j = 0; j < AM_UNROLL; ++j) v[j] = i + j * stride < n4 ? __ldg(x4 + i + j * stride) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int j = 0; j < AM_UNROLL; ++j)
        m[SLOTS - 1] = fmaxf(m[SLOTS - 1], fmaxf(fmaxf(fabsf(v[j].x), fabsf(v[j].y)), fmaxf(fabsf(v[j].z), fabsf(v[j].w))));
    }
    if (at < job.n1 - 4 * n4) m[SLOTS - 1] = fmaxf(m[SLOTS - 1], fabsf(__ldg(job.image1 + 4 * n4 + at)));
  }
  if constexpr (MAGNITUDES) {
    __shared__ float red[AM_THREADS / 32][SLOTS];
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m[s] = fmaxf(m[s], __shfl_xor_sync(0xffffffffu, m[s], o));
      if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][s] = m[s];
    }
    __syncthreads();
    if (threadIdx.x < SLOTS) {
      const int s = threadIdx.x;
      float most = red[0][s];
#pragma unroll
      for (int i = 1; i < AM_THREADS / 32; ++i) most = fmaxf(most, red[i][s]);
      if (s == SLOTS - 1) most *= fabsf(job.premul1);
      const int slot = s == SLOTS - 1 ? SCALE_AMAX_F1 : s * SCALE_LEVEL + SCALE_AMAX_F2;
      if (most > 0.f) atomicMax(reinterpret_cast<unsigned*>(scales) + slot, __float_as_uint(most));
      __threadfence();
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    unsigned* ticket = reinterpret_cast<unsigned*>(scales) + SCALE_TICKET;
    if (atomicAdd(ticket, 1u) != gridDim.x - 1) return;
    __threadfence();
    for (int l = 0; l <= job.levels; ++l) feature_scales(scales + l * SCALE_LEVEL, scales + SCALE_AMAX_F1);
    *ticket = 0;
  }
}

static cudaError_t launch_pool(const Dims* d, int levels, const float* fmap1, const float* fmap2, float* const* pooled,
                               float premul1, bool magnitudes, float* scales, cudaStream_t stream) {
  PoolJob job{};
  job.in = fmap2;
  for (int l = 1; l < levels; ++l) job.out[l - 1] = pooled[l];
  job.planes = d[0].B * d[0].C;
  job.H = d[0].H2;
  job.W = d[0].W2;
  job.levels = levels - 1;
  job.image1 = fmap1;
  job.n1 = (size_t)d[0].B * d[0].N1() * d[0].C;
  job.premul1 = premul1;
  const long long regions = (long long)job.planes * ((job.H + 7) / 8) * ((job.W + 7) / 8);
  const long long blocks2 = (regions + AM_THREADS - 1) / AM_THREADS;
  const size_t per_block = (size_t)AM_THREADS * 4 * AM_UNROLL;
  const long long blocks1 = magnitudes ? (long long)std::max<size_t>(1, std::min<size_t>((job.n1 + per_block - 1) / per_block, 148 * 8)) : 0;
  if (blocks1 + blocks2 > INT_MAX) return cudaErrorInvalidConfiguration;
  job.blocks2 = (int)blocks2;
  const bool vec = job.W % 4 == 0 && reinterpret_cast<uintptr_t>(job.in) % 16 == 0;
  auto kern = magnitudes ? (vec ? pool_levels_kernel<true, true> : pool_levels_kernel<false, true>)
                         : (vec ? pool_levels_kernel<true, false> : pool_levels_kernel<false, false>);
  launch_next(kern, (unsigned)(blocks1 + blocks2), AM_THREADS, 0, stream, job, scales);
  return cudaGetLastError();
}

cudaError_t launch_pool_levels(const Dims* d, int levels, const float* fmap2, float* const* pooled, cudaStream_t stream) {
  return launch_pool(d, levels, nullptr, fmap2, pooled, 1.f, false, nullptr, stream);
}

// Gradient of image 2 from those of its pooled levels, in place on level 0's: every level's gradient spreads evenly over the 2 x 2 entries
// it averaged, the coarsest first, as the chain of avg_pool2d's adjoints adds them up.  Four neighbouring columns a thread.
// grid (ceil(ceil(W/4) * H / 256), planes), block 256.
struct UnpoolJob {
  float* g0;
  const float* g[MAX_FUSED_LEVELS - 1];
  int H, W, levels;
};
__global__ void __launch_bounds__(256)
unpool_levels_kernel(const __grid_constant__ UnpoolJob job) {
  follow_previous_kernel();
  const int H = job.H, W = job.W, quads = (W + 3) / 4;
  const int i = blockIdx.x * 256 + threadIdx.x, y = i / quads, x0 = (i - y * quads) * 4;
  if (y >= H) return;
  const size_t plane = blockIdx.y;
  float add[4] = {0.f, 0.f, 0.f, 0.f};
  for (int l = job.levels; l >= 1; --l) {
    const int h = H >> l, w = W >> l;
    const float* g = job.g[l - 1] + (plane * h + (y >> l)) * w;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int x = (x0 + j) >> l;
      // (an entry that the floor of an odd size drops has no parent at this level, and what it would have had of a coarser one
      // does not exist either)
      add[j] = (y >> l) < h && x < w ? (__ldg(g + x) + add[j]) * 0.25f : 0.f;
    }
  }
  float* dst = job.g0 + (plane * H + y) * W + x0;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (x0 + j < W) dst[j] += add[j];
}
cudaError_t launch_unpool_levels(const Dims* d, int levels, float* g0, const float* const* g, cudaStream_t stream) {
  UnpoolJob job{};
  job.g0 = g0;
  for (int l = 1; l < levels; ++l) job.g[l - 1] = g[l];
  job.H = d[0].H2;
  job.W = d[0].W2;
  job.levels = levels - 1;
  const int quads = (job.W + 3) / 4;
  const long long planes = (long long)d[0].B * d[0].C;
  for (long long p0 = 0; p0 < planes; p0 += 65535) {
    const unsigned n = (unsigned)std::min<long long>(planes - p0, 65535);
    launch_next(unpool_levels_kernel, dim3((unsigned)(((long long)quads * job.H + 255) / 256), n), 256, 0, stream, job);
    if (cudaError_t err = cudaGetLastError(); err != cudaSuccess) return err;
    job.g0 += (size_t)n * d[0].N2();
    for (int l = 1; l < levels; ++l) job.g[l - 1] += (size_t)n * d[l].N2();
  }
  return cudaSuccess;
}

cudaError_t launch_absmax(const AbsmaxSource* src, int count, float* scales, int levels, bool gradients, cudaStream_t stream) {
  if (count < 1 || count > ABSMAX_MAX) return cudaErrorInvalidValue;
  AbsmaxJobs jobs;
  const size_t per_block = (size_t)AM_THREADS * 4 * AM_UNROLL;
  long long blocks = 0;
  for (int i = 0; i < ABSMAX_MAX; ++i) {
    jobs.src[i] = src[i < count ? i : 0];
    jobs.first[i] = i < count ? (int)blocks : INT_MAX;
    jobs.blocks[i] = 1;
    if (i >= count) continue;
    if (src[i].sb == (long long)src[i].n) {   // samples that follow one another are one array
      jobs.src[i].n *= src[i].samples;
      jobs.src[i].samples = 1;
    }
    jobs.blocks[i] = (int)std::max<size_t>(1, std::min<size_t>((jobs.src[i].n + per_block - 1) / per_block, 148 * 8));
    blocks += (long long)jobs.blocks[i] * jobs.src[i].samples;
    if (blocks > INT_MAX) return cudaErrorInvalidConfiguration;
  }
  launch_next(absmax_kernel, (unsigned)blocks, AM_THREADS, 0, stream, jobs, scales, levels, gradients ? 1 : 0);
  return cudaGetLastError();
}

// Both images of a call: rounded to TF32 in `out`, or in `outh` as 16-bit operands of kind `op16` (BF16, or FP16 of the value times the
// device scalar *scale16); the one that is not wanted is null.
struct RoundJob {
  const float4* in;
  float4* out;
  uint2* outh;
  const float* scale16;
  size_t n4;
};
__device__ __forceinline__ void round_copy(const RoundJob& j, int op16, int block, int blocks) {
  const size_t stride = (size_t)blocks * blockDim.x;
  const float sc = (j.outh != nullptr && j.scale16 != nullptr) ? __ldg(j.scale16) : 1.f;
  for (size_t i = (size_t)block * blockDim.x + threadIdx.x; i < j.n4; i += stride) {
    float4 v = __ldg(j.in + i);
    if (j.outh != nullptr) {
      if (op16 == OP16_FP16) j.outh[i] = make_uint2(pack_fp16x2(v.x * sc, v.y * sc), pack_fp16x2(v.z * sc, v.w * sc));
      else j.outh[i] = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
    }
    if (j.out != nullptr) {
      v.x = round_tf32(v.x); v.y = round_tf32(v.y); v.z = round_tf32(v.z); v.w = round_tf32(v.w);
      j.out[i] = v;
    }
  }
}

// One mean row, in the two forms the sweeps may read it: TF32 in `aux` or 16-bit in `auxh` (each may be null).
__device__ __forceinline__ void store_mean(float mean, size_t at, float* aux, uint16_t* auxh, int op16, float sc16) {
  if (aux != nullptr) aux[at] = round_tf32(mean);
  if (auxh != nullptr) auxh[at] = to_op16(mean * sc16, op16);
}

// From pixel-major features, in one launch with the copies (1 x 48 x 64, C = 256: 4 + 4.5 us apart, 3.6 together).  A block owns one mean
// row; four groups of 64 threads take every fourth pixel of it, a
// thread four channels at a time, so that the pixels' loads are in flight side by side.  The blocks of the mean rows come first.
// grid (mean_rows * B + copies1 + copies2), block 256.
constexpr int FM_GROUPS = 4, FM_QUADS = 64;
__global__ void __launch_bounds__(FM_GROUPS * FM_QUADS)
round_means_kernel(const RoundJob j1, const RoundJob j2, int copies1, int copies2, const float* __restrict__ F2, float* __restrict__ aux, int mean_rows,
                   int B, int H2, int W2, int C, uint16_t* __restrict__ auxh, int op16, const float* __restrict__ scale16) {
  follow_previous_kernel();
  __shared__ float4 red[FM_GROUPS][FM_QUADS];
  const int block = (int)blockIdx.x - mean_rows * B;
  if (block >= 0) {
    if (block < copies1) round_copy(j1, op16, block, copies1);
    else round_copy(j2, op16, block - copies1, copies2);
    return;
  }
  const int b = blockIdx.x / mean_rows, r = blockIdx.x - b * mean_rows, g = threadIdx.x / FM_QUADS, q = threadIdx.x % FM_QUADS;
  const float sc16 = (op16 == OP16_FP16 && scale16 != nullptr) ? __ldg(scale16) : 1.f;
  const int count = r < H2 ? W2 : H2;
  const size_t step = r < H2 ? (size_t)C : (size_t)W2 * C;   // between the pixels of the row / column
  const float* base = F2 + (size_t)b * H2 * W2 * C + (r < H2 ? (size_t)r * W2 * C : (size_t)(r - H2) * C);
  for (int c0 = 0; c0 < C; c0 += 4 * FM_QUADS) {   // C is a multiple of 4
    const int c = c0 + 4 * q;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < C) {
#pragma unroll 4
      for (int i = g; i < count; i += FM_GROUPS) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(base + i * step + c));
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
      }
    }
    red[g][q] = acc;
    __syncthreads();
    if (g == 0 && c < C) {
#pragma unroll
      for (int i = 1; i < FM_GROUPS; ++i) {
        const float4 v = red[i][q];
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
      }
      const float n = (float)count;
      const size_t at = ((size_t)b * (H2 + W2) + r) * C + c;
      store_mean(acc.x / n, at, aux, auxh, op16, sc16);
      store_mean(acc.y / n, at + 1, aux, auxh, op16, sc16);
      store_mean(acc.z / n, at + 2, aux, auxh, op16, sc16);
      store_mean(acc.w / n, at + 3, aux, auxh, op16, sc16);
    }
    __syncthreads();
  }
}

// From channel-major feature maps: a block owns one channel plane; its warps take every eighth row, ROWS rows at a time, a
// lane every 32nd column.  NV = ceil(W2 / 32) rounded up to a power of two: the column sums of a lane stay in registers, so
// that the plane is read once, with ROWS * NV loads of a lane in flight (one walk for the rows and one for the
// columns took 162 us at 8 x 135 x 240, C = 256; 62 now).  Bound by the latency of a block's few steps: at four columns a lane four rows a step
// take 6.6 us for the levels of 1 x 55 x 128 where two take 9.8; at two columns (2 x 48 x 64) four take 10.7 and two 8.3, the coarse
// levels having few rows; at eight (8 x 135 x 240) one takes 66 and four 73.  NV = 0: any width, in the two walks.  Both add in the same order.
// grid (C, B, levels), block 256.
struct MeansJobs {
  struct Job {
    const float* fmap2;
    float* aux;
    uint16_t* auxh;
    const float* scale16;
    int H2, W2;
  } j[MAX_FUSED_LEVELS];
};
template <int NV>
__global__ void __launch_bounds__(256)
f2_means_cf_kernel(const __grid_constant__ MeansJobs jobs, int C, int op16) {
  follow_previous_kernel();
  const MeansJobs::Job& job = jobs.j[blockIdx.z];
  const float* const fmap2 = job.fmap2;
  float* const aux = job.aux;
  uint16_t* const auxh = job.auxh;
  const float* const scale16 = job.scale16;
  const int H2 = job.H2, W2 = job.W2;
  __shared__ float red[8][NV > 0 ? NV : 1][33];
  const int c = blockIdx.x, b = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float sc16 = (op16 == OP16_FP16 && scale16 != nullptr) ? __ldg(scale16) : 1.f;
  const float* plane = fmap2 + ((size_t)b * C + c) * H2 * W2;
  const size_t out0 = (size_t)b * (H2 + W2) * C + c;
  if constexpr (NV > 0) {
    float col[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) col[i] = 0.f;
    constexpr int ROWS = NV == 4 ? 4 : 2;
    for (int u0 = warp; u0 < H2; u0 += 8 * ROWS) {
      float v[ROWS][NV], acc[ROWS];
#pragma unroll
      for (int r = 0; r < ROWS; ++r)
#pragma unroll
        for (int i = 0; i < NV; ++i)
          v[r][i] = u0 + 8 * r < H2 && lane + 32 * i < W2 ? __ldg(plane + (size_t)(u0 + 8 * r) * W2 + lane + 32 * i) : 0.f;
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        acc[r] = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          acc[r] += v[r][i];
          if (u0 + 8 * r < H2) col[i] += v[r][i];
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < ROWS; ++r) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
#pragma unroll
      for (int r = 0; r < ROWS; ++r)
        if (lane == 0 && u0 + 8 * r < H2) store_mean(acc[r] / (float)W2, out0 + (size_t)(u0 + 8 * r) * C, aux, auxh, op16, sc16);
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) red[warp][i][lane] = col[i];
    __syncthreads();
    for (int v = threadIdx.x; v < W2; v += 256) {
      float acc = red[0][v >> 5][v & 31];
#pragma unroll
      for (int i = 1; i < 8; ++i) acc += red[i][v >> 5][v & 31];
      store_mean(acc / (float)H2, out0 + (size_t)(H2 + v) * C, aux, auxh, op16, sc16);
    }
  } else {
    auto store_row = [&](int u, float acc) {   // acc: this lane's share of row u
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) store_mean(acc / (float)W2, out0 + (size_t)u * C, aux, auxh, op16, sc16);
    };
    for (int u = warp; u < H2; u += 8) {
      float acc = 0.f;
#pragma unroll 4
      for (int v = lane; v < W2; v += 32) acc += __ldg(plane + (size_t)u * W2 + v);
      store_row(u, acc);
    }
    for (int v0 = 0; v0 < W2; v0 += 32) {
      const int v = v0 + lane;
      float acc = 0.f;
      if (v < W2) {
#pragma unroll 4
        for (int u = warp; u < H2; u += 8) acc += __ldg(plane + (size_t)u * W2 + v);
      }
      red[warp][0][lane] = acc;
      __syncthreads();
      if (warp == 0 && v < W2) {
#pragma unroll
        for (int i = 1; i < 8; ++i) acc += red[i][0][lane];
        store_mean(acc / (float)H2, out0 + (size_t)(H2 + v) * C, aux, auxh, op16, sc16);
      }
      __syncthreads();
    }
  }
}

// Tiled transposes between the reference's per-pixel layout (B, N1, K, D) (displacement d fastest) and the
// packed layout (B, D, R, n1p) (pixel fastest) the kernels use.  A block moves a patch of 128 pixels (PX) x 32
// displacements through shared memory so that both sides are coalesced; every thread keeps 16 loads in flight,
// and the displacement tiles are the fastest so that blocks running together read neighbouring
// 128-byte pieces of the same rows.  One launch for all tensors of a call (a launch of a small one is mostly latency: the four outputs of
// 2 x 48 x 64 took 31 us in four launches, 10 in one).
// Launches of less than four such blocks per SM move 32 pixels a block: they are over sooner than a block's instructions for sixteen loads and stores
// have been fetched (drop-in operators 2 x 48 x 64, three conversions and two packs, 365 -> 349 us; up to 16 blocks per SM
// 4 x 48 x 64 with three channels takes 577 instead of 562).
// grid: ceil(D/32) * n1p/PX * B*K blocks per tensor, block (32, 8).
struct PatchJobs {
  PatchJob j[MAX_PATCH_JOBS];
  int first[MAX_PATCH_JOBS];   // blocks; tensors that do not exist start past the end of the grid
};
struct Patch {
  int b, k, d0, p0;
};
template <int PX>
__device__ __forceinline__ Patch patch_of(const PatchJobs& jobs, int n1p, int& job) {
  job = 0;
#pragma unroll
  for (int i = 1; i < MAX_PATCH_JOBS; ++i) job = (int)blockIdx.x >= jobs.first[i] ? i : job;
  const PatchJob& j = jobs.j[job];
  const int r = blockIdx.x - jobs.first[job], nd = (j.D + 31) / 32, np = n1p / PX;
  const int q = r / nd, z = q / np, b = z / j.K;
  return Patch{b, z - b * j.K, (r - q * nd) * 32, (q - z * np) * PX};
}

template <int PX>
__global__ void __launch_bounds__(256) pack_kernel(const __grid_constant__ PatchJobs jobs, int N1, int n1p) {
  follow_previous_kernel();
  __shared__ uint32_t tile[PX][33];
  int ji;
  const Patch t = patch_of<PX>(jobs, n1p, ji);
  const PatchJob& j = jobs.j[ji];
  const int tx = threadIdx.x, ty = threadIdx.y, D = j.D;
  const uint32_t* src = static_cast<const uint32_t*>(j.pixels) + (((size_t)t.b * N1 + t.p0) * j.Kpix + j.k0 + t.k) * D + t.d0 + tx;
#pragma unroll
  for (int i = ty; i < PX; i += 8) {
    uint32_t v = 0;
    if (t.p0 + i < N1 && t.d0 + tx < D) v = __ldg(src + (size_t)i * j.Kpix * D);
    tile[i][tx] = v;
  }
  __syncthreads();
  uint32_t* dst = reinterpret_cast<uint32_t*>(j.packed) + (((size_t)t.b * D + t.d0) * j.R + j.r0 + t.k) * n1p + t.p0;
#pragma unroll
  for (int i = ty; i < 32 * (PX / 32); i += 8) {
    const int d = i / (PX / 32), p = (i % (PX / 32)) * 32 + tx;
    if (t.d0 + d < D) dst[(size_t)d * j.R * n1p + p] = tile[p][d];
  }
}

template <int PX>
__global__ void __launch_bounds__(256) unpack_kernel(const __grid_constant__ PatchJobs jobs, int N1, int n1p) {
  follow_previous_kernel();
  __shared__ uint32_t tile[PX][33];
  int ji;
  const Patch t = patch_of<PX>(jobs, n1p, ji);
  const PatchJob& j = jobs.j[ji];
  const int tx = threadIdx.x, ty = threadIdx.y, D = j.D;
  const uint32_t* src = reinterpret_cast<const uint32_t*>(j.packed) + (((size_t)t.b * D + t.d0) * j.R + j.r0 + t.k) * n1p + t.p0;
#pragma unroll
  for (int i = ty; i < 32 * (PX / 32); i += 8) {
    const int d = i / (PX / 32), p = (i % (PX / 32)) * 32 + tx;
    tile[p][d] = t.d0 + d < D ? __ldg(src + (size_t)d * j.R * n1p + p) : 0u;
  }
  __syncthreads();
  uint32_t* dst = static_cast<uint32_t*>(const_cast<void*>(j.pixels)) + (((size_t)t.b * N1 + t.p0) * j.Kpix + j.k0 + t.k) * D + t.d0 + tx;
#pragma unroll
  for (int i = ty; i < PX; i += 8)
    if (t.p0 + i < N1 && t.d0 + tx < D) dst[(size_t)i * j.Kpix * D] = tile[i][tx];
}

template <class Kernel>
static cudaError_t launch_patches(Kernel kern, int px, const PatchJob* job, int count, int B, int N1, int n1p, cudaStream_t stream) {
  PatchJobs jobs;
  long long blocks = 0;
  for (int i = 0; i < MAX_PATCH_JOBS; ++i) {
    jobs.j[i] = job[i < count ? i : 0];
    jobs.first[i] = i < count ? (int)blocks : INT_MAX;
    if (i < count) blocks += (long long)((job[i].D + 31) / 32) * (n1p / px) * B * job[i].K;
    if (blocks > INT_MAX) return cudaErrorInvalidConfiguration;
  }
  launch_next(kern, (unsigned)blocks, dim3(32, 8), 0, stream, jobs, N1, n1p);
  return cudaGetLastError();
}
static bool short_patches(const PatchJob* job, int count, int B, int n1p) {
  long long blocks = 0;   // of 128 pixels
  for (int i = 0; i < count; ++i) blocks += (long long)((job[i].D + 31) / 32) * (n1p / 128) * B * job[i].K;
  return blocks < 4 * SM_COUNT;
}
cudaError_t launch_pack(const PatchJob* jobs, int count, int B, int N1, int n1p, cudaStream_t stream) {
  if (count < 1 || count > MAX_PATCH_JOBS) return cudaErrorInvalidValue;
  if (short_patches(jobs, count, B, n1p)) return launch_patches(pack_kernel<32>, 32, jobs, count, B, N1, n1p, stream);
  return launch_patches(pack_kernel<128>, 128, jobs, count, B, N1, n1p, stream);
}
cudaError_t launch_unpack(const PatchJob* jobs, int count, int B, int N1, int n1p, cudaStream_t stream) {
  if (count < 1 || count > MAX_PATCH_JOBS) return cudaErrorInvalidValue;
  if (short_patches(jobs, count, B, n1p)) return launch_patches(unpack_kernel<32>, 32, jobs, count, B, N1, n1p, stream);
  return launch_patches(unpack_kernel<128>, 128, jobs, count, B, N1, n1p, stream);
}

// Interleaved pack of groups of four slots: every block transposes a 32-pixel x 32-displacement patch of each of a group's sources through
// shared memory, then writes, per displacement, the four slots of its 32 pixels as one contiguous run.  All groups of a call in one
// launch.  grid (ceil(largest D/32), n1p/32, groups * B), block (32, 8).
__global__ void __launch_bounds__(256)
pack_interleaved_kernel(const __grid_constant__ PackGroups groups, int B, int N1, int n1p) {
  follow_previous_kernel();
  constexpr int RS = 32 * 33 + 32 / 4;  // slot stride chosen so that the interleaved read below is conflict-free
  __shared__ uint32_t tile[4 * RS];
  const int gi = blockIdx.z / B, b = blockIdx.z - gi * B;
  const PackGroup& g = groups.g[gi];
  const int D = g.D, d0 = blockIdx.x * 32, p0 = blockIdx.y * 32;  // displacement tiles fastest
  if (d0 >= D) return;
  const int tx = threadIdx.x, ty = threadIdx.y;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const SlotSource& ss = g.s[r];
    const uint32_t* s = ss.src == nullptr ? nullptr : static_cast<const uint32_t*>(ss.src) + (((size_t)b * N1 + p0) * ss.Ksrc + ss.k) * D + d0 + tx;
    const float dev = ss.dev != 0 ? __ldg(g.dev_scales + ss.dev - 1) : 1.f;
#pragma unroll
    for (int j = ty; j < 32; j += 8) {
      uint32_t v = 0;
      if (p0 + j < N1 && d0 + tx < D) {
        if (s == nullptr) {
          v = __float_as_uint(ss.scale);  // constant slot
        } else {
          v = __ldg(s + (size_t)j * ss.Ksrc * D);
          if (ss.scale != 0.f) v = __float_as_uint(__uint_as_float(v) * ss.scale);
          if (ss.dev != 0) v = __float_as_uint(__uint_as_float(v) * dev);
        }
      }
      tile[r * RS + j * 33 + tx] = v;
    }
  }
  __syncthreads();
  // per displacement: 32 pixels x 4 slots = 128 consecutive words, half a block each
  const int t = ty * 32 + tx, w = t % 128;
  uint32_t* dst = reinterpret_cast<uint32_t*>(g.dst) + ((((size_t)b * D + d0) * g.Qtot + g.q) * n1p + p0) * 4 + w;
#pragma unroll 4
  for (int j = t / 128; j < 32; j += 2) {
    if (d0 + j >= D) break;
    dst[(size_t)j * g.Qtot * n1p * 4] = tile[(w & 3) * RS + (w >> 2) * 33 + j];
  }
}

// Launches of at most as many groups as grid.z takes.
template <class Launch>
static cudaError_t launch_groups(const PackGroups& groups, int B, Launch&& launch) {
  const int per_launch = pack_groups_per_launch(B);
  for (int first = 0; first < groups.count; first += per_launch) {
    PackGroups some = groups;
    some.count = std::min(per_launch, groups.count - first);
    int D = 1;
    for (int i = 0; i < some.count; ++i) {
      some.g[i] = groups.g[first + i];
      D = std::max(D, some.g[i].D);
    }
    launch(some, D);
    if (cudaError_t err = cudaGetLastError(); err != cudaSuccess) return err;
  }
  return cudaSuccess;
}

cudaError_t launch_pack_interleaved(const PackGroups& groups, int B, int N1, int n1p, cudaStream_t stream) {
  return launch_groups(groups, B, [&](const PackGroups& some, int D) {
    launch_next(pack_interleaved_kernel, dim3((D + 31) / 32, n1p / 32, some.count * B), dim3(32, 8), 0, stream, some, B, N1, n1p);
  });
}

// Channels-first sources are already pixel-fastest: one thread per pixel gathers the four slots of a group
// and stores them as one 16-byte word, for PI_DB displacements at a time (all loads issued before the stores,
// so that a thread keeps 4*PI_DB loads in flight).  One launch for all groups of a call's operands (a training step on small
// crops is bound by the number of launches): in place of four, 1720 -> 1400 us at 8 x 135 x 240 with four channels, 142 -> 111 at
// 8 x 47 x 156 with two, 60 -> 21 for the four levels of 2 x 48 x 64.
// grid (ceil(n1p/256), ceil(largest D/PI_DB), groups * B), block 256.  grid.z takes 65535 blocks: larger batches are packed by
// several launches of fewer groups.  (The groups on grid.x, next to one another: 1500 us at 8 x 135 x 240; a loop over
// (group, sample) pairs in the kernel: 1750.)
constexpr int PI_DB = 4;

__global__ void __launch_bounds__(256)
pack_interleaved_cf_kernel(const __grid_constant__ PackGroups groups, int B, int N1, int n1p) {
  follow_previous_kernel();
  const int gi = blockIdx.z / B, b = blockIdx.z - gi * B;
  const PackGroup& g = groups.g[gi];
  const int p = blockIdx.x * 256 + threadIdx.x, d0 = blockIdx.y * PI_DB, D = g.D;
  if (p >= n1p || d0 >= D) return;
  const bool in = p < N1;
  // per slot: where its values are (null: a constant), and the factor they are multiplied by (0 = raw 32-bit copy): host
  // scale times device scale
  const uint32_t* src[4];
  float fac[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const SlotSource& ss = g.s[j];
    src[j] = ss.src == nullptr ? nullptr : static_cast<const uint32_t*>(ss.src) + (((size_t)b * ss.Ksrc + ss.k) * D + d0) * N1 + p;
    fac[j] = ss.scale;
    if (ss.dev != 0 && ss.src != nullptr) fac[j] = (ss.scale != 0.f ? ss.scale : 1.f) * __ldg(g.dev_scales + ss.dev - 1);
  }
  uint32_t w[PI_DB][4];
#pragma unroll
  for (int i = 0; i < PI_DB; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      w[i][j] = 0;
      if (src[j] != nullptr && in && d0 + i < D) w[i][j] = __ldg(src[j] + (size_t)i * N1);
      else if (src[j] == nullptr && in) w[i][j] = __float_as_uint(fac[j]);
    }
  float4* dst = g.dst + (((size_t)b * D + d0) * g.Qtot + g.q) * n1p + p;
#pragma unroll
  for (int i = 0; i < PI_DB; ++i) {
    if (d0 + i >= D) break;
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      v[j] = (fac[j] != 0.f && src[j] != nullptr) ? __uint_as_float(w[i][j]) * fac[j] : __uint_as_float(w[i][j]);
    dst[(size_t)i * g.Qtot * n1p] = make_float4(v[0], v[1], v[2], v[3]);
  }
}

cudaError_t launch_pack_interleaved_cf(const PackGroups& groups, int B, int N1, int n1p, cudaStream_t stream) {
  return launch_groups(groups, B, [&](const PackGroups& some, int D) {
    launch_next(pack_interleaved_cf_kernel, dim3((n1p + 255) / 256, (D + PI_DB - 1) / PI_DB, some.count * B), 256, 0, stream, some, B, N1, n1p);
  });
}

// (B, C, N) -> (B, N, C) for all images of a call in one launch, scaled: as TF32 in `out` or as 16-bit operands in `outh` (the one
// that is not wanted is null).  Tiles of 64 channels x 32 pixels through shared memory, so that a warp writes 64 channels
// of a pixel, two per lane; image j has the blocks first[j] .. of a row.  grid (sum of the images' ceil(N/32), ceil(C/64), B), block
// (32, 8).
struct TransposeJob { const float* in; float* out; uint16_t* outh; const float* scale16; float scale; int N; };
struct TransposeJobs {
  TransposeJob j[1 + MAX_FUSED_LEVELS];
  int first[1 + MAX_FUSED_LEVELS];   // images that do not exist start past the end of the grid
};
__global__ void __launch_bounds__(256)
transpose_round_kernel(const __grid_constant__ TransposeJobs jobs, int C, int op16) {
  follow_previous_kernel();
  __shared__ float tile[64][33];
  int image = 0;
#pragma unroll
  for (int i = 1; i <= MAX_FUSED_LEVELS; ++i) image = (int)blockIdx.x >= jobs.first[i] ? i : image;
  const TransposeJob& j = jobs.j[image];
  const int N = j.N;
  const float sc16 = (j.outh != nullptr && op16 == OP16_FP16 && j.scale16 != nullptr) ? __ldg(j.scale16) : 1.f;
  const int b = blockIdx.z, p0 = ((int)blockIdx.x - jobs.first[image]) * 32, c0 = blockIdx.y * 64;
  const int tx = threadIdx.x, ty = threadIdx.y;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int c = c0 + ty + 8 * i, p = p0 + tx;
    tile[ty + 8 * i][tx] = (c < C && p < N) ? __ldg(j.in + ((size_t)b * C + c) * N + p) * j.scale : 0.f;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int p = p0 + ty + 8 * i, c = c0 + 2 * tx;   // C is even
    if (p < N && c < C) {
      const float lo = tile[2 * tx][ty + 8 * i], hi = tile[2 * tx + 1][ty + 8 * i];
      const size_t at = ((size_t)b * N + p) * C + c;
      if (j.out != nullptr) *reinterpret_cast<float2*>(j.out + at) = make_float2(round_tf32(lo), round_tf32(hi));
      if (j.outh != nullptr)
        *reinterpret_cast<uint32_t*>(j.outh + at) = op16 == OP16_FP16 ? pack_fp16x2(lo * sc16, hi * sc16) : pack_bf16x2(lo, hi);
    }
  }
}

// Channel-major copies straight from the model's feature maps (B, C, rows*width), times `scale`: as 16-bit operands (FP16: times the device
// scalar as well) or TF32.  The layouts of channel_major_kernel, padding included (zeros), two values per store.  A thread makes CM_PAIRS
// pairs, 512 values apart, with all loads first: with one pair a thread HBM waited for them (8 x 47 x 156, C = 256: 81 us, 39 now; with eight
// pairs 33, but 10.6 instead of 9.4 for the levels of 2 x 48 x 64).  The two values of a pair are one load where every pair of a copy lies on
// 8 bytes.  One grid row per channel of a sample: grid (sum over the copies of ceil(pairs per channel / (256 * CM_PAIRS)), C, B).
constexpr int CM_PAIRS = 4;
struct MapCopies {
  MapCopy c[MAX_MAP_COPIES];
  int first[MAX_MAP_COPIES];   // of grid.x; copies that do not exist start past its end
  bool vec[MAX_MAP_COPIES];
};
__host__ __device__ inline int map_copy_channel(const MapCopy& c) { return c.blocked ? (c.width + 15) / 16 * c.pitch * 16 : c.pitch; }
__global__ void __launch_bounds__(256)
channel_major_cf_kernel(const __grid_constant__ MapCopies copies, int C, int op16) {
  follow_previous_kernel();
  int ci = 0;
#pragma unroll
  for (int i = 1; i < MAX_MAP_COPIES; ++i) ci = (int)blockIdx.x >= copies.first[i] ? i : ci;
  const MapCopy& copy = copies.c[ci];
  const bool vec = copies.vec[ci];
  const int per_channel = map_copy_channel(copy), width = copy.width;
  const int i0 = (blockIdx.x - copies.first[ci]) * (256 * 2 * CM_PAIRS) + threadIdx.x * 2;
  if (i0 >= per_channel) return;
  const float sc16 = (op16 == OP16_FP16 && copy.scale16 != nullptr) ? __ldg(copy.scale16) : 1.f;
  const size_t chan = (size_t)blockIdx.z * C + blockIdx.y;
  const float* const src = copy.src + chan * copy.rows * width;
  float2 v[CM_PAIRS];
#pragma unroll
  for (int k = 0; k < CM_PAIRS; ++k) {
    const int i = i0 + k * 512;
    int row = 0, x = i;
    if (copy.blocked) {
      const int xb = (unsigned)i / ((unsigned)copy.pitch * 16u), r = i - xb * copy.pitch * 16;
      row = r / 16;
      x = xb * 16 + (r & 15);
    }
    const bool ok = i < per_channel && row < copy.rows && x < width;
    const float* const p = src + (size_t)row * width + x;
    if (vec) v[k] = ok ? __ldg(reinterpret_cast<const float2*>(p)) : make_float2(0.f, 0.f);   // (width is even)
    else v[k] = make_float2(ok ? __ldg(p) : 0.f, ok && x + 1 < width ? __ldg(p + 1) : 0.f);
  }
#pragma unroll
  for (int k = 0; k < CM_PAIRS; ++k) {
    const int i = i0 + k * 512;
    if (i >= per_channel) return;
    const float lo = v[k].x * copy.scale, hi = v[k].y * copy.scale;
    const size_t at = (chan * per_channel + i) / 2;
    if (op16 == 0) static_cast<float2*>(copy.dst)[at] = make_float2(round_tf32(lo), round_tf32(hi));
    else static_cast<uint32_t*>(copy.dst)[at] = op16 == OP16_FP16 ? pack_fp16x2(lo * sc16, hi * sc16) : pack_bf16x2(lo, hi);
  }
}

cudaError_t launch_channel_major_cf(const MapCopy* copy, int count, int B, int C, int op16, cudaStream_t stream) {
  if (count < 1 || count > MAX_MAP_COPIES) return cudaErrorInvalidValue;
  MapCopies copies;
  int blocks = 0;
  for (int i = 0; i < MAX_MAP_COPIES; ++i) {
    copies.c[i] = copy[i < count ? i : 0];
    copies.vec[i] = copies.c[i].width % 2 == 0 && reinterpret_cast<uintptr_t>(copies.c[i].src) % 8 == 0;
    copies.first[i] = i < count ? blocks : INT_MAX;
    if (i < count) blocks += (map_copy_channel(copy[i]) / 2 + 256 * CM_PAIRS - 1) / (256 * CM_PAIRS);
  }
  launch_next(channel_major_cf_kernel, dim3(blocks, C, B), 256, 0, stream, copies, C, op16);
  return cudaGetLastError();
}

// Channel-major copies of pixel-major feature arrays (B, rows*width, C), the K-major B operands of the gradient GEMMs.
//   blocked = 0: dst (B, C, pitch), pixel index = row*width + x (image 1: rows = 1, width = N1, pitch = n1p)
//   blocked = 1: dst (B, C, ceil(width/16), pitch, 16): columns in blocks of 16, so that the 4 rows x 16 columns of one
//                K block of the image-1-major GEMM are 64 consecutive values (image 2: pitch = H2 rounded up to 4)
// Padding is zero.  Tiles of CMK_PX pixels x 32 channels through shared memory, both images in one launch; grid (sum over the images of tiles of
// their padded rows, ceil(C/32), B), block (32, 8).  A thread has eight
// loads under way and stores two pixels at once; with tiles of 32 pixels, one to a store, the drop-in operators took 348 us instead of 346 at
// 2 x 48 x 64, 3024 instead of 2978 at 8 x 47 x 156 (BF16) and 5767 instead of 5692 at 1 x 135 x 240.
__host__ __device__ inline int map_copy_columns(const MapCopy& c) { return c.blocked ? (c.width + 15) / 16 * 16 : c.pitch; }   // of a padded row
__host__ __device__ inline int map_copy_rows(const MapCopy& c) { return c.blocked ? c.pitch : 1; }
constexpr int CMK_PX = 64;
template <typename T>
__global__ void __launch_bounds__(256) channel_major_kernel(const MapCopy c1, const MapCopy c2, int blocks1, int C, int op16) {
  follow_previous_kernel();
  __shared__ float tile[CMK_PX][33];
  const bool first = (int)blockIdx.x < blocks1;
  const MapCopy& c = first ? c1 : c2;
  const float sc16 = (op16 == OP16_FP16 && c.scale16 != nullptr) ? __ldg(c.scale16) : 1.f;
  const int columns = map_copy_columns(c), per_row = (columns + CMK_PX - 1) / CMK_PX, r = blockIdx.x - (first ? 0 : blocks1);
  const int row = r / per_row, x0 = (r - row * per_row) * CMK_PX, c0 = blockIdx.y * 32, b = blockIdx.z;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const float* src = c.src + (((size_t)b * c.rows + row) * c.width + x0) * C + c0 + tx;
#pragma unroll
  for (int j = ty; j < CMK_PX; j += 8) tile[j][tx] = (row < c.rows && x0 + j < c.width && c0 + tx < C) ? __ldg(src + (size_t)j * C) : 0.f;
  __syncthreads();
  const size_t per_channel = (size_t)map_copy_rows(c) * columns;
  const int x = x0 + 2 * tx;   // and x + 1, next to it: columns and blocks of them are even
  if (x >= columns) return;
  const size_t off = c.blocked ? ((size_t)(x >> 4) * c.pitch + row) * 16 + (x & 15) : (size_t)x;
  T* dst = static_cast<T*>(c.dst) + ((size_t)b * C + c0) * per_channel + off;
#pragma unroll
  for (int j = ty; j < 32; j += 8) {
    if (c0 + j >= C) return;
    const float lo = tile[2 * tx][j], hi = tile[2 * tx + 1][j];
    T* const at = dst + (size_t)j * per_channel;
    if constexpr (sizeof(T) == 2) {
      *reinterpret_cast<uint32_t*>(at) = op16 == OP16_FP16 ? pack_fp16x2(lo * sc16, hi * sc16) : pack_bf16x2(lo * sc16, hi * sc16);
    } else {
      *reinterpret_cast<float2*>(at) = make_float2(lo, hi);
    }
  }
}

cudaError_t launch_channel_major(const MapCopy& c1, const MapCopy& c2, int B, int C, int op16, cudaStream_t stream) {
  auto blocks = [](const MapCopy& c) { return (map_copy_columns(c) + CMK_PX - 1) / CMK_PX * map_copy_rows(c); };
  const dim3 grid(blocks(c1) + blocks(c2), (C + 31) / 32, B), block(32, 8);
  if (op16) launch_next(channel_major_kernel<uint16_t>, grid, block, 0, stream, c1, c2, blocks(c1), C, op16);
  else launch_next(channel_major_kernel<float>, grid, block, 0, stream, c1, c2, blocks(c1), C, 0);
  return cudaGetLastError();
}

// Zeros for the workspace header.  A kernel: launches wait for a memory operation as a whole, with the device idle on either side of it (drop-in
// operators 2 x 48 x 64, four calls, 357 -> 348 us, max/mean channels 1 x 48 x 64 50 -> 37, infer 1 x 55 x 128 238 -> 235).  grid 1, block 32.
__global__ void __launch_bounds__(32) clear_header_kernel(int* words, int n) {
  follow_previous_kernel();
  for (int i = threadIdx.x; i < n; i += 32) words[i] = 0;
}
static cudaError_t clear_header(int levels, int* status, cudaStream_t stream) {
  launch_next(clear_header_kernel, 1, 32, 0, stream, status, (int)(WS_SCALES_OFFSET / sizeof(int)) + levels * SCALE_LEVEL);
  return cudaGetLastError();
}
// Clears the workspace header (status word, scale slots) and, for FP16 operands, finds the feature scales.
static cudaError_t begin_prepare(const Dims* d, int levels, const float* F1, const float* const* F2, float premul1, int* status, int op16,
                                 float* scales, cudaStream_t stream) {
  cudaError_t err = clear_header(levels, status, stream);
  if (err != cudaSuccess || op16 != OP16_FP16 || scales == nullptr) return err;
  AbsmaxSource src[1 + MAX_FUSED_LEVELS];
  src[0] = absmax_array(F1, (size_t)d[0].B * d[0].N1() * d[0].C, premul1, SCALE_AMAX_F1);
  for (int l = 0; l < levels; ++l)
    src[1 + l] = absmax_array(F2[l], (size_t)d[l].B * d[l].N2() * d[l].C, 1.f, l * SCALE_LEVEL + SCALE_AMAX_F2);
  return launch_absmax(src, 1 + levels, scales, levels, false, stream);
}

cudaError_t launch_prepare_cf(const Dims* d, int levels, const float* fmap1, const float* const* fmap2, float scale1,
                              const LevelOperands* out, float* F1r, uint16_t* F1h, int* status, cudaStream_t stream, int op16, float* scales,
                              float* const* pooled) {
  if (levels < 1 || levels > MAX_FUSED_LEVELS) return cudaErrorInvalidValue;
  cudaError_t err;
  if (pooled != nullptr) {
    err = clear_header(levels, status, stream);
    if (err == cudaSuccess) err = launch_pool(d, levels, fmap1, fmap2[0], pooled, scale1, op16 == OP16_FP16 && scales != nullptr, scales, stream);
  } else {
    err = begin_prepare(d, levels, fmap1, fmap2, scale1, status, op16, scales, stream);
  }
  if (err != cudaSuccess) return err;
  const bool scaled = op16 == OP16_FP16 && scales != nullptr;
  const int B = d[0].B, C = d[0].C;
  if (F1r != nullptr || F1h != nullptr) {
    TransposeJobs jobs;
    int blocks = (d[0].N1() + 31) / 32;
    jobs.j[0] = TransposeJob{fmap1, F1r, F1h, scaled ? scales + SCALE_F1 : nullptr, scale1, d[0].N1()};
    jobs.first[0] = 0;
    for (int l = 0; l < MAX_FUSED_LEVELS; ++l) {
      jobs.first[1 + l] = l < levels ? blocks : INT_MAX;
      jobs.j[1 + l] = jobs.j[0];
      if (l >= levels) continue;
      jobs.j[1 + l] = TransposeJob{fmap2[l], out[l].F2r, out[l].F2h, scaled ? scales + l * SCALE_LEVEL + SCALE_F2 : nullptr, 1.f, d[l].N2()};
      blocks += (d[l].N2() + 31) / 32;
    }
    launch_next(transpose_round_kernel, dim3(blocks, (C + 63) / 64, B), dim3(32, 8), 0, stream, jobs, C, op16);
  }
  if (out[0].aux != nullptr || out[0].auxh != nullptr) {
    MeansJobs jobs;
    int W2 = 0;
    for (int l = 0; l < MAX_FUSED_LEVELS; ++l) {
      jobs.j[l] = jobs.j[0];
      if (l >= levels) continue;
      jobs.j[l] = MeansJobs::Job{fmap2[l], out[l].aux, out[l].auxh, scaled ? scales + l * SCALE_LEVEL + SCALE_F2 : nullptr, d[l].H2, d[l].W2};
      W2 = std::max(W2, d[l].W2);
    }
    auto kern = W2 <= 32    ? f2_means_cf_kernel<1>
                : W2 <= 64  ? f2_means_cf_kernel<2>
                : W2 <= 128 ? f2_means_cf_kernel<4>
                : W2 <= 256 ? f2_means_cf_kernel<8>
                            : f2_means_cf_kernel<0>;
    launch_next(kern, dim3(C, B, levels), 256, 0, stream, jobs, C, op16);
  }
  return cudaGetLastError();
}

cudaError_t launch_prepare(const Dims& d, const float* F1, const float* F2, float* F1r, float* F2r, float* aux,
                           int* status, cudaStream_t stream, uint16_t* F1h, uint16_t* F2h, uint16_t* auxh, int op16,
                           float* scales) {
  cudaError_t err = begin_prepare(&d, 1, F1, &F2, 1.f, status, op16, scales, stream);
  if (err != cudaSuccess) return err;
  const float* s1 = (op16 == OP16_FP16 && scales != nullptr) ? scales + SCALE_F1 : nullptr;
  const float* s2 = (op16 == OP16_FP16 && scales != nullptr) ? scales + SCALE_F2 : nullptr;
  const size_t n1 = (size_t)d.B * d.N1() * d.C / 4, n2 = (size_t)d.B * d.N2() * d.C / 4;  // C % 4 == 0
  const int threads = 256;
  auto blocks = [&](size_t n) { return (unsigned)std::min<size_t>((n + threads - 1) / threads, 148 * 16); };
  const bool copies = F1r != nullptr || F1h != nullptr, means = aux != nullptr || auxh != nullptr;
  if (!copies && !means) return cudaSuccess;
  const RoundJob j1{reinterpret_cast<const float4*>(F1), reinterpret_cast<float4*>(F1r), reinterpret_cast<uint2*>(F1h), s1, n1};
  const RoundJob j2{reinterpret_cast<const float4*>(F2), reinterpret_cast<float4*>(F2r), reinterpret_cast<uint2*>(F2h), s2, n2};
  const unsigned c1 = copies ? blocks(n1) : 0, c2 = copies ? blocks(n2) : 0;
  const int mean_rows = means ? d.H2 + d.W2 : 0;
  const long long grid = (long long)mean_rows * d.B + c1 + c2;
  if (grid > INT_MAX) return cudaErrorInvalidConfiguration;
  launch_next(round_means_kernel, (unsigned)grid, threads, 0, stream, j1, j2, (int)c1, (int)c2, F2, aux, mean_rows, d.B, d.H2, d.W2, d.C, auxh,
              op16, s2);
  return cudaGetLastError();
}

}  // namespace sfb
