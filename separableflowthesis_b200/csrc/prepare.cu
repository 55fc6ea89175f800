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
// multipliers.  One launch in place of one per array and one for the multipliers.  grid (blocks, rows: the samples of every array),
// block 256.
constexpr int AM_THREADS = 256, AM_UNROLL = 4;
struct AbsmaxJobs {
  AbsmaxSource src[ABSMAX_MAX];
  int first_row[ABSMAX_MAX];   // of grid.y; sources that do not exist start past its end
};
__global__ void __launch_bounds__(AM_THREADS)
absmax_kernel(const __grid_constant__ AbsmaxJobs jobs, float* scales, int levels, int gradients) {
  __shared__ float red[AM_THREADS / 32];
  int job = 0;
#pragma unroll
  for (int j = 1; j < ABSMAX_MAX; ++j) job = (int)blockIdx.y >= jobs.first_row[j] ? j : job;
  const AbsmaxSource& src = jobs.src[job];
  const float* x = src.p + (size_t)(blockIdx.y - jobs.first_row[job]) * src.sb;
  // a sample's channels may start off a 16-byte boundary: up to three values before the first vector, up to three behind the last
  const size_t n = src.n, head = min((size_t)((16u - (reinterpret_cast<uintptr_t>(x) & 15u)) & 15u) / 4, n);
  const size_t n4 = (n - head) / 4, stride = (size_t)gridDim.x * AM_THREADS;
  const float4* x4 = reinterpret_cast<const float4*>(x + head);
  float m = 0.f;
  for (size_t i = (size_t)blockIdx.x * AM_THREADS + threadIdx.x; i < n4; i += AM_UNROLL * stride) {
    float4 v[AM_UNROLL];
#pragma unroll
    for (int j = 0; j < AM_UNROLL; ++j) v[j] = i + j * stride < n4 ? __ldg(x4 + i + j * stride) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < AM_UNROLL; ++j)
      m = fmaxf(m, fmaxf(fmaxf(fabsf(v[j].x), fabsf(v[j].y)), fmaxf(fabsf(v[j].z), fabsf(v[j].w))));
  }
  if (blockIdx.x == 0 && threadIdx.x < head) m = fmaxf(m, fabsf(__ldg(x + threadIdx.x)));
  if (blockIdx.x == 0 && threadIdx.x < n - head - 4 * n4) m = fmaxf(m, fabsf(__ldg(x + head + 4 * n4 + threadIdx.x)));
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
  if (atomicAdd(ticket, 1u) != gridDim.x * gridDim.y - 1) return;
  __threadfence();
  for (int l = 0; l < levels; ++l) {
    if (gradients) grad_scales(scales + l * SCALE_LEVEL);
    else feature_scales(scales + l * SCALE_LEVEL, scales + SCALE_AMAX_F1);
  }
  *ticket = 0;
}

cudaError_t launch_absmax(const AbsmaxSource* src, int count, float* scales, int levels, bool gradients, cudaStream_t stream) {
  if (count < 1 || count > ABSMAX_MAX) return cudaErrorInvalidValue;
  AbsmaxJobs jobs;
  size_t most = 0;
  long long rows = 0;
  for (int i = 0; i < ABSMAX_MAX; ++i) {
    jobs.src[i] = src[i < count ? i : 0];
    jobs.first_row[i] = i < count ? (int)rows : INT_MAX;
    if (i >= count) continue;
    if (src[i].sb == (long long)src[i].n) {   // samples that follow one another are one array
      jobs.src[i].n *= src[i].samples;
      jobs.src[i].samples = 1;
    }
    rows += jobs.src[i].samples;
    most = std::max(most, jobs.src[i].n);
  }
  if (rows > 65535) return cudaErrorInvalidConfiguration;
  const size_t per_block = (size_t)AM_THREADS * 4 * AM_UNROLL;
  const unsigned blocks = (unsigned)std::max<size_t>(1, std::min<size_t>((most + per_block - 1) / per_block, 148 * 8));
  absmax_kernel<<<dim3(blocks, (unsigned)rows), AM_THREADS, 0, stream>>>(jobs, scales, levels, gradients ? 1 : 0);
  return cudaGetLastError();
}

// `outh` (optional): the same values as 16-bit operands of kind `op16` instead (BF16, or FP16 of the value times the
// device scalar *scale16).
__global__ void round_copy_kernel(const float4* __restrict__ in, float4* __restrict__ out, size_t n4,
                                  uint2* __restrict__ outh, int op16, const float* __restrict__ scale16) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const float sc = (outh != nullptr && scale16 != nullptr) ? __ldg(scale16) : 1.f;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += stride) {
    float4 v = __ldg(in + i);
    if (outh != nullptr) {
      if (op16 == OP16_FP16) outh[i] = make_uint2(pack_fp16x2(v.x * sc, v.y * sc), pack_fp16x2(v.z * sc, v.w * sc));
      else outh[i] = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
    }
    if (out != nullptr) {
      v.x = round_tf32(v.x); v.y = round_tf32(v.y); v.z = round_tf32(v.z); v.w = round_tf32(v.w);
      out[i] = v;
    }
  }
}

// One mean row, in the two forms the sweeps may read it: TF32 in `aux` or 16-bit in `auxh` (each may be null).
__device__ __forceinline__ void store_mean(float mean, size_t at, float* aux, uint16_t* auxh, int op16, float sc16) {
  if (aux != nullptr) aux[at] = round_tf32(mean);
  if (auxh != nullptr) auxh[at] = to_op16(mean * sc16, op16);
}

// From pixel-major features.  A block owns one mean row; four groups of 64 threads take every fourth pixel of it, a
// thread four channels at a time, so that the pixels' loads are in flight side by side.  grid (H2 + W2, B), block 256.
constexpr int FM_GROUPS = 4, FM_QUADS = 64;
__global__ void __launch_bounds__(FM_GROUPS * FM_QUADS)
f2_means_kernel(const float* __restrict__ F2, float* __restrict__ aux, int H2, int W2, int C,
                uint16_t* __restrict__ auxh, int op16, const float* __restrict__ scale16) {
  __shared__ float4 red[FM_GROUPS][FM_QUADS];
  const int r = blockIdx.x, b = blockIdx.y, g = threadIdx.x / FM_QUADS, q = threadIdx.x % FM_QUADS;
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

// From channel-major feature maps: a block owns one channel plane; its warps take every eighth row, FC_ROWS rows at a time, a
// lane every 32nd column.  NV = ceil(W2 / 32) rounded up to a power of two: the column sums of a lane stay in registers, so
// that the plane is read once, with FC_ROWS * NV loads of a lane in flight (HBM-bound; one walk for the rows and one for the
// columns took 162 us at 8 x 135 x 240, C = 256).  NV = 0: any width, in the two walks.  Both add in the same order.
// grid (C, B, levels), block 256.
constexpr int FC_ROWS = 2;
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
  auto store_row = [&](int u, float acc) {   // acc: this lane's share of row u
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) store_mean(acc / (float)W2, out0 + (size_t)u * C, aux, auxh, op16, sc16);
  };
  if constexpr (NV > 0) {
    float col[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) col[i] = 0.f;
    for (int u0 = warp; u0 < H2; u0 += 8 * FC_ROWS) {
      float v[FC_ROWS][NV];
#pragma unroll
      for (int r = 0; r < FC_ROWS; ++r)
#pragma unroll
        for (int i = 0; i < NV; ++i)
          v[r][i] = u0 + 8 * r < H2 && lane + 32 * i < W2 ? __ldg(plane + (size_t)(u0 + 8 * r) * W2 + lane + 32 * i) : 0.f;
#pragma unroll
      for (int r = 0; r < FC_ROWS; ++r) {
        if (u0 + 8 * r >= H2) break;
        float acc = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          acc += v[r][i];
          col[i] += v[r][i];
        }
        store_row(u0 + 8 * r, acc);
      }
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
// packed layout (B, D, R, n1p) (pixel fastest) the kernels use.  A block moves a patch of 128 pixels x 32
// displacements through shared memory so that both sides are coalesced; every thread keeps 16 loads in flight,
// and the displacement tiles are the fastest grid dimension so that blocks running together read neighbouring
// 128-byte pieces of the same rows.  grid (ceil(D/32), n1p/128, B*K), block (32, 8).
constexpr int PACK_PX = 128;

__global__ void pack_kernel(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst, int N1, int n1p, int Ksrc,
                            int ksrc0, int K, int D, int R, int r0, int rstride, float scale) {
  __shared__ uint32_t tile[PACK_PX][33];
  const int b = blockIdx.z / K, k = blockIdx.z - b * K, d0 = blockIdx.x * 32, p0 = blockIdx.y * PACK_PX;
  const int tx = threadIdx.x, ty = threadIdx.y;
#pragma unroll
  for (int j = ty; j < PACK_PX; j += 8) {
    const int p = p0 + j, d = d0 + tx;
    uint32_t v = 0;
    if (p < N1 && d < D) v = __ldg(src + (((size_t)b * N1 + p) * Ksrc + ksrc0 + k) * D + d);
    tile[j][tx] = v;
  }
  __syncthreads();
  const int r = r0 + k * rstride;
#pragma unroll
  for (int i = ty; i < 32 * (PACK_PX / 32); i += 8) {
    const int d = d0 + i / (PACK_PX / 32), p = (i % (PACK_PX / 32)) * 32 + tx;
    if (d < D) {
      uint32_t v = tile[p][i / (PACK_PX / 32)];
      if (scale != 0.f) v = __float_as_uint(__uint_as_float(v) * scale);
      dst[(((size_t)b * D + d) * R + r) * n1p + p0 + p] = v;
    }
  }
}

__global__ void unpack_kernel(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst, int N1, int n1p, int K,
                              int D, int R, int r0, int rstride, int Kdst, int kdst0) {
  __shared__ uint32_t tile[PACK_PX][33];
  const int b = blockIdx.z / K, k = blockIdx.z - b * K, d0 = blockIdx.x * 32, p0 = blockIdx.y * PACK_PX;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int r = r0 + k * rstride;
#pragma unroll
  for (int i = ty; i < 32 * (PACK_PX / 32); i += 8) {
    const int dl = i / (PACK_PX / 32), p = (i % (PACK_PX / 32)) * 32 + tx;
    tile[p][dl] = (d0 + dl < D) ? __ldg(src + (((size_t)b * D + d0 + dl) * R + r) * n1p + p0 + p) : 0u;
  }
  __syncthreads();
#pragma unroll
  for (int j = ty; j < PACK_PX; j += 8) {
    const int p = p0 + j, d = d0 + tx;
    if (p < N1 && d < D) dst[(((size_t)b * N1 + p) * Kdst + kdst0 + k) * D + d] = tile[j][tx];
  }
}

// Interleaved pack: every block transposes a 32-pixel x 32-displacement patch of each source through
// shared memory, then writes, per displacement, the R4 slots of its 32 pixels as one contiguous run.
template <int R4>
__global__ void pack_interleaved_kernel(const SlotSources src, uint32_t* __restrict__ dst, int N1, int n1p, int D,
                                        int Qtot, int q0) {
  constexpr int RS = 32 * 33 + 32 / R4;  // slot stride chosen so that the interleaved read below is conflict-free
  __shared__ uint32_t tile[R4 * RS];
  const int b = blockIdx.z, d0 = blockIdx.x * 32, p0 = blockIdx.y * 32;  // displacement tiles fastest
  const int tx = threadIdx.x, ty = threadIdx.y;
#pragma unroll
  for (int r = 0; r < R4; ++r) {
    const uint32_t* s = static_cast<const uint32_t*>(src.s[r].src);
    for (int j = ty; j < 32; j += 8) {
      const int p = p0 + j, d = d0 + tx;
      uint32_t v = 0;
      if (p < N1 && d < D) {
        if (s == nullptr) {
          v = __float_as_uint(src.s[r].scale);  // constant slot
        } else {
          v = __ldg(s + (((size_t)b * N1 + p) * src.s[r].Ksrc + src.s[r].k) * D + d);
          if (src.s[r].scale != 0.f) v = __float_as_uint(__uint_as_float(v) * src.s[r].scale);
          if (src.s[r].dev != 0) v = __float_as_uint(__uint_as_float(v) * __ldg(src.dev_scales + src.s[r].dev - 1));
        }
      }
      tile[r * RS + j * 33 + tx] = v;
    }
  }
  __syncthreads();
  // per displacement and group of four slots: 32 pixels x 4 slots = 128 consecutive words
  const int t = ty * 32 + tx;
  for (int j = 0; j < 32; ++j) {
    const int d = d0 + j;
    if (d >= D) break;
    for (int i = t; i < 32 * R4; i += 256) {
      const int q = i / 128, w = i % 128;  // group, word inside the group's 32-pixel run
      dst[((((size_t)b * D + d) * Qtot + q0 + q) * n1p + p0) * 4 + w] = tile[(q * 4 + (w & 3)) * RS + (w >> 2) * 33 + j];
    }
  }
}

cudaError_t launch_pack_interleaved(const SlotSources& src, float* dst, int B, int N1, int n1p, int D, int R4,
                                    int Qtot, int q0, cudaStream_t stream) {
  const dim3 grid((D + 31) / 32, n1p / 32, B), block(32, 8);
  uint32_t* out = reinterpret_cast<uint32_t*>(dst);
  if (R4 == 4) pack_interleaved_kernel<4><<<grid, block, 0, stream>>>(src, out, N1, n1p, D, Qtot, q0);
  else if (R4 == 8) pack_interleaved_kernel<8><<<grid, block, 0, stream>>>(src, out, N1, n1p, D, Qtot, q0);
  else return cudaErrorInvalidValue;
  return cudaGetLastError();
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
  const int per_launch = pack_groups_per_launch(B);
  for (int first = 0; first < groups.count; first += per_launch) {
    PackGroups some = groups;
    some.count = std::min(per_launch, groups.count - first);
    int D = 1;
    for (int i = 0; i < some.count; ++i) {
      some.g[i] = groups.g[first + i];
      D = std::max(D, some.g[i].D);
    }
    const dim3 grid((n1p + 255) / 256, (D + PI_DB - 1) / PI_DB, some.count * B);
    pack_interleaved_cf_kernel<<<grid, 256, 0, stream>>>(some, B, N1, n1p);
    if (cudaError_t err = cudaGetLastError(); err != cudaSuccess) return err;
  }
  return cudaSuccess;
}

cudaError_t launch_pack(const void* src, float* dst, int B, int N1, int n1p, int Ksrc, int ksrc0, int K, int D,
                        int R, int r0, int rstride, float scale, cudaStream_t stream) {
  const dim3 grid((D + 31) / 32, n1p / PACK_PX, B * K), block(32, 8);
  pack_kernel<<<grid, block, 0, stream>>>(static_cast<const uint32_t*>(src), reinterpret_cast<uint32_t*>(dst), N1,
                                          n1p, Ksrc, ksrc0, K, D, R, r0, rstride, scale);
  return cudaGetLastError();
}

cudaError_t launch_unpack(const float* src, void* dst, int B, int N1, int n1p, int K, int D, int R, int r0,
                          int rstride, int Kdst, int kdst0, cudaStream_t stream) {
  const dim3 grid((D + 31) / 32, n1p / PACK_PX, B * K), block(32, 8);
  unpack_kernel<<<grid, block, 0, stream>>>(reinterpret_cast<const uint32_t*>(src), static_cast<uint32_t*>(dst), N1,
                                            n1p, K, D, R, r0, rstride, Kdst, kdst0);
  return cudaGetLastError();
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
// scalar as well) or TF32.  The layouts of channel_major_kernel, padding included (zeros), two values per store.  One grid row per
// channel of a sample: grid (sum over the copies of ceil(pairs per channel / 256), C, B).
struct MapCopies {
  MapCopy c[MAX_MAP_COPIES];
  int first[MAX_MAP_COPIES];   // of grid.x; copies that do not exist start past its end
};
__host__ __device__ inline int map_copy_channel(const MapCopy& c) { return c.blocked ? (c.width + 15) / 16 * c.pitch * 16 : c.pitch; }
__global__ void __launch_bounds__(256)
channel_major_cf_kernel(const __grid_constant__ MapCopies copies, int C, int op16) {
  int ci = 0;
#pragma unroll
  for (int i = 1; i < MAX_MAP_COPIES; ++i) ci = (int)blockIdx.x >= copies.first[i] ? i : ci;
  const MapCopy& copy = copies.c[ci];
  const int per_channel = map_copy_channel(copy), width = copy.width;
  const int i = ((blockIdx.x - copies.first[ci]) * 256 + threadIdx.x) * 2;
  if (i >= per_channel) return;
  const float sc16 = (op16 == OP16_FP16 && copy.scale16 != nullptr) ? __ldg(copy.scale16) : 1.f;
  int row = 0, x = i;
  if (copy.blocked) {
    const int xb = i / (copy.pitch * 16), r = i - xb * copy.pitch * 16;
    row = r / 16;
    x = xb * 16 + (r & 15);
  }
  const size_t chan = (size_t)blockIdx.z * C + blockIdx.y;
  const float* src = copy.src + (chan * copy.rows + row) * width + x;
  const bool ok = row < copy.rows;
  const float lo = ok && x < width ? __ldg(src) * copy.scale : 0.f, hi = ok && x + 1 < width ? __ldg(src + 1) * copy.scale : 0.f;
  const size_t at = (chan * per_channel + i) / 2;
  if (op16 == 0) static_cast<float2*>(copy.dst)[at] = make_float2(round_tf32(lo), round_tf32(hi));
  else static_cast<uint32_t*>(copy.dst)[at] = op16 == OP16_FP16 ? pack_fp16x2(lo * sc16, hi * sc16) : pack_bf16x2(lo, hi);
}

cudaError_t launch_channel_major_cf(const MapCopy* copy, int count, int B, int C, int op16, cudaStream_t stream) {
  if (count < 1 || count > MAX_MAP_COPIES) return cudaErrorInvalidValue;
  MapCopies copies;
  int blocks = 0;
  for (int i = 0; i < MAX_MAP_COPIES; ++i) {
    copies.c[i] = copy[i < count ? i : 0];
    copies.first[i] = i < count ? blocks : INT_MAX;
    if (i < count) blocks += (map_copy_channel(copy[i]) / 2 + 255) / 256;
  }
  channel_major_cf_kernel<<<dim3(blocks, C, B), 256, 0, stream>>>(copies, C, op16);
  return cudaGetLastError();
}

// Channel-major copies of a pixel-major feature array (B, rows*width, C), the K-major B operands of the gradient GEMMs.
//   blocked = 0: dst (B, C, pitch), pixel index = row*width + x (image 1: rows = 1, width = N1, pitch = n1p)
//   blocked = 1: dst (B, C, ceil(width/16), pitch, 16): columns in blocks of 16, so that the 4 rows x 16 columns of one
//                K block of the image-1-major GEMM are 64 consecutive values (image 2: pitch = H2 rounded up to 4)
// Padding is not written (the caller clears the array).  32 x 32 tiles through shared memory; grid (ceil(width/32),
// ceil(C/32), B*rows), block (32, 8).
template <typename T>
__global__ void channel_major_kernel(const float* __restrict__ in, T* __restrict__ out, int rows, int width,
                                     int pitch, int C, int blocked, int op16, const float* __restrict__ scale16) {
  __shared__ float tile[32][33];
  const float sc16 = (op16 == OP16_FP16 && scale16 != nullptr) ? __ldg(scale16) : 1.f;
  const int b = blockIdx.z / rows, row = blockIdx.z - b * rows, x0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const float* src = in + ((size_t)b * rows + row) * width * C;
#pragma unroll
  for (int j = ty; j < 32; j += 8) {
    const int x = x0 + j, c = c0 + tx;
    tile[j][tx] = (x < width && c < C) ? __ldg(src + (size_t)x * C + c) : 0.f;
  }
  __syncthreads();
  const size_t per_channel = blocked ? (size_t)((width + 15) / 16) * pitch * 16 : (size_t)pitch;
#pragma unroll
  for (int j = ty; j < 32; j += 8) {
    const int c = c0 + j, x = x0 + tx;
    if (c < C && x < width) {
      const size_t off = blocked ? ((size_t)(x >> 4) * pitch + row) * 16 + (x & 15) : (size_t)x;
      if constexpr (sizeof(T) == 2) out[((size_t)b * C + c) * per_channel + off] = to_op16(tile[tx][j] * sc16, op16);
      else out[((size_t)b * C + c) * per_channel + off] = tile[tx][j];
    }
  }
}

cudaError_t launch_channel_major(const float* src, void* dst, int B, int rows, int width, int pitch, int C,
                                 int blocked, int op16, const float* scale16, cudaStream_t stream) {
  const dim3 grid((width + 31) / 32, (C + 31) / 32, B * rows), block(32, 8);
  if (op16)
    channel_major_kernel<<<grid, block, 0, stream>>>(src, static_cast<uint16_t*>(dst), rows, width, pitch, C, blocked,
                                                     op16, scale16);
  else
    channel_major_kernel<<<grid, block, 0, stream>>>(src, static_cast<float*>(dst), rows, width, pitch, C, blocked, 0,
                                                     nullptr);
  return cudaGetLastError();
}

// Clears the workspace header (status word, scale slots) and, for FP16 operands, finds the feature scales.
static cudaError_t begin_prepare(const Dims* d, int levels, const float* F1, const float* const* F2, float premul1, int* status, int op16,
                                 float* scales, cudaStream_t stream) {
  cudaError_t err = cudaMemsetAsync(status, 0, WS_SCALES_OFFSET + (size_t)levels * SCALE_LEVEL * sizeof(float), stream);
  if (err != cudaSuccess || op16 != OP16_FP16 || scales == nullptr) return err;
  AbsmaxSource src[1 + MAX_FUSED_LEVELS];
  src[0] = absmax_array(F1, (size_t)d[0].B * d[0].N1() * d[0].C, premul1, SCALE_AMAX_F1);
  for (int l = 0; l < levels; ++l)
    src[1 + l] = absmax_array(F2[l], (size_t)d[l].B * d[l].N2() * d[l].C, 1.f, l * SCALE_LEVEL + SCALE_AMAX_F2);
  return launch_absmax(src, 1 + levels, scales, levels, false, stream);
}

cudaError_t launch_prepare_cf(const Dims* d, int levels, const float* fmap1, const float* const* fmap2, float scale1,
                              const LevelOperands* out, float* F1r, uint16_t* F1h, int* status, cudaStream_t stream, int op16, float* scales) {
  if (levels < 1 || levels > MAX_FUSED_LEVELS) return cudaErrorInvalidValue;
  cudaError_t err = begin_prepare(d, levels, fmap1, fmap2, scale1, status, op16, scales, stream);
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
    transpose_round_kernel<<<dim3(blocks, (C + 63) / 64, B), dim3(32, 8), 0, stream>>>(jobs, C, op16);
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
    kern<<<dim3(C, B, levels), 256, 0, stream>>>(jobs, C, op16);
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
  if (F1r != nullptr || F1h != nullptr) {
    round_copy_kernel<<<blocks(n1), threads, 0, stream>>>(reinterpret_cast<const float4*>(F1),
                                                          reinterpret_cast<float4*>(F1r), n1,
                                                          reinterpret_cast<uint2*>(F1h), op16, s1);
    round_copy_kernel<<<blocks(n2), threads, 0, stream>>>(reinterpret_cast<const float4*>(F2),
                                                          reinterpret_cast<float4*>(F2r), n2,
                                                          reinterpret_cast<uint2*>(F2h), op16, s2);
  }
  if (aux != nullptr || auxh != nullptr)
    f2_means_kernel<<<dim3(d.H2 + d.W2, d.B), FM_GROUPS * FM_QUADS, 0, stream>>>(F2, aux, d.H2, d.W2, d.C, auxh, op16, s2);
  return cudaGetLastError();
}

}  // namespace sfb
