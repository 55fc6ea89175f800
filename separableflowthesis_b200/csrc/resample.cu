// Placement of one pyramid level's separated volumes into the concatenated, level-0-sized outputs of the call site
// (core/corr.py:459-475): F.interpolate(..., mode='trilinear', align_corners=True) to [D0, H1, W1] followed by
// torch.cat over the levels.  H1 and W1 do not change, so the resampling is linear interpolation along the
// displacement axis only; the arithmetic follows torch's upsample_trilinear3d (source index = d * (Dl-1)/(D0-1) in
// float, lower neighbour by truncation, the upper neighbour clamped to the last row).  HBM-bound streaming kernels;
// every output element is written once, the backward (the adjoint) has one thread per (sample, channel, pixel) walk
// the displacement axis, so it needs no atomics.
#include <climits>

#include "kernels.h"
#include "sm100_primitives.cuh"

namespace sfb {

constexpr int RS_THREADS = 128;

__device__ __forceinline__ void resample_source(int d, float scale, int Dl, int& i0, int& i1, float& l0, float& l1) {
  const float src = scale * (float)d;
  i0 = (int)src;
  if (i0 > Dl - 1) i0 = Dl - 1;
  i1 = i0 + (i0 < Dl - 1 ? 1 : 0);
  l1 = fmaf(scale, (float)d, -(float)i0);   // in every kernel alike, so that what they add up is the same
  l0 = 1.f - l1;
}

// A thread produces its output rows of four pixels, all loads first: RS_DB rows of four neighbours with 16-byte loads and stores where the
// planes allow it (VEC), else RS_DB1 rows of four that are RS_THREADS apart.  HBM-bound with four pixels to share what a row costs
// beside its loads, its source rows and weights; with one pixel a thread 3 x 47 x 155 (three levels of five channels, 342 MB) took 112 us,
// 72 now.  grid (ceil(N1/(128*4)), sum over the volumes of ceil(D0/rows), B*K)
constexpr int RS_DB = 8, RS_DB1 = 4, RS_PX = 4;
struct ResampleJobs {
  ResampleJob j[MAX_RESAMPLE_JOBS];
  float scale[MAX_RESAMPLE_JOBS];
  int first[MAX_RESAMPLE_JOBS];   // of grid.y; volumes that do not exist start past its end
};

__device__ __forceinline__ float rs_mix(float a, float b, float l0, float l1) { return l0 * a + l1 * b; }
__device__ __forceinline__ float4 rs_mix(const float4& a, const float4& b, float l0, float l1) {
  return make_float4(rs_mix(a.x, b.x, l0, l1), rs_mix(a.y, b.y, l0, l1), rs_mix(a.z, b.z, l0, l1), rs_mix(a.w, b.w, l0, l1));
}
// Four pixels of a row: neighbours (16-byte aligned), or RS_THREADS apart and `n` of them in the plane.
template <bool VEC>
__device__ __forceinline__ float4 rs_load(const float* p, int n) {
  if (VEC) return __ldg(reinterpret_cast<const float4*>(p));
  return make_float4(__ldg(p), n > 1 ? __ldg(p + RS_THREADS) : 0.f, n > 2 ? __ldg(p + 2 * RS_THREADS) : 0.f, n > 3 ? __ldg(p + 3 * RS_THREADS) : 0.f);
}
template <bool VEC>
__device__ __forceinline__ void rs_store(float* p, const float4& v, int n) {
  if (VEC) {
    *reinterpret_cast<float4*>(p) = v;
    return;
  }
  p[0] = v.x;
  if (n > 1) p[RS_THREADS] = v.y;
  if (n > 2) p[2 * RS_THREADS] = v.z;
  if (n > 3) p[3 * RS_THREADS] = v.w;
}

template <bool VEC>
__global__ void __launch_bounds__(RS_THREADS)
upsample_displacement_kernel(const __grid_constant__ ResampleJobs jobs, int K, int N1) {
  follow_previous_kernel();
  constexpr int DB = VEC ? RS_DB : RS_DB1;
  int ji = 0;
#pragma unroll
  for (int i = 1; i < MAX_RESAMPLE_JOBS; ++i) ji = (int)blockIdx.y >= jobs.first[i] ? i : ji;
  const ResampleJob& job = jobs.j[ji];
  const int Dl = job.Dl, D0 = job.D0;
  const float scale = jobs.scale[ji];
  const int p = blockIdx.x * (RS_THREADS * RS_PX) + threadIdx.x * (VEC ? RS_PX : 1), d0 = (blockIdx.y - jobs.first[ji]) * DB;
  if (p >= N1) return;
  const int n = (N1 - p + RS_THREADS - 1) / RS_THREADS;
  const int b = blockIdx.z / K, k = blockIdx.z - b * K;
  const float* src = job.in + ((size_t)blockIdx.z * Dl) * N1 + p;
  float4 v0[DB], v1[DB];
  float l0[DB], l1[DB];
#pragma unroll
  for (int j = 0; j < DB; ++j) {
    int i0, i1;
    resample_source(min(d0 + j, D0 - 1), scale, Dl, i0, i1, l0[j], l1[j]);
    v0[j] = rs_load<VEC>(src + (size_t)i0 * N1, n);
    v1[j] = rs_load<VEC>(src + (size_t)i1 * N1, n);
  }
  float* dst = job.out + (size_t)b * job.out_sb + ((size_t)k * D0 + d0) * N1 + p;
#pragma unroll
  for (int j = 0; j < DB; ++j)
    if (d0 + j < D0) rs_store<VEC>(dst + (size_t)j * N1, rs_mix(v0[j], v1[j], l0[j], l1[j]), n);
}

// gin[b][k][i][p] = sum over d of the weights with which output row d read input row i, added in the order of d.  A
// thread walks its pixel's whole column, or (CUT) produces the RS_IB rows from r0 on by walking the output rows whose lower
// neighbour is r0 - 1 .. r0 + RS_IB - 1.  Pieces re-read rows at their ends (twice the rows at Dl = D0, batches included),
// so only launches of fewer than RS_CUT_BELOW blocks are cut, which on their own leave HBM idle.  Whole and cut, us:
// 55 blocks (1 x 55 x 128, 128 -> 128 rows) 35 and 10, 464 (8 x 47 x 156, 156 rows) 50 and 39, 1016 (4 x 135 x 240, 240 rows)
// 100 and 115, 2784 (six channels of 8 x 47 x 156) 153 and 197, 6096 (six of 4 x 135 x 240) 472 and 647.
// The volumes of a launch are cut together or not at all.  Launches of RS_WIDE_FROM such blocks or more take RS_PX pixels a thread, RS_THREADS apart,
// which share what a row costs beside its load: three levels of 2 x 48 x 64 (1152 blocks of one pixel a thread) 19 us with one and 21 with four,
// 1 x 55 x 128 (1980) 44 and 44, 2 x 55 x 128 (3960) 79 and 52, 3 x 47 x 155 110 and 67, 2 x 135 x 240 692 and 360.
// grid (ceil(N1/(128*PX)), B*K, sum over the volumes of CUT ? ceil(Dl/RS_IB) : 1)
constexpr int RS_IB = 8, RS_CUT_BELOW = 6 * SM_COUNT, RS_WIDE_FROM = 16 * SM_COUNT;
struct ResampleAdjointJobs {
  ResampleAdjointJob j[MAX_RESAMPLE_JOBS];
  float scale[MAX_RESAMPLE_JOBS];
  int first[MAX_RESAMPLE_JOBS];   // of grid.z; volumes that do not exist start past its end
};

template <bool CUT, int PX>
__global__ void __launch_bounds__(RS_THREADS)
upsample_displacement_adjoint_kernel(const __grid_constant__ ResampleAdjointJobs jobs, int K, int N1) {
  follow_previous_kernel();
  int ji = 0;
#pragma unroll
  for (int i = 1; i < MAX_RESAMPLE_JOBS; ++i) ji = (int)blockIdx.z >= jobs.first[i] ? i : ji;
  const ResampleAdjointJob& job = jobs.j[ji];
  const int Dl = job.Dl, D0 = job.D0;
  const float scale = jobs.scale[ji];
  const int p = blockIdx.x * (RS_THREADS * PX) + threadIdx.x;
  if (p >= N1) return;
  const int n = (N1 - p + RS_THREADS - 1) / RS_THREADS;   // of the thread's PX pixels, RS_THREADS apart
  const int b = blockIdx.y / K, k = blockIdx.y - b * K;
  const int r0 = CUT ? (blockIdx.z - jobs.first[ji]) * RS_IB : 0, r1 = CUT ? min(r0 + RS_IB, Dl) : Dl;
  const float* g = job.gout + (size_t)b * job.gout_sb + ((size_t)k * D0) * N1 + p;
  float* dst = job.gin + ((size_t)blockIdx.y * Dl) * N1 + p;
  // first output row with lower neighbour >= r0 - 1: an estimate, corrected with the exact rule (neighbours never fall
  // as d grows)
  int first = 0;
  if (CUT && r0 > 1) {
    int i0, i1;
    float l0, l1;
    first = max(0, min(D0 - 1, (int)((float)(r0 - 1) / scale) - 1));
    for (; first > 0; --first) {
      resample_source(first - 1, scale, Dl, i0, i1, l0, l1);
      if (i0 < r0 - 1) break;
    }
    for (; first < D0; ++first) {
      resample_source(first, scale, Dl, i0, i1, l0, l1);
      if (i0 >= r0 - 1) break;
    }
  }
  // the source row grows by at most one per output row (Dl <= D0): two running sums cover rows cur and cur + 1
  int cur = CUT && r0 > 0 ? r0 - 1 : 0;
  float acc0[PX], acc1[PX];
#pragma unroll
  for (int k = 0; k < PX; ++k) acc0[k] = acc1[k] = 0.f;
  auto put = [&](int i, const float (&v)[PX]) {
    if (CUT && (i < r0 || i >= r1)) return;
#pragma unroll
    for (int k = 0; k < PX; ++k)
      if (k < n) dst[(size_t)i * N1 + k * RS_THREADS] = v[k];
  };
  constexpr int DB = PX == 1 ? 8 : 4;  // output rows loaded per batch
  bool done = false;
  for (int d0 = first; d0 < D0 && !done; d0 += DB) {
    float gv[DB][PX];
#pragma unroll
    for (int j = 0; j < DB; ++j)
#pragma unroll
      for (int k = 0; k < PX; ++k) gv[j][k] = d0 + j < D0 && k < n ? __ldg(g + (size_t)(d0 + j) * N1 + k * RS_THREADS) : 0.f;
#pragma unroll
    for (int j = 0; j < DB; ++j) {
      if (d0 + j >= D0) break;
      int i0, i1;
      float l0, l1;
      resample_source(d0 + j, scale, Dl, i0, i1, l0, l1);
      if (CUT && i0 >= r1) { done = true; break; }
      while (cur < i0) {  // at most one step
        put(cur, acc0);
#pragma unroll
        for (int k = 0; k < PX; ++k) {
          acc0[k] = acc1[k];
          acc1[k] = 0.f;
        }
        ++cur;
      }
#pragma unroll
      for (int k = 0; k < PX; ++k) {
        acc0[k] = fmaf(l0, gv[j][k], acc0[k]);
        if (i1 != i0) acc1[k] = fmaf(l1, gv[j][k], acc1[k]);
        else acc0[k] = fmaf(l1, gv[j][k], acc0[k]);
      }
    }
  }
  put(cur, acc0);
  if (cur + 1 < r1) put(cur + 1, acc1);
#pragma unroll
  for (int k = 0; k < PX; ++k) acc0[k] = 0.f;
  for (int i = cur + 2; i < r1; ++i) put(i, acc0);
}

static float resample_scale(int Dl, int D0) { return D0 > 1 ? (float)(Dl - 1) / (float)(D0 - 1) : 0.f; }

cudaError_t launch_upsample_displacement(const ResampleJob* job, int count, int B, int K, int N1, cudaStream_t st) {
  if (count < 1 || count > MAX_RESAMPLE_JOBS) return cudaErrorInvalidValue;
  ResampleJobs jobs;
  bool vec = N1 % 4 == 0;
  for (int i = 0; i < count; ++i)
    vec = vec && job[i].out_sb % 4 == 0 && ((reinterpret_cast<uintptr_t>(job[i].in) | reinterpret_cast<uintptr_t>(job[i].out)) & 15u) == 0;
  const int per_block = vec ? RS_DB : RS_DB1;
  int rows = 0;
  for (int i = 0; i < MAX_RESAMPLE_JOBS; ++i) {
    jobs.j[i] = job[i < count ? i : 0];
    jobs.first[i] = i < count ? rows : INT_MAX;
    jobs.scale[i] = resample_scale(jobs.j[i].Dl, jobs.j[i].D0);
    if (i < count) rows += (job[i].D0 + per_block - 1) / per_block;
  }
  const dim3 grid((N1 + RS_THREADS * RS_PX - 1) / (RS_THREADS * RS_PX), rows, B * K);
  auto kern = vec ? upsample_displacement_kernel<true> : upsample_displacement_kernel<false>;
  launch_next(kern, grid, RS_THREADS, 0, st, jobs, K, N1);
  return cudaGetLastError();
}

cudaError_t launch_upsample_displacement_adjoint(const ResampleAdjointJob* job, int count, int B, int K, int N1, cudaStream_t st) {
  if (count < 1 || count > MAX_RESAMPLE_JOBS) return cudaErrorInvalidValue;
  const int blocks = (N1 + RS_THREADS - 1) / RS_THREADS;
  bool cut = false;
  for (int i = 0; i < count; ++i) cut = cut || job[i].Dl > RS_IB;
  cut = cut && (long long)blocks * B * K * count < RS_CUT_BELOW;
  ResampleAdjointJobs jobs;
  int pieces = 0;
  for (int i = 0; i < MAX_RESAMPLE_JOBS; ++i) {
    jobs.j[i] = job[i < count ? i : 0];
    jobs.first[i] = i < count ? pieces : INT_MAX;
    jobs.scale[i] = resample_scale(jobs.j[i].Dl, jobs.j[i].D0);
    if (i < count) pieces += cut ? (job[i].Dl + RS_IB - 1) / RS_IB : 1;
  }
  // whole columns of a large launch: several pixels a thread
  const int px = cut || (long long)blocks * B * K * count < RS_WIDE_FROM ? 1 : RS_PX;
  auto kern = cut ? upsample_displacement_adjoint_kernel<true, 1>
                  : (px == 1 ? upsample_displacement_adjoint_kernel<false, 1> : upsample_displacement_adjoint_kernel<false, RS_PX>);
  launch_next(kern, dim3((N1 + RS_THREADS * px - 1) / (RS_THREADS * px), B * K, pieces), RS_THREADS, 0, st, jobs, K, N1);
  return cudaGetLastError();
}

}  // namespace sfb
