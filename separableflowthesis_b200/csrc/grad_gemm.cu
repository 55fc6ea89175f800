// Gradient GEMMs of the backward ops:  gF1 = G * F2  and  gF2 = G^T * F1,  where
// G = dLoss/dS (N1 x N2 per sample) is never stored: each 128 x 32 block of it is generated by CUDA
// cores as the A operand of tcgen05.mma, while TMA streams the matching block of the other image's
// features as the B operand.  The 128 x C output tile accumulates in TMEM over the whole K sweep and is
// written once, so the result is deterministic (no atomics), unlike the reference's atomicAdd scatter
// (MemorySaver_kernel_max_avg_argmax_backward.cu:305-310, MemorySaver_kernel_compression_backward.cu:477-488).
//
//   image2_major = 0 : rows = 128 consecutive image-1 pixels, K = image-2 pixels in blocks of
//                      2 rows x 16 columns (column blocks outermost), output gF1.  A generator thread owns one
//                      row = one TMEM lane, so the generated blocks go to tensor memory (tcgen05.st) next to the
//                      accumulator and the tensor core reads A from TMEM: no shared-memory stores, fences or
//                      operand reads for A.
//   image2_major = 1 : rows = an 8 x 16 block of image-2 pixels, K = 32 consecutive image-1 pixels,
//                      output gF2.  A generator thread owns one K column (pixel), so the blocks are written to
//                      shared memory in the swizzled K-major layout.
// B operand, both forms: K-major, like the operands of the correlation sweeps: one TMA box of 32*ceil(C/32) channel
// rows x 32 K-values from channel-major copies of the rounded features (image 1: (C, pixels); image 2: (C, column
// blocks of 16, rows, 16), so that the 2 rows x 16 columns of a K block are 32 consecutive values).  The MN-major
// form (pixel-major features) issues about 1.4x slower per tcgen05.mma and was dropped.
// G for the max/avg op (MemorySaver_kernel_max_avg_argmax_backward.cu:200-251):
//   G[p,u,v] = gMax_u[p,u]*[v==AM_u[p,u]] + gAvg_u[p,u]/W2 + gMax_v[p,v]*[u==AM_v[p,v]] + gAvg_v[p,v]/H2
// G for the compression op (MemorySaver_kernel_compression_backward.cu:464-488):
//   G[p,u,v] = sum_k gC_u[p,k,u]*A_u[p,k,v] + A_v[p,k,u]*gC_v[p,k,v]
// GRAD_FUSED generates the sum of both, so one GEMM pair serves both backward ops.
// The per-pixel inputs come from the interleaved operands XU / XV (kernels.h); the blocks a K step needs are
// copied into shared memory by TMA a few steps ahead, so the generator's reads have shared-memory latency.
//
// 16-bit form (GradArgs::op16 = BF16 or FP16): the same kernels with tcgen05.mma kind::f16.  G is rounded to the 16-bit
// type as it is generated (two values per 32-bit TMEM column / 64-byte shared-memory rows) and the feature copies are
// 16-bit (64-byte rows, 64-byte swizzle), so a block is two instructions of K = 16 instead of four of K = 8.
// Accumulation stays FP32.  With FP16 the operands carry power-of-two scales (kernels.h, SCALE_*) that the drain undoes.
//
// Tail tiles: like the correlation sweeps, the tiles past the last full wave of 148 CTAs are cut into `pieces` CTAs, each
// a range of the K sweep.  Piece 0 drains to the output, the others to scratch, and the CTA that finishes a tile last
// (a counter per tile, nobody waits) adds them to the output in piece order: deterministic.
//
// Warp roles: warp 0 feature (B operand) producer, warp 1 TMEM allocation + MMA issue, warps 2..9 generate G
// and, at the end, drain the accumulator (two warps per TMEM lane quarter, alternating 16-column chunks),
// warp 10 producer of the XU / XV blocks.
#include <cuda_bf16.h>

#include "kernels.h"
#include "sm100_primitives.cuh"

namespace sfb {

constexpr int GG_GEN_WARPS = 8;
constexpr int GG_THREADS = (3 + GG_GEN_WARPS) * 32;
constexpr int GG_VH = GG_VT / (GG_GEN_WARPS / 4);          // columns of one image-1-major generator thread
constexpr uint32_t GG_YBLOCK_BYTES = GG_KJ * KBLK * 4;     // 4 KB: 32 channel rows x 32 K-values
constexpr uint32_t GG_ACC_COLS = 256;                      // accumulator columns (the feature dimension)

// Ring depths.  Every kind of block has its own ring, sized by how long a stage stays in use:
//   NY   feature blocks (B operand, 32 KB at C = 256): freed when the MMAs of the block have completed
//   NG   generated blocks (A operand): image-1-major in TMEM columns 256 + 32*stage .., image-2-major in shared memory
//   NXU  (pixel, u) operand blocks: read row by row while the block is computed, freed after the computation
//   NXV  (pixel, v) operand blocks (image-2-major only; the image-1-major form keeps those slots in registers): read
//        into registers at the start of a block and freed at once, so that the next load has the whole computation
//        of the block to arrive
// The image-2-major form's two generator groups hold two operand blocks at a time and a TMA load takes about as long
// as one block's computation: with fewer than four (pixel, u) stages the generators wait for their operands.
template <int Q, int I2MAJOR> struct GradCfg;
template <> struct GradCfg<1, 0> { static constexpr int NY = 6, NG = 6, NXU = 4, NXV = 1; };
template <> struct GradCfg<2, 0> { static constexpr int NY = 5, NG = 5, NXU = 4, NXV = 1; };
template <> struct GradCfg<3, 0> { static constexpr int NY = 5, NG = 5, NXU = 4, NXV = 1; };
template <> struct GradCfg<1, 1> { static constexpr int NY = 3, NG = 2, NXU = 4, NXV = 2; };
template <> struct GradCfg<2, 1> { static constexpr int NY = 3, NG = 2, NXU = 4, NXV = 2; };
template <> struct GradCfg<3, 1> { static constexpr int NY = 3, NG = 2, NXU = 4, NXV = 2; };
template <int I2MAJOR> __host__ __device__ constexpr uint32_t gg_tmem_cols() { return I2MAJOR ? 256u : 512u; }

template <int Q, int I2MAJOR>
struct GradSmem {
  using Cfg = GradCfg<Q, I2MAJOR>;
  static constexpr int AT = I2MAJOR ? 0 : 1;   // A blocks in tensor memory
  static_assert(GG_ACC_COLS + (AT ? Cfg::NG * GG_KJ : 0) <= gg_tmem_cols<I2MAJOR>(), "A stages exceed TMEM");
  // one operand block: [displacement][group of 4 slots][pixel][4]; image-1-major 2 x Q x 128, image-2-major 8 x Q x 32
  static constexpr int XU_FLOATS = (I2MAJOR ? GG_ROW_UT * GG_KJ : GG_UT * TILE_M) * Q * 4;
  static constexpr int XV_FLOATS = I2MAJOR ? GG_ROW_VT * GG_KJ * Q * 4 : 4;  // image-1-major keeps XV in registers
  float y[Cfg::NY][MAX_KB * KBLK * GG_KJ];    // feature blocks [channel][32 K-values], K-major, 128B swizzle
  float g[AT ? 1 : Cfg::NG][AT ? 32 : TILE_M * GG_KJ];  // generated A blocks (image-2-major form), K-major, 128B swizzle
  float xu[Cfg::NXU][XU_FLOATS];
  float xv[Cfg::NXV][XV_FLOATS];
  uint64_t y_full[Cfg::NY];
  uint64_t y_empty[Cfg::NY];
  uint64_t g_full[Cfg::NG];
  uint64_t g_empty[Cfg::NG];
  uint64_t xu_full[Cfg::NXU];
  uint64_t xu_empty[Cfg::NXU];
  uint64_t xv_full[Cfg::NXV];
  uint64_t xv_empty[Cfg::NXV];
  uint64_t acc_full;
  uint32_t tmem_base;
  int last_piece;                             // this CTA finished its tail tile last: it adds the pieces up
  WaitCtl ctl;
};

struct GradSched {
  int b, nkb;
  int t0, n_blocks;  // first block of the K sweep this CTA does, and how many
  int tail, piece;   // tail tile this CTA has a piece of (-1: a whole tile) and which piece
  int m0;            // image-1-major: first pixel of the row tile
  int u0, v0;        // image-2-major: origin of the 8 x 16 row tile
  int n_ub2;         // image-1-major: number of 2-row blocks along u
  int h2p;           // image-1-major: rows of the column-blocked channel-major copy of image 2 (H2 rounded up to even)
};

// The 4*Q slots of one (pixel, displacement) pair as 2*Q packed float pairs.
template <int Q>
struct Slots {
  uint64_t v[2 * Q];
  // global memory: group q of this pixel is `group_stride` floats after group q-1
  __device__ __forceinline__ void load_global(const float* p, size_t group_stride, bool ok) {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      ulonglong2 t = make_ulonglong2(0ull, 0ull);
      if (ok) t = __ldg(reinterpret_cast<const ulonglong2*>(p + q * group_stride));
      v[2 * q] = t.x;
      v[2 * q + 1] = t.y;
    }
  }
  // shared memory block [group][pixel][4]
  __device__ __forceinline__ void load_shared(const float* p, int group_stride) {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(p + q * group_stride);
      v[2 * q] = t.x;
      v[2 * q + 1] = t.y;
    }
  }
};

// TF32 rounding of a value that goes straight to the tensor core: tcgen05.mma kind::tf32 ignores the low 13
// mantissa bits, so adding half a TF32 ulp is all it takes (round_tf32 without the mask).
__device__ __forceinline__ float round_for_mma(float x) { return __uint_as_float(__float_as_uint(x) + 0x1000u); }

// x += add when a == b, as one compare and one predicated add (a select followed by an add costs a third instruction
// per term, and the generator is bound by instruction issue).
__device__ __forceinline__ void add_if_equal(float& x, int a, int b, float add) {
  asm("{\n\t.reg .pred p;\n\t"
      "setp.eq.s32 p, %1, %2;\n\t"
      "@p add.f32 %0, %0, %3;\n\t}"
      : "+f"(x)
      : "r"(a), "r"(b), "f"(add));
}

__device__ __forceinline__ float pair_lo(uint64_t v) { return __uint_as_float(static_cast<uint32_t>(v)); }
__device__ __forceinline__ int pair_hi_bits(uint64_t v) { return static_cast<int>(static_cast<uint32_t>(v >> 32)); }

// The part of a G value that is a sum of products of the two pixels' slots, as one packed multiply-add chain.
// Max/avg group (slots 0..3 of XU: mean-gradient/W2, 1, max-gradient, argmax; of XV: 1, mean-gradient/H2,
// max-gradient, argmax): pair 0 multiplies to (mean-gradient_u, mean-gradient_v), whose two halves the final
// horizontal add sums; pair 1 takes no part in the chain.  Compression groups: every pair is a product.
template <int MODE, int Q>
__device__ __forceinline__ float g_products(const Slots<Q>& xu, const Slots<Q>& xv) {
  uint64_t acc = mul2(xu.v[0], xv.v[0]);
#pragma unroll
  for (int q = (MODE == GRAD_COMPRESS ? 1 : 2); q < 2 * Q; ++q) acc = fma2(xu.v[q], xv.v[q], acc);
  return sum2(acc);
}

// rows = image-1 pixels.  Thread (pl, vh): row pl of the tile, columns vh*8 .. vh*8+7 of every 2 x 16 block.
// The (pixel, v) slots stay in registers across the inner sweep over u; the (pixel, u) slots of each block
// arrive in shared memory by TMA.  The finished values go to this thread's TMEM lane (A operand in tensor memory).
template <int MODE, int Q, int BF16>
__device__ void generator_image1(GradSmem<Q, 0>& sm, const GradArgs& a, const GradSched& sc, int warp, int gw, int lane) {
  using Cfg = GradCfg<Q, 0>;
  const int W2 = a.d.W2;
  const size_t group_stride = (size_t)a.n1p * 4, row_stride = group_stride * Q;
  const int pl = (warp & 3) * 32 + lane, vh = gw >> 2;
  const float* xv_p = a.xv + (size_t)sc.b * W2 * row_stride + (size_t)(sc.m0 + pl) * 4;
  Slots<Q> xv[GG_VH];
  // TMEM address of this thread's lane quarter, first A column of stage 0, this thread's 8 columns
  // (BF16: two values per column, so the thread's 8 values of a row are 4 columns)
  const uint32_t ta0 = sm.tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + GG_ACC_COLS +
                       vh * (BF16 ? GG_VH / 2 : GG_VH);
  int vb = sc.t0 / sc.n_ub2, ub2 = sc.t0 - vb * sc.n_ub2;
  for (int t = 0; t < sc.n_blocks; ++t) {
    const uint32_t so = t % Cfg::NXU, pho = (t / Cfg::NXU) & 1u;
    const uint32_t s = t % Cfg::NG, ph = (t / Cfg::NG) & 1u;
    const int vbase = vb * GG_VT + vh * GG_VH;
    if (ub2 == 0 || t == 0) {
#pragma unroll
      for (int i = 0; i < GG_VH; ++i)
        xv[i].load_global(xv_p + (size_t)(vbase + i) * row_stride, group_stride, vbase + i < W2);
    }
    if (!mbar_wait(&sm.xu_full[so], pho, &sm.ctl, a.status, DEV_TIMEOUT_GENERATOR)) return;
    float g[GG_UT][GG_VH];
#pragma unroll
    for (int ul = 0; ul < GG_UT; ++ul) {
      Slots<Q> xu;  // block layout [pixel half][ul][group][64 pixels][4]; rows past the image are zero-filled by TMA
      xu.load_shared(sm.xu[so] + ((((pl >> 6) * GG_UT + ul) * Q) * 64 + (pl & 63)) * 4, 64 * 4);
      const int u = ub2 * GG_UT + ul;
      // the arg-max column of (pixel, u) relative to this thread's first column: equals i for at most one i
      const int cu = MODE != GRAD_COMPRESS ? pair_hi_bits(xu.v[1]) - vbase : -1;
      const float gu_max = MODE != GRAD_COMPRESS ? pair_lo(xu.v[1]) : 0.f;
#pragma unroll
      for (int i = 0; i < GG_VH; ++i) {
        float x = g_products<MODE, Q>(xu, xv[i]);
        if (MODE != GRAD_COMPRESS) {
          add_if_equal(x, cu, i, gu_max);
          add_if_equal(x, pair_hi_bits(xv[i].v[1]), u, pair_lo(xv[i].v[1]));
        }
        g[ul][i] = BF16 ? x : round_for_mma(x);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.xu_empty[so]);  // operands are in registers
    if (!mbar_wait(&sm.g_empty[s], ph ^ 1u, &sm.ctl, a.status, DEV_TIMEOUT_GENERATOR)) return;
    tc_fence_after();  // the MMAs that read this stage's TMEM columns have completed
    if constexpr (BF16) {
#pragma unroll
      for (int ul = 0; ul < GG_UT; ++ul) {
        uint32_t h[GG_VH / 2];
#pragma unroll
        for (int j = 0; j < GG_VH / 2; ++j)
          h[j] = BF16 == OP16_FP16 ? pack_fp16x2(g[ul][2 * j], g[ul][2 * j + 1]) : pack_bf16x2(g[ul][2 * j], g[ul][2 * j + 1]);
        tmem_st4(ta0 + s * GG_KJ + ul * (GG_VT / 2), h);
      }
    } else {
#pragma unroll
      for (int ul = 0; ul < GG_UT; ++ul) tmem_st8(ta0 + s * GG_KJ + ul * GG_VT, g[ul]);
    }
    tmem_st_wait();
    tc_fence_before();  // stores complete and ordered before the tensor core's reads, which follow the arrive
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.g_full[s]);
    if (++ub2 == sc.n_ub2) { ub2 = 0; ++vb; }
  }
}

// rows = an 8 x 16 block of image-2 pixels, K = 32 image-1 pixels.  A group of four warps fills one block; the two
// groups work on alternate blocks.  A warp covers 16 K columns (pixels) x 8 columns of the row tile: lane = (pixel
// pl % 16, column half vh), each thread 8 rows x 4 columns.  The two lanes of a pixel read the same (pixel, u) slots,
// which shared memory serves as one broadcast, so a warp's loads of those slots touch half as many bytes as with
// one pixel per lane.
template <int MODE, int Q, int BF16>
__device__ void generator_image2(GradSmem<Q, 1>& sm, const GradArgs& a, const GradSched& sc, int gw, int lane) {
  using Cfg = GradCfg<Q, 1>;
  constexpr int VQ = GG_ROW_VT / 4;  // columns per thread
  const int group = gw >> 2, sub = gw & 3;
  const int pl = (sub >> 1) * 16 + (lane & 15);          // K column of this thread
  const int vloc = ((sub & 1) * 2 + (lane >> 4)) * VQ;   // first of its four columns inside the row tile
  const int vbase = sc.v0 + vloc;
  // element (row, K column) of the swizzled block: row = ul*16 + vloc + i, so row % 8 == (vloc + i) % 8.
  // FP32: 128-byte rows, 16-byte chunk index ^ (row % 8).  BF16: 64-byte rows, chunk index ^ ((row % 8) / 2).
  uint32_t coff[VQ];
#pragma unroll
  for (int i = 0; i < VQ; ++i) {
    const uint32_t r = (uint32_t)(vloc + i), k = (uint32_t)pl;
    coff[i] = BF16 ? r * 64u + ((((k >> 3) ^ ((r & 7u) >> 1)) & 3u) << 4) + ((k & 7u) << 1)
                   : r * 128u + (((k >> 2) ^ (r & 7u)) << 4) + ((k & 3u) << 2);
  }
  // No more groups than ring stages: a group two fills ahead of a stage would see the parity of the fill before
  // last and pass its wait early.
  static_assert(GG_GEN_WARPS / 4 <= Cfg::NXU && GG_GEN_WARPS / 4 <= Cfg::NXV && GG_GEN_WARPS / 4 <= Cfg::NG,
                "more generator groups than ring stages");
  for (int t = group; t < sc.n_blocks; t += GG_GEN_WARPS / 4) {
    const uint32_t su = t % Cfg::NXU, phu = (t / Cfg::NXU) & 1u;
    const uint32_t sv = t % Cfg::NXV, phv = (t / Cfg::NXV) & 1u;
    const uint32_t s = t % Cfg::NG, ph = (t / Cfg::NG) & 1u;
    if (!mbar_wait(&sm.xv_full[sv], phv, &sm.ctl, a.status, DEV_TIMEOUT_GENERATOR)) return;
    Slots<Q> xv[VQ];  // block layouts [displacement][group][pixel][4]
    int du[VQ];       // arg-max row of (pixel, v) relative to the tile's first row: equals ul for at most one ul
#pragma unroll
    for (int i = 0; i < VQ; ++i) {
      xv[i].load_shared(sm.xv[sv] + ((vloc + i) * Q * GG_KJ + pl) * 4, GG_KJ * 4);
      du[i] = MODE != GRAD_COMPRESS ? pair_hi_bits(xv[i].v[1]) - sc.u0 : -1;
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.xv_empty[sv]);  // the (pixel, v) slots are in registers: the next load may start
    if (!mbar_wait(&sm.xu_full[su], phu, &sm.ctl, a.status, DEV_TIMEOUT_GENERATOR)) return;
    float g[GG_ROW_UT][VQ];
#pragma unroll
    for (int ul = 0; ul < GG_ROW_UT; ++ul) {
      Slots<Q> xu;
      xu.load_shared(sm.xu[su] + (ul * Q * GG_KJ + pl) * 4, GG_KJ * 4);
      const int cu = MODE != GRAD_COMPRESS ? pair_hi_bits(xu.v[1]) - vbase : -1;
      const float gu_max = MODE != GRAD_COMPRESS ? pair_lo(xu.v[1]) : 0.f;
#pragma unroll
      for (int i = 0; i < VQ; ++i) {
        float x = g_products<MODE, Q>(xu, xv[i]);
        if (MODE != GRAD_COMPRESS) {
          add_if_equal(x, cu, i, gu_max);
          add_if_equal(x, du[i], ul, pair_lo(xv[i].v[1]));
        }
        g[ul][i] = BF16 ? x : round_for_mma(x);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.xu_empty[su]);
    if (!mbar_wait(&sm.g_empty[s], ph ^ 1u, &sm.ctl, a.status, DEV_TIMEOUT_GENERATOR)) return;
    uint8_t* base = reinterpret_cast<uint8_t*>(sm.g[s]);
#pragma unroll
    for (int ul = 0; ul < GG_ROW_UT; ++ul)
#pragma unroll
      for (int i = 0; i < VQ; ++i) {
        if constexpr (BF16)
          *reinterpret_cast<uint16_t*>(base + ul * (GG_ROW_VT * 64) + coff[i]) = to_op16(g[ul][i], BF16);
        else
          *reinterpret_cast<float*>(base + ul * (GG_ROW_VT * 128) + coff[i]) = g[ul][i];
      }
    fence_proxy_async_smem();  // generic-proxy writes -> visible to the tensor core's async-proxy reads
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.g_full[s]);
  }
}

// B operand: one box of 32*nkb channel rows x 32 K-values of the other image's channel-major feature copy per block.
// Image 2 is stored in column blocks of 16 with an even number of rows, so block (vb, ub2) of the image-1-major form
// (2 rows x 16 columns) is 32 consecutive values.
template <int Q, int I2MAJOR, int BF16>
__device__ void feature_producer(GradSmem<Q, I2MAJOR>& sm, const GradArgs& a, const GradSched& sc,
                                 const CUtensorMap* tm_y) {
  using Cfg = GradCfg<Q, I2MAJOR>;
  int vb = 0, ub2 = 0;
  if (I2MAJOR == 0) { vb = sc.t0 / sc.n_ub2; ub2 = sc.t0 - vb * sc.n_ub2; }
  for (int t = 0; t < sc.n_blocks; ++t) {
    const uint32_t s = t % Cfg::NY, ph = (t / Cfg::NY) & 1u;
    if (!mbar_wait(&sm.y_empty[s], ph ^ 1u, &sm.ctl, a.status, DEV_TIMEOUT_PRODUCER)) return;
    mbar_expect_tx(&sm.y_full[s], sc.nkb * (BF16 ? GG_YBLOCK_BYTES / 2 : GG_YBLOCK_BYTES));
    if (I2MAJOR == 0) {
      tma_load_3d(sm.y[s], tm_y, &sm.y_full[s], (vb * sc.h2p + ub2 * GG_UT) * GG_VT, 0, sc.b);
      if (++ub2 == sc.n_ub2) { ub2 = 0; ++vb; }
    } else {
      tma_load_3d(sm.y[s], tm_y, &sm.y_full[s], (sc.t0 + t) * GG_KJ, 0, sc.b);
    }
  }
}

// Interleaved operand blocks.  Tensor maps are 4-D (4*n1p, Q, D, B); a box is (4*pixels, Q, displacements, 1)
// with at most 64 pixels (256 floats) per box, so the image-1-major form copies its 128 pixels as two boxes.
template <int Q, int I2MAJOR>
__device__ void operand_producer(GradSmem<Q, I2MAJOR>& sm, const GradArgs& a, const GradSched& sc,
                                 const CUtensorMap* tm_xu, const CUtensorMap* tm_xv) {
  using Cfg = GradCfg<Q, I2MAJOR>;
  using Smem = GradSmem<Q, I2MAJOR>;
  int ub2 = I2MAJOR == 0 ? sc.t0 % sc.n_ub2 : 0;
  for (int t = 0; t < sc.n_blocks; ++t) {
    const uint32_t su = t % Cfg::NXU, phu = (t / Cfg::NXU) & 1u;
    if (!mbar_wait(&sm.xu_empty[su], phu ^ 1u, &sm.ctl, a.status, DEV_TIMEOUT_PRODUCER)) return;
    mbar_expect_tx(&sm.xu_full[su], Smem::XU_FLOATS * 4);
    if (I2MAJOR == 0) {
      tma_load_4d(sm.xu[su], tm_xu, &sm.xu_full[su], sc.m0 * 4, 0, ub2 * GG_UT, sc.b);
      tma_load_4d(sm.xu[su] + Smem::XU_FLOATS / 2, tm_xu, &sm.xu_full[su], (sc.m0 + 64) * 4, 0, ub2 * GG_UT, sc.b);
      if (++ub2 == sc.n_ub2) ub2 = 0;
    } else {
      tma_load_4d(sm.xu[su], tm_xu, &sm.xu_full[su], (sc.t0 + t) * GG_KJ * 4, 0, sc.u0, sc.b);
      const uint32_t sv = t % Cfg::NXV, phv = (t / Cfg::NXV) & 1u;
      if (!mbar_wait(&sm.xv_empty[sv], phv ^ 1u, &sm.ctl, a.status, DEV_TIMEOUT_PRODUCER)) return;
      mbar_expect_tx(&sm.xv_full[sv], Smem::XV_FLOATS * 4);
      tma_load_4d(sm.xv[sv], tm_xv, &sm.xv_full[sv], (sc.t0 + t) * GG_KJ * 4, 0, sc.v0, sc.b);
    }
  }
}

template <int Q, int I2MAJOR, int BF16>
__device__ void grad_mma(GradSmem<Q, I2MAJOR>& sm, const GradArgs& a, const GradSched& sc) {
  using Cfg = GradCfg<Q, I2MAJOR>;
  // A: generated block, K-major: TMEM columns 256 + 32*stage .. (image-1-major) or shared memory (image-2-major).
  // B: feature block [channels][32 K-values], K-major, 8-row groups 1024 B apart.  K = 8 per instruction: 8 TMEM
  // columns / 32 bytes along a row of A, 32 bytes along a row of B.
  // BF16: 64-byte rows with the 64-byte swizzle (8-row groups 512 B apart), K = 16 per instruction: 8 TMEM columns
  // of two values / 32 bytes along a row.
  const uint32_t idesc = BF16 ? make_idesc_op16(BF16, TILE_M, sc.nkb * KBLK) : make_idesc_tf32(TILE_M, sc.nkb * KBLK, false, false);
  constexpr int NK = BF16 ? GG_KJ / 16 : GG_KJ / 8;  // instructions per block
  for (int t = 0; t < sc.n_blocks; ++t) {
    const uint32_t sy = t % Cfg::NY, phy = (t / Cfg::NY) & 1u;
    const uint32_t sg = t % Cfg::NG, phg = (t / Cfg::NG) & 1u;
    if (!mbar_wait(&sm.y_full[sy], phy, &sm.ctl, a.status, DEV_TIMEOUT_MMA)) return;
    if (!mbar_wait(&sm.g_full[sg], phg, &sm.ctl, a.status, DEV_TIMEOUT_MMA)) return;
    tc_fence_after();
    const uint64_t bdesc = BF16 ? make_smem_desc_sw128(smem_u32(sm.y[sy]), 16, 512, 4)
                                : make_smem_desc_sw128(smem_u32(sm.y[sy]), 16, 1024);
    if constexpr (I2MAJOR == 0) {
      const uint32_t a_tmem = sm.tmem_base + GG_ACC_COLS + sg * GG_KJ;
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        if constexpr (BF16) umma_bf16_ts(sm.tmem_base, a_tmem + k * 8, desc_advance(bdesc, k * 32), idesc, (t | k) != 0);
        else umma_tf32_ts(sm.tmem_base, a_tmem + k * 8, desc_advance(bdesc, k * 32), idesc, (t | k) != 0);
      }
    } else {
      const uint64_t adesc = BF16 ? make_smem_desc_sw128(smem_u32(sm.g[sg]), 16, 512, 4)
                                  : make_smem_desc_sw128(smem_u32(sm.g[sg]), 16, 1024);
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        if constexpr (BF16) umma_bf16(sm.tmem_base, desc_advance(adesc, k * 32), desc_advance(bdesc, k * 32), idesc, (t | k) != 0);
        else umma_tf32(sm.tmem_base, desc_advance(adesc, k * 32), desc_advance(bdesc, k * 32), idesc, (t | k) != 0);
      }
    }
    umma_commit(&sm.y_empty[sy]);  // both stages are reusable once these MMAs have read them
    umma_commit(&sm.g_empty[sg]);
  }
  umma_commit(&sm.acc_full);
}

// Where output row m of this CTA's tile lives (null: past the image); consecutive channels are cstride floats apart.
template <int I2MAJOR>
__device__ float* grad_row(const GradArgs& a, const GradSched& sc, int m, size_t& cstride) {
  const int C = a.d.C;
  cstride = 1;
  if (I2MAJOR == 0) {
    const int p = sc.m0 + m;
    if (p >= a.d.N1()) return nullptr;
    if (!a.out_cf) return a.out + ((size_t)sc.b * a.d.N1() + p) * C;
    cstride = (size_t)a.d.N1();
    return a.out + (size_t)sc.b * C * a.d.N1() + p;
  }
  const int u = sc.u0 + m / GG_ROW_VT, v = sc.v0 + m % GG_ROW_VT;
  if (u >= a.d.H2 || v >= a.d.W2) return nullptr;
  if (!a.out_cf) return a.out + (((size_t)sc.b * a.d.H2 + u) * a.d.W2 + v) * C;
  cstride = (size_t)a.d.N2();
  return a.out + (size_t)sc.b * C * a.d.N2() + (size_t)u * a.d.W2 + v;
}
// Scratch of pieces 1.. of the tail tiles: [tail][piece - 1][channel][128 rows] or [tail][piece - 1][128 rows][channel], as the
// output has it, so that the fold reads both in runs (channel-major pieces under a pixel-major output, 16-byte accesses 1 KB
// apart, made the launch for 1 x 55 x 128 against 27 x 64 take 58 us; 47 now, 48 with whole tiles).
__device__ __forceinline__ float* grad_part(const GradArgs& a, int tail, int piece) {
  return a.part + ((size_t)tail * (a.pieces - 1) + piece - 1) * a.d.C * TILE_M;
}

template <int Q, int I2MAJOR>
__device__ void grad_drain(GradSmem<Q, I2MAJOR>& sm, const GradArgs& a, const GradSched& sc, int warp, int gw, int lane) {
  const bool ok = mbar_wait(&sm.acc_full, 0, &sm.ctl, a.status, DEV_TIMEOUT_EPILOGUE);
  if (!__all_sync(0xffffffffu, ok)) return;
  tc_fence_after();
  const int C = a.d.C;
  const int q = warp & 3;  // TMEM lane quarter this warp may read
  const int m = q * 32 + lane;
  size_t cstride;
  float* dst = grad_row<I2MAJOR>(a, sc, m, cstride);
  const bool channel_major = a.out_cf != 0;
  bool accumulate = a.accumulate != 0;
  if (sc.piece > 0) {
    if (dst != nullptr) dst = grad_part(a, sc.tail, sc.piece) + (channel_major ? m : m * C);
    cstride = TILE_M;
    accumulate = false;
  }
  const uint32_t tbase = sm.tmem_base + (static_cast<uint32_t>(q * 32) << 16);
  const float osc = a.out_scale * (a.dev_scale != nullptr ? __ldg(a.dev_scale) : 1.f);
  // the two warps of a quarter take alternate 16-column chunks; C is a multiple of 4 and the
  // accumulator has 32*nkb >= C columns
  for (int c0 = (gw >> 2) * 16; c0 < C; c0 += 16 * (GG_GEN_WARPS / 4)) {
    float s[16];
    tmem_ld16(tbase + c0, s);
    if (dst == nullptr) continue;
    if (channel_major) {  // a warp's 32 rows are 32 neighbouring pixels of one channel plane
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (c0 + j < C) {
          float* d1 = dst + (size_t)(c0 + j) * cstride;
          float v1 = s[j] * osc;
          if (accumulate) v1 += *d1;
          *d1 = v1;
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        if (c0 + j < C) {
          float4* d4 = reinterpret_cast<float4*>(dst + c0 + j);
          float4 v4 = make_float4(s[j] * osc, s[j + 1] * osc, s[j + 2] * osc, s[j + 3] * osc);
          if (accumulate) {
            const float4 o = *d4;
            v4.x += o.x; v4.y += o.y; v4.z += o.z; v4.w += o.w;
          }
          *d4 = v4;
        }
      }
    }
  }
}

// Pieces 1.. of a finished tail tile added to the output, in piece order (all threads of the CTA that finished last).  One
// SM's loads move all of it, so a thread takes sixteen values at once and asks for several pieces' values before it uses any.
constexpr int FOLD_PIECES = 2;
__device__ __forceinline__ void fold_add(const float* const (&part)[4], const bool (&in)[4], size_t step, int pieces, float4 (&sum)[4]) {
  for (int s0 = 1; s0 < pieces; s0 += FOLD_PIECES) {
    float4 o[FOLD_PIECES][4];
#pragma unroll
    for (int q = 0; q < FOLD_PIECES; ++q)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        o[q][j] = s0 + q < pieces && in[j] ? __ldcg(reinterpret_cast<const float4*>(part[j] + (s0 + q - 1) * step))
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int q = 0; q < FOLD_PIECES; ++q) {
      if (s0 + q >= pieces) break;
#pragma unroll
      for (int j = 0; j < 4; ++j) add4(sum[j], o[q][j]);
    }
  }
}

template <int I2MAJOR>
__device__ void grad_fold_pieces(const GradArgs& a, const GradSched& sc) {
  const int C = a.d.C;   // a multiple of 4
  const float* const part0 = grad_part(a, sc.tail, 1);
  const size_t step = (size_t)C * TILE_M;
  float4 sum[4];
  const float* part[4];
  bool in[4];
  size_t cstride;
  if (a.out_cf) {   // channel-major: four rows, neighbours in the image (the ones that exist come first), of four channels
    constexpr int QUADS = TILE_M / 4;
    for (int i = threadIdx.x; i < C / 4 * QUADS; i += GG_THREADS) {
      const int m = i % QUADS * 4, c0 = i / QUADS * 4;
      float* const row = grad_row<I2MAJOR>(a, sc, m, cstride);
      if (row == nullptr) continue;
      const int cnt = min(4, I2MAJOR ? a.d.W2 - (sc.v0 + m % GG_ROW_VT) : a.d.N1() - (sc.m0 + m));
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        sum[j] = load4_cg(row + (c0 + j) * cstride, cnt);
        part[j] = part0 + (size_t)(c0 + j) * TILE_M + m;
        in[j] = true;
      }
      fold_add(part, in, step, a.pieces, sum);
#pragma unroll
      for (int j = 0; j < 4; ++j) store4(row + (c0 + j) * cstride, sum[j], cnt);
    }
  } else {          // pixel-major, as the pieces are: runs of four channels of a row, neighbouring runs to neighbouring threads
    const int runs = C / 4, n = runs * TILE_M;
    for (int i0 = threadIdx.x; i0 < n; i0 += 4 * GG_THREADS) {
      float* row[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int i = i0 + j * GG_THREADS, m = i / runs;
        row[j] = i < n ? grad_row<I2MAJOR>(a, sc, m, cstride) : nullptr;
        in[j] = row[j] != nullptr;
        if (in[j]) row[j] += (i - m * runs) * 4;
        sum[j] = load4_cg(row[j], in[j] ? 4 : 0);
        part[j] = part0 + (size_t)i * 4;
      }
      fold_add(part, in, step, a.pieces, sum);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (in[j]) store4(row[j], sum[j], 4);
    }
  }
}

template <int MODE, int Q, int I2MAJOR, int BF16>
__global__ void __launch_bounds__(GG_THREADS, 1)
grad_gemm_kernel(const __grid_constant__ CUtensorMap tm_y, const __grid_constant__ CUtensorMap tm_xu,
                 const __grid_constant__ CUtensorMap tm_xv, const GradArgs a) {
  if (*reinterpret_cast<volatile int*>(a.status) != 0) return;
  using Smem = GradSmem<Q, I2MAJOR>;
  using Cfg = GradCfg<Q, I2MAJOR>;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t pad = (1024u - (smem_u32(smem_raw) & 1023u)) & 1023u;
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw + pad);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  GradSched sc;
  sc.nkb = (a.d.C + KBLK - 1) / KBLK;
  int tile = blockIdx.x;
  sc.tail = -1;
  sc.piece = 0;
  if (tile >= a.whole_tiles) {  // pieces of the tail tiles follow the whole tiles
    const int r = tile - a.whole_tiles;
    sc.tail = r / a.pieces;
    sc.piece = r - sc.tail * a.pieces;
    tile = a.whole_tiles + sc.tail;
  }
  int all_blocks;
  if (I2MAJOR == 0) {
    const int tiles = (a.d.N1() + TILE_M - 1) / TILE_M;
    sc.b = tile / tiles;
    sc.m0 = (tile - sc.b * tiles) * TILE_M;
    sc.u0 = sc.v0 = 0;
    sc.n_ub2 = (a.d.H2 + GG_UT - 1) / GG_UT;
    sc.h2p = sc.n_ub2 * GG_UT;
    all_blocks = sc.n_ub2 * ((a.d.W2 + GG_VT - 1) / GG_VT);
  } else {
    const int n_ub = (a.d.H2 + GG_ROW_UT - 1) / GG_ROW_UT, n_vb = (a.d.W2 + GG_ROW_VT - 1) / GG_ROW_VT;
    sc.b = tile / (n_ub * n_vb);
    const int r = tile - sc.b * (n_ub * n_vb);
    sc.u0 = (r / n_vb) * GG_ROW_UT;
    sc.v0 = (r % n_vb) * GG_ROW_VT;
    sc.m0 = 0;
    sc.n_ub2 = 0;
    sc.h2p = 0;
    all_blocks = (a.d.N1() + GG_KJ - 1) / GG_KJ;
  }
  const int n_pieces = sc.tail >= 0 ? a.pieces : 1;
  {
    const int per = all_blocks / n_pieces, extra = all_blocks - per * n_pieces;  // the first `extra` pieces have one more
    sc.t0 = sc.piece * per + min(sc.piece, extra);
    sc.n_blocks = per + (sc.piece < extra ? 1 : 0);
  }

  if (threadIdx.x == 0) {
    constexpr int gen_arrivals = I2MAJOR ? 4 : GG_GEN_WARPS;  // one arrival per warp that writes / reads a block
    for (int s = 0; s < Cfg::NY; ++s) { mbar_init(&sm.y_full[s], 1); mbar_init(&sm.y_empty[s], 1); }
    for (int s = 0; s < Cfg::NG; ++s) { mbar_init(&sm.g_full[s], gen_arrivals); mbar_init(&sm.g_empty[s], 1); }
    for (int s = 0; s < Cfg::NXU; ++s) { mbar_init(&sm.xu_full[s], 1); mbar_init(&sm.xu_empty[s], gen_arrivals); }
    for (int s = 0; s < Cfg::NXV; ++s) { mbar_init(&sm.xv_full[s], 1); mbar_init(&sm.xv_empty[s], gen_arrivals); }
    mbar_init(&sm.acc_full, 1);
    wait_ctl_init(&sm.ctl, a.wait_limit_ns);
    fence_barrier_init();
    prefetch_tensormap(&tm_y);
    prefetch_tensormap(&tm_xu);
    if (I2MAJOR) prefetch_tensormap(&tm_xv);
  }
  if (warp == 1) {
    tmem_alloc(&sm.tmem_base, gg_tmem_cols<I2MAJOR>());
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  if (warp == 0) {
    if (lane == 0) feature_producer<Q, I2MAJOR, BF16>(sm, a, sc, &tm_y);
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) grad_mma<Q, I2MAJOR, BF16>(sm, a, sc);
    __syncwarp();
  } else if (warp == 2 + GG_GEN_WARPS) {
    if (lane == 0) operand_producer<Q, I2MAJOR>(sm, a, sc, &tm_xu, &tm_xv);
    __syncwarp();
  } else {
    const int gw = warp - 2;
    if constexpr (I2MAJOR == 0) generator_image1<MODE, Q, BF16>(sm, a, sc, warp, gw, lane);
    else generator_image2<MODE, Q, BF16>(sm, a, sc, gw, lane);
    grad_drain<Q, I2MAJOR>(sm, a, sc, warp, gw, lane);
  }

  tc_fence_before();
  __syncthreads();
  if (wait_ctl_aborted(&sm.ctl)) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(sm.tmem_base, gg_tmem_cols<I2MAJOR>());
  }
  if (n_pieces > 1 && !wait_ctl_aborted(&sm.ctl)) {  // uniform over the CTA after the barrier above
    __threadfence();  // this thread's results before the count ...
    __syncthreads();
    if (threadIdx.x == 0) sm.last_piece = atomicAdd(a.tail_count + sc.tail, 1) == n_pieces - 1;
    __syncthreads();
    if (sm.last_piece) {
      __threadfence();  // ... and the count before the other pieces' results
      grad_fold_pieces<I2MAJOR>(a, sc);
      if (threadIdx.x == 0) a.tail_count[sc.tail] = 0;  // as the next launch expects it
    }
  }
}

static int grad_tiles(const Dims& d, int image2_major) {
  return image2_major ? d.B * ((d.H2 + GG_ROW_UT - 1) / GG_ROW_UT) * ((d.W2 + GG_ROW_VT - 1) / GG_ROW_VT)
                      : d.B * ((d.N1() + TILE_M - 1) / TILE_M);
}

// How the tail tiles are cut, in units of one K block's time (32 values, about 0.6 us): a CTA costs about eight blocks of
// prologue and drain, a fold reads 128 KB per piece through one SM (about two blocks).  Pieces must save a quarter of the
// tail (see sweep_split) and at least twelve blocks to be used: with predicted savings of seven and eleven, launches of 23
// (2 x 33 x 70 against 16 x 35) and 33 us (3 x 55 x 128 against 13 x 32) got one or two us slower.  Whole and cut tiles
// measured, image-1-major and image-2-major form (us per launch, C = 256, FP16): 1 x 48 x 64: 60 and
// 37, 62 and 38; 1 x 55 x 128: 150 and 104, 148 and 107; 4 x 55 x 128: 300 and 246, 299 and 280; 8 x 47 x 156: 508 and
// 438, 541 and 476; 1 x 55 x 128 against 27 x 64: 48 and 40, 147 and 49; 1 x 135 x 240 against 67 x 120: 350 whole, 634 and
// 335.
TileSplit grad_split(const Dims& d, int image2_major) {
  const int tiles = grad_tiles(d, image2_major), rest = tiles % SM_COUNT;
  const int blocks = image2_major ? (d.N1() + GG_KJ - 1) / GG_KJ
                                  : ((d.H2 + GG_UT - 1) / GG_UT) * ((d.W2 + GG_VT - 1) / GG_VT);
  TileSplit r{tiles, tiles, 1, 0, 0};
  if (rest == 0) return r;
  double best = 0, whole = 0;
  for (int n = 1; n <= blocks && n <= MAX_PIECES; ++n) {
    const double waves = (rest * n + SM_COUNT - 1) / SM_COUNT;
    const double cost = waves * ((blocks + n - 1) / n + 8) + (n > 1 ? 2.0 * n * d.C / MAX_C + 2 : 0.0);
    if (n == 1) best = whole = cost;
    if (cost < best && cost < 0.75 * whole && cost < whole - 12) { best = cost; r.pieces = n; }
  }
  if (r.pieces > 1) {
    r.whole_tiles = tiles - rest;
    r.parts = r.pieces - 1;
    r.part_floats = (size_t)rest * (r.pieces - 1) * d.C * TILE_M;
  }
  return r;
}

template <int MODE, int Q, int I2MAJOR, int BF16>
static cudaError_t launch_one(const GradArgs& a, const CUtensorMap& tm_y, const CUtensorMap& tm_xu,
                              const CUtensorMap& tm_xv, cudaStream_t stream) {
  auto kern = grad_gemm_kernel<MODE, Q, I2MAJOR, BF16>;
  constexpr size_t smem_bytes = sizeof(GradSmem<Q, I2MAJOR>) + 1024;
  static_assert(smem_bytes <= 232448, "shared memory of one CTA");
  static DeviceOnce configured;  // the attribute is per device and stays set
  cudaError_t err = configured.run([&] {
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes);
  });
  if (err != cudaSuccess) return err;
  const int ctas = a.whole_tiles + (grad_tiles(a.d, I2MAJOR) - a.whole_tiles) * a.pieces;
  kern<<<dim3(ctas), GG_THREADS, smem_bytes, stream>>>(tm_y, tm_xu, tm_xv, a);
  return cudaGetLastError();
}

template <int MODE, int Q>
static cudaError_t launch_major(const GradArgs& a, const CUtensorMap& tm_y, const CUtensorMap& tm_xu,
                                const CUtensorMap& tm_xv, cudaStream_t stream) {
  if (a.op16 == OP16_FP16)
    return a.image2_major ? launch_one<MODE, Q, 1, OP16_FP16>(a, tm_y, tm_xu, tm_xv, stream)
                          : launch_one<MODE, Q, 0, OP16_FP16>(a, tm_y, tm_xu, tm_xv, stream);
  if (a.op16 == OP16_BF16)
    return a.image2_major ? launch_one<MODE, Q, 1, OP16_BF16>(a, tm_y, tm_xu, tm_xv, stream)
                          : launch_one<MODE, Q, 0, OP16_BF16>(a, tm_y, tm_xu, tm_xv, stream);
  return a.image2_major ? launch_one<MODE, Q, 1, 0>(a, tm_y, tm_xu, tm_xv, stream)
                        : launch_one<MODE, Q, 0, 0>(a, tm_y, tm_xu, tm_xv, stream);
}

cudaError_t launch_grad_gemm(const GradArgs& a, const CUtensorMap& tm_y, const CUtensorMap& tm_xu,
                             const CUtensorMap& tm_xv, cudaStream_t stream) {
  const int Q = a.R4 / 4;
  if (a.mode == GRAD_MAXAVG && Q == 1) return launch_major<GRAD_MAXAVG, 1>(a, tm_y, tm_xu, tm_xv, stream);
  if (a.mode == GRAD_COMPRESS && Q == 1) return launch_major<GRAD_COMPRESS, 1>(a, tm_y, tm_xu, tm_xv, stream);
  if (a.mode == GRAD_COMPRESS && Q == 2) return launch_major<GRAD_COMPRESS, 2>(a, tm_y, tm_xu, tm_xv, stream);
  if (a.mode == GRAD_FUSED && Q == 2) return launch_major<GRAD_FUSED, 2>(a, tm_y, tm_xu, tm_xv, stream);
  if (a.mode == GRAD_FUSED && Q == 3) return launch_major<GRAD_FUSED, 3>(a, tm_y, tm_xu, tm_xv, stream);
  return cudaErrorInvalidValue;
}

}  // namespace sfb
