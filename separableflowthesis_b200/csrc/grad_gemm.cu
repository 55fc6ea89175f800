// Gradient GEMMs of the backward ops:  gF1 = G * F2  and  gF2 = G^T * F1,  where
// G = dLoss/dS (N1 x N2 per sample) is made block by block: each, 128 rows x 64 (image-1-major) or 32 (image-2-major)
// K-values, is generated by CUDA cores as the A operand of tcgen05.mma, while TMA streams the matching block of the other image's
// features as the B operand.  The 128 x C output tile accumulates in TMEM over the whole K sweep and is
// written once, so the result is deterministic (no atomics), unlike the reference's atomicAdd scatter
// (MemorySaver_kernel_max_avg_argmax_backward.cu:305-310, MemorySaver_kernel_compression_backward.cu:477-488).
//
//   image2_major = 0 : rows = 128 consecutive image-1 pixels, K = image-2 pixels in blocks of
//                      4 rows x 16 columns (column blocks outermost), output gF1.  A generator thread owns one
//                      row = one TMEM lane, so the generated blocks go to tensor memory (tcgen05.st) next to the
//                      accumulator and the tensor core reads A from TMEM: no shared-memory stores, fences or
//                      operand reads for A.
//   image2_major = 1 : rows = an 8 x 16 block of image-2 pixels, K = 32 consecutive image-1 pixels,
//                      output gF2.  A generator thread owns one K column (pixel), so the blocks are written to
//                      shared memory, swizzled, K-major (TF32) or MN-major (16-bit).
//   With 16-bit operands G is generated once.  It costs the CUDA cores several times what its multiply-adds cost the tensor core, and the
//   image-2-major generator, which shares no operand across a block, is the dearer one:
//   storing          : image-1-major, but the blocks go to shared memory, where the tensor core reads them as they are and from where
//                      one bulk copy per block takes them to memory (16 KB per 128 x 64 values, beside some 1900 cycles of generating
//                      them).  Written to tensor memory as well, they took 418 instead of 404 us at 8 x 47 x 156.
//   stored           : rows = 256 image-2 pixels (four blocks of 4 x 16, two accumulators), K = 64 image-1 pixels.  A block is 128-byte
//                      rows of 64 image-2 pixels, MN-major, and is loaded as it lies in memory.  A plain GEMM: bound by the HBM
//                      that G comes from, next to the tensor core.  With tiles of 128 rows it would read 1.5 times as much of image 1
//                      through L2 per multiply-add as it gives the tensor core time for.
//   G generated twice and once (the pair, us): 8 x 135 x 240 with four channels 17.6 ms and 13.1, 8 x 47 x 156 with two 782 and
//   614 (BF16); the rule is grad_hands_over in c_abi.cu.
// B operand, all forms: K-major, like the operands of the correlation sweeps: TMA boxes of 32*ceil(C/32) channel
// rows x the K-values of a block from channel-major copies of the rounded features (image 1: (C, pixels); image 2: (C, column
// blocks of 16, rows, 16), so that the 4 rows x 16 columns of a K block are 64 consecutive values).  The MN-major
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
// type as it is generated (two values per 32-bit TMEM column) and the feature copies are 16-bit, so 32 K-values are two
// instructions of K = 16 instead of four of K = 8.
// Accumulation stays FP32.  With FP16 the operands carry power-of-two scales (kernels.h, SCALE_*) that the drain undoes.
//
// Tail tiles: like the correlation sweeps, the tiles past the last full wave of 148 CTAs are cut into `pieces` CTAs, each
// a range of the K sweep.  Piece 0 drains to the output, the others to scratch, and grad_fold_kernel adds them to the output
// in piece order: deterministic.
//
// The levels of a pyramid share a launch: the tiles of a level follow those of the one before, with maps and arguments of their own.
// gF1 is the sum over the levels, whose tiles beyond the first level's go to scratch like pieces.
//
// Warp roles: warp 0 feature (B operand) producer, warp 1 TMEM allocation + MMA issue, warps 2..9 generate G
// and, at the end, drain the accumulator (two warps per TMEM lane quarter, alternating 16-column chunks),
// warp 10 producer of the XU / XV blocks; storing: warp 11 copies the blocks to memory.
#include <climits>

#include <cuda_bf16.h>

#include "kernels.h"
#include "sm100_primitives.cuh"

namespace sfb {

constexpr int GG_GEN_WARPS = 8;
template <int FORM> __host__ __device__ constexpr int gg_threads() { return (3 + GG_GEN_WARPS + (FORM == GRAD_IMAGE1_STORING ? 1 : 0)) * 32; }
constexpr int GG_VH = GG_VT / (GG_GEN_WARPS / 4);          // columns of one image-1-major generator thread
constexpr uint32_t GG_YBLOCK_BYTES = KBLK * 128;           // 4 KB: 128 bytes of K-values of 32 channel rows
constexpr uint32_t GG_A_MBLOCK = GG_KJ * 128;              // image-2-major 16-bit A block: 64 rows x 32 K-values
constexpr int GG_KJ1 = GG_UT * GG_VT;                      // K extent of one image-1-major block
static_assert(GG_KJ1 == 64, "one 128-byte row of 16-bit values, two of FP32");
constexpr uint32_t GG_ACC_COLS = 256;                      // accumulator columns (the feature dimension)

// Ring depths.  Every kind of block has its own ring, sized by how long a stage stays in use:
//   NY   feature blocks (B operand, 32 KB at C = 256): freed when the MMAs of the block have completed
//   NG   generated blocks (A operand): image-1-major in TMEM columns 256 + 64*stage .. (32*stage with 16-bit values),
//        image-2-major in shared memory
//   NXU  (pixel, u) operand blocks: read row by row while the block is computed, freed when its values are stored
//   NXV  (pixel, v) operand blocks (image-2-major only; the image-1-major form keeps those slots in registers): read
//        into registers at the start of a block and freed at once, so that the next load has the whole computation
//        of the block to arrive
// The image-2-major form's two generator groups hold two operand blocks at a time and a TMA load takes about as long
// as one block's computation: with fewer than four (pixel, u) stages the generators wait for their operands.
// The storing form has a ring (NST) of blocks that the multiply-adds and the copy to memory both read, and gives it what it takes from the
// others (three (pixel, u) stages and four of these: 412 us instead of 404 at 8 x 47 x 156, 10.99 ms instead of 9.5 at 8 x 135 x 240); the
// stored form has one ring, a feature block and the four blocks of G that go with it to a stage.
template <int Q, int FORM> struct GradCfg;
template <> struct GradCfg<1, GRAD_IMAGE1> { static constexpr int NY = 6, NG = 4, NXU = 4, NXV = 1; };
template <> struct GradCfg<2, GRAD_IMAGE1> { static constexpr int NY = 5, NG = 4, NXU = 4, NXV = 1; };
template <> struct GradCfg<3, GRAD_IMAGE1> { static constexpr int NY = 4, NG = 4, NXU = 4, NXV = 1; };
template <> struct GradCfg<1, GRAD_IMAGE1_STORING> { static constexpr int NY = 4, NG = 1, NXU = 4, NXV = 1; };
template <> struct GradCfg<2, GRAD_IMAGE1_STORING> { static constexpr int NY = 3, NG = 1, NXU = 4, NXV = 1; };
template <> struct GradCfg<3, GRAD_IMAGE1_STORING> { static constexpr int NY = 3, NG = 1, NXU = 3, NXV = 1; };
template <int Q> struct GradCfg<Q, GRAD_IMAGE2> { static constexpr int NY = 3, NG = 2, NXU = 4, NXV = 2; };
template <int Q> struct GradCfg<Q, GRAD_IMAGE2_STORED> { static constexpr int NY = 3, NG = 3, NXU = 1, NXV = 1; };
constexpr uint32_t GG_SBLOCK_BYTES = GG_SJ * 128;          // stored form: 64 pixels of one block of G
template <int FORM> __host__ __device__ constexpr uint32_t gg_tmem_cols() { return FORM == GRAD_IMAGE2 || FORM == GRAD_IMAGE1_STORING ? 256u : 512u; }

template <int Q, int FORM>
struct GradSmem {
  using Cfg = GradCfg<Q, FORM>;
  static constexpr bool STORING = FORM == GRAD_IMAGE1_STORING, STORED = FORM == GRAD_IMAGE2_STORED;
  static constexpr bool AT = FORM == GRAD_IMAGE1;   // A blocks in tensor memory
  static constexpr bool I1 = !grad_is_image2(FORM);
  static constexpr int NST = STORING ? (Q == 1 ? 4 : 3) : 1;
  static_assert(GG_ACC_COLS + (AT ? Cfg::NG * GG_KJ1 : 0) <= gg_tmem_cols<FORM>(), "A stages exceed TMEM");
  // one operand block: [displacement][group of 4 slots][pixel][4]; image-1-major 4 x Q x 128, image-2-major 8 x Q x 32
  static constexpr int XU_FLOATS = STORED ? 4 : (I1 ? GG_UT * TILE_M : GG_ROW_UT * GG_KJ) * Q * 4;
  static constexpr int XV_FLOATS = FORM == GRAD_IMAGE2 ? GG_ROW_VT * GG_KJ * Q * 4 : 4;  // image-1-major keeps XV in registers
  float y[Cfg::NY][MAX_KB * GG_YBLOCK_BYTES / 4];  // feature stages [channel][K-values], K-major, swizzled
  // A blocks in shared memory, 128B swizzle: generated ones, K-major (TF32) or MN-major (16-bit); stored ones, MN-major
  float g[I1 ? 1 : Cfg::NG][I1 ? (STORING ? 256 : 32) : (STORED ? GG_SM * GG_SBLOCK_BYTES / 4 : TILE_M * GG_KJ)];
  uint8_t st[NST][STORING ? TILE_M * 128 : 128];   // the storing form's A blocks, K-major, 128B swizzle, as they go to memory
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
  uint64_t st_full[NST];
  uint64_t st_empty[NST];
  uint64_t acc_full;
  uint32_t tmem_base;
  WaitCtl ctl;
};

struct GradSched {
  int b, nkb;
  int t0, n_blocks;  // first block of the K sweep this CTA does, and how many
  int tail, piece;   // tail tile this CTA has a piece of (-1: a whole tile) and which piece
  int m0;            // image-1-major: first pixel of the row tile
  int u0, v0;        // image-2-major: origin of the 8 x 16 row tile
  int kb;            // over a stored G: the first of the tile's blocks of 4 x 16 (of 128 rows, once they are drained)
  int n_ub2;         // number of 4-row blocks along u
  int h2p;           // image-1-major: rows of the column-blocked channel-major copy of image 2 (H2 rounded up to a multiple of 4)
};

// The 4*Q slots of one (pixel, displacement) pair.
template <int Q>
struct Slots {
  float f[4 * Q];
  // shared memory block [group][pixel][4]
  __device__ __forceinline__ void load_shared(const float* p, int group_stride) {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const float4 t = *reinterpret_cast<const float4*>(p + q * group_stride);
      f[4 * q] = t.x; f[4 * q + 1] = t.y; f[4 * q + 2] = t.z; f[4 * q + 3] = t.w;
    }
  }
};

// The slots of N columns from column v0 on (p: of column 0, a column `column_stride` floats after the one before, group q
// `group_stride` floats after group q-1); zero past column W - 1.  As 16-byte loads that are all under way before the first value is
// used; with one load per value, and columns waiting for one another, a CTA took some 12,000 cycles for the slots of 16 columns (three groups, every 34
// blocks at 8 x 135 x 240; 6,100 with two groups, every 12 blocks at 8 x 47 x 156), and every CTA asks for them at about the same time:
// operand_producer brings them into L2 before that, which leaves 6,800 and 3,700.  The selection also moves every value to a register of
// its own: a 16-byte load puts the four slots of a column into neighbouring registers, and then a slot of all columns lies in the same
// register bank as their sums, which costs every other multiply-add a cycle.  Image-1-major GEMMs, 8 x 47 x 156 (BF16) 403 -> 383 us,
// 3 x 47 x 155 (TF32) 333 -> 320, 8 x 135 x 240 within 2 %.
template <int Q, int N>
__device__ __forceinline__ void load_columns(Slots<Q> (&xv)[N], const float* p, size_t column_stride, size_t group_stride, int v0, int W) {
  float4 raw[N][Q];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const float* column = p + (size_t)min(v0 + i, W - 1) * column_stride;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const float4* src = reinterpret_cast<const float4*>(column + q * group_stride);
      asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(raw[i][q].x), "=f"(raw[i][q].y), "=f"(raw[i][q].z), "=f"(raw[i][q].w) : "l"(src));
    }
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const bool ok = v0 + i < W;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      xv[i].f[4 * q] = ok ? raw[i][q].x : 0.f;
      xv[i].f[4 * q + 1] = ok ? raw[i][q].y : 0.f;
      xv[i].f[4 * q + 2] = ok ? raw[i][q].z : 0.f;
      xv[i].f[4 * q + 3] = ok ? raw[i][q].w : 0.f;
    }
  }
}

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

// The part of the G values of one (pixel, u) and N (pixel, v) that is a sum of products of the two pixels' slots.
// Max/avg group (slots 0..3 of XU: mean-gradient/W2, 1, max-gradient, argmax; of XV: 1, mean-gradient/H2,
// max-gradient, argmax): the two mean-gradients are added (the constants beside them, which a product would need, are not read).
// Columns past the image so hold the (pixel, u) mean-gradient, and meet the zero padding of the features.  Compression groups: every slot is a product.
// Scalar multiply-adds, a slot of the (pixel, u) at a time: it stays in the operand's register port while the N columns take
// theirs, and such a multiply-add issues every cycle.  A packed one (fma.rn.f32x2) with three different operands takes three.
template <int MODE, int Q, int N>
__device__ __forceinline__ void g_products(const Slots<Q>& xu, const Slots<Q> (&xv)[N], float (&x)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) x[i] = MODE == GRAD_COMPRESS ? xu.f[0] * xv[i].f[0] : xu.f[0] + xv[i].f[1];
#pragma unroll
  for (int k = MODE == GRAD_COMPRESS ? 1 : 4; k < 4 * Q; ++k)
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = fmaf(xu.f[k], xv[i].f[k], x[i]);
}

// Eight values as pairs of the 16-bit type.
template <int OP>
__device__ __forceinline__ void pack_row(const float (&g)[GG_VH], uint32_t (&h)[GG_VH / 2]) {
#pragma unroll
  for (int j = 0; j < GG_VH / 2; ++j) h[j] = OP == OP16_FP16 ? pack_fp16x2(g[2 * j], g[2 * j + 1]) : pack_bf16x2(g[2 * j], g[2 * j + 1]);
}

// rows = image-1 pixels.  Thread (pl, vh): row pl of the tile, columns vh*8 .. vh*8+7 of every 4 x 16 block.
// Bound: issue.  A value takes 8 multiply-adds, 3 additions, 2 compares and half a conversion at four channels; blocks of four
// rows instead of two halve what the barriers and waits of a block cost beside them (353 instead of 430 instructions per 16
// values with the scalar multiply-adds; 8 x 135 x 240: 8.4 -> 7.3 ms, 8 x 47 x 156: 436 -> 346 us).
// The (pixel, v) slots stay in registers across the inner sweep over u; the (pixel, u) slots of each block
// arrive in shared memory by TMA.  The finished values go to this thread's TMEM lane (A operand in tensor memory).
template <int MODE, int Q, int BF16, int FORM>
__device__ void generator_image1(GradSmem<Q, FORM>& sm, const GradArgs& a, const GradSched& sc, int warp, int gw, int lane) {
  using Cfg = GradCfg<Q, FORM>;
  constexpr bool STORING = FORM == GRAD_IMAGE1_STORING;
  const int W2 = a.d.W2;
  const size_t group_stride = (size_t)a.n1p * 4, row_stride = group_stride * Q;
  const int pl = (warp & 3) * 32 + lane, vh = gw >> 2;
  const float* xv_p = a.xv + (size_t)sc.b * W2 * row_stride + (size_t)(sc.m0 + pl) * 4;
  Slots<Q> xv[GG_VH];
  // TMEM address of this thread's lane quarter, first A column of stage 0, this thread's 8 columns
  // (BF16: two values per column, so the thread's 8 values of a row are 4 columns)
  const uint32_t ta0 = sm.tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + GG_ACC_COLS +
                       vh * (BF16 ? GG_VH / 2 : GG_VH);
  constexpr uint32_t A_COLS = BF16 ? GG_KJ1 / 2 : GG_KJ1;   // tensor-memory columns of one stage
  int vb = sc.t0 / sc.n_ub2, ub2 = sc.t0 - vb * sc.n_ub2;
  for (int t = 0; t < sc.n_blocks; ++t) {
    const uint32_t so = t % Cfg::NXU, pho = (t / Cfg::NXU) & 1u;
    const int vbase = vb * GG_VT + vh * GG_VH;
    if (ub2 == 0 || t == 0) load_columns(xv, xv_p, row_stride, group_stride, vbase, W2);
    if (!mbar_wait_warp(&sm.xu_full[so], pho, &sm.ctl, a.status, DEV_TIMEOUT_GENERATOR)) return;
    float g[GG_UT][GG_VH];
#pragma unroll
    for (int ul = 0; ul < GG_UT; ++ul) {
      Slots<Q> xu;  // block layout [pixel half][ul][group][64 pixels][4]; rows past the image are zero-filled by TMA
      xu.load_shared(sm.xu[so] + ((((pl >> 6) * GG_UT + ul) * Q) * 64 + (pl & 63)) * 4, 64 * 4);
      const int u = ub2 * GG_UT + ul;
      // the arg-max column of (pixel, u) relative to this thread's first column: equals i for at most one i
      const int cu = MODE != GRAD_COMPRESS ? __float_as_int(xu.f[3]) - vbase : -1;
      const float gu_max = MODE != GRAD_COMPRESS ? xu.f[2] : 0.f;
      float x[GG_VH];
      g_products<MODE, Q>(xu, xv, x);
#pragma unroll
      for (int i = 0; i < GG_VH; ++i) {
        if (MODE != GRAD_COMPRESS) {
          add_if_equal(x[i], cu, i, gu_max);
          add_if_equal(x[i], __float_as_int(xv[i].f[3]), u, xv[i].f[2]);
        }
        g[ul][i] = BF16 ? x[i] : round_for_mma(x[i]);
      }
    }
    if constexpr (STORING) {
      // the multiply-adds and the copy that read this stage have completed
      const uint32_t d = t % GradSmem<Q, FORM>::NST;
      if (!mbar_wait_warp(&sm.st_empty[d], ((t / GradSmem<Q, FORM>::NST) & 1u) ^ 1u, &sm.ctl, a.status, DEV_TIMEOUT_GENERATOR)) return;
#pragma unroll
      for (int ul = 0; ul < GG_UT; ++ul) {
        uint32_t h[GG_VH / 2];
        pack_row<BF16>(g[ul], h);
        // eight values = chunk 2 * ul + vh of the pixel's row; eight lanes' chunks lie in different banks
        *reinterpret_cast<uint4*>(sm.st[d] + pl * 128 + ((((uint32_t)ul * 2 + vh) ^ ((uint32_t)pl & 7u)) << 4)) = make_uint4(h[0], h[1], h[2], h[3]);
      }
      fence_proxy_async_smem();   // before the tensor core's and the bulk copy's reads; the operand stage has been read, too
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&sm.st_full[d]);
        mbar_arrive(&sm.xu_empty[so]);
      }
    } else {
      const uint32_t s = t % Cfg::NG, ph = (t / Cfg::NG) & 1u;
      if (!mbar_wait_warp(&sm.g_empty[s], ph ^ 1u, &sm.ctl, a.status, DEV_TIMEOUT_GENERATOR)) return;
      tc_fence_after();  // the MMAs that read this stage's TMEM columns have completed
#pragma unroll
      for (int ul = 0; ul < GG_UT; ++ul) {
        if constexpr (BF16) {
          uint32_t h[GG_VH / 2];
          pack_row<BF16>(g[ul], h);
          tmem_st4(ta0 + s * A_COLS + ul * (GG_VT / 2), h);
        } else {
          tmem_st8(ta0 + s * A_COLS + ul * GG_VT, g[ul]);
        }
      }
      tmem_st_wait();
      tc_fence_before();  // stores complete and ordered before the tensor core's reads, which follow the arrive
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.g_full[s]);
      hand_back_stage(&sm.xu_empty[so], lane);
    }
    if (++ub2 == sc.n_ub2) { ub2 = 0; ++vb; }
  }
}

// rows = an 8 x 16 block of image-2 pixels, K = 32 image-1 pixels.  A group of four warps fills one block; the two
// groups work on alternate blocks.  A warp covers 16 K columns (pixels) x 8 columns of the row tile: lane = (pixel
// pl % 16, column half vh), each thread 8 rows x 4 columns.  The two lanes of a pixel read the same (pixel, u) slots,
// which shared memory serves as one broadcast, so a warp's loads of those slots touch half as many bytes as with
// one pixel per lane.
template <int MODE, int Q, int BF16>
__device__ void generator_image2(GradSmem<Q, GRAD_IMAGE2>& sm, const GradArgs& a, const GradSched& sc, int gw, int lane) {
  using Cfg = GradCfg<Q, GRAD_IMAGE2>;
  constexpr int VQ = GG_ROW_VT / 4;  // columns per thread
  const int group = gw >> 2, sub = gw & 3;
  const int pl = (sub >> 1) * 16 + (lane & 15);          // K column of this thread
  const int vloc = ((sub & 1) * 2 + (lane >> 4)) * VQ;   // first of its four columns inside the row tile
  const int vbase = sc.v0 + vloc;
  // Element (row m, K column) of the block, m = ul*16 + vloc + i.  FP32: K-major, 128-byte rows m, 16-byte chunk index ^ (m % 8)
  // (m % 8 == (vloc + i) % 8).  16-bit: MN-major, two blocks of 64 m, 128-byte rows K, chunk index ^ (K % 8), so that the four
  // columns of a row are one 8-byte store; as 2-byte stores of a K-major block (a thread has one K column) the stores alone
  // took as many shared-memory cycles as the operands' loads (445 -> 403 us at 8 x 47 x 156; at 8 x 135 x 240, which runs against
  // the power cap, 8.7 ms with either).
  uint32_t coff[VQ];
#pragma unroll
  for (int i = 0; i < VQ; ++i) {
    const uint32_t r = (uint32_t)(vloc + i), k = (uint32_t)pl;
    coff[i] = r * 128u + (((k >> 2) ^ (r & 7u)) << 4) + ((k & 3u) << 2);
  }
  const uint32_t row16 = (uint32_t)pl * 128u + (((uint32_t)vloc & 7u) << 1), chunk16 = (uint32_t)vloc >> 3, flip16 = (uint32_t)pl & 7u;
  // No more groups than ring stages: a group two fills ahead of a stage would see the parity of the fill before
  // last and pass its wait early.
  static_assert(GG_GEN_WARPS / 4 <= Cfg::NXU && GG_GEN_WARPS / 4 <= Cfg::NXV && GG_GEN_WARPS / 4 <= Cfg::NG,
                "more generator groups than ring stages");
  for (int t = group; t < sc.n_blocks; t += GG_GEN_WARPS / 4) {
    const uint32_t su = t % Cfg::NXU, phu = (t / Cfg::NXU) & 1u;
    const uint32_t sv = t % Cfg::NXV, phv = (t / Cfg::NXV) & 1u;
    const uint32_t s = t % Cfg::NG, ph = (t / Cfg::NG) & 1u;
    if (!mbar_wait_warp(&sm.xv_full[sv], phv, &sm.ctl, a.status, DEV_TIMEOUT_GENERATOR)) return;
    Slots<Q> xv[VQ];  // block layouts [displacement][group][pixel][4]
    int du[VQ];       // arg-max row of (pixel, v) relative to the tile's first row: equals ul for at most one ul
#pragma unroll
    for (int i = 0; i < VQ; ++i) {
      xv[i].load_shared(sm.xv[sv] + ((vloc + i) * Q * GG_KJ + pl) * 4, GG_KJ * 4);
      du[i] = MODE != GRAD_COMPRESS ? __float_as_int(xv[i].f[3]) - sc.u0 : -1;
    }
    // The (pixel, v) slots are in registers: the next load may start.  At once, since it has only this block's computation to
    // arrive in: handed back after the next wait, the launch takes 437 instead of 426 us (8 x 47 x 156, BF16).
    hand_back_stage(&sm.xv_empty[sv], lane);
    if (!mbar_wait_warp(&sm.xu_full[su], phu, &sm.ctl, a.status, DEV_TIMEOUT_GENERATOR)) return;
    float g[GG_ROW_UT][VQ];
#pragma unroll
    for (int ul = 0; ul < GG_ROW_UT; ++ul) {
      Slots<Q> xu;
      xu.load_shared(sm.xu[su] + (ul * Q * GG_KJ + pl) * 4, GG_KJ * 4);
      const int cu = MODE != GRAD_COMPRESS ? __float_as_int(xu.f[3]) - vbase : -1;
      const float gu_max = MODE != GRAD_COMPRESS ? xu.f[2] : 0.f;
      float x[VQ];
      g_products<MODE, Q>(xu, xv, x);
#pragma unroll
      for (int i = 0; i < VQ; ++i) {
        if (MODE != GRAD_COMPRESS) {
          add_if_equal(x[i], cu, i, gu_max);
          add_if_equal(x[i], du[i], ul, xv[i].f[2]);
        }
        g[ul][i] = BF16 ? x[i] : round_for_mma(x[i]);
      }
    }
    if (!mbar_wait_warp(&sm.g_empty[s], ph ^ 1u, &sm.ctl, a.status, DEV_TIMEOUT_GENERATOR)) return;
    uint8_t* base = reinterpret_cast<uint8_t*>(sm.g[s]);
#pragma unroll
    for (int ul = 0; ul < GG_ROW_UT; ++ul) {
      if constexpr (BF16) {
        const uint2 h = BF16 == OP16_FP16 ? make_uint2(pack_fp16x2(g[ul][0], g[ul][1]), pack_fp16x2(g[ul][2], g[ul][3]))
                                          : make_uint2(pack_bf16x2(g[ul][0], g[ul][1]), pack_bf16x2(g[ul][2], g[ul][3]));
        *reinterpret_cast<uint2*>(base + (ul >> 2) * GG_A_MBLOCK + row16 + (((((uint32_t)ul & 3u) * 2 + chunk16) ^ flip16) << 4)) = h;
      } else {
#pragma unroll
        for (int i = 0; i < VQ; ++i) *reinterpret_cast<float*>(base + ul * (GG_ROW_VT * 128) + coff[i]) = g[ul][i];
      }
    }
    fence_proxy_async_smem();  // generic-proxy writes -> visible to the tensor core's async-proxy reads
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(&sm.g_full[s]);
      mbar_arrive(&sm.xu_empty[su]);   // behind the same fence
    }
  }
}

// B operand, a ring of 32 KB stages: one box of 32*nkb channel rows of the other image's channel-major feature copy each.
// Image-1-major: 128 bytes of a row, i.e. the 64 K-values of a block (16-bit) or half of them; image 2 is stored in column
// blocks of 16 with a multiple of four rows, so block (vb, ub2) (4 rows x 16 columns) is 64 consecutive values.
// Image-2-major: the 32 pixels of a block (64 bytes of 16-bit values).
// Over a stored G: the 64 pixels of a block and, with them, four blocks of G.
template <int FORM, int BF16> __device__ constexpr int y_stages_per_block() { return !grad_is_image2(FORM) && !BF16 ? 2 : 1; }
template <int Q, int FORM, int BF16>
__device__ void feature_producer(GradSmem<Q, FORM>& sm, const GradArgs& a, const GradSched& sc,
                                 const CUtensorMap* tm_y) {
  using Cfg = GradCfg<Q, FORM>;
  constexpr int PER = y_stages_per_block<FORM, BF16>();
  int vb = 0, ub2 = 0;
  if (!grad_is_image2(FORM)) { vb = sc.t0 / sc.n_ub2; ub2 = sc.t0 - vb * sc.n_ub2; }
  const int n_kb = sc.n_ub2 * ((a.d.W2 + GG_VT - 1) / GG_VT);
  uint32_t s = 0, ph = 0;
  for (int t = 0; t < sc.n_blocks; ++t) {
#pragma unroll
    for (int h = 0; h < PER; ++h) {
      if (!mbar_wait(&sm.y_empty[s], ph ^ 1u, &sm.ctl, a.status, DEV_TIMEOUT_PRODUCER)) return;
      if constexpr (FORM == GRAD_IMAGE2_STORED) {
        mbar_expect_tx(&sm.y_full[s], sc.nkb * GG_YBLOCK_BYTES + GG_SM * GG_SBLOCK_BYTES);
        tma_load_3d(sm.y[s], tm_y, &sm.y_full[s], (sc.t0 + t) * GG_SJ, 0, sc.b);
#pragma unroll
        for (int i = 0; i < GG_SM; ++i) {   // (rows past the last block are not stored: they may hold any)
          const size_t kb = (size_t)(sc.b - a.b0) * n_kb + min(sc.kb + i, n_kb - 1);
          bulk_load(reinterpret_cast<uint8_t*>(sm.g[s]) + i * GG_SBLOCK_BYTES, a.stored + (kb * a.n1p + (sc.t0 + t) * GG_SJ) * 128, GG_SBLOCK_BYTES,
                    &sm.y_full[s]);
        }
      } else {
        mbar_expect_tx(&sm.y_full[s], sc.nkb * (FORM == GRAD_IMAGE2 && BF16 ? GG_YBLOCK_BYTES / 2 : GG_YBLOCK_BYTES));
        if (!grad_is_image2(FORM))
          tma_load_3d(sm.y[s], tm_y, &sm.y_full[s], (vb * sc.h2p + ub2 * GG_UT) * GG_VT + h * KBLK, 0, sc.b);
        else
          tma_load_3d(sm.y[s], tm_y, &sm.y_full[s], (sc.t0 + t) * GG_KJ, 0, sc.b);
      }
      if (++s == Cfg::NY) { s = 0; ph ^= 1u; }
    }
    if (!grad_is_image2(FORM) && ++ub2 == sc.n_ub2) { ub2 = 0; ++vb; }
  }
}

// Interleaved operand blocks.  Tensor maps are 4-D (4*n1p, Q, D, B); a box is (4*pixels, Q, displacements, 1)
// with at most 64 pixels (256 floats) per box, so the image-1-major form copies its 128 pixels as two boxes.
template <int Q, int FORM>
__device__ void operand_producer(GradSmem<Q, FORM>& sm, const GradArgs& a, const GradSched& sc,
                                 const CUtensorMap* tm_xu, const CUtensorMap* tm_xv) {
  using Cfg = GradCfg<Q, FORM>;
  using Smem = GradSmem<Q, FORM>;
  constexpr int I2MAJOR = grad_is_image2(FORM) ? 1 : 0;
  int vb = 0, ub2 = 0;
  if (I2MAJOR == 0) { vb = sc.t0 / sc.n_ub2; ub2 = sc.t0 - vb * sc.n_ub2; }
  const size_t xv_group = (size_t)a.n1p * 4;
  const float* const xv_p = a.xv + (size_t)sc.b * a.d.W2 * Q * xv_group + (size_t)sc.m0 * 4;
  const int ahead = min(sc.n_ub2, GG_VT), quiet = sc.n_ub2 - ahead;   // the last blocks of a column of blocks, and the ones before
  for (int t = 0; t < sc.n_blocks; ++t) {
    const uint32_t su = t % Cfg::NXU, phu = (t / Cfg::NXU) & 1u;
    if (!mbar_wait(&sm.xu_empty[su], phu ^ 1u, &sm.ctl, a.status, DEV_TIMEOUT_PRODUCER)) return;
    mbar_expect_tx(&sm.xu_full[su], Smem::XU_FLOATS * 4);
    if (I2MAJOR == 0) {
      tma_load_4d(sm.xu[su], tm_xu, &sm.xu_full[su], sc.m0 * 4, 0, ub2 * GG_UT, sc.b);
      tma_load_4d(sm.xu[su] + Smem::XU_FLOATS / 2, tm_xu, &sm.xu_full[su], (sc.m0 + 64) * 4, 0, ub2 * GG_UT, sc.b);
      // The (pixel, v) slots of the next 16 columns, which all CTAs read at about the same time, are brought into L2 a few columns per block.
      if (ub2 >= quiet) {
        const int v0 = (vb + 1) * GG_VT + (ub2 - quiet) * GG_VT / ahead, v1 = min((vb + 1) * GG_VT + (ub2 - quiet + 1) * GG_VT / ahead, a.d.W2);
        for (int v = v0; v < v1; ++v)
#pragma unroll
          for (int q = 0; q < Q; ++q) bulk_prefetch_l2(xv_p + ((size_t)v * Q + q) * xv_group, TILE_M * 16);
      }
      if (++ub2 == sc.n_ub2) { ub2 = 0; ++vb; }
    } else {
      tma_load_4d(sm.xu[su], tm_xu, &sm.xu_full[su], (sc.t0 + t) * GG_KJ * 4, 0, sc.u0, sc.b);
      const uint32_t sv = t % Cfg::NXV, phv = (t / Cfg::NXV) & 1u;
      if (!mbar_wait(&sm.xv_empty[sv], phv ^ 1u, &sm.ctl, a.status, DEV_TIMEOUT_PRODUCER)) return;
      mbar_expect_tx(&sm.xv_full[sv], Smem::XV_FLOATS * 4);
      tma_load_4d(sm.xv[sv], tm_xv, &sm.xv_full[sv], (sc.t0 + t) * GG_KJ * 4, 0, sc.v0, sc.b);
    }
  }
}

template <int Q, int FORM, int BF16>
__device__ void grad_mma(GradSmem<Q, FORM>& sm, const GradArgs& a, const GradSched& sc) {
  using Cfg = GradCfg<Q, FORM>;
  // A: generated block, K-major: TMEM columns from 256 on (image-1-major; a 16-bit column holds two values) or shared memory
  // (image-2-major).  B: feature block [channels][K-values], K-major.  Rows of 128 bytes have the 128-byte swizzle (8-row
  // groups 1024 B apart); the 64-byte rows of 16-bit image-2-major blocks the 64-byte swizzle (512 B apart).  An instruction
  // takes K = 8 TF32 or 16 16-bit values: 8 TMEM columns / 32 bytes along a row of A, 32 bytes along a row of B.  The 16-bit
  // image-2-major A block is MN-major (generator_image2): 8-K groups 1024 B apart, two of them to an instruction.
  constexpr bool I2MAJOR = grad_is_image2(FORM);
  const uint32_t idesc = BF16 ? make_idesc_op16(BF16, TILE_M, sc.nkb * KBLK, I2MAJOR) : make_idesc_tf32(TILE_M, sc.nkb * KBLK, false, false);
  constexpr int PER = y_stages_per_block<FORM, BF16>();
  constexpr int NK = FORM == GRAD_IMAGE2 && BF16 ? 2 : 4;   // instructions per feature stage
  constexpr uint32_t A_COLS = BF16 ? GG_KJ1 / 2 : GG_KJ1;
  uint32_t sy = 0, phy = 0;
  constexpr bool STORING = FORM == GRAD_IMAGE1_STORING;
  constexpr int N_A = STORING ? GradSmem<Q, FORM>::NST : Cfg::NG;
  uint64_t *const a_full = STORING ? sm.st_full : sm.g_full, *const a_empty = STORING ? sm.st_empty : sm.g_empty;
  for (int t = 0; t < sc.n_blocks; ++t) {
    const uint32_t sg = t % N_A, phg = (t / N_A) & 1u;
#pragma unroll
    for (int h = 0; h < PER; ++h) {
      if (!mbar_wait(&sm.y_full[sy], phy, &sm.ctl, a.status, DEV_TIMEOUT_MMA)) return;
      if (FORM != GRAD_IMAGE2_STORED && h == 0 && !mbar_wait(&a_full[sg], phg, &sm.ctl, a.status, DEV_TIMEOUT_MMA)) return;
      tc_fence_after();
      const uint64_t bdesc = FORM == GRAD_IMAGE2 && BF16 ? make_smem_desc_sw128(smem_u32(sm.y[sy]), 16, 512, 4)
                                                         : make_smem_desc_sw128(smem_u32(sm.y[sy]), 16, 1024);
      if constexpr (STORING) {
        const uint64_t adesc = make_smem_desc_sw128(smem_u32(sm.st[sg]), 16, 1024);
#pragma unroll
        for (int k = 0; k < NK; ++k)
          umma_bf16(sm.tmem_base, desc_advance(adesc, k * 32), desc_advance(bdesc, k * 32), idesc, (t | k) != 0);
      } else if constexpr (!I2MAJOR) {
        const uint32_t a_tmem = sm.tmem_base + GG_ACC_COLS + sg * A_COLS + h * 32;
#pragma unroll
        for (int k = 0; k < NK; ++k) {
          if constexpr (BF16) umma_bf16_ts(sm.tmem_base, a_tmem + k * 8, desc_advance(bdesc, k * 32), idesc, (t | k) != 0);
          else umma_tf32_ts(sm.tmem_base, a_tmem + k * 8, desc_advance(bdesc, k * 32), idesc, (t | h | k) != 0);
        }
      } else if constexpr (FORM == GRAD_IMAGE2_STORED) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {   // 128 rows = two blocks each
          const uint64_t adesc = make_smem_desc_sw128(smem_u32(sm.g[sy]) + half * 2 * GG_SBLOCK_BYTES, GG_SBLOCK_BYTES, 1024);
#pragma unroll
          for (int k = 0; k < NK; ++k)
            umma_bf16(sm.tmem_base + half * GG_ACC_COLS, desc_advance(adesc, k * 2048), desc_advance(bdesc, k * 32), idesc, (t | k) != 0);
        }
      } else {
        const uint64_t adesc = make_smem_desc_sw128(smem_u32(sm.g[sg]), BF16 ? GG_A_MBLOCK : 16, 1024);
#pragma unroll
        for (int k = 0; k < NK; ++k) {
          if constexpr (BF16) umma_bf16(sm.tmem_base, desc_advance(adesc, k * 2048), desc_advance(bdesc, k * 32), idesc, (t | k) != 0);
          else umma_tf32(sm.tmem_base, desc_advance(adesc, k * 32), desc_advance(bdesc, k * 32), idesc, (t | k) != 0);
        }
      }
      umma_commit(&sm.y_empty[sy]);  // reusable once these MMAs have read it
      if (++sy == Cfg::NY) { sy = 0; phy ^= 1u; }
    }
    if constexpr (FORM != GRAD_IMAGE2_STORED) umma_commit(&a_empty[sg]);
  }
  umma_commit(&sm.acc_full);
}

// The storing form's blocks, from shared memory to their place in memory.  A thread of its own: as a duty of the MMA thread, which then
// waits for a copy to have read its block before it issues the next block's multiply-adds, the copies cost a third of the launch.
template <int Q>
__device__ void block_storer(GradSmem<Q, GRAD_IMAGE1_STORING>& sm, const GradArgs& a, const GradSched& sc) {
  constexpr uint32_t NST = GradSmem<Q, GRAD_IMAGE1_STORING>::NST;
  // the tile's pixels in the first of its blocks, and bytes from one block to the next
  const size_t step = (size_t)a.n1p * 128;
  uint8_t* dst = a.stored + ((size_t)(sc.b - a.b0) * sc.n_ub2 * ((a.d.W2 + GG_VT - 1) / GG_VT) + sc.t0) * step + (size_t)sc.m0 * 128;
  for (int t = 0; t < sc.n_blocks; ++t, dst += step) {
    const uint32_t s = t % NST, ph = (t / NST) & 1u;
    if (!mbar_wait(&sm.st_full[s], ph, &sm.ctl, a.status, DEV_TIMEOUT_PRODUCER)) return;
    bulk_store(dst, sm.st[s], TILE_M * 128);
    bulk_wait_read<1>();   // the block before this one has been read
    if (t > 0) mbar_arrive(&sm.st_empty[(t - 1) % NST]);
  }
  bulk_wait_all();
}


// Where output row m of this CTA's tile lives (null: past the image); consecutive channels are cstride floats apart.
template <int FORM>
__device__ float* grad_row(const GradArgs& a, const GradSched& sc, int m, size_t& cstride) {
  const int C = a.d.C;
  cstride = 1;
  if (!grad_is_image2(FORM)) {
    const int p = sc.m0 + m;
    if (p >= a.d.N1()) return nullptr;
    if (!a.out_cf) return a.out + ((size_t)sc.b * a.d.N1() + p) * C;
    cstride = (size_t)a.d.N1();
    return a.out + (size_t)sc.b * C * a.d.N1() + p;
  }
  int u = sc.u0 + m / GG_ROW_VT, v = sc.v0 + m % GG_ROW_VT;
  if constexpr (FORM == GRAD_IMAGE2_STORED) {
    const int kb = sc.kb + m / GG_KJ1, vb = kb / sc.n_ub2, r = m % GG_KJ1;
    u = (kb - vb * sc.n_ub2) * GG_UT + r / GG_VT;
    v = vb * GG_VT + r % GG_VT;   // a block past the last lies past the last column
  }
  if (u >= a.d.H2 || v >= a.d.W2) return nullptr;
  if (!a.out_cf) return a.out + (((size_t)sc.b * a.d.H2 + u) * a.d.W2 + v) * C;
  cstride = (size_t)a.d.N2();
  return a.out + (size_t)sc.b * C * a.d.N2() + (size_t)u * a.d.W2 + v;
}
// Scratch of the parts of a tile that do not go straight to the output (a cut tile's pieces 1.., the other levels' pieces):
// [tail][part][channel][128 rows] or [tail][part][128 rows][channel], as the
// output has it, so that the fold reads both in runs (with channel-major pieces under a pixel-major output, 16-byte accesses 1 KB
// apart, the form that folded in the tile's last CTA took 58 instead of 47 us for 1 x 55 x 128 against 27 x 64).
__device__ __forceinline__ float* grad_part(const GradArgs& a, int tail, int part) {
  return a.part + ((size_t)tail * a.parts + part) * a.d.C * TILE_M;
}

template <int Q, int FORM>
__device__ void grad_drain(GradSmem<Q, FORM>& sm, const GradArgs& a, GradSched sc, int warp, int gw, int lane) {
  constexpr bool STORED = FORM == GRAD_IMAGE2_STORED;
  const bool ok = mbar_wait(&sm.acc_full, 0, &sm.ctl, a.status, DEV_TIMEOUT_EPILOGUE);
  if (!__all_sync(0xffffffffu, ok)) return;
  tc_fence_after();
  const int C = a.d.C;
  const int q = warp & 3;  // TMEM lane quarter this warp may read
  const int m = q * 32 + lane;
  size_t cstride;
  const int half = STORED ? gw >> 2 : 0;   // of the 256 rows: an accumulator each, drained by four warps
  if (STORED) sc.kb += half * (TILE_M / GG_KJ1);
  float* dst = grad_row<FORM>(a, sc, m, cstride);
  const bool channel_major = a.out_cf != 0;
  bool accumulate = a.accumulate != 0;
  if (a.part0 + sc.piece >= 0) {
    if (dst != nullptr) dst = grad_part(a, STORED ? sc.tail * 2 + half : sc.tail, a.part0 + sc.piece) + (channel_major ? m : m * C);
    cstride = TILE_M;
    accumulate = false;
  }
  const uint32_t tbase = sm.tmem_base + (static_cast<uint32_t>(q * 32) << 16) + half * GG_ACC_COLS;
  const float osc = a.out_scale * (a.dev_scale != nullptr ? __ldg(a.dev_scale) : 1.f);
  // the two warps of a quarter take alternate 16-column chunks; C is a multiple of 4 and the
  // accumulator has 32*nkb >= C columns
  for (int c0 = STORED ? 0 : (gw >> 2) * 16; c0 < C; c0 += STORED ? 16 : 16 * (GG_GEN_WARPS / 4)) {
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

// Sample and origin of a row tile; returns the blocks of its K sweep.
template <int FORM>
__device__ __forceinline__ int grad_tile(const GradArgs& a, int tile, GradSched& sc) {
  sc.m0 = sc.u0 = sc.v0 = sc.kb = 0;
  sc.n_ub2 = (a.d.H2 + GG_UT - 1) / GG_UT;
  sc.h2p = sc.n_ub2 * GG_UT;
  if (!grad_is_image2(FORM)) {
    const int tiles = (a.d.N1() + TILE_M - 1) / TILE_M;
    sc.b = tile / tiles;
    sc.m0 = (tile - sc.b * tiles) * TILE_M;
    sc.b += a.b0;
    return sc.n_ub2 * ((a.d.W2 + GG_VT - 1) / GG_VT);
  }
  if constexpr (FORM == GRAD_IMAGE2_STORED) {
    const int tiles = (sc.n_ub2 * ((a.d.W2 + GG_VT - 1) / GG_VT) + GG_SM - 1) / GG_SM;
    sc.b = tile / tiles;
    sc.kb = (tile - sc.b * tiles) * GG_SM;
    sc.b += a.b0;
    return (a.d.N1() + GG_SJ - 1) / GG_SJ;
  }
  const int n_ub = (a.d.H2 + GG_ROW_UT - 1) / GG_ROW_UT, n_vb = (a.d.W2 + GG_ROW_VT - 1) / GG_ROW_VT;
  sc.b = tile / (n_ub * n_vb);
  const int r = tile - sc.b * (n_ub * n_vb);
  sc.u0 = (r / n_vb) * GG_ROW_UT;
  sc.v0 = (r % n_vb) * GG_ROW_VT;
  sc.b += a.b0;
  return (a.d.N1() + GG_KJ - 1) / GG_KJ;
}

// What a launch works on: one pair of images, or the levels of a pyramid over the same image 1.
template <int LEVELS>
struct GradLaunch {
  CUtensorMap y[LEVELS], xu[LEVELS], xv[LEVELS];
  GradArgs a[LEVELS];
  int first_block[LEVELS + 1], first_tail[LEVELS + 1];   // of the GEMM and of the fold; levels that do not exist have none
};
template <int LEVELS>
__device__ __forceinline__ int grad_level(const int (&first)[LEVELS + 1], int block) {
  int level = 0;
#pragma unroll
  for (int l = 1; l < LEVELS; ++l) level = block >= first[l] ? l : level;
  return level;
}

// The parts of a tile in scratch added to the output, in their order, four values to a thread.  A kernel of its own: added up by
// the CTA that finished a tile last, the 128 KB of every piece came through that one SM.
// grid (tails * grad_fold_blocks): the levels of a large batch have more tails than grid.y takes.
constexpr int GG_FOLD_THREADS = 256;
__host__ __device__ constexpr int grad_fold_blocks(int C) { return (C * (TILE_M / 4) + GG_FOLD_THREADS - 1) / GG_FOLD_THREADS; }
template <int FORM, int LEVELS>
__global__ void __launch_bounds__(GG_FOLD_THREADS) grad_fold_kernel(const __grid_constant__ GradLaunch<LEVELS> launch) {
  follow_previous_kernel();
  const int C = launch.a[0].d.C, per_tail = grad_fold_blocks(C), t = blockIdx.x / per_tail;   // C is a multiple of 4
  const int level = grad_level<LEVELS>(launch.first_tail, t);
  const GradArgs& a = launch.a[level];
  if (*reinterpret_cast<volatile int*>(a.status) != 0) return;
  const int tail = LEVELS == 1 ? t : t - launch.first_tail[level];
  const int i = (blockIdx.x - t * per_tail) * GG_FOLD_THREADS + threadIdx.x;   // four neighbours of the parts' layout (grad_part)
  if (i >= C * (TILE_M / 4)) return;
  GradSched sc;
  constexpr bool STORED = FORM == GRAD_IMAGE2_STORED;   // tails are halves of a tile
  grad_tile<FORM>(a, a.whole_tiles + (STORED ? tail / 2 : tail), sc);
  if (STORED) sc.kb += tail % 2 * (TILE_M / GG_KJ1);
  size_t cstride;
  float* dst;
  int cnt = 4;
  if (a.out_cf) {   // channel-major: four rows, neighbours in the image (the ones that exist come first), of one channel
    const int c = i / (TILE_M / 4), m = i % (TILE_M / 4) * 4;
    dst = grad_row<FORM>(a, sc, m, cstride);
    if (dst == nullptr) return;
    dst += c * cstride;
    const int v0 = STORED ? (sc.kb + m / GG_KJ1) / sc.n_ub2 * GG_VT : sc.v0;   // (16 columns a row in either)
    cnt = min(4, grad_is_image2(FORM) ? a.d.W2 - (v0 + m % GG_ROW_VT) : a.d.N1() - (sc.m0 + m));
  } else {          // pixel-major: four channels of a row
    const int m = i / (C / 4);
    dst = grad_row<FORM>(a, sc, m, cstride);
    if (dst == nullptr) return;
    dst += (i - m * (C / 4)) * 4;
  }
  const float* part = grad_part(a, tail, 0) + (size_t)i * 4;
  const size_t step = (size_t)C * TILE_M;
  float4 sum = load4_cg(dst, cnt);
#pragma unroll 4
  for (int k = 0; k < a.parts; ++k, part += step) add4(sum, *reinterpret_cast<const float4*>(part));
  store4(dst, sum, cnt);
}

template <int MODE, int Q, int FORM, int BF16, int LEVELS>
__global__ void __launch_bounds__(gg_threads<FORM>(), 1)
grad_gemm_kernel(const __grid_constant__ GradLaunch<LEVELS> launch, int* status) {
  if (!cta_has_work(status)) return;
  const int level = grad_level<LEVELS>(launch.first_block, blockIdx.x);
  const GradArgs& a = launch.a[level];
  const CUtensorMap *const tm_y = &launch.y[level], *const tm_xu = &launch.xu[level], *const tm_xv = &launch.xv[level];
  using Smem = GradSmem<Q, FORM>;
  using Cfg = GradCfg<Q, FORM>;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t pad = (1024u - (smem_u32(smem_raw) & 1023u)) & 1023u;
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw + pad);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  GradSched sc;
  sc.nkb = (a.d.C + KBLK - 1) / KBLK;
  int tile = LEVELS == 1 ? blockIdx.x : blockIdx.x - launch.first_block[level];
  sc.tail = -1;
  sc.piece = 0;
  if (tile >= a.whole_tiles) {  // pieces of the tail tiles follow the whole tiles
    const int r = tile - a.whole_tiles;
    sc.tail = r / a.pieces;
    sc.piece = r - sc.tail * a.pieces;
    tile = a.whole_tiles + sc.tail;
  }
  const int all_blocks = grad_tile<FORM>(a, tile, sc);
  const int n_pieces = sc.tail >= 0 ? a.pieces : 1;
  {
    const int per = all_blocks / n_pieces, extra = all_blocks - per * n_pieces;  // the first `extra` pieces have one more
    sc.t0 = sc.piece * per + min(sc.piece, extra);
    sc.n_blocks = per + (sc.piece < extra ? 1 : 0);
  }

  if (threadIdx.x == 0) {
    constexpr int gen_arrivals = FORM == GRAD_IMAGE2 ? 4 : GG_GEN_WARPS;  // one arrival per warp that writes / reads a block
    for (int s = 0; s < Cfg::NY; ++s) { mbar_init(&sm.y_full[s], 1); mbar_init(&sm.y_empty[s], 1); }
    for (int s = 0; s < Cfg::NG; ++s) { mbar_init(&sm.g_full[s], gen_arrivals); mbar_init(&sm.g_empty[s], 1); }
    for (int s = 0; s < Cfg::NXU; ++s) { mbar_init(&sm.xu_full[s], 1); mbar_init(&sm.xu_empty[s], gen_arrivals); }
    for (int s = 0; s < Cfg::NXV; ++s) { mbar_init(&sm.xv_full[s], 1); mbar_init(&sm.xv_empty[s], gen_arrivals); }
    for (int s = 0; s < Smem::NST; ++s) { mbar_init(&sm.st_full[s], gen_arrivals); mbar_init(&sm.st_empty[s], 2); }   // read by two
    mbar_init(&sm.acc_full, 1);
    wait_ctl_init(&sm.ctl, a.wait_limit_ns);
    fence_barrier_init();
    prefetch_tensormap(tm_y);
    if (FORM != GRAD_IMAGE2_STORED) prefetch_tensormap(tm_xu);
    if (FORM == GRAD_IMAGE2) prefetch_tensormap(tm_xv);
  }
  if (warp == 1) {
    tmem_alloc(&sm.tmem_base, gg_tmem_cols<FORM>());
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  if (warp == 0) {
    if (lane == 0) feature_producer<Q, FORM, BF16>(sm, a, sc, tm_y);
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) grad_mma<Q, FORM, BF16>(sm, a, sc);
    __syncwarp();
  } else if (warp == 2 + GG_GEN_WARPS) {
    if constexpr (FORM != GRAD_IMAGE2_STORED) {
      if (lane == 0) operand_producer<Q, FORM>(sm, a, sc, tm_xu, tm_xv);
    }
    __syncwarp();
  } else if (FORM == GRAD_IMAGE1_STORING && warp == 3 + GG_GEN_WARPS) {
    if constexpr (FORM == GRAD_IMAGE1_STORING) {
      if (lane == 0) block_storer<Q>(sm, a, sc);
    }
    __syncwarp();
  } else {
    const int gw = warp - 2;
    if constexpr (!grad_is_image2(FORM)) generator_image1<MODE, Q, BF16, FORM>(sm, a, sc, warp, gw, lane);
    else if constexpr (FORM == GRAD_IMAGE2) generator_image2<MODE, Q, BF16>(sm, a, sc, gw, lane);
    grad_drain<Q, FORM>(sm, a, sc, warp, gw, lane);
  }

  tc_fence_before();
  __syncthreads();
  if (wait_ctl_aborted(&sm.ctl)) {
    let_copies_land();
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(sm.tmem_base, gg_tmem_cols<FORM>());
  }
}

// Row tiles of a launch, and blocks of a tile's K sweep with the time of one in units of 32 generated K-values (a block of the stored
// form's 256 rows takes about as long).
static int grad_tiles(const Dims& d, int form) {
  switch (form) {
    case GRAD_IMAGE2: return d.B * ((d.H2 + GG_ROW_UT - 1) / GG_ROW_UT) * ((d.W2 + GG_ROW_VT - 1) / GG_ROW_VT);
    case GRAD_IMAGE2_STORED: return d.B * ((((d.H2 + GG_UT - 1) / GG_UT) * ((d.W2 + GG_VT - 1) / GG_VT) + GG_SM - 1) / GG_SM);
    default: return d.B * ((d.N1() + TILE_M - 1) / TILE_M);
  }
}
static int grad_blocks(const Dims& d, int form, int* unit) {
  *unit = grad_is_image2(form) ? 1 : GG_KJ1 / GG_KJ;
  switch (form) {
    case GRAD_IMAGE2: return (d.N1() + GG_KJ - 1) / GG_KJ;
    case GRAD_IMAGE2_STORED: return (d.N1() + GG_SJ - 1) / GG_SJ;
    default: return ((d.H2 + GG_UT - 1) / GG_UT) * ((d.W2 + GG_VT - 1) / GG_VT);
  }
}
static int grad_tail_rows(int form) { return form == GRAD_IMAGE2_STORED ? 2 * TILE_M : TILE_M; }

// How the tail tiles are cut, in units of the time of 32 K-values (about 0.6 us): a CTA costs about eight of prologue and drain,
// the fold is a launch of 4 to 11 us.  Pieces must save a quarter of the tail (see sweep_split) and at least twelve units to be
// used.  Whole and cut tiles measured, the fold with the latter, image-1-major and image-2-major form (us, C = 256, FP16):
// 1 x 48 x 64: 46 and 25, 50 and 24; 1 x 55 x 128: 122 and 79, 133 and 81; 4 x 55 x 128: 255 and 209, 268 and 249;
// 3 x 47 x 155: 266 and 177, 273 and 189; 8 x 47 x 156: 418 and 350, 472 and 407; 1 x 55 x 128 against 27 x 64: 40 and 33,
// 125 and 30; 1 x 135 x 240 against 67 x 120: 303 whole, 565 and 308; 2 x 33 x 70 against 16 x 35: 20 whole, 40 and 18.
TileSplit grad_split(const Dims& d, int form) {
  const int tiles = grad_tiles(d, form), rest = tiles % SM_COUNT;
  int unit;
  const int blocks = grad_blocks(d, form, &unit);
  TileSplit r{tiles, tiles, 1, 0, 0};
  if (rest == 0) return r;
  double best = 0, whole = 0;
  for (int n = 1; n <= blocks && n <= MAX_PIECES; ++n) {
    const double waves = (rest * n + SM_COUNT - 1) / SM_COUNT;
    const double cost = waves * ((blocks + n - 1) / n * unit + 8) + (n > 1 ? 6.0 : 0.0);
    if (n == 1) best = whole = cost;
    if (cost < best && cost < 0.75 * whole && cost < whole - 12) { best = cost; r.pieces = n; }
  }
  if (r.pieces > 1) {
    r.whole_tiles = tiles - rest;
    r.parts = r.pieces - 1;
    r.part_floats = (size_t)rest * (r.pieces - 1) * d.C * grad_tail_rows(form);
  }
  return r;
}

// How the tiles of a pyramid's levels are cut when they share a launch, in the same units: all tiles of a level alike, the first two
// levels of the image-1-major form into pieces of their own, all levels of the image-2-major form, whose K sweeps are equally
// long, into the same number.  The cut with the smallest makespan; nothing is cut where the tiles make more than a few waves.
void grad_split_levels(const Dims* d, int levels, int form, TileSplit* out) {
  const bool image2_major = grad_is_image2(form);
  int tiles[MAX_FUSED_LEVELS], blocks[MAX_FUSED_LEVELS], all = 0, unit = 1;
  for (int l = 0; l < levels; ++l) {
    tiles[l] = grad_tiles(d[l], form);
    blocks[l] = grad_blocks(d[l], form, &unit);
    all += tiles[l];
    out[l] = TileSplit{tiles[l], tiles[l], 1, 0, 0};
  }
  int cut[MAX_FUSED_LEVELS] = {1, 1, 1, 1};
  static_assert(MAX_FUSED_LEVELS == 4, "cut");
  if (all <= 4 * SM_COUNT) {
    const auto pieces = [&](int l, int n0, int n1) { return l == 0 || image2_major ? n0 : (l == 1 ? n1 : 1); };
    const LevelCut c = cheapest_cut(std::min(blocks[0], MAX_PIECES), image2_major || levels < 2 ? 1 : blocks[1], [&](auto& work, int n0, int n1) {
      for (int l = 0; l < levels; ++l) {
        const int n = pieces(l, n0, n1);
        work.add(tiles[l] * n, (double)blocks[l] / n * unit + 8);
      }
      return image2_major && n0 > 1 ? 6.0 : 0.0;
    });
    for (int l = 0; l < levels; ++l) cut[l] = pieces(l, c.n0, c.n1);
  }
  int parts = -1;   // the image-1-major form: of all levels, less the one that goes to the output
  for (int l = 0; l < levels; ++l) parts += cut[l];
  for (int l = 0; l < levels; ++l) {
    if (image2_major && cut[l] == 1) continue;
    out[l].whole_tiles = 0;
    out[l].pieces = cut[l];
    out[l].parts = image2_major ? cut[l] - 1 : parts;
    out[l].part_floats = image2_major || l == 0 ? (size_t)tiles[l] * out[l].parts * d[l].C * grad_tail_rows(form) : 0;   // image 1: one array for all
  }
}

template <int MODE, int Q, int FORM, int BF16, int LEVELS>
static cudaError_t launch_one(GradLaunch<LEVELS>& launch, int levels, cudaStream_t stream) {
  auto kern = grad_gemm_kernel<MODE, Q, FORM, BF16, LEVELS>;
  constexpr size_t smem_bytes = sizeof(GradSmem<Q, FORM>) + 1024;
  static_assert(smem_bytes <= 232448, "shared memory of one CTA");
  static DeviceOnce configured;  // the attribute is per device and stays set
  cudaError_t err = configured.run([&] {
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes);
  });
  if (err != cudaSuccess) return err;
  int blocks = 0, tails = 0;
  for (int l = 0; l < LEVELS; ++l) {
    launch.first_block[l] = blocks;
    launch.first_tail[l] = tails;
    if (l >= levels) continue;
    const GradArgs& a = launch.a[l];
    const int cut = grad_tiles(a.d, FORM) - a.whole_tiles;
    blocks += a.whole_tiles + cut * a.pieces;
    if (a.parts > 0 && a.part0 < 0) tails += cut * grad_tail_rows(FORM) / TILE_M;   // the level whose piece 0 is in the output adds up the parts
  }
  launch.first_block[LEVELS] = blocks;
  launch.first_tail[LEVELS] = tails;
  launch_next(kern, blocks, gg_threads<FORM>(), smem_bytes, stream, launch, launch.a[0].status);
  if (tails > 0) {
    if ((err = cudaGetLastError()) != cudaSuccess) return err;
    const long long fold_blocks = (long long)tails * grad_fold_blocks(launch.a[0].d.C);
    if (fold_blocks > INT_MAX) return cudaErrorInvalidConfiguration;
    launch_next(grad_fold_kernel<FORM, LEVELS>, (unsigned)fold_blocks, GG_FOLD_THREADS, 0, stream, launch);
  }
  return cudaGetLastError();
}

template <int MODE, int Q, int FORM, int BF16>
static cudaError_t launch_levels(const GradArgs* a, int levels, const GradMaps& maps, cudaStream_t stream) {
  auto fill = [&](auto& launch) {
    for (int l = 0; l < levels; ++l) {
      launch.y[l] = maps.y[l];
      launch.xu[l] = maps.xu[l];
      launch.xv[l] = maps.xv[l];
      launch.a[l] = a[l];
    }
  };
  if constexpr (MODE == GRAD_FUSED) {
    if (levels > 1) {
      GradLaunch<MAX_FUSED_LEVELS> launch{};
      fill(launch);
      return launch_one<MODE, Q, FORM, BF16>(launch, levels, stream);
    }
  }
  if (levels != 1) return cudaErrorInvalidValue;
  GradLaunch<1> launch{};
  fill(launch);
  return launch_one<MODE, Q, FORM, BF16>(launch, 1, stream);
}

template <int MODE, int Q, int BF16>
static cudaError_t launch_form(const GradArgs* a, int levels, const GradMaps& maps, cudaStream_t stream) {
  switch (a->form) {
    case GRAD_IMAGE1: return launch_levels<MODE, Q, GRAD_IMAGE1, BF16>(a, levels, maps, stream);
    case GRAD_IMAGE2: return launch_levels<MODE, Q, GRAD_IMAGE2, BF16>(a, levels, maps, stream);
    case GRAD_IMAGE1_STORING:
      if constexpr (BF16 != 0) return launch_levels<MODE, Q, GRAD_IMAGE1_STORING, BF16>(a, levels, maps, stream);
      break;
    case GRAD_IMAGE2_STORED:   // whatever G is a sum of
      if constexpr (BF16 != 0) return launch_levels<GRAD_FUSED, 1, GRAD_IMAGE2_STORED, BF16>(a, levels, maps, stream);
      break;
  }
  return cudaErrorInvalidValue;
}

template <int MODE, int Q>
static cudaError_t launch_major(const GradArgs* a, int levels, const GradMaps& maps, cudaStream_t stream) {
  if (a->op16 == OP16_FP16) return launch_form<MODE, Q, OP16_FP16>(a, levels, maps, stream);
  if (a->op16 == OP16_BF16) return launch_form<MODE, Q, OP16_BF16>(a, levels, maps, stream);
  return launch_form<MODE, Q, 0>(a, levels, maps, stream);
}

cudaError_t launch_grad_gemm(const GradArgs* a, int levels, const GradMaps& maps, cudaStream_t stream) {
  if (levels < 1 || levels > MAX_FUSED_LEVELS) return cudaErrorInvalidValue;
  const int Q = a->R4 / 4;
  if (a->mode == GRAD_MAXAVG && Q == 1) return launch_major<GRAD_MAXAVG, 1>(a, levels, maps, stream);
  if (a->mode == GRAD_COMPRESS && Q == 1) return launch_major<GRAD_COMPRESS, 1>(a, levels, maps, stream);
  if (a->mode == GRAD_COMPRESS && Q == 2) return launch_major<GRAD_COMPRESS, 2>(a, levels, maps, stream);
  if (a->mode == GRAD_FUSED && Q == 2) return launch_major<GRAD_FUSED, 2>(a, levels, maps, stream);
  if (a->mode == GRAD_FUSED && Q == 3) return launch_major<GRAD_FUSED, 3>(a, levels, maps, stream);
  return cudaErrorInvalidValue;
}

}  // namespace sfb
