// Correlation sweep: S = F1 * F2^T computed tile by tile on the tcgen05 tensor cores with the
// accumulator in TMEM, reduced in the epilogue so that S never reaches HBM.
//
// One CTA owns 128 consecutive image-1 pixels of one sample (the rows / TMEM lanes of every
// accumulator tile) and sweeps all image-2 pixels in tiles of 8 rows x 32 columns (256 accumulator columns) or, over narrow
// images, 16 x 16 (Tile), column-blocks outermost.  Warp roles:
//   warp 0      TMA producer: F1 tile once (stays resident), F2 tiles through a ring of stages
//   warp 1      allocates TMEM, issues tcgen05.mma (TF32 or 16-bit in, FP32 accumulate), 2 accumulators in flight
//   warps 2, 3  idle: they make up a warpgroup, the unit in which registers are handed to the epilogues
//   warps 4..11 two epilogue warpgroups; in each, one thread per image-1 pixel reads its accumulator lane with
//               tcgen05.ld.  Both groups consume every tile and split its work.
// Everything indexed by an image-1 pixel is read and written in the packed, pixel-fastest layout
// (kernels.h), so a warp's 32 lanes touch one 128-byte line per access.
// Epilogues
//   max/avg      : group g takes one half of a tile's rows.  Running column-direction max(+argmax) in
//                  registers across the inner row-block loop (the two groups' partial results are put together
//                  once per column block), row-direction max(+argmax) merged through the packed output
//                  once per tile.  The two mean channels come from extra tiles whose "image-2 pixels"
//                  are the row-mean and column-mean feature rows of F2 (mean_v S[u,v] = F1 . mean_v F2[u,v]).
//   compression  : OU[k,u] = sum_v S*w_u[k,v] (reduced per tile, accumulated with red.add), OV[k,v] = sum_u S*w_v[k,u]
//                  (register accumulators across the inner loop); two channels to a thread.
// Code that runs once per CTA or column block is fetched cold and is kept short (loops, running pointers, no branch per
// element): unrolled, the mean channels alone took as long as the tiles of a 55 x 128 launch.
// Tail tiles: a grid that is not a multiple of 148 tiles leaves SMs idle in its last wave (and a single 55 x 128 pair has
// 55 tiles in all), so the tiles past the last full wave are cut into `pieces` CTAs, each a range of column blocks.  Column
// results are complete within a piece; row results of pieces 1.. go to scratch, and sweep_fold_kernel folds them into piece
// 0's results in piece order, so the result does not depend on timing.
// Replaces the reference kernels MemorySaver_kernel_forward.cu:128-313, :328-533, :550-753.
#include <math_constants.h>

#include <type_traits>

#include "kernels.h"
#include "sm100_primitives.cuh"

namespace sfb {

constexpr int SW_NACC = 2;                      // 2 x 256 TMEM columns
constexpr int SW_TILE_N = SWEEP_UT * SWEEP_VT;  // 256 accumulator columns: tcgen05.mma issues at a fixed
                                                // rate per instruction, so the widest N does the most work
// Rows and columns of a tile.  Half as many row results leave a wide tile per cell, but image 2 is padded to whole tiles, and a
// narrow one (up to 16 columns, or one such block behind a few of 32) in half as many rows.  Both make 16 rows of 16 cells, the unit
// that the epilogues read from tensor memory; HALVES of them lie side by side.
template <bool NARROW>
struct Tile {
  static constexpr int UT = NARROW ? SWEEP_UT_NARROW : SWEEP_UT, VT = NARROW ? SWEEP_VT_NARROW : SWEEP_VT;
  static constexpr int HALVES = VT / 16;
  static constexpr int RW = UT / 2;   // rows of one epilogue warpgroup when the two split a tile's rows
};
static_assert(Tile<false>::UT * Tile<false>::VT == SW_TILE_N && Tile<true>::UT * Tile<true>::VT == SW_TILE_N, "accumulator columns");
static_assert(Tile<false>::HALVES == 2 && Tile<true>::HALVES == 1 && Tile<false>::RW == 4 && Tile<true>::RW == 8, "see the epilogues");
constexpr int SW_EPI_WARPS = 8;                 // two epilogue warpgroups
constexpr int SW_THREADS = 128 + SW_EPI_WARPS * 32;
// Registers a thread (setmaxnreg): the launch has 168 for each of its 384 threads; the four warps of the first warpgroup
// (TMA, MMA, two idle) need few, and the epilogues keep two channels' weights and sums of 32 columns (128 registers).
constexpr int SW_REGS_LAUNCH = 168, SW_REGS_ISSUE = 40, SW_REGS_EPI = 232;
constexpr bool register_split_fits(int regs_per_thread) {   // at launch
  return regs_per_thread * SW_THREADS >= 128 * SW_REGS_ISSUE + SW_EPI_WARPS * 32 * SW_REGS_EPI;
}
static_assert(register_split_fits(SW_REGS_LAUNCH) && !register_split_fits(SW_REGS_LAUNCH - 1), "more registers than the launch has");
constexpr int SW_NMERGE = 4;                    // ring of column-merge barriers (> SW_NACC tiles of run-ahead)
constexpr uint32_t SW_STAGE_BYTES = SW_TILE_N * KBLK * 4;
constexpr uint32_t SW_F1_BLOCK_BYTES = TILE_M * KBLK * 4;
constexpr uint32_t SW_TMEM_COLS = 512;
// Image-2 blocks (32 KB) in flight: what the resident image-1 tile leaves.  128 KB of it (TF32, 256 channels) leave three,
// 64 KB (16-bit) five, and four beside the 8 to 32 KB of row sums on their way to memory (compression, TMA rows).
constexpr int SW_MAX_STAGES = 6;
constexpr uint32_t SW_RING_BYTES = MAX_KB * SW_F1_BLOCK_BYTES + 3 * SW_STAGE_BYTES;   // image-1 tile and ring together
__host__ __device__ constexpr uint32_t sw_stages(int nkb, uint32_t row_bytes) {
  const uint32_t n = (SW_RING_BYTES - row_bytes - nkb * SW_F1_BLOCK_BYTES) / SW_STAGE_BYTES;
  return n < SW_MAX_STAGES ? n : SW_MAX_STAGES;
}
// Row sums on their way to memory (the compression with KC channels, TMA rows): behind the ring, two buffers per epilogue warp of the
// rows x channels of 32 pixels that it has of a tile.
__host__ __device__ constexpr int sw_channels(int KC) { return KC == 1 ? 1 : 2; }           // of a thread
__host__ __device__ constexpr int sw_rows(int KC) { return KC <= 2 ? SWEEP_UT / 2 : SWEEP_UT; }   // with one or two channels the two groups share a tile's rows
__host__ __device__ constexpr uint32_t sw_row_bytes(int KC) { return 2 * SW_EPI_WARPS * sw_rows(KC) * sw_channels(KC) * 32 * sizeof(float); }
static_assert(sw_stages((MAX_KB + 1) / 2, sw_row_bytes(4)) >= 3 && sw_row_bytes(4) >= sw_row_bytes(2), "image-2 blocks in flight beside the row sums");
static_assert(SW_NACC * SW_TILE_N <= 512, "accumulators exceed TMEM");
static_assert(SW_NMERGE > SW_NACC, "a warpgroup can run SW_NACC tiles ahead of the other");

struct SweepSmem {
  uint8_t ring[SW_RING_BYTES];            // image-1 tile, one 128B-swizzled block per 128 bytes of channels; then the ring of
                                          // image-2 tile blocks
  uint64_t f1_full;
  uint64_t full[SW_MAX_STAGES];
  uint64_t empty[SW_MAX_STAGES];
  uint64_t acc_full[SW_NACC];
  uint64_t acc_empty[SW_NACC];
  uint64_t merge[2][SW_NMERGE];           // to group g: the other group's part of g's columns is in memory
  uint32_t tmem_base;
  WaitCtl ctl;
  __device__ __forceinline__ uint8_t* f1(int kb) { return ring + kb * SW_F1_BLOCK_BYTES; }
  __device__ __forceinline__ uint8_t* f2(int nkb, uint32_t stage) { return ring + nkb * SW_F1_BLOCK_BYTES + stage * SW_STAGE_BYTES; }
};
constexpr size_t SW_SMEM_BYTES = sizeof(SweepSmem) + 1024;  // + slack to align the base to 1024 B

struct SweepSched {
  int b, m0, nkb, n_ub;
  int vb0, vb1;         // column blocks vb0 .. vb1 - 1 of this CTA
  int t_main, t_total;  // tiles of its column blocks; the same plus the tiles of the mean rows
  int tail, piece;      // tail tile this CTA has a piece of (-1: a whole tile) and which piece
  int part_vb0;         // first column block of piece 1
};

// Scratch of the tail tiles: [tail][part][slot][row u][128 pixels].  The parts of a tile are its pieces 1.. (row maxima) or
// the column blocks of its pieces 1.. (row sums, which are then folded block by block, in the order of a whole tile).
__device__ __forceinline__ float* sweep_part(const SweepArgs& a, int tail, int part, int slot) {
  return a.part + (((size_t)tail * a.parts + part) * a.part_slots + slot) * a.d.H2 * TILE_M;
}
// Column blocks of the pieces of a cut tile: the first n_vb % pieces have one more than the others.
__host__ __device__ __forceinline__ int piece_start(int n_vb, int pieces, int piece) {
  const int per = n_vb / pieces, extra = n_vb - per * pieces;
  return piece * per + (piece < extra ? piece : extra);
}

// What the CTA of a block index does.
template <int MODE, bool CUT, bool NARROW>
__device__ __forceinline__ SweepSched sweep_sched(const SweepArgs& a, int block) {
  const int tiles_per_sample = (a.d.N1() + TILE_M - 1) / TILE_M;
  SweepSched sc;
  int tile = block;
  sc.tail = -1;
  sc.piece = 0;
  if (CUT && tile >= a.whole_tiles) {  // pieces of the tail tiles follow the whole tiles
    const int r = tile - a.whole_tiles;
    sc.tail = r / a.pieces;
    sc.piece = r - sc.tail * a.pieces;
    tile = a.whole_tiles + sc.tail;
  }
  sc.b = tile / tiles_per_sample;
  sc.m0 = (tile - sc.b * tiles_per_sample) * TILE_M;
  sc.nkb = a.op16 ? (a.d.C + 2 * KBLK - 1) / (2 * KBLK) : (a.d.C + KBLK - 1) / KBLK;
  using T = Tile<NARROW>;
  sc.n_ub = (a.d.H2 + T::UT - 1) / T::UT;
  const int n_vb = (a.d.W2 + T::VT - 1) / T::VT;
  const int n_pieces = CUT && sc.tail >= 0 ? a.pieces : 1;
  sc.vb0 = piece_start(n_vb, n_pieces, sc.piece);
  sc.part_vb0 = piece_start(n_vb, n_pieces, 1);
  sc.vb1 = piece_start(n_vb, n_pieces, sc.piece + 1);
  sc.t_main = sc.n_ub * (sc.vb1 - sc.vb0);
  const bool has_aux = (MODE == SWEEP_MAXAVG || MODE == SWEEP_MAXARGAVG);
  const bool does_aux = has_aux && sc.piece == n_pieces - 1;       // the mean rows go to the last, smallest piece
  sc.t_total = sc.t_main + (does_aux ? (a.d.H2 + a.d.W2 + SW_TILE_N - 1) / SW_TILE_N : 0);
  return sc;
}

// ---------------------------------------------------------------------------------- producer
template <bool NARROW>
__device__ void sweep_producer(SweepSmem& sm, const SweepArgs& a, const SweepSched& sc, const CUtensorMap* tm_f1,
                               const CUtensorMap* tm_f2, const CUtensorMap* tm_aux, uint32_t row_bytes) {
  const int kel = a.op16 ? 2 * KBLK : KBLK;  // channels in one 128-byte row
  mbar_expect_tx(&sm.f1_full, sc.nkb * SW_F1_BLOCK_BYTES);
  for (int kb = 0; kb < sc.nkb; ++kb) tma_load_3d(sm.f1(kb), tm_f1, &sm.f1_full, kb * kel, sc.m0, sc.b);
  const uint32_t n_stages = sw_stages(sc.nkb, row_bytes);
  uint32_t s = 0, ph = 0;
  int vb = sc.vb0, ub = 0;
  for (int t = 0; t < sc.t_total; ++t) {
    const bool main_tile = t < sc.t_main;
    for (int kb = 0; kb < sc.nkb; ++kb) {
      if (!mbar_wait(&sm.empty[s], ph ^ 1u, &sm.ctl, a.status, DEV_TIMEOUT_PRODUCER)) return;
      if (a.drop_last_load && t == sc.t_total - 1 && kb == sc.nkb - 1) return;  // test hook: this block never arrives
      mbar_expect_tx(&sm.full[s], SW_STAGE_BYTES);
      if (main_tile)
        tma_load_4d(sm.f2(sc.nkb, s), tm_f2, &sm.full[s], kb * kel, vb * Tile<NARROW>::VT, ub * Tile<NARROW>::UT, sc.b);
      else
        tma_load_3d(sm.f2(sc.nkb, s), tm_aux, &sm.full[s], kb * kel, (t - sc.t_main) * SW_TILE_N, sc.b);
      if (++s == n_stages) { s = 0; ph ^= 1u; }
    }
    if (++ub == sc.n_ub) { ub = 0; ++vb; }
  }
}

// ---------------------------------------------------------------------------------- MMA issuer
__device__ void sweep_mma(SweepSmem& sm, const SweepArgs& a, const SweepSched& sc, uint32_t row_bytes) {
  constexpr uint32_t idesc_tf32 = make_idesc_tf32(TILE_M, SW_TILE_N, false, false);
  const uint32_t idesc_16 = make_idesc_op16(a.op16, TILE_M, SW_TILE_N);  // BF16 or FP16 operands
  const bool op16 = a.op16 != 0;
  if (!mbar_wait(&sm.f1_full, 0, &sm.ctl, a.status, DEV_TIMEOUT_MMA)) return;
  tc_fence_after();
  const uint32_t n_stages = sw_stages(sc.nkb, row_bytes);
  uint32_t s = 0, ph = 0;
  for (int t = 0; t < sc.t_total; ++t) {
    const uint32_t acc = t % SW_NACC, aph = (t / SW_NACC) & 1u;
    if (!mbar_wait(&sm.acc_empty[acc], aph ^ 1u, &sm.ctl, a.status, DEV_TIMEOUT_MMA)) return;
    tc_fence_after();
    const uint32_t d_tmem = sm.tmem_base + acc * SW_TILE_N;
    for (int kb = 0; kb < sc.nkb; ++kb) {
      if (!mbar_wait(&sm.full[s], ph, &sm.ctl, a.status, DEV_TIMEOUT_MMA)) return;
      tc_fence_after();
      const uint64_t adesc = make_smem_desc_sw128(smem_u32(sm.f1(kb)), 16, 1024);
      const uint64_t bdesc = make_smem_desc_sw128(smem_u32(sm.f2(sc.nkb, s)), 16, 1024);
      if (op16) {
#pragma unroll
        for (int k = 0; k < 4; ++k)  // one instruction consumes K = 16 16-bit values = 32 bytes of each row
          umma_bf16(d_tmem, desc_advance(adesc, k * 32), desc_advance(bdesc, k * 32), idesc_16, (kb | k) != 0);
      } else {
#pragma unroll
        for (int k = 0; k < KBLK / 8; ++k)  // one instruction consumes K = 8 TF32 values = 32 bytes of each row
          umma_tf32(d_tmem, desc_advance(adesc, k * 32), desc_advance(bdesc, k * 32), idesc_tf32, (kb | k) != 0);
      }
      umma_commit(&sm.empty[s]);  // stage reusable once these MMAs have read it
      if (++s == n_stages) { s = 0; ph ^= 1u; }
    }
    umma_commit(&sm.acc_full[acc]);
  }
}

// ---------------------------------------------------------------------------------- epilogues
struct EpiCtx {
  int wg;           // epilogue warpgroup 0 / 1
  int lane;
  int p;            // pixel index inside the sample: m0 + 32*quarter + lane
  bool valid;       // p < n_valid: lanes past the end compute but never touch memory
  uint32_t tbase;   // TMEM address of this warp's lane quarter, column 0
  float osc;        // every stored value is multiplied by this (1, or the inverse of the FP16 operands' scaling: a
                    // power of two, so the order of values and exact ties are unchanged)
};

// Waits for accumulator `t`; the result is warp-uniform so that the warp-collective tcgen05.ld that
// follows is executed by all lanes or by none.
__device__ __forceinline__ bool epi_wait(SweepSmem& sm, const SweepArgs& a, int t) {
  const uint32_t acc = t % SW_NACC, aph = (t / SW_NACC) & 1u;
  const bool ok = mbar_wait(&sm.acc_full[acc], aph, &sm.ctl, a.status, DEV_TIMEOUT_EPILOGUE);
  const bool all_ok = __all_sync(0xffffffffu, ok);
  if (all_ok) tc_fence_after();
  return all_ok;
}
__device__ __forceinline__ void epi_release(SweepSmem& sm, int t, int lane) {
  tc_fence_before();
  __syncwarp();
  if (lane == 0) mbar_arrive(&sm.acc_empty[t % SW_NACC]);
}

// Column results of a block that the two groups hold parts of: each stores its part of the other's 16 columns to the output
// and arrives, waits for the other, reads its own columns' other part back (all of it before it stores anything: a load that
// follows a store waits for it, and one memory latency per column took longer than the block's tiles) and stores the two
// together.
__device__ __forceinline__ void merge_publish(SweepSmem& sm, const SweepSched& sc, int vb, const EpiCtx& e) {
  __threadfence_block();
  __syncwarp();
  if (e.lane == 0) mbar_arrive(&sm.merge[1 - e.wg][(vb - sc.vb0) % SW_NMERGE]);
}
__device__ __forceinline__ bool merge_wait(SweepSmem& sm, const SweepArgs& a, const SweepSched& sc, int vb, const EpiCtx& e) {
  const bool ok = mbar_wait(&sm.merge[e.wg][(vb - sc.vb0) % SW_NMERGE], ((vb - sc.vb0) / SW_NMERGE) & 1u, &sm.ctl, a.status,
                            DEV_TIMEOUT_EPILOGUE);
  return __all_sync(0xffffffffu, ok);
}

// Largest of 16 values; NaNs are passed over.
__device__ __forceinline__ float max16(const uint32_t (&r)[16]) {
  float m = fmax3(__uint_as_float(r[0]), __uint_as_float(r[1]), __uint_as_float(r[2]));
#pragma unroll
  for (int i = 3; i + 1 < 16; i += 2) m = fmax3(m, __uint_as_float(r[i]), __uint_as_float(r[i + 1]));
  return fmaxf(m, __uint_as_float(r[15]));
}
// Which of the values equal m, as a sum of powers of two: value j of the first n - 1 counts 2^(n-1-j).  The lowest j is then the
// leading bit, and the last value is the one when no bit is set.  One comparison on the ALU pipe and one multiply-add on the
// FMA pipe per value, where carrying an index through a tournament takes a comparison and two selects, all on the ALU pipe
// (half rate), which set the pace: 3 ALU operations per cell and direction.
__device__ __forceinline__ float equal_bits16(const uint32_t (&r)[16], float m) {
  float bits = 0.f;
#pragma unroll
  for (int j = 0; j < 15; ++j) bits = fmaf(is_equal(__uint_as_float(r[j]), m), static_cast<float>(1 << (15 - j)), bits);
  return bits;
}
__device__ __forceinline__ int first_of16(float bits) {   // 2^15 .. 2^1: 0 .. 14; zero: 15
  return min(142 - static_cast<int>(__float_as_uint(bits) >> 23), 15);
}

// Max / arg-max / mean.  Bound: the tensor core (some 2400 cycles per tile) without arg-max, and with it the ALU pipe (half
// rate: about 480 of its instructions per warp and tile, 1900 cycles) beside what two warps per scheduler cannot hide.
// 135 x 240, one pair, without / with arg-max: 590 -> 465 / 868 -> 630 us; 55 x 128: 81 -> 38 / 81 -> 50.
// Group g takes half of a tile's rows, as two units of 4 rows x 16 columns (side by side, or in a narrow tile one above the
// other), the second one being loaded while the first is worked on.  State across the row blocks: the running maximum of each column and (ARG) where it
// lies, as the float 8 * (row / 4) + (bits of the row inside its four rows), which is exact up to 2^24.
// NaN entries are passed over; a row that holds nothing else has the maximum NaN at index 0, such a column -inf at index 0.
template <bool ARG, bool CUT, bool NARROW>
__device__ void epilogue_maxavg(SweepSmem& sm, const SweepArgs& a, const SweepSched& sc, const EpiCtx& e) {
  using T = Tile<NARROW>;
  constexpr int RW = T::RW, VT = T::VT;
  const int H2 = a.d.H2, W2 = a.d.W2;
  // per-thread views: value of (displacement d, slot) at ptr[d*sd + slot*ss]
  float* pu = a.pu.base + sc.b * a.pu.sb + e.p;
  float* pv = a.pv.base + sc.b * a.pv.sb + e.p;
  float* pum = pu + a.pu.ss;   // the mean channel: written by one piece, straight to its place
  float* pua = ARG ? a.pu_arg.base + sc.b * a.pu_arg.sb + e.p : nullptr;
  float* pva = ARG ? a.pv_arg.base + sc.b * a.pv_arg.sb + e.p : nullptr;
  uint32_t usd = a.pu.sd, uasd = a.pu_arg.sd;
  const uint32_t umsd = a.pu.sd, vsd = a.pv.sd, vss = a.pv.ss, vasd = a.pv_arg.sd;
  if (CUT && sc.piece > 0) {   // row maxima of a later piece: scratch slots 0 (value) and 1 (arg-max)
    pu = sweep_part(a, sc.tail, sc.piece - 1, 0) + (e.p - sc.m0);
    if (ARG) pua = sweep_part(a, sc.tail, sc.piece - 1, 1) + (e.p - sc.m0);
    usd = uasd = TILE_M;
  }
  const bool valid = e.valid;
  const bool all_valid = sc.m0 + TILE_M <= a.n_valid;

  float rnext[RW];
  auto load_rows = [&](int ub, bool none) {
    const int u0 = ub * T::UT + e.wg * RW;
#pragma unroll
    for (int r = 0; r < RW; ++r) rnext[r] = valid && !none && u0 + r < H2 ? pu[(u0 + r) * usd] : -CUDART_INF_F;
  };
#pragma unroll
  for (int r = 0; r < RW; ++r) rnext[r] = -CUDART_INF_F;
  int main_tiles = 0;
  for (int vb = sc.vb0; vb < sc.vb1; ++vb) {
   const int v0 = vb * VT, nv = min(VT, W2 - v0);
   const bool first = vb == sc.vb0;
   float cm[VT], ca[VT];
#pragma unroll
   for (int j = 0; j < VT; ++j) { cm[j] = -CUDART_INF_F; ca[j] = 4.f; }
   for (int ub = 0; ub < sc.n_ub; ++ub, ++main_tiles) {
    const int t = main_tiles;
    const int ubase = ub * T::UT + e.wg * RW;
    const int nu = min(RW, H2 - ubase);  // may be <= 0
    // row-direction state of earlier column blocks: asked for one tile ahead, unless that tile has the same rows
    if (sc.n_ub == 1) load_rows(ub, first);
    float rold[RW];
#pragma unroll
    for (int r = 0; r < RW; ++r) rold[r] = rnext[r];
    if (sc.n_ub > 1) load_rows(ub + 1 < sc.n_ub ? ub + 1 : 0, first && ub + 1 < sc.n_ub);
    const float qbase = static_cast<float>(ubase / 4 * 8);

    if (!epi_wait(sm, a, t)) return;
    const uint32_t tacc = e.tbase + (t % SW_NACC) * SW_TILE_N + e.wg * (RW * VT);
    // two units of 4 rows x 16 columns; half of the second one is on its way while the first is worked on (all of it would
    // cost the arg-max form registers that it does not have)
    uint32_t s[2][4][16];
    auto load = [&](int h, int r) { tmem_ld16_issue(tacc + (NARROW ? (h * 4 + r) * VT : r * VT + h * 16), s[h][r]); };
    float rmax[4], rbits[4];
    auto unit = [&](auto half, auto whole) {   // whole: every lane, row and column of this thread's part of the tile exists
      constexpr int h = decltype(half)::value;
      constexpr bool WHOLE = decltype(whole)::value;
      constexpr int ROW = NARROW ? h * 4 : 0, COL = NARROW ? 0 : h * 16;   // of the unit in this thread's part
      uint32_t(&x)[4][16] = s[h];
      if (!WHOLE) {  // cells outside the image are passed over
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (ROW + r >= nu || COL + j >= nv) x[r][j] = 0x7FFFFFFFu;
      }
      // rows
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float mh = max16(x[r]), bits = ARG ? equal_bits16(x[r], mh) : 0.f;
        if (!NARROW && h == 0) {
          rmax[r] = mh;
          rbits[r] = bits;
          continue;
        }
        const float m = NARROW ? mh : fmaxf(rmax[r], mh);
        int arg = 0;
        if (ARG) {
          const bool left = !NARROW && rmax[r] == m;
          arg = first_of16(left ? rbits[r] : bits) + (NARROW || left ? v0 : v0 + 16);
          arg = m == m ? arg : 0;
        }
        const float ms = m * e.osc;  // memory holds scaled-back values; compare and store in that domain
        float* const dst = pu + (ubase + ROW + r) * usd;
        float* const dst_arg = ARG ? pua + (ubase + ROW + r) * uasd : nullptr;
        const bool more = ms > fmaxf(rold[ROW + r], -CUDART_INF_F);  // strict: the lowest column block wins ties
        if ((WHOLE || (valid && ROW + r < nu)) && (first || more)) {
          *dst = ms;
          if (ARG) *dst_arg = __int_as_float(arg);
        }
      }
      // columns
      const float qbits = qbase + 2 * ROW;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float x0 = __uint_as_float(x[0][j]), x1 = __uint_as_float(x[1][j]);
        const float x2 = __uint_as_float(x[2][j]), x3 = __uint_as_float(x[3][j]);
        float &c = cm[COL + j], &where = ca[COL + j];
        if (ARG) {
          const float m = fmaxf(fmax3(x0, x1, x2), x3);
          const float bits = fmaf(is_equal(x0, m), 4.f, fmaf(is_equal(x1, m), 2.f, qbits + is_equal(x2, m)));
          const bool more = m > c;  // strict: the lowest rows win ties
          c = more ? m : c;
          where = more ? bits : where;
        } else {
          c = fmax3(fmax3(c, x0, x1), x2, x3);
        }
      }
    };
    auto tile = [&](auto whole) {
#pragma unroll
      for (int r = 0; r < 4; ++r) load(0, r);
#pragma unroll
      for (int r = 0; r < 4; ++r) tmem_ld_wait16(s[0][r]);
#pragma unroll
      for (int r = 0; r < 2; ++r) load(1, r);
      unit(std::integral_constant<int, 0>{}, whole);
#pragma unroll
      for (int r = 2; r < 4; ++r) load(1, r);
#pragma unroll
      for (int r = 0; r < 4; ++r) tmem_ld_wait16(s[1][r]);
      epi_release(sm, t, e.lane);  // all values are in registers: hand the accumulator back
      unit(std::integral_constant<int, 1>{}, whole);
    };
    if (all_valid && nu == RW && nv == VT) tile(std::true_type{});
    else tile(std::false_type{});
   }
    // end of a column block: group 0 puts the first half of the columns together, group 1 the others
    {
      auto row = [&](int j) {
        const int code = static_cast<int>(ca[j]);
        return (code >> 3) * 4 + __clz(code & 7) - 29;   // 4, 2, 1, 0 stand for rows 0 .. 3 of the four
      };
      const int cols = valid ? nv : 0;   // columns this lane has
      auto merge = [&](auto own_half) -> bool {
        constexpr int HALF = VT / 2, OWN = decltype(own_half)::value * HALF, OTHER = HALF - OWN;
        float* q = pv + (v0 + OTHER) * vsd;
        float* qa = ARG ? pva + (v0 + OTHER) * vasd : nullptr;
#pragma unroll
        for (int j = OTHER; j < OTHER + HALF; ++j, q += vsd, qa += ARG ? vasd : 0) {
          if (j < cols) *q = cm[j] * e.osc;
          if (ARG && j < cols) *qa = __int_as_float(row(j));
        }
        merge_publish(sm, sc, vb, e);
        if (!merge_wait(sm, a, sc, vb, e)) return false;
        q = pv + (v0 + OWN) * vsd;
        if (ARG) qa = pva + (v0 + OWN) * vasd;
        float om[HALF], oa[HALF];
#pragma unroll
        for (int j = 0; j < HALF; ++j, q += vsd, qa += ARG ? vasd : 0) {
          om[j] = OWN + j < cols ? __ldcg(q) : 0.f;
          if (ARG) oa[j] = OWN + j < cols ? __ldcg(qa) : 0.f;
        }
        q = pv + (v0 + OWN) * vsd;
        if (ARG) qa = pva + (v0 + OWN) * vasd;
#pragma unroll
        for (int j = 0; j < HALF; ++j, q += vsd, qa += ARG ? vasd : 0) {
          const float mine = cm[OWN + j] * e.osc;
          if (ARG) {
            const int o = __float_as_int(oa[j]), own = row(OWN + j);
            const bool other = om[j] > mine || (om[j] == mine && o < own);  // lowest u on ties
            if (OWN + j < cols) *q = other ? om[j] : mine;
            if (OWN + j < cols) *qa = __int_as_float(other ? o : own);
          } else {
            if (OWN + j < cols) *q = fmaxf(mine, om[j]);
          }
        }
        return true;
      };
      if (!(e.wg == 0 ? merge(std::integral_constant<int, 0>{}) : merge(std::integral_constant<int, 1>{}))) return;
    }
  }
  // mean channels: accumulator column r of an aux tile is F1[p] . (row-mean u=r | column-mean v=r-H2).  A loop over 16 columns
  // at a time: this code runs once per CTA, so its instructions are fetched cold, and unrolled over 128 columns with a branch
  // each it took 33,000 cycles, as long as the tiles of a 55 x 128 launch.
  const int naux = H2 + W2;
  float* const pvm = pv + vss;
  for (int t = sc.t_main; t < sc.t_total; ++t) {
    if (!epi_wait(sm, a, t)) return;
    const uint32_t tacc = e.tbase + (t % SW_NACC) * SW_TILE_N + e.wg * 128;
    const int r_end = min(naux, (t - sc.t_main) * SW_TILE_N + e.wg * 128 + 128);
#pragma unroll 1
    for (int r0 = (t - sc.t_main) * SW_TILE_N + e.wg * 128, c0 = 0; r0 < r_end; r0 += 16, c0 += 16) {
      float s[16];
      tmem_ld16(tacc + c0, s);
      if (!valid) continue;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int r = r0 + j;
        float* const dst = r < H2 ? pum + r * umsd : pvm + (r - H2) * vsd;
        if (r < r_end) *dst = s[j] * e.osc;
      }
    }
    epi_release(sm, t, e.lane);
  }
}

// acc += (lo, hi) * w on a packed pair; lo and hi are tcgen05.ld registers: volatile keeps the multiply-add behind the
// tcgen05.wait::ld before it.
__device__ __forceinline__ void fma2_tmem(uint64_t& acc, uint32_t lo, uint32_t hi, uint64_t w) {
  asm volatile("{\n\t.reg .b64 s;\n\tmov.b64 s, {%1, %2};\n\tfma.rn.f32x2 %0, s, %3, %0;\n\t}" : "+l"(acc) : "r"(lo), "r"(hi), "l"(w));
}

// Where the row sums of a level go by TMA: the output, and the scratch of later pieces.  (pixel, displacement, channel, sample or part)
struct RowMaps {
  CUtensorMap out, part;
};

// Compression sums.  A thread does CPT channels of its pixel.  With three or four channels the two groups take two each and read
// whole tiles; with one or two (SPLIT) both do all of them and share a tile's rows, and the column sums of a block are put
// together at its end.
//   au2[c][j] = (w_u[v0+2j], w_u[v0+2j+1])         weights of this column block, per column pair
//   cv2[c][j] = running (OV[v0+2j], OV[v0+2j+1])   over the rows of the column block
// Cells outside the image hold S = 0 (TMA zero-fills the missing F2 rows) and get weight 0, so every tile is processed
// whole and only the stores at the edges are predicated.
// Bound: the FMA pipe and the register ports.  A cell takes a packed multiply-add (fma.rn.f32x2) per channel and direction;
// with three different 64-bit operands that instruction takes 3 cycles of a scheduler (measured; 2.2 with one operand kept),
// 3072 cycles per tile and scheduler at four channels, where the tensor core needs some 2600.  As scalar multiply-adds, twice
// as many instructions at 1 cycle, the same loop was slower (780 .. 910 us): it is then issue that runs short.
// What else mattered: one value per row of 32 columns and channel leaves a tile, instead of one per 16 (16 x 16 tiles); 16
// columns are loaded while 16 others are worked on; loops nested by column block, so that the 128 registers of weights and
// sums are not moved around at every tile (450 of 1860 instructions per warp and tile were moves); the row weights of the
// next tile are asked for before the wait for this one.  135 x 240, one pair, four channels: 897 -> 717 us (8 pairs, two
// sweeps: 14.2 -> 10.9 ms); 8 x 47 x 156, two channels: 337 -> 290 us.
template <int KC, bool CUT, bool NARROW, bool TMA_ROWS>
__device__ void epilogue_compress(SweepSmem& sm, const SweepArgs& a, const SweepSched& sc, const EpiCtx& e, const RowMaps* maps) {
  constexpr int CPT = sw_channels(KC);
  constexpr bool SPLIT = KC <= 2;
  using T = Tile<NARROW>;
  constexpr int VT = T::VT, HALVES = T::HALVES;
  constexpr int NR = SPLIT ? T::RW : T::UT;      // tile rows of this thread
  const int H2 = a.d.H2, W2 = a.d.W2;
  const int k_first = SPLIT ? 0 : e.wg * CPT;    // its first channel among those of this launch
  const int n_ch = min(CPT, a.kc - k_first);     // how many of them exist
  const uint32_t xusd = a.xu.sd, xvsd = a.xv.sd, ovsd = a.ov.sd;
  uint32_t ousd = a.ou.sd, ouss = a.ou.ss;
  const uint32_t wuss = (uint32_t)a.w_stride * a.xv.ss, wvss = (uint32_t)a.w_stride * a.xu.ss, ovss = a.ov.ss;
  // this thread's pixel and first channel in sample b of each view; displacement d at ptr[d*sd], 32-bit offsets.  Weights that
  // do not exist (lanes past the image, a second channel past the last) are read from the nearest that do.
  const int k = a.k0 + k_first, p_in = min(e.p, a.n_valid - 1);
  const float* wu = a.xv.base + sc.b * a.xv.sb + p_in + (a.wu_slot0 + k * a.w_stride) * a.xv.ss;  // w_u[k][v]
  const float* wv = a.xu.base + sc.b * a.xu.sb + p_in + (a.wv_slot0 + k * a.w_stride) * a.xu.ss;  // w_v[k][u]
  float* ou = a.ou.base + sc.b * a.ou.sb + e.p + k * a.ou.ss;
  float* ov = a.ov.base + sc.b * a.ov.sb + e.p + k * a.ov.ss;
  // The first column block initialises the row sums, the others are added to them (same thread, same address in every block,
  // hence ordered).  A later piece stores every block, into a part of its own (slot = channel of this launch).
  uint32_t part_step = 0;
  if (CUT && sc.piece > 0) {
    ou = sweep_part(a, sc.tail, sc.vb0 - sc.part_vb0, k_first) + (e.p - sc.m0);
    ousd = TILE_M;
    ouss = (uint32_t)H2 * TILE_M;
    part_step = (uint32_t)a.part_slots * H2 * TILE_M;
  }
  const int row0 = SPLIT ? e.wg * T::RW : 0;
  // TMA_ROWS: a tile's row sums go to one of the warp's two buffers, from where a TMA store (first column block, and every one of a later
  // piece) or add takes them to memory.  A buffer is used again, and a row added to again, when the copies of two tiles ago are complete
  // (of one row block: of the tile before), so the sums of a row are added up in the order of its column blocks.  Every tile is a bulk group,
  // also one of which a group of warps has no row (SPLIT, 1 to 4 rows in the last block): without it the wait for all groups but the last
  // would leave the one of two tiles ago under way.  With red.global from the
  // registers the sixteen of a warp and tile, their 64-bit addresses and conditions took an eighth of the launch (135 x 240, one pair, four
  // levels and channels 965 -> 860 us, 4 x 55 x 128 228 -> 203; 8 x 47 x 156, one level, two channels, both sweeps 514 -> 487).
  const int warp = e.wg * 4 + (e.p - e.lane - sc.m0) / 32;
  float* const row_buffer = reinterpret_cast<float*>(sm.ring + SW_RING_BYTES - sw_row_bytes(KC)) + warp * (2 * NR * CPT * 32) + e.lane;
  const bool later_piece = CUT && sc.piece > 0;
  float av[CPT][NR];   // w_v of the coming tile's rows (past the image: the last row's)
  auto load_av = [&](int u0) {
#pragma unroll
    for (int c = 0; c < CPT; ++c)
#pragma unroll
      for (int ul = 0; ul < NR; ++ul) av[c][ul] = __ldg(wv + (c < n_ch ? c * wvss : 0u) + min(u0 + ul, H2 - 1) * xusd);
  };
  load_av(row0);
  int t = 0;
  for (int vb = sc.vb0; vb < sc.vb1; ++vb, ou += part_step) {
    const int v0 = vb * VT, nv = min(VT, W2 - v0);
    const bool first = vb == 0 || part_step != 0;
    uint64_t au2[CPT][VT / 2], cv2[CPT][VT / 2];
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
      const float* wu_t = wu + v0 * xvsd + (c < n_ch ? c * wuss : 0u);
#pragma unroll
      for (int j = 0; j < VT; j += 2) {
        au2[c][j / 2] = pack2(j < nv ? __ldg(wu_t + j * xvsd) : 0.f, j + 1 < nv ? __ldg(wu_t + (j + 1) * xvsd) : 0.f);
        cv2[c][j / 2] = 0ull;
      }
    }
    for (int ub = 0; ub < sc.n_ub; ++ub, ++t) {
      const int u0 = ub * T::UT + row0, nu = min(NR, H2 - u0);   // nu may be <= 0
      uint64_t a2[CPT][NR];
#pragma unroll
      for (int c = 0; c < CPT; ++c)
#pragma unroll
        for (int ul = 0; ul < NR; ++ul) {
          const float w = ul < nu ? av[c][ul] : 0.f;   // rows past the image hold S = 0; their weight must not be an infinity
          a2[c][ul] = pack2(w, w);
        }
      load_av((ub + 1 == sc.n_ub ? 0 : ub + 1) * T::UT + row0);
      int rows[CPT];   // rows of each channel that are stored
      float* dst[CPT];
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        rows[c] = e.valid && c < n_ch ? nu : 0;
        dst[c] = ou + u0 * ousd + c * ouss;
      }
      float* const to_rows = row_buffer + (t & 1) * (NR * CPT * 32);
      if (!epi_wait(sm, a, t)) return;
      if constexpr (TMA_ROWS) {
        if (e.lane == 0) {
          if (sc.n_ub > 1) bulk_wait<1>();
          else bulk_wait<0>();
        }
        __syncwarp();
      }
      const uint32_t tacc = e.tbase + (t % SW_NACC) * SW_TILE_N + row0 * VT;
      uint32_t s[2][16];
      uint64_t r2[CPT];
      tmem_ld16_issue(tacc, s[0]);
#pragma unroll
      for (int i = 0; i < HALVES * NR; ++i) {   // 16 columns of a row at a time, the next ones on their way
        const int ul = i / HALVES, h = i % HALVES;
        tmem_ld_wait();
        if (i + 1 < HALVES * NR) tmem_ld16_issue(tacc + (i + 1) * 16, s[(i + 1) % 2]);
        else epi_release(sm, t, e.lane);   // last read of this tile
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          if (h == 0) r2[c] = 0ull;
#pragma unroll
          for (int j = 0; j < 8; ++j) fma2_tmem(cv2[c][h * 8 + j], s[i % 2][2 * j], s[i % 2][2 * j + 1], a2[c][ul]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int c = 0; c < CPT; ++c) fma2_tmem(r2[c], s[i % 2][2 * j], s[i % 2][2 * j + 1], au2[c][h * 8 + j]);
        if (h == HALVES - 1) {
#pragma unroll
          for (int c = 0; c < CPT; ++c, dst[c - 1] += ousd) {
            if constexpr (TMA_ROWS) {
              to_rows[(c * NR + ul) * 32] = sum2(r2[c]) * e.osc;
            } else if (rows[c] > ul) {
              const float x = sum2(r2[c]) * e.osc;
              if (first) *dst[c] = x;
              else atomicAdd(dst[c], x);
            }
          }
        }
      }
      if constexpr (TMA_ROWS) {
        fence_proxy_async_smem();
        __syncwarp();
        if (e.lane == 0 && (!SPLIT || nu > 0) && e.valid) {
          if (later_piece) tma_store_4d(&maps->part, to_rows, e.p - sc.m0, u0, k_first, sc.tail * a.parts + vb - sc.part_vb0);
          else if (first) tma_store_4d(&maps->out, to_rows, e.p, u0, k, sc.b);
          else tma_add_4d(&maps->out, to_rows, e.p, u0, k, sc.b);
        }
        bulk_commit();   // in every tile: the wait above counts groups (by all lanes: in lane 0's branch the 135 x 240 launch takes 866 us, not 860)
      }
    }
    float cv[CPT][VT];
#pragma unroll
    for (int c = 0; c < CPT; ++c)
#pragma unroll
      for (int j = 0; j < VT / 2; ++j) unpack2(cv2[c][j], cv[c][2 * j], cv[c][2 * j + 1]);
    auto column = [&](int c, int j) { return ov + (v0 + j) * ovsd + c * ovss; };
    auto columns = [&](int c) { return e.valid && c < n_ch ? nv : 0; };   // how many of them this thread has
    if constexpr (!SPLIT) {
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        float* q = column(c, 0);
        const int n = columns(c);
#pragma unroll
        for (int j = 0; j < VT; ++j, q += ovsd)
          if (j < n) *q = cv[c][j] * e.osc;
      }
    } else {
      auto merge = [&](auto own_half) -> bool {
        constexpr int HALF = VT / 2, OWN = decltype(own_half)::value * HALF, OTHER = HALF - OWN;
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          float* q = column(c, OTHER);
          const int n = columns(c);
#pragma unroll
          for (int j = OTHER; j < OTHER + HALF; ++j, q += ovsd)
            if (j < n) *q = cv[c][j] * e.osc;
        }
        merge_publish(sm, sc, vb, e);
        if (!merge_wait(sm, a, sc, vb, e)) return false;
        float o[CPT][HALF];
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          const float* q = column(c, OWN);
          const int n = columns(c);
#pragma unroll
          for (int j = 0; j < HALF; ++j, q += ovsd) o[c][j] = OWN + j < n ? __ldcg(q) : 0.f;
        }
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          float* q = column(c, OWN);
          const int n = columns(c);
#pragma unroll
          for (int j = 0; j < HALF; ++j, q += ovsd)
            if (OWN + j < n) *q = cv[c][OWN + j] * e.osc + o[c][j];
        }
        return true;
      };
      if (!(e.wg == 0 ? merge(std::integral_constant<int, 0>{}) : merge(std::integral_constant<int, 1>{}))) return;
    }
  }
  if (TMA_ROWS && e.lane == 0) bulk_wait_all();
}

// Test aid: writes the dense volume of a (small) problem so the tensor-core plumbing can be checked alone.
template <bool NARROW>
__device__ void epilogue_dump(SweepSmem& sm, const SweepArgs& a, const SweepSched& sc, const EpiCtx& e) {
  using T = Tile<NARROW>;
  const int H2 = a.d.H2, W2 = a.d.W2, N1 = a.d.N1();
  const bool valid = e.p < N1;
  float* out = a.dump + ((size_t)sc.b * N1 + (valid ? e.p : 0)) * H2 * W2;
  int vb = 0, ub = 0;
  for (int t = 0; t < sc.t_main; ++t) {
    const int v0 = vb * T::VT, ubase = ub * T::UT + e.wg * T::RW;
    const int nu = min(T::RW, H2 - ubase), nv = min(T::VT, W2 - v0);
    if (!epi_wait(sm, a, t)) return;
    const uint32_t tacc = e.tbase + (t % SW_NACC) * SW_TILE_N + e.wg * 128;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float s[64];
      tmem_ld64(tacc + half * 64, s);
      if (half == 1) epi_release(sm, t, e.lane);
      if (valid) {
#pragma unroll
        for (int hl = 0; hl < T::RW / 2; ++hl)
#pragma unroll
          for (int j = 0; j < T::VT; ++j) {
            const int ul = half * (T::RW / 2) + hl;
            if (ul < nu && j < nv) out[(size_t)(ubase + ul) * W2 + v0 + j] = s[hl * T::VT + j] * e.osc;
          }
      }
    }
    if (++ub == sc.n_ub) { ub = 0; ++vb; }
  }
}

// ---------------------------------------------------------------------------------- kernel
// What a launch works on: one pair of images, or the levels of a pyramid over the same image 1, whose tiles follow one another.
template <int LEVELS>
struct SweepLaunch {
  CUtensorMap f1, f2[LEVELS], aux[LEVELS];
  RowMaps rows[LEVELS];
  SweepArgs a[LEVELS];
  int first_block[LEVELS + 1], first_tail[LEVELS + 1];   // of the sweep and of the fold; levels that do not exist have none
};
template <int LEVELS>
__device__ __forceinline__ int level_of(const int (&first)[LEVELS + 1], int block) {
  int level = 0;
#pragma unroll
  for (int l = 1; l < LEVELS; ++l) level = block >= first[l] ? l : level;
  return level;
}
enum TileForm : int { TILES_WIDE = 0, TILES_NARROW = 1, TILES_BY_LEVEL = 2 };
// f(std::true_type) for narrow tiles, f(std::false_type) for wide ones
template <int FORM, class F>
__device__ __forceinline__ void by_tile_form(const SweepArgs& a, F&& f) {
  if constexpr (FORM == TILES_WIDE) f(std::false_type{});
  else if constexpr (FORM == TILES_NARROW) f(std::true_type{});
  else if (a.narrow) f(std::true_type{});
  else f(std::false_type{});
}

// CUT: the launch has tail pieces.  A launch without any runs the kernel without their bookkeeping.
// KC (compression): channels of the launch, 1, 2 or (three or four) 4.
// LEVELS > 1: the levels of a pyramid in one launch.  The coarse ones have too few cells to fill the SMs (55 x 128: 8, 2 and 1 tiles per
// pixel tile beside 28), and the finest leaves SMs idle in its last wave, which their tiles fill.  Both sweeps of four levels with their
// folds, levels one after the other and together (us, four channels, FP16): 1 x 55 x 128 172 and 134, 4 x 55 x 128 422 and 360,
// 1 x 135 x 240 1675 and 1558.
// TMA_ROWS (compression): the row sums go to memory by TMA (wide tiles; narrow ones of a pyramid's levels do not).
template <int MODE, bool CUT, int KC, int FORM, int LEVELS, bool TMA_ROWS>
__global__ void __launch_bounds__(SW_THREADS, 1)
sweep_kernel(const __grid_constant__ SweepLaunch<LEVELS> launch, int* status) {
  if (!cta_has_work(status)) return;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t pad = (1024u - (smem_u32(smem_raw) & 1023u)) & 1023u;
  SweepSmem& sm = *reinterpret_cast<SweepSmem*>(smem_raw + pad);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int level = level_of<LEVELS>(launch.first_block, blockIdx.x);
  const SweepArgs& a = launch.a[level];
  const int block = LEVELS == 1 ? blockIdx.x : blockIdx.x - launch.first_block[level];
  const CUtensorMap *const tm_f1 = &launch.f1, *const tm_f2 = &launch.f2[level], *const tm_aux = &launch.aux[level];

  if (threadIdx.x == 0) {
    mbar_init(&sm.f1_full, 1);
    for (int s = 0; s < SW_MAX_STAGES; ++s) { mbar_init(&sm.full[s], 1); mbar_init(&sm.empty[s], 1); }
    for (int i = 0; i < SW_NACC; ++i) { mbar_init(&sm.acc_full[i], 1); mbar_init(&sm.acc_empty[i], SW_EPI_WARPS); }
    for (int i = 0; i < SW_NMERGE; ++i) { mbar_init(&sm.merge[0][i], 4); mbar_init(&sm.merge[1][i], 4); }  // four warps of a group
    wait_ctl_init(&sm.ctl, a.wait_limit_ns);
    fence_barrier_init();
    prefetch_tensormap(tm_f1);
    prefetch_tensormap(tm_f2);
    if (MODE == SWEEP_MAXAVG || MODE == SWEEP_MAXARGAVG) prefetch_tensormap(tm_aux);
  }
  if (warp == 1) {
    tmem_alloc(&sm.tmem_base, SW_TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  // Every role is through: its copies have landed, or, where a wait ran out, get time to.
  auto meet = [&] {
    tc_fence_before();
    __syncthreads();
    if (wait_ctl_aborted(&sm.ctl)) {
      let_copies_land();
      __syncthreads();
    }
  };
  // The two kinds of warps do not meet in common code again: what follows here is compiled for SW_REGS_ISSUE registers, what
  // follows there for SW_REGS_EPI.
  constexpr uint32_t row_bytes = TMA_ROWS ? sw_row_bytes(KC) : 0;
  if (warp < 4) {
    set_max_registers<SW_REGS_ISSUE, false>();
    by_tile_form<FORM>(a, [&](auto narrow) {
      constexpr bool NARROW = decltype(narrow)::value;
      const SweepSched sc = sweep_sched<MODE, CUT, NARROW>(a, block);
      if (warp == 0) {
        if (lane == 0) sweep_producer<NARROW>(sm, a, sc, tm_f1, tm_f2, tm_aux, row_bytes);
      } else if (warp == 1) {
        if (lane == 0) sweep_mma(sm, a, sc, row_bytes);
      }
    });
    __syncwarp();
    meet();
    if (warp == 1) {
      tc_fence_after();
      tmem_dealloc(sm.tmem_base, SW_TMEM_COLS);
    }
    return;
  }
  set_max_registers<SW_REGS_EPI, true>();
  by_tile_form<FORM>(a, [&](auto narrow) {
    constexpr bool NARROW = decltype(narrow)::value;
    const SweepSched sc = sweep_sched<MODE, CUT, NARROW>(a, block);
    EpiCtx e;
    const int q = warp & 3;  // tcgen05.ld lets a warp read TMEM lanes 32*(warp%4) .. +31 only
    e.wg = (warp >> 2) - 1;
    e.lane = lane;
    e.p = sc.m0 + q * 32 + lane;
    e.valid = e.p < a.n_valid;
    e.tbase = sm.tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    e.osc = a.out_scale != nullptr ? __ldg(a.out_scale) : 1.f;
    if constexpr (MODE == SWEEP_MAXAVG) epilogue_maxavg<false, CUT, NARROW>(sm, a, sc, e);
    else if constexpr (MODE == SWEEP_MAXARGAVG) epilogue_maxavg<true, CUT, NARROW>(sm, a, sc, e);
    else if constexpr (MODE == SWEEP_COMPRESS) epilogue_compress<KC, CUT, NARROW, TMA_ROWS && !NARROW>(sm, a, sc, e, &launch.rows[level]);
    else epilogue_dump<NARROW>(sm, a, sc, e);
  });
  __syncwarp();
  meet();
}

// The parts of the cut tiles folded into their piece 0's row results, in order.  Maxima: a later piece has the higher columns,
// so only a strictly larger value replaces (a NaN counts as -inf, as it does between the column blocks of a tile).  Sums:
// block by block, the order in which a whole tile adds them, so that a sample's sums do not depend on the cut, which follows
// the batch and the row range.  A kernel of its own, one thread per pixel and FOLD_ROWS rows: folded by the CTA that finished a
// tile last, the 0.3 MB of a 55 x 128 tile with four channels took that one SM 16 us, most of it memory latency.
constexpr int FOLD_ROWS = 4;
template <int MODE, int LEVELS>
__global__ void __launch_bounds__(TILE_M) sweep_fold_kernel(const __grid_constant__ SweepLaunch<LEVELS> launch) {
  follow_previous_kernel();
  constexpr bool SUM = MODE == SWEEP_COMPRESS, ARG = MODE == SWEEP_MAXARGAVG;
  const int level = level_of<LEVELS>(launch.first_tail, blockIdx.y);
  const SweepArgs& a = launch.a[level];
  if (*reinterpret_cast<volatile int*>(a.status) != 0) return;
  const int tiles_per_sample = (a.d.N1() + TILE_M - 1) / TILE_M, H2 = a.d.H2;
  const int tail = LEVELS == 1 ? blockIdx.y : blockIdx.y - launch.first_tail[level], tile = a.whole_tiles + tail, b = tile / tiles_per_sample;
  const int px = threadIdx.x, p = (tile - b * tiles_per_sample) * TILE_M + px;
  if (p >= a.n_valid) return;
  const PixView& out = SUM ? a.ou : a.pu;
  const size_t slot = (size_t)H2 * TILE_M, step = slot * a.part_slots;
  float *dst[FOLD_ROWS], *arg_dst[FOLD_ROWS], v[FOLD_ROWS], va[FOLD_ROWS];
  const float* src[FOLD_ROWS];
  bool in[FOLD_ROWS];
#pragma unroll
  for (int r = 0; r < FOLD_ROWS; ++r) {
    const int q = blockIdx.x * FOLD_ROWS + r, k = q / H2, u = q - k * H2;   // slot (channel of the launch) and row
    in[r] = k < (SUM ? a.kc : 1);
    dst[r] = out.base + b * out.sb + p + (SUM ? (a.k0 + k) * out.ss : 0u) + u * out.sd;
    arg_dst[r] = ARG ? a.pu_arg.base + b * a.pu_arg.sb + p + u * a.pu_arg.sd : nullptr;
    src[r] = sweep_part(a, tail, 0, k) + (size_t)u * TILE_M + px;
    v[r] = in[r] ? *dst[r] : 0.f;
    va[r] = ARG && in[r] ? *arg_dst[r] : 0.f;
  }
#pragma unroll 4
  for (int part = 0; part < a.parts; ++part) {
#pragma unroll
    for (int r = 0; r < FOLD_ROWS; ++r) {
      if (!in[r]) continue;
      const float o = src[r][part * step];
      if (SUM) {
        v[r] += o;
      } else if (o > fmaxf(v[r], -CUDART_INF_F)) {
        v[r] = o;
        if (ARG) va[r] = src[r][part * step + slot];
      }
    }
  }
#pragma unroll
  for (int r = 0; r < FOLD_ROWS; ++r) {
    if (!in[r]) continue;
    *dst[r] = v[r];
    if (ARG) *arg_dst[r] = va[r];
  }
}

// How the tail tiles are cut, in units of one 256-column tile's time: a CTA costs about two tiles of prologue.  Pieces must save
// a quarter of the tail and a whole tile to be used: a wave with idle SMs runs its tiles faster than a full one, and the fold
// is a launch of 4 to 10 us.
// Whole and cut tiles measured (us per call with the fold, C = 256, FP16, max/arg-max/avg and compression; Kc = 4 but for two
// channels at 8 x 47 x 156 and three at 3 x 47 x 155): 1 x 48 x 64: 37 and 27, 33 and 26; 1 x 55 x 128: 76 and 50, 72 and 53;
// 4 x 55 x 128: 158 and 134, 155 and 145; 3 x 47 x 155: 179 and 130, 164 and 116; 8 x 47 x 156: 355 and 302, 277 and 244;
// 1 x 55 x 128 against 27 x 64: 30 and 25, 25 and 21; 3 x 20 x 27 against 18 x 50: 25 and 19, 19 and 14.
TileSplit sweep_split(const Dims& d, int slots, bool sums) {
  const long long tiles = (long long)d.B * ((d.N1() + TILE_M - 1) / TILE_M);
  const bool narrow = sweep_narrow(d, sums);
  const int ut = narrow ? SWEEP_UT_NARROW : SWEEP_UT, vt = narrow ? SWEEP_VT_NARROW : SWEEP_VT;
  const int n_ub = (d.H2 + ut - 1) / ut, n_vb = (d.W2 + vt - 1) / vt;
  const int rest = (int)(tiles % SM_COUNT);
  TileSplit r{(int)tiles, (int)tiles, 1, 0, 0};
  if (rest == 0) return r;
  double best = 0, whole = 0;
  for (int n = 1; n <= n_vb && n <= MAX_PIECES; ++n) {
    const double waves = (rest * n + SM_COUNT - 1) / SM_COUNT;
    const int parts = sums ? n_vb - piece_start(n_vb, n, 1) : n - 1;
    const double cost = waves * ((n_vb + n - 1) / n * n_ub + 2) + (n > 1 ? 0.5 : 0.0);
    if (n == 1) best = whole = cost;
    if (cost < best && cost < 0.75 * whole && cost < whole - 1) { best = cost; r.pieces = n; r.parts = parts; }
  }
  if (r.pieces > 1) {
    r.whole_tiles = (int)tiles - rest;
    r.part_floats = (size_t)rest * r.parts * slots * d.H2 * TILE_M;
  }
  return r;
}

// How the tiles of a pyramid's levels are cut when they share a launch, in the units of sweep_split.  The blocks start in the
// order of the levels, so the short tiles of the coarse levels fill the gaps that the finest leaves: nothing is cut where its tiles
// make more than a few waves.  Else the cut (the same for all tiles of a level) with the smallest makespan of that order.
void sweep_split_levels(const Dims* d, int levels, int slots, bool sums, TileSplit* out) {
  int n_ub[MAX_FUSED_LEVELS], n_vb[MAX_FUSED_LEVELS];
  const int tiles = (int)((long long)d[0].B * ((d[0].N1() + TILE_M - 1) / TILE_M));
  for (int l = 0; l < levels; ++l) {
    const bool narrow = sweep_narrow(d[l], sums);
    const int ut = narrow ? SWEEP_UT_NARROW : SWEEP_UT, vt = narrow ? SWEEP_VT_NARROW : SWEEP_VT;
    n_ub[l] = (d[l].H2 + ut - 1) / ut;
    n_vb[l] = (d[l].W2 + vt - 1) / vt;
    out[l] = TileSplit{tiles, tiles, 1, 0, 0};
  }
  if (tiles > 4 * SM_COUNT) return;
  const LevelCut cut = cheapest_cut(std::min(n_vb[0], MAX_PIECES), levels > 1 ? n_vb[1] : 1, [&](auto& work, int n0, int n1) {
    for (int l = 0; l < levels; ++l) {
      const int n = l == 0 ? n0 : (l == 1 ? n1 : 1), per = n_vb[l] / n, extra = n_vb[l] - per * n;
      work.add(tiles * extra, (per + 1) * n_ub[l] + 2);   // (the order inside a level does not matter much)
      work.add(tiles * (n - extra), per * n_ub[l] + 2);
    }
    return n0 > 1 || n1 > 1 ? 2.0 : 0.0;
  });
  for (int l = 0; l < std::min(levels, 2); ++l) {
    const int n = l == 0 ? cut.n0 : cut.n1;
    if (n == 1) continue;
    const int parts = sums ? n_vb[l] - piece_start(n_vb[l], n, 1) : n - 1;
    out[l] = TileSplit{tiles, 0, n, parts, (size_t)tiles * parts * slots * d[l].H2 * TILE_M};
  }
}

// Maps of the row sums of a level.  Not all views have the alignment that a tensor map asks for (planes of a multiple of 4 pixels); and with
// TF32 operands the image-1 tile leaves no room for the buffers beside a ring of three stages.
static bool row_maps(const SweepArgs& a, int rows, int channels, RowMaps* maps, cudaError_t* err) {
  const auto aligned = [](long long elements) { return elements % 4 == 0; };
  if ((reinterpret_cast<uintptr_t>(a.ou.base) & 15u) != 0 || !aligned(a.ou.sb) || !aligned(a.ou.sd) || !aligned(a.ou.ss)) return false;
  const uint32_t box[4] = {32, (uint32_t)rows, (uint32_t)channels, 1};
  const uint64_t dims[4] = {(uint64_t)a.n_valid, (uint64_t)a.d.H2, (uint64_t)(a.k0 + a.kc), (uint64_t)a.d.B};
  const uint64_t strides[3] = {a.ou.sd * 4ull, a.ou.ss * 4ull, (uint64_t)a.ou.sb * 4ull};
  if ((*err = encode_plain_map(&maps->out, a.ou.base, 4, dims, strides, box)) != cudaSuccess) return false;
  if (a.pieces == 1) return true;
  const int tails = a.d.B * ((a.d.N1() + TILE_M - 1) / TILE_M) - a.whole_tiles;
  const uint64_t part_dims[4] = {TILE_M, (uint64_t)a.d.H2, (uint64_t)a.part_slots, (uint64_t)tails * a.parts};
  const uint64_t part_strides[3] = {TILE_M * 4ull, a.d.H2 * (TILE_M * 4ull), (uint64_t)a.part_slots * a.d.H2 * (TILE_M * 4ull)};
  return (*err = encode_plain_map(&maps->part, a.part, 4, part_dims, part_strides, box)) == cudaSuccess;
}

template <int MODE, bool CUT, int KC, int FORM, int LEVELS, bool TMA_ROWS = false>
static cudaError_t launch_one(SweepLaunch<LEVELS>& launch, int levels, cudaStream_t stream) {
  if constexpr (MODE == SWEEP_COMPRESS && FORM != TILES_NARROW && !TMA_ROWS) {
    bool tma = launch.a[0].op16 != 0;
    cudaError_t err = cudaSuccess;
    for (int l = 0; l < levels && tma; ++l)
      tma = launch.a[l].narrow || row_maps(launch.a[l], sw_rows(KC), sw_channels(KC), &launch.rows[l], &err);
    if (err != cudaSuccess) return err;
    if (tma) return launch_one<MODE, CUT, KC, FORM, LEVELS, true>(launch, levels, stream);
  }
  auto kern = sweep_kernel<MODE, CUT, KC, FORM, LEVELS, TMA_ROWS>;
  static DeviceOnce configured;  // the attribute is per device and stays set
  cudaError_t err = configured.run([&] {
    // A kernel that was compiled for fewer registers than the split takes would wait in setmaxnreg.inc without a limit.
    cudaFuncAttributes built;
    if (cudaError_t e = cudaFuncGetAttributes(&built, kern); e != cudaSuccess) return e;
    if (!register_split_fits(built.numRegs)) return cudaErrorInvalidKernelImage;
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SW_SMEM_BYTES);
  });
  if (err != cudaSuccess) return err;
  int blocks = 0, tails = 0, rows = 0;
  for (int l = 0; l < LEVELS; ++l) {
    launch.first_block[l] = blocks;
    launch.first_tail[l] = tails;
    if (l >= levels) continue;
    const SweepArgs& a = launch.a[l];
    const int cut = a.d.B * ((a.d.N1() + TILE_M - 1) / TILE_M) - a.whole_tiles;
    blocks += a.whole_tiles + cut * a.pieces;
    if (a.pieces > 1) {
      tails += cut;
      rows = std::max(rows, (MODE == SWEEP_COMPRESS ? a.kc : 1) * a.d.H2);
    }
  }
  launch.first_block[LEVELS] = blocks;
  launch.first_tail[LEVELS] = tails;
  launch_next(kern, blocks, SW_THREADS, SW_SMEM_BYTES, stream, launch, launch.a[0].status);
  if constexpr (CUT) {
    if (tails == 0) return cudaGetLastError();
    if ((err = cudaGetLastError()) != cudaSuccess) return err;
    launch_next(sweep_fold_kernel<MODE, LEVELS>, dim3((rows + FOLD_ROWS - 1) / FOLD_ROWS, tails), TILE_M, 0, stream, launch);
  }
  return cudaGetLastError();
}

template <int MODE, int KC>
static cudaError_t launch_mode(const SweepArgs* a, int levels, const CUtensorMap& tm_f1, const CUtensorMap* tm_f2,
                               const CUtensorMap* tm_aux, cudaStream_t stream) {
  auto fill = [&](auto& launch) {
    launch.f1 = tm_f1;
    for (int l = 0; l < levels; ++l) {
      launch.f2[l] = tm_f2[l];
      launch.aux[l] = tm_aux[l];
      launch.a[l] = a[l];
      launch.a[l].narrow = sweep_narrow(a[l].d, MODE == SWEEP_COMPRESS);
    }
  };
  if constexpr (MODE != SWEEP_DUMP) {
    if (levels > 1) {
      SweepLaunch<MAX_FUSED_LEVELS> launch{};
      fill(launch);
      return launch_one<MODE, true, KC, TILES_BY_LEVEL>(launch, levels, stream);
    }
  }
  SweepLaunch<1> launch{};
  fill(launch);
  const bool narrow = launch.a[0].narrow;
  if constexpr (MODE != SWEEP_DUMP) {
    if (a->pieces > 1)
      return narrow ? launch_one<MODE, true, KC, TILES_NARROW>(launch, 1, stream) : launch_one<MODE, true, KC, TILES_WIDE>(launch, 1, stream);
  }
  return narrow ? launch_one<MODE, false, KC, TILES_NARROW>(launch, 1, stream) : launch_one<MODE, false, KC, TILES_WIDE>(launch, 1, stream);
}

cudaError_t launch_sweep_levels(const SweepArgs* a, int levels, const CUtensorMap& tm_f1, const CUtensorMap* tm_f2,
                                const CUtensorMap* tm_aux, cudaStream_t stream) {
  if (levels < 1 || levels > MAX_FUSED_LEVELS) return cudaErrorInvalidValue;
  switch (a->mode) {
    case SWEEP_MAXAVG: return launch_mode<SWEEP_MAXAVG, 0>(a, levels, tm_f1, tm_f2, tm_aux, stream);
    case SWEEP_MAXARGAVG: return launch_mode<SWEEP_MAXARGAVG, 0>(a, levels, tm_f1, tm_f2, tm_aux, stream);
    case SWEEP_DUMP: return levels == 1 ? launch_mode<SWEEP_DUMP, 0>(a, 1, tm_f1, tm_f2, tm_aux, stream) : cudaErrorInvalidValue;
    case SWEEP_COMPRESS:
      switch (a->kc) {
        case 1: return launch_mode<SWEEP_COMPRESS, 1>(a, levels, tm_f1, tm_f2, tm_aux, stream);
        case 2: return launch_mode<SWEEP_COMPRESS, 2>(a, levels, tm_f1, tm_f2, tm_aux, stream);
        case 3: case 4: return launch_mode<SWEEP_COMPRESS, 4>(a, levels, tm_f1, tm_f2, tm_aux, stream);
        default: return cudaErrorInvalidValue;
      }
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_sweep(const SweepArgs& a, const CUtensorMap& tm_f1, const CUtensorMap& tm_f2,
                         const CUtensorMap& tm_aux, cudaStream_t stream) {
  return launch_sweep_levels(&a, 1, tm_f1, &tm_f2, &tm_aux, stream);
}

}  // namespace sfb
