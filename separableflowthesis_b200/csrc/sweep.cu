// Correlation sweep: S = F1 * F2^T computed tile by tile on the tcgen05 tensor cores with the
// accumulator in TMEM, reduced in the epilogue so that S never reaches HBM.
//
// One CTA owns 128 consecutive image-1 pixels of one sample (the rows / TMEM lanes of every
// accumulator tile) and sweeps all image-2 pixels in tiles of SWEEP_UT x SWEEP_VT (16 rows x 16
// columns = 256 accumulator columns), column-blocks outermost.  Warp roles:
//   warp 0      TMA producer: F1 tile once (stays resident), F2 tiles through a ring of stages
//   warp 1      allocates TMEM, issues tcgen05.mma (TF32 in, FP32 accumulate), 2 accumulators in flight
//   warps 2..   epilogue warpgroups (two, or four for the compression epilogue); in each, one thread per
//               image-1 pixel reads its accumulator lane with tcgen05.ld.  All groups consume every tile and
//               split its work.
// Everything indexed by an image-1 pixel is read and written in the packed, pixel-fastest layout
// (kernels.h), so a warp's 32 lanes touch one 128-byte line per access.
// Epilogues
//   max/avg      : group g takes tile rows 8g..8g+7.  Running column-direction max(+argmax) in
//                  registers across the inner row-block loop (the two groups' partial results are merged
//                  once per column block), row-direction max(+argmax) merged through the packed output
//                  once per tile.  The two mean channels come from extra tiles whose "image-2 pixels"
//                  are the row-mean and column-mean feature rows of F2 (mean_v S[u,v] = F1 . mean_v F2[u,v]).
// Tail tiles: a grid that is not a multiple of 148 tiles leaves SMs idle in its last wave (and a single 55 x 128 pair has
// 55 tiles in all), so the tiles past the last full wave are cut into `pieces` CTAs, each a range of column blocks.  Column
// results are complete within a piece; row results of pieces 1.. go to scratch, and the CTA that finishes a tile last (a
// counter per tile, nobody waits) folds them into piece 0's results in piece order, so the result does not depend on timing.
//   compression  : group g takes channel g.  OU[k,u] = sum_v S*w_u[k,v] (reduced per tile, accumulated
//                  with red.add), OV[k,v] = sum_u S*w_v[k,u] (register accumulators across the inner loop).
// Replaces the reference kernels MemorySaver_kernel_forward.cu:128-313, :328-533, :550-753.
#include <math_constants.h>

#include "kernels.h"
#include "sm100_primitives.cuh"

namespace sfb {

constexpr int SW_NSTAGE = 3;                    // 3 x 32 KB of F2 blocks next to the 128 KB resident F1 tile
constexpr int SW_NACC = 2;                      // 2 x 256 TMEM columns
constexpr int SW_TILE_N = SWEEP_UT * SWEEP_VT;  // 256 accumulator columns: tcgen05.mma issues at a fixed
                                                // rate per instruction, so the widest N does the most work
// Epilogue warps: two warpgroups for the max/avg and dump epilogues (each takes half of a tile's rows), four for
// the compression epilogue (each takes one channel and reads the whole tile): its work per cell is 2 FMAs per
// channel, and with 16 warps the FP32 pipes keep up with the tensor pipe.
__host__ __device__ constexpr int sw_epi_warps(int mode) { return mode == SWEEP_COMPRESS ? 16 : 8; }
__host__ __device__ constexpr int sw_threads(int mode) { return 64 + sw_epi_warps(mode) * 32; }
constexpr int SW_RW = SWEEP_UT / 2;             // tile rows of one epilogue warpgroup
constexpr int SW_NMERGE = 4;                    // ring of column-merge barriers (> SW_NACC tiles of run-ahead)
constexpr uint32_t SW_STAGE_BYTES = SW_TILE_N * KBLK * 4;
constexpr uint32_t SW_F1_BLOCK_BYTES = TILE_M * KBLK * 4;
constexpr uint32_t SW_TMEM_COLS = 512;
static_assert(SW_NACC * SW_TILE_N <= 512, "accumulators exceed TMEM");
static_assert(SW_NMERGE > SW_NACC, "a warpgroup can run SW_NACC tiles ahead of the other");
static_assert(SW_TILE_N == 256 && SW_RW * SWEEP_VT == 128, "epilogues read two 64-column halves per warpgroup");

struct SweepSmem {
  float f1[MAX_KB][TILE_M * KBLK];        // resident image-1 tile, one 128B-swizzled block per 32 channels
  float f2[SW_NSTAGE][SW_TILE_N * KBLK];  // ring of image-2 tile blocks
  uint64_t f1_full;
  uint64_t full[SW_NSTAGE];
  uint64_t empty[SW_NSTAGE];
  uint64_t acc_full[SW_NACC];
  uint64_t acc_empty[SW_NACC];
  uint64_t merge[SW_NMERGE];              // group 1 -> group 0: partial column results are in memory
  uint32_t tmem_base;
  int last_piece;                         // this CTA finished its tail tile last: it folds the pieces together
  WaitCtl ctl;
};
constexpr size_t SW_SMEM_BYTES = sizeof(SweepSmem) + 1024;  // + slack to align the base to 1024 B

struct SweepSched {
  int b, m0, nkb, n_ub;
  int vb0;              // first column block of this CTA
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
template <int MODE, bool CUT>
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
  sc.n_ub = (a.d.H2 + SWEEP_UT - 1) / SWEEP_UT;
  const int n_vb = (a.d.W2 + SWEEP_VT - 1) / SWEEP_VT;
  const int n_pieces = CUT && sc.tail >= 0 ? a.pieces : 1;
  sc.vb0 = piece_start(n_vb, n_pieces, sc.piece);
  sc.part_vb0 = piece_start(n_vb, n_pieces, 1);
  sc.t_main = sc.n_ub * (piece_start(n_vb, n_pieces, sc.piece + 1) - sc.vb0);
  const bool has_aux = (MODE == SWEEP_MAXAVG || MODE == SWEEP_MAXARGAVG);
  const bool does_aux = has_aux && sc.piece == n_pieces - 1;       // the mean rows go to the last, smallest piece
  sc.t_total = sc.t_main + (does_aux ? (a.d.H2 + a.d.W2 + SW_TILE_N - 1) / SW_TILE_N : 0);
  return sc;
}

// ---------------------------------------------------------------------------------- producer
__device__ void sweep_producer(SweepSmem& sm, const SweepArgs& a, const SweepSched& sc, const CUtensorMap* tm_f1,
                               const CUtensorMap* tm_f2, const CUtensorMap* tm_aux) {
  const int kel = a.op16 ? 2 * KBLK : KBLK;  // channels in one 128-byte row
  mbar_expect_tx(&sm.f1_full, sc.nkb * SW_F1_BLOCK_BYTES);
  for (int kb = 0; kb < sc.nkb; ++kb) tma_load_3d(sm.f1[kb], tm_f1, &sm.f1_full, kb * kel, sc.m0, sc.b);
  uint32_t it = 0;
  int vb = sc.vb0, ub = 0;
  for (int t = 0; t < sc.t_total; ++t) {
    const bool main_tile = t < sc.t_main;
    for (int kb = 0; kb < sc.nkb; ++kb, ++it) {
      const uint32_t s = it % SW_NSTAGE, ph = (it / SW_NSTAGE) & 1u;
      if (!mbar_wait(&sm.empty[s], ph ^ 1u, &sm.ctl, a.status, DEV_TIMEOUT_PRODUCER)) return;
      if (a.drop_last_load && t == sc.t_total - 1 && kb == sc.nkb - 1) return;  // test hook: this block never arrives
      mbar_expect_tx(&sm.full[s], SW_STAGE_BYTES);
      if (main_tile)
        tma_load_4d(sm.f2[s], tm_f2, &sm.full[s], kb * kel, vb * SWEEP_VT, ub * SWEEP_UT, sc.b);
      else
        tma_load_3d(sm.f2[s], tm_aux, &sm.full[s], kb * kel, (t - sc.t_main) * SW_TILE_N, sc.b);
    }
    if (++ub == sc.n_ub) { ub = 0; ++vb; }
  }
}

// ---------------------------------------------------------------------------------- MMA issuer
__device__ void sweep_mma(SweepSmem& sm, const SweepArgs& a, const SweepSched& sc) {
  constexpr uint32_t idesc_tf32 = make_idesc_tf32(TILE_M, SW_TILE_N, false, false);
  const uint32_t idesc_16 = make_idesc_op16(a.op16, TILE_M, SW_TILE_N);  // BF16 or FP16 operands
  const bool op16 = a.op16 != 0;
  if (!mbar_wait(&sm.f1_full, 0, &sm.ctl, a.status, DEV_TIMEOUT_MMA)) return;
  tc_fence_after();
  uint32_t it = 0;
  for (int t = 0; t < sc.t_total; ++t) {
    const uint32_t acc = t % SW_NACC, aph = (t / SW_NACC) & 1u;
    if (!mbar_wait(&sm.acc_empty[acc], aph ^ 1u, &sm.ctl, a.status, DEV_TIMEOUT_MMA)) return;
    tc_fence_after();
    const uint32_t d_tmem = sm.tmem_base + acc * SW_TILE_N;
    for (int kb = 0; kb < sc.nkb; ++kb, ++it) {
      const uint32_t s = it % SW_NSTAGE, ph = (it / SW_NSTAGE) & 1u;
      if (!mbar_wait(&sm.full[s], ph, &sm.ctl, a.status, DEV_TIMEOUT_MMA)) return;
      tc_fence_after();
      const uint64_t adesc = make_smem_desc_sw128(smem_u32(sm.f1[kb]), 16, 1024);
      const uint64_t bdesc = make_smem_desc_sw128(smem_u32(sm.f2[s]), 16, 1024);
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

// Maximum of 16 values and the LOWEST index holding it: pairwise tournament, the left (lower-index)
// entry survives ties.  Same comparison count as a linear scan but only four dependent steps.
__device__ __forceinline__ void max16_first(const float* r, float& m, int& arg) {
  float v8[8], v4[4], v2[2];
  int i8[8], i4[4], i2[2];
#pragma unroll
  for (int i = 0; i < 8; ++i) { const bool g = r[2 * i + 1] > r[2 * i]; v8[i] = g ? r[2 * i + 1] : r[2 * i]; i8[i] = g ? 2 * i + 1 : 2 * i; }
#pragma unroll
  for (int i = 0; i < 4; ++i) { const bool g = v8[2 * i + 1] > v8[2 * i]; v4[i] = g ? v8[2 * i + 1] : v8[2 * i]; i4[i] = g ? i8[2 * i + 1] : i8[2 * i]; }
#pragma unroll
  for (int i = 0; i < 2; ++i) { const bool g = v4[2 * i + 1] > v4[2 * i]; v2[i] = g ? v4[2 * i + 1] : v4[2 * i]; i2[i] = g ? i4[2 * i + 1] : i4[2 * i]; }
  const bool g = v2[1] > v2[0];
  m = g ? v2[1] : v2[0];
  arg = g ? i2[1] : i2[0];
}

template <bool ARG, bool CUT>
__device__ void epilogue_maxavg(SweepSmem& sm, const SweepArgs& a, const SweepSched& sc, const EpiCtx& e) {
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

  // A NaN of a piece's first block must not stand in for a later piece (nothing compares greater than it, and the fold would
  // drop the piece): read back, it counts as -inf there.  It stays in a whole tile and in piece 0, as it always has.
  const float least = CUT && sc.piece > 0 ? -CUDART_INF_F : CUDART_NAN_F;   // fmaxf(x, NaN) is x

  float cm[SWEEP_VT];
  int ca[SWEEP_VT];
  int vb = sc.vb0, ub = 0;
  for (int t = 0; t < sc.t_main; ++t) {
    const int v0 = vb * SWEEP_VT, ubase = ub * SWEEP_UT + e.wg * SW_RW;
    const int nu = min(SW_RW, H2 - ubase), nv = min(SWEEP_VT, W2 - v0);  // nu may be <= 0
    if (ub == 0) {
#pragma unroll
      for (int j = 0; j < SWEEP_VT; ++j) { cm[j] = -CUDART_INF_F; ca[j] = 0; }
    }
    // row-direction state of earlier column blocks (issued before the wait to hide the latency)
    float rold[SW_RW];
#pragma unroll
    for (int ul = 0; ul < SW_RW; ++ul)
      rold[ul] = (valid && vb > sc.vb0 && ul < nu) ? pu[(ubase + ul) * usd] : -CUDART_INF_F;
    if (CUT) {
#pragma unroll
      for (int ul = 0; ul < SW_RW; ++ul) rold[ul] = fmaxf(rold[ul], least);
    }

    if (!epi_wait(sm, a, t)) return;
    const uint32_t tacc = e.tbase + (t % SW_NACC) * SW_TILE_N + e.wg * (SW_RW * SWEEP_VT);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float s[64];
      tmem_ld64(tacc + half * 64, s);
      if (half == 1) epi_release(sm, t, e.lane);  // all values are in registers: hand the accumulator back
#pragma unroll
      for (int hl = 0; hl < SW_RW / 2; ++hl) {
        const int ul = half * (SW_RW / 2) + hl;
        if (ul < nu) {  // warp-uniform
          float* r = &s[hl * SWEEP_VT];
          if (nv < SWEEP_VT) {
#pragma unroll
            for (int j = 0; j < SWEEP_VT; ++j)
              if (j >= nv) r[j] = -CUDART_INF_F;  // padded columns never win a max
          }
          const int u = ubase + ul;
          float m;
          int arg;
          if (ARG) {
            max16_first(r, m, arg);
#pragma unroll
            for (int j = 0; j < SWEEP_VT; ++j) {
              if (r[j] > cm[j]) { cm[j] = r[j]; ca[j] = u; }  // strict: lowest u of this group wins ties
            }
          } else {
            m = r[0];
            arg = 0;
#pragma unroll
            for (int j = 1; j < SWEEP_VT; ++j) m = fmaxf(m, r[j]);
#pragma unroll
            for (int j = 0; j < SWEEP_VT; ++j) cm[j] = fmaxf(cm[j], r[j]);
          }
          m *= e.osc;  // memory holds scaled-back values; compare and store in that domain
          if (valid && (vb == sc.vb0 || m > rold[ul])) {  // strict: the lowest column block wins ties
            pu[u * usd] = m;
            if (ARG) pua[u * uasd] = __int_as_float(v0 + arg);
          }
        }
      }
    }
    if (ub == sc.n_ub - 1) {
      // end of a column block: group 1 publishes its partial column maxima, group 0 merges and stores
      uint64_t* bar = &sm.merge[(vb - sc.vb0) % SW_NMERGE];
      if (e.wg == 1) {
#pragma unroll
        for (int j = 0; j < SWEEP_VT; ++j) {
          if (valid && j < nv) {
            pv[(v0 + j) * vsd] = cm[j] * e.osc;
            if (ARG) pva[(v0 + j) * vasd] = __int_as_float(ca[j]);
          }
        }
        __threadfence_block();
        __syncwarp();
        if (e.lane == 0) mbar_arrive(bar);
      } else {
        const bool ok = mbar_wait(bar, ((vb - sc.vb0) / SW_NMERGE) & 1u, &sm.ctl, a.status, DEV_TIMEOUT_EPILOGUE);
        if (!__all_sync(0xffffffffu, ok)) return;
#pragma unroll
        for (int j = 0; j < SWEEP_VT; ++j) {
          if (valid && j < nv) {
            float* dst = pv + (v0 + j) * vsd;
            const float om = __ldcg(dst);
            float best = cm[j] * e.osc;
            int besta = ca[j];
            if (ARG) {
              float* dsta = pva + (v0 + j) * vasd;
              const int oa = __float_as_int(__ldcg(dsta));
              if (om > best || (om == best && oa < besta)) { best = om; besta = oa; }  // lowest u on ties
              *dsta = __int_as_float(besta);
            } else {
              best = fmaxf(best, om);
            }
            dst[0] = best;
          }
        }
      }
    }
    if (++ub == sc.n_ub) { ub = 0; ++vb; }
  }
  // mean channels: accumulator column r of an aux tile is F1[p] . (row-mean u=r | column-mean v=r-H2)
  const int naux = H2 + W2;
  for (int t = sc.t_main; t < sc.t_total; ++t) {
    if (!epi_wait(sm, a, t)) return;
    const uint32_t tacc = e.tbase + (t % SW_NACC) * SW_TILE_N + e.wg * 128;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int r0 = (t - sc.t_main) * SW_TILE_N + e.wg * 128 + half * 64;
      if (r0 < naux) {  // warp-uniform
        float s[64];
        tmem_ld64(tacc + half * 64, s);
#pragma unroll
        for (int j = 0; j < 64; ++j) {
          const int r = r0 + j;
          if (!valid) continue;
          if (r < H2) pum[r * umsd] = s[j] * e.osc;
          else if (r < naux) pv[(r - H2) * vsd + vss] = s[j] * e.osc;
        }
      }
    }
    epi_release(sm, t, e.lane);
  }
}

template <bool CUT>
__device__ void epilogue_compress(SweepSmem& sm, const SweepArgs& a, const SweepSched& sc, const EpiCtx& e) {
  const int H2 = a.d.H2, W2 = a.d.W2;
  const bool active = e.wg < a.kc;            // this warpgroup's channel exists (warp-uniform)
  const bool valid = e.valid && active;
  const uint32_t xusd = a.xu.sd, xvsd = a.xv.sd, ovsd = a.ov.sd;
  uint32_t ousd = a.ou.sd;
  // this thread's pixel and channel in sample b of each view; displacement d at ptr[d*sd], 32-bit offsets
  const int k = a.k0 + e.wg;
  const float* wu = a.xv.base + sc.b * a.xv.sb + e.p + (a.wu_slot0 + k * a.w_stride) * a.xv.ss;  // w_u[k][v]
  const float* wv = a.xu.base + sc.b * a.xu.sb + e.p + (a.wv_slot0 + k * a.w_stride) * a.xu.ss;  // w_v[k][u]
  float* ou = a.ou.base + sc.b * a.ou.sb + e.p + k * a.ou.ss;
  float* ov = a.ov.base + sc.b * a.ov.sb + e.p + k * a.ov.ss;
  // The first column block initialises the row sums, the others are added to them.  A later piece stores every block, into
  // a part of its own (slot = channel of this launch).
  uint32_t part_step = 0;
  if (CUT && sc.piece > 0) {
    ou = sweep_part(a, sc.tail, sc.vb0 - sc.part_vb0, e.wg) + (e.p - sc.m0);
    ousd = TILE_M;
    part_step = (uint32_t)a.part_slots * H2 * TILE_M;
  }

  // Both sums run on packed FP32 pairs (two neighbouring columns per fma.rn.f32x2), which halves the
  // instructions per cell: the epilogue warps share their schedulers' issue slots, and with scalar FMAs
  // those slots, not the tensor pipe, set the pace of this sweep.
  //   au2[j] = (w_u[v0+2j], w_u[v0+2j+1])         weights of this column block, per column pair
  //   cv2[j] = running (OV[v0+2j], OV[v0+2j+1])   over the rows of the column block
  // Cells outside the image hold S = 0 (TMA zero-fills the missing F2 rows) and get weight 0, so every
  // tile is processed whole and only the loads and stores at the edges are predicated.
  uint64_t au2[SWEEP_VT / 2], cv2[SWEEP_VT / 2];
  int vb = sc.vb0, ub = 0;
  for (int t = 0; t < sc.t_main; ++t) {
    const int v0 = vb * SWEEP_VT, u0 = ub * SWEEP_UT;
    const int nu = min(SWEEP_UT, H2 - u0), nv = min(SWEEP_VT, W2 - v0);
    if (ub == 0) {
      const float* wu_t = wu + v0 * xvsd;
#pragma unroll
      for (int j = 0; j < SWEEP_VT / 2; ++j) {
        const float lo = (valid && 2 * j < nv) ? __ldg(wu_t + (2 * j) * xvsd) : 0.f;
        const float hi = (valid && 2 * j + 1 < nv) ? __ldg(wu_t + (2 * j + 1) * xvsd) : 0.f;
        au2[j] = pack2(lo, hi);
        cv2[j] = 0ull;
      }
    }
    float av[SWEEP_UT];
    {
      const float* wv_t = wv + u0 * xusd;
#pragma unroll
      for (int ul = 0; ul < SWEEP_UT; ++ul) av[ul] = (valid && ul < nu) ? __ldg(wv_t + ul * xusd) : 0.f;
    }

    if (!epi_wait(sm, a, t)) return;
    const uint32_t tacc = e.tbase + (t % SW_NACC) * SW_TILE_N;
    if (active) {
      float* ou_t = ou + u0 * ousd;
      const bool first = vb == 0 || part_step != 0;
#pragma unroll
      for (int pr = 0; pr < SWEEP_UT / 2; ++pr) {
        float s[2 * SWEEP_VT];
        tmem_ld32(tacc + pr * 2 * SWEEP_VT, s);
        if (pr == SWEEP_UT / 2 - 1) epi_release(sm, t, e.lane);  // last read of this tile
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int ul = 2 * pr + h;
          const uint64_t av2 = pack2(av[ul], av[ul]);
          uint64_t r2 = 0ull;
#pragma unroll
          for (int j = 0; j < SWEEP_VT / 2; ++j) {
            const uint64_t s2 = pack2(s[h * SWEEP_VT + 2 * j], s[h * SWEEP_VT + 2 * j + 1]);
            r2 = j == 0 ? mul2(s2, au2[0]) : fma2(s2, au2[j], r2);
            cv2[j] = fma2(s2, av2, cv2[j]);
          }
          if (valid && ul < nu) {
            float* dst = ou_t + ul * ousd;
            const float r = sum2(r2) * e.osc;
            if (first) *dst = r;
            else atomicAdd(dst, r);  // same thread, same address in every column block: ordered
          }
        }
      }
    } else {
      epi_release(sm, t, e.lane);
    }
    if (ub == sc.n_ub - 1) {
      float* ov_t = ov + v0 * ovsd;
#pragma unroll
      for (int j = 0; j < SWEEP_VT / 2; ++j) {
        float lo, hi;
        unpack2(cv2[j], lo, hi);
        if (valid && 2 * j < nv) ov_t[(2 * j) * ovsd] = lo * e.osc;
        if (valid && 2 * j + 1 < nv) ov_t[(2 * j + 1) * ovsd] = hi * e.osc;
      }
    }
    if (++ub == sc.n_ub) { ub = 0; ++vb; ou += part_step; }
  }
}

// Test aid: writes the dense volume of a (small) problem so the tensor-core plumbing can be checked alone.
__device__ void epilogue_dump(SweepSmem& sm, const SweepArgs& a, const SweepSched& sc, const EpiCtx& e) {
  const int H2 = a.d.H2, W2 = a.d.W2, N1 = a.d.N1();
  const bool valid = e.p < N1;
  float* out = a.dump + ((size_t)sc.b * N1 + (valid ? e.p : 0)) * H2 * W2;
  int vb = 0, ub = 0;
  for (int t = 0; t < sc.t_main; ++t) {
    const int v0 = vb * SWEEP_VT, ubase = ub * SWEEP_UT + e.wg * SW_RW;
    const int nu = min(SW_RW, H2 - ubase), nv = min(SWEEP_VT, W2 - v0);
    if (!epi_wait(sm, a, t)) return;
    const uint32_t tacc = e.tbase + (t % SW_NACC) * SW_TILE_N + e.wg * 128;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float s[64];
      tmem_ld64(tacc + half * 64, s);
      if (half == 1) epi_release(sm, t, e.lane);
      if (valid) {
#pragma unroll
        for (int hl = 0; hl < SW_RW / 2; ++hl)
#pragma unroll
          for (int j = 0; j < SWEEP_VT; ++j) {
            const int ul = half * (SW_RW / 2) + hl;
            if (ul < nu && j < nv) out[(size_t)(ubase + ul) * W2 + v0 + j] = s[hl * SWEEP_VT + j] * e.osc;
          }
      }
    }
    if (++ub == sc.n_ub) { ub = 0; ++vb; }
  }
}

// The parts of a finished tail tile folded into piece 0's row results, in order (all threads of the CTA that finished last).
// Maxima: a later piece has the higher columns, so only a strictly larger value replaces.  Sums: block by block, the order
// in which a whole tile adds them, so that a sample's sums do not depend on the cut, which follows the batch and the row
// range.  One SM's loads are all that moves these bytes, so a thread takes four pixels of up to FOLD_ROWS rows at once and
// asks for several parts' values before it uses any (with one 4-byte load at a time a fold of 135 rows x 4 channels took as
// long as the sweep).
__device__ __forceinline__ void max4_first(float& v, float& arg, float o, float oarg) {
  if (o > v) { v = o; arg = oarg; }
}
template <int MODE>
__device__ void sweep_fold_pieces(const SweepArgs& a, const SweepSched& sc) {
  constexpr int NT = sw_threads(MODE), QUADS = TILE_M / 4, FOLD_ROWS = MODE == SWEEP_MAXAVG ? 4 : 2, FOLD_PARTS = MODE == SWEEP_COMPRESS ? 6 : 2;
  const int H2 = a.d.H2, n = (MODE == SWEEP_COMPRESS ? a.kc : 1) * H2 * QUADS;
  for (int i0 = threadIdx.x; i0 < n; i0 += FOLD_ROWS * NT) {
    float* dst[FOLD_ROWS];
    float* arg_dst[FOLD_ROWS];
    const float* part[FOLD_ROWS];   // the first part's values; part s is s * part_slots slots further on
    int cnt[FOLD_ROWS];
    float4 v[FOLD_ROWS], va[FOLD_ROWS];
#pragma unroll
    for (int r = 0; r < FOLD_ROWS; ++r) {
      const int i = i0 + r * NT, px = i % QUADS * 4, q = i / QUADS, k = q / H2, u = q - k * H2, p = sc.m0 + px;
      cnt[r] = i < n ? min(4, a.n_valid - p) : 0;
      if (cnt[r] <= 0) { cnt[r] = 0; dst[r] = arg_dst[r] = nullptr; part[r] = a.part; continue; }
      if (MODE == SWEEP_COMPRESS) dst[r] = a.ou.base + sc.b * a.ou.sb + p + (a.k0 + k) * a.ou.ss + u * a.ou.sd;
      else dst[r] = a.pu.base + sc.b * a.pu.sb + p + u * a.pu.sd;
      arg_dst[r] = MODE == SWEEP_MAXARGAVG ? a.pu_arg.base + sc.b * a.pu_arg.sb + p + u * a.pu_arg.sd : nullptr;
      part[r] = sweep_part(a, sc.tail, 0, k) + (size_t)u * TILE_M + px;
      v[r] = load4_cg(dst[r], cnt[r]);
      if (MODE == SWEEP_MAXARGAVG) va[r] = load4_cg(arg_dst[r], cnt[r]);
    }
    const size_t slot = (size_t)H2 * TILE_M, step = slot * a.part_slots;
    for (int s0 = 0; s0 < a.parts; s0 += FOLD_PARTS) {
      float4 o[FOLD_PARTS][FOLD_ROWS], oa[MODE == SWEEP_MAXARGAVG ? FOLD_PARTS : 1][FOLD_ROWS];
#pragma unroll
      for (int j = 0; j < FOLD_PARTS; ++j)
#pragma unroll
        for (int r = 0; r < FOLD_ROWS; ++r) {
          const bool ok = s0 + j < a.parts && cnt[r] > 0;
          const float* src = part[r] + (s0 + j) * step;
          // lanes past the image were never written: their values are loaded and dropped
          o[j][r] = ok ? __ldcg(reinterpret_cast<const float4*>(src)) : make_float4(0.f, 0.f, 0.f, 0.f);
          if (MODE == SWEEP_MAXARGAVG)
            oa[j][r] = ok ? __ldcg(reinterpret_cast<const float4*>(src + slot)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
      for (int j = 0; j < FOLD_PARTS; ++j) {
        if (s0 + j >= a.parts) break;
#pragma unroll
        for (int r = 0; r < FOLD_ROWS; ++r) {
          if (MODE == SWEEP_COMPRESS) {
            add4(v[r], o[j][r]);
          } else if (MODE == SWEEP_MAXARGAVG) {
            max4_first(v[r].x, va[r].x, o[j][r].x, oa[j][r].x);
            max4_first(v[r].y, va[r].y, o[j][r].y, oa[j][r].y);
            max4_first(v[r].z, va[r].z, o[j][r].z, oa[j][r].z);
            max4_first(v[r].w, va[r].w, o[j][r].w, oa[j][r].w);
          } else {
            v[r] = make_float4(o[j][r].x > v[r].x ? o[j][r].x : v[r].x, o[j][r].y > v[r].y ? o[j][r].y : v[r].y,
                               o[j][r].z > v[r].z ? o[j][r].z : v[r].z, o[j][r].w > v[r].w ? o[j][r].w : v[r].w);
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < FOLD_ROWS; ++r) {
      if (cnt[r] == 0) continue;
      store4(dst[r], v[r], cnt[r]);
      if (MODE == SWEEP_MAXARGAVG) store4(arg_dst[r], va[r], cnt[r]);
    }
  }
}

// ---------------------------------------------------------------------------------- kernel
// CUT: the launch has tail pieces.  A launch without any runs the kernel without their bookkeeping, whose registers cost
// the compression epilogue 10 % (it is at its register limit: 897 -> 990 us at 135 x 240).
template <int MODE, bool CUT>
__global__ void __launch_bounds__(sw_threads(MODE), 1)
sweep_kernel(const __grid_constant__ CUtensorMap tm_f1, const __grid_constant__ CUtensorMap tm_f2,
             const __grid_constant__ CUtensorMap tm_aux, const SweepArgs a) {
  if (*reinterpret_cast<volatile int*>(a.status) != 0) return;  // an earlier CTA gave up: do not pile on

  extern __shared__ uint8_t smem_raw[];
  const uint32_t pad = (1024u - (smem_u32(smem_raw) & 1023u)) & 1023u;
  SweepSmem& sm = *reinterpret_cast<SweepSmem*>(smem_raw + pad);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const SweepSched sc = sweep_sched<MODE, CUT>(a, blockIdx.x);

  if (threadIdx.x == 0) {
    mbar_init(&sm.f1_full, 1);
    for (int s = 0; s < SW_NSTAGE; ++s) { mbar_init(&sm.full[s], 1); mbar_init(&sm.empty[s], 1); }
    for (int i = 0; i < SW_NACC; ++i) { mbar_init(&sm.acc_full[i], 1); mbar_init(&sm.acc_empty[i], sw_epi_warps(MODE)); }
    for (int i = 0; i < SW_NMERGE; ++i) mbar_init(&sm.merge[i], 4);  // the four warps of max/avg group 1
    wait_ctl_init(&sm.ctl, a.wait_limit_ns);
    fence_barrier_init();
    prefetch_tensormap(&tm_f1);
    prefetch_tensormap(&tm_f2);
    if (MODE == SWEEP_MAXAVG || MODE == SWEEP_MAXARGAVG) prefetch_tensormap(&tm_aux);
  }
  if (warp == 1) {
    tmem_alloc(&sm.tmem_base, SW_TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  if (warp == 0) {
    if (lane == 0) sweep_producer(sm, a, sc, &tm_f1, &tm_f2, &tm_aux);
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) sweep_mma(sm, a, sc);
    __syncwarp();
  } else {
    EpiCtx e;
    const int q = warp & 3;  // tcgen05.ld lets a warp read TMEM lanes 32*(warp%4) .. +31 only
    e.wg = (warp - 2) >> 2;
    e.lane = lane;
    e.p = sc.m0 + q * 32 + lane;
    e.valid = e.p < a.n_valid;
    e.tbase = sm.tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    e.osc = a.out_scale != nullptr ? __ldg(a.out_scale) : 1.f;
    if (MODE == SWEEP_MAXAVG) epilogue_maxavg<false, CUT>(sm, a, sc, e);
    else if (MODE == SWEEP_MAXARGAVG) epilogue_maxavg<true, CUT>(sm, a, sc, e);
    else if (MODE == SWEEP_COMPRESS) epilogue_compress<CUT>(sm, a, sc, e);
    else epilogue_dump(sm, a, sc, e);
  }

  tc_fence_before();
  __syncthreads();
  if (wait_ctl_aborted(&sm.ctl)) {
    // A wait ran out.  Give copies that are still in flight time to land before the CTA's shared
    // memory is released (TMA latency is a few microseconds), then free TMEM as usual.
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(sm.tmem_base, SW_TMEM_COLS);
  }
  if constexpr (CUT) {
    const SweepSched tail_sc = [&] {
      if constexpr (MODE == SWEEP_COMPRESS) {
        // worked out again: kept over the compression epilogue, its registers would be spilled there
        int block;
        asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(block));
        return sweep_sched<MODE, CUT>(a, block);
      } else {
        return sc;
      }
    }();
    if (tail_sc.tail >= 0 && !wait_ctl_aborted(&sm.ctl)) {  // uniform over the CTA after the barrier above
      __threadfence();  // this thread's results before the count ...
      __syncthreads();
      if (threadIdx.x == 0) sm.last_piece = atomicAdd(a.tail_count + tail_sc.tail, 1) == a.pieces - 1;
      __syncthreads();
      if (sm.last_piece) {
        __threadfence();  // ... and the count before the other pieces' results
        sweep_fold_pieces<MODE>(a, tail_sc);
        if (threadIdx.x == 0) a.tail_count[tail_sc.tail] = 0;  // as the next launch expects it
      }
    }
  }
}

// How the tail tiles are cut, in units of one 256-column tile's time: a CTA costs about two tiles of prologue, a fold
// reads (parts + 1) * slots * H2 rows of 128 values through one SM (about 677 rows per tile time).  Pieces must save a quarter
// of the tail and a whole tile to be used: a wave with idle SMs runs its tiles faster than a full one, so little is left of
// smaller predicted savings (106 tail tiles of 135 x 240 in four pieces, predicted 0.86: max/avg sweep 588 -> 551 us, but
// the compression sweep no faster).  Whole and cut tiles measured (us per launch, C = 256, FP16, max/avg and compression):
// 1 x 48 x 64: 65 and 44, 40 and 25; 1 x 55 x 128: 122 and 81, 113 and 83; 4 x 55 x 128: 240 and 199, 231 and 218;
// 3 x 47 x 155: 246 and 171, 199 and 158; 8 x 47 x 156: 486 and 414, 349 and 339; 1 x 55 x 128 against 27 x 64: 54 and 46,
// 37 and 31.  Adding the sums block by block costs a compression sweep 1 to 7 us against one sum per piece.
TileSplit sweep_split(const Dims& d, int slots, bool sums) {
  const long long tiles = (long long)d.B * ((d.N1() + TILE_M - 1) / TILE_M);
  const int n_ub = (d.H2 + SWEEP_UT - 1) / SWEEP_UT, n_vb = (d.W2 + SWEEP_VT - 1) / SWEEP_VT;
  const int rest = (int)(tiles % SM_COUNT);
  TileSplit r{(int)tiles, (int)tiles, 1, 0, 0};
  if (rest == 0) return r;
  double best = 0, whole = 0;
  for (int n = 1; n <= n_vb && n <= MAX_PIECES; ++n) {
    const double waves = (rest * n + SM_COUNT - 1) / SM_COUNT;
    const int parts = sums ? n_vb - piece_start(n_vb, n, 1) : n - 1;
    const double cost = waves * ((n_vb + n - 1) / n * n_ub + 2) + (n > 1 ? (parts + 1) * (double)slots * d.H2 / 677.0 + 0.5 : 0.0);
    if (n == 1) best = whole = cost;
    if (cost < best && cost < 0.75 * whole && cost < whole - 1) { best = cost; r.pieces = n; r.parts = parts; }
  }
  if (r.pieces > 1) {
    r.whole_tiles = (int)tiles - rest;
    r.part_floats = (size_t)rest * r.parts * slots * d.H2 * TILE_M;
  }
  return r;
}

template <int MODE, bool CUT>
static cudaError_t launch_one(const SweepArgs& a, const CUtensorMap& tm_f1, const CUtensorMap& tm_f2,
                              const CUtensorMap& tm_aux, cudaStream_t stream) {
  auto kern = sweep_kernel<MODE, CUT>;
  static DeviceOnce configured;  // the attribute is per device and stays set
  cudaError_t err = configured.run([&] {
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SW_SMEM_BYTES);
  });
  if (err != cudaSuccess) return err;
  const int tiles_per_sample = (a.d.N1() + TILE_M - 1) / TILE_M;
  const int tiles = a.d.B * tiles_per_sample;
  const dim3 grid(a.whole_tiles + (tiles - a.whole_tiles) * a.pieces);
  kern<<<grid, sw_threads(MODE), SW_SMEM_BYTES, stream>>>(tm_f1, tm_f2, tm_aux, a);
  return cudaGetLastError();
}

template <int MODE>
static cudaError_t launch_mode(const SweepArgs& a, const CUtensorMap& tm_f1, const CUtensorMap& tm_f2,
                               const CUtensorMap& tm_aux, cudaStream_t stream) {
  return a.pieces > 1 ? launch_one<MODE, true>(a, tm_f1, tm_f2, tm_aux, stream)
                      : launch_one<MODE, false>(a, tm_f1, tm_f2, tm_aux, stream);
}

cudaError_t launch_sweep(const SweepArgs& a, const CUtensorMap& tm_f1, const CUtensorMap& tm_f2,
                         const CUtensorMap& tm_aux, cudaStream_t stream) {
  switch (a.mode) {
    case SWEEP_MAXAVG: return launch_mode<SWEEP_MAXAVG>(a, tm_f1, tm_f2, tm_aux, stream);
    case SWEEP_MAXARGAVG: return launch_mode<SWEEP_MAXARGAVG>(a, tm_f1, tm_f2, tm_aux, stream);
    case SWEEP_DUMP: return launch_one<SWEEP_DUMP, false>(a, tm_f1, tm_f2, tm_aux, stream);
    case SWEEP_COMPRESS:
      if (a.kc < 1 || a.kc > KC_MAX_PER_SWEEP) return cudaErrorInvalidValue;
      return launch_mode<SWEEP_COMPRESS>(a, tm_f1, tm_f2, tm_aux, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace sfb
