// Internal launcher interface between the C-ABI layer (c_abi.cu) and the kernel files.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <utility>

namespace sfb {

// Host side.  Runs a per-device set-up step (cudaFuncSetAttribute and the like) once per device instead of before every launch.
// Racing first calls may both run it, which is harmless for idempotent settings.
struct DeviceOnce {
  std::atomic<bool> done[64];
  DeviceOnce() { for (auto& d : done) d.store(false); }
  template <class F>
  cudaError_t run(F&& f) {
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    if (dev < 0 || dev >= 64) return f();
    if (done[dev].load(std::memory_order_acquire)) return cudaSuccess;
    err = f();
    if (err == cudaSuccess) done[dev].store(true, std::memory_order_release);
    return err;
  }
};

// Host side.  Launch of a kernel that begins with follow_previous_kernel(): it may be brought onto the device while the kernel before it in the
// stream is still running, and waits there for that kernel's end instead of being launched after it.  Errors are those of cudaGetLastError, as
// after <<<>>>.  A call is up to 39 launches that depend on one another, some 1.4 us apart when each is launched after the one before: max/mean
// channels 1 x 48 x 64 47.2 -> 40.0 us, inference 1 x 55 x 128 with four levels 262 -> 239, 4 x 55 x 128 697 -> 687, the drop-in operators of a
// training step 2 x 48 x 64 409 -> 384, twelve lookups 4 x 55 x 128 135 -> 114.
template <class... Params, class... Args>
void launch_with(bool early, void (*kernel)(Params...), dim3 grid, dim3 block, size_t shared_bytes, cudaStream_t stream, Args&&... args) {
  cudaLaunchAttribute attribute{};
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config{};
  config.gridDim = grid;
  config.blockDim = block;
  config.dynamicSmemBytes = shared_bytes;
  config.stream = stream;
  config.attrs = &attribute;
  config.numAttrs = early ? 1 : 0;
  (void)cudaLaunchKernelEx(&config, kernel, std::forward<Args>(args)...);
}
template <class... Params, class... Args>
void launch_next(void (*kernel)(Params...), dim3 grid, dim3 block, size_t shared_bytes, cudaStream_t stream, Args&&... args) {
  launch_with(true, kernel, grid, block, shared_bytes, stream, std::forward<Args>(args)...);
}
// The same when the device is empty again: for few long blocks behind a kernel that holds the SMs unevenly, which would come to lie two to an SM
// while others have none.
template <class... Params, class... Args>
void launch_after(void (*kernel)(Params...), dim3 grid, dim3 block, size_t shared_bytes, cudaStream_t stream, Args&&... args) {
  launch_with(false, kernel, grid, block, shared_bytes, stream, std::forward<Args>(args)...);
}

// Problem size of one op call (one pyramid level).  N1 = H1*W1 image-1 pixels, N2 = H2*W2.
struct Dims {
  int B, H1, W1, H2, W2, C, Kc;
  __host__ __device__ int N1() const { return H1 * W1; }
  __host__ __device__ int N2() const { return H2 * W2; }
  __host__ __device__ int aux_rows() const { return H2 + W2; }
};

// Tile constants shared by host and device code.
constexpr int TILE_M = 128;   // TMEM lanes = rows of one accumulator tile
constexpr int KBLK = 32;      // fp32 elements in one 128-byte swizzled row
#ifndef SFB_MAX_KB
#define SFB_MAX_KB 8
#endif
constexpr int MAX_KB = SFB_MAX_KB;  // feature dimension C <= MAX_KB * KBLK
constexpr int MAX_C = MAX_KB * KBLK;
// Image-2 rows and columns of a correlation tile (256 accumulator columns): wide, or narrow where that needs clearly fewer tiles
// (sweep_narrow).
constexpr int SWEEP_UT = 8, SWEEP_VT = 32;
constexpr int SWEEP_UT_NARROW = 16, SWEEP_VT_NARROW = 16;
constexpr int GG_ROW_UT = 8;  // row tile of the image-2-major gradient GEMM: 8 x 16 image-2 pixels = 128 TMEM lanes
constexpr int GG_ROW_VT = 16;
constexpr int GG_UT = 4;      // a K block of the image-1-major gradient GEMM: 4 image-2 rows x 16 columns
constexpr int GG_VT = 16;
constexpr int GG_KJ = 32;     // and of the image-2-major one: 32 image-1 pixels
constexpr int GG_SJ = 64, GG_SM = 4;  // over a stored G: 64 pixels, tiles of 4 blocks of 4 x 16 image-2 pixels
constexpr int KC_MAX_PER_SWEEP = 4;  // attention channels handled by one compression sweep
constexpr int MAX_FUSED_LEVELS = 4;  // levels of a pyramid that the kernels of a call take in one launch

// 16-bit operand kinds of the contractions (0 = none: TF32 operands in FP32 storage).
#ifndef SFB_OP16_KINDS
#define SFB_OP16_KINDS
enum : int { OP16_NONE = 0, OP16_BF16 = 1, OP16_FP16 = 2 };
#endif
enum SweepMode : int { SWEEP_MAXAVG = 0, SWEEP_MAXARGAVG = 1, SWEEP_COMPRESS = 2, SWEEP_DUMP = 3 };
enum GradMode : int { GRAD_MAXAVG = 0, GRAD_COMPRESS = 1, GRAD_FUSED = 2 };
// Forms of the gradient GEMM.  Rows are image-1 pixels (output gF1) or image-2 pixels (gF2); G is generated, or, with 16-bit operands,
// generated once: the image-1-major form stores its blocks and the image-2-major form reads them back.
enum GradForm : int { GRAD_IMAGE1 = 0, GRAD_IMAGE2 = 1, GRAD_IMAGE1_STORING = 2, GRAD_IMAGE2_STORED = 3 };
__host__ __device__ constexpr bool grad_is_image2(int form) { return form == GRAD_IMAGE2 || form == GRAD_IMAGE2_STORED; }

// A tensor indexed by (sample b, displacement d, slot, image-1 pixel p) with the pixel fastest:
// element at base + b*sb + d*sd + slot*ss + p.  Two instances of this are used:
//   "packed"         workspace arrays (B, D, slots, n1p): sb = D*slots*n1p, sd = slots*n1p, ss = n1p
//   "channels-first" user tensors   (B, slots, D, N1)  : sb = slots*D*N1,  sd = N1,        ss = D*N1
// (the layout torch's Conv3d produces and consumes at the call site, core/corr.py:437-446).
struct PixView {
  float* base;
  long long sb;      // elements between samples
  uint32_t sd, ss;   // elements between displacements / slots (one sample spans < 2^32 elements: host-checked)
};

// Correlation sweep.  Everything indexed by an image-1 pixel is read and written through PixViews, so a
// warp's 32 lanes (32 consecutive pixels) touch one or two 128-byte lines per access.
//   max/avg    : outputs pu (per u) / pv (per v): slots 0 = max, 1 = mean; argmax (int32 bits) in pu_arg / pv_arg
//   compression: weights  w_v[k][u] = xu(b, u, wv_slot0 + k*w_stride, p),  w_u[k][v] = xv(b, v, wu_slot0 + k*w_stride, p)
//                outputs  ou(b, u, k, p) = sum_v S*w_u,  ov(b, v, k, p) = sum_u S*w_v
// Lanes with p >= n_valid compute but never touch memory (n_valid = n1p for packed arrays, N1 otherwise).
struct SweepArgs {
  Dims d;
  int mode;
  int n_valid;
  int k0, kc;            // compression: first channel and number of channels (<= KC_MAX_PER_SWEEP) of this launch
  PixView pu, pv, pu_arg, pv_arg;
  PixView xu, xv;
  int wu_slot0, wv_slot0, w_stride;
  PixView ou, ov;
  int op16;              // operands are 16-bit copies (64 channels per 128-byte row, tcgen05.mma kind::f16) instead of
                         // TF32: OP16_BF16 or OP16_FP16
  const float* out_scale;  // device scalar every output value is multiplied by before it is stored (null = 1): undoes
                           // the power-of-two scaling of FP16 operands
  float* dump;           // SWEEP_DUMP: dense S (B,N1,H2,W2), test use only
  int* status;           // device status word
  unsigned long long wait_limit_ns;  // time limit of one device-side wait; 0 = the default (2 s)
  int drop_last_load;    // test hook: the producer leaves out its last F2 block, so that one wait runs out
  // Tiles past `whole_tiles` are done by `pieces` CTAs each (TileSplit); part is unused when pieces is 1.
  int whole_tiles, pieces, parts, part_slots;
  float* part;
  bool narrow;           // sweep_narrow of this shape and mode (set by the launcher)
};

// How a launch of equal tiles fills the SMs: whole_tiles CTAs do one tile each, every further tile is done by `pieces`
// CTAs, which need part_floats floats of scratch.
constexpr int SM_COUNT = 148;
constexpr int MAX_PIECES = 16;
struct TileSplit { int tiles, whole_tiles, pieces, parts; size_t part_floats; };   // parts: results in scratch per tile and slot
// Whether a sweep over this image 2 runs on narrow tiles; sums: the compression, whose row results are added up.  It follows the
// shape of image 2 alone: the width of a tile is the order in which the compression adds up a row, and a sample's sums must not
// depend on the batch or the row range.  A narrow tile takes as long as a wide one for max (/ arg-max) and 1.36 (two channels) to
// 1.6 (four) times as long for the sums.  4 x 55 x 128 against 128 x 16, wide and narrow (us): maxima with arg-max 109 and 57,
// sums of two and four channels 66 and 42, 83 and 61; against 128 x 48: 155 and 117, 112 and 115, 164 and 197.
// What the line costs: sums over 2 x 48 x 64 against 64 x 48, where three narrow blocks cut the tail better than two wide ones, take
// 26 and 35 us instead of 20 and 30.
__host__ __device__ inline bool sweep_narrow(const Dims& d, bool sums) {
  const int wide = ((d.H2 + SWEEP_UT - 1) / SWEEP_UT) * ((d.W2 + SWEEP_VT - 1) / SWEEP_VT);
  const int narrow = ((d.H2 + SWEEP_UT_NARROW - 1) / SWEEP_UT_NARROW) * ((d.W2 + SWEEP_VT_NARROW - 1) / SWEEP_VT_NARROW);
  return sums ? 5 * narrow <= 3 * wide : 4 * narrow <= 3 * wide;
}
// slots: row results per pixel (max and argmax; channels of a launch); sums: they are added up, not compared
TileSplit sweep_split(const Dims& d, int slots, bool sums);
// The same for the levels of a pyramid that share a launch (same image 1).
void sweep_split_levels(const Dims* d, int levels, int slots, bool sums, TileSplit* out);

// Host side.  Makespan of a launch on SM_COUNT SMs with one block each at a time: groups of equal blocks, which start in the
// order in which they are added wherever an SM is free.
class BlockQueue {
 public:
  void add(int blocks, double length) {
    while (blocks > 0) {
      std::pop_heap(free_, free_ + n_, later);   // the SMs that are free first
      Sms& first = free_[n_ - 1];
      if (blocks >= first.count || n_ == MAX_GROUPS) {
        blocks -= first.count;
        first.at += length;
      } else {
        first.count -= blocks;
        free_[n_] = Sms{first.at + length, blocks};
        blocks = 0;
        std::push_heap(free_, free_ + n_, later);
        ++n_;
      }
      std::push_heap(free_, free_ + n_, later);
    }
  }
  double makespan() const {
    double most = 0;
    for (int i = 0; i < n_; ++i) most = std::max(most, free_[i].at);
    return most;
  }

 private:
  struct Sms { double at; int count; };
  static bool later(const Sms& x, const Sms& y) { return x.at > y.at; }
  static constexpr int MAX_GROUPS = 32;   // SMs that become free together; past that many groups a remainder counts as a whole one
  Sms free_[MAX_GROUPS] = {{0.0, SM_COUNT}};
  int n_ = 1;
};

// What a makespan is not below: no SM idle, and the longest block.
class BlockWork {
 public:
  void add(int blocks, double length) {
    if (blocks <= 0) return;
    total_ += blocks * length;
    longest_ = std::max(longest_, length);
  }
  double bound() const { return std::max(total_ / SM_COUNT, longest_); }

 private:
  double total_ = 0, longest_ = 0;
};
// Host side.  The cut (n0, n1) of the blocks of two groups, 1 <= n0 <= most0 and 1 <= n1 <= min(n0, most1), that clearly (by a twentieth)
// undercuts the ones before it.  fill(blocks, n0, n1) adds a cut's blocks and returns what the launch costs beside them.  Of up to 136 cuts
// those whose work alone shows that they do not are left out: the size query of a backward of 2 x 55 x 128 with four levels, four searches, took
// 130 us with all of them, 7 now.
struct LevelCut { int n0, n1; };
template <class Fill>
LevelCut cheapest_cut(int most0, int most1, Fill&& fill) {
  LevelCut cut{1, 1};
  double best = 0;
  for (int n0 = 1; n0 <= most0; ++n0) {
    for (int n1 = 1; n1 <= std::min(n0, most1); ++n1) {
      if (best > 0) {
        BlockWork work;
        const double beside = fill(work, n0, n1);
        if (work.bound() * (1 - 1e-9) + beside >= 0.95 * best) continue;   // (less than the rounding of either)
      }
      BlockQueue queue;
      const double beside = fill(queue, n0, n1), cost = queue.makespan() + beside;
      if (best == 0 || cost < 0.95 * best) {
        best = cost;
        cut = LevelCut{n0, n1};
      }
    }
  }
  return cut;
}

// Gradient GEMM.  G = dLoss/dS is generated from two "interleaved" operand sets: for every displacement
// and image-1 pixel the R4 values (slots) that pixel contributes, in groups of four:
//   XU (B, H2, R4/4, n1p, 4)  values that depend on (pixel, u);  XV (B, W2, R4/4, n1p, 4)  (pixel, v)
// n1p = N1 rounded up to a multiple of 128 (padding is zero), R4 = slots rounded up to a multiple of 4.
// One group of four slots of 32 consecutive pixels is 512 contiguous bytes: a 16-byte load per lane, or one
// TMA box row, and conflict-free 16-byte shared-memory reads after a TMA copy.
//   GRAD_COMPRESS: G[p,u,v] = sum_r XU[u,p,r] * XV[v,p,r]            (2 slots per channel, zero padded)
//   GRAD_MAXAVG  : XU slots (mean-gradient / W2, 1, max-gradient, argmax bits), XV slots (1, mean-gradient / H2,
//                  max-gradient, argmax bits); the mean terms are added, the constants are not read:
//                  G[p,u,v] = XU[u,p,0] + XV[v,p,1]
//                             + (XU[u,p,3]==v ? XU[u,p,2] : 0) + (XV[v,p,3]==u ? XV[v,p,2] : 0)
//   GRAD_FUSED   : group 0 as GRAD_MAXAVG, groups 1.. as GRAD_COMPRESS; G is the sum of both
struct GradArgs {
  Dims d;
  int mode;
  int form;              // GradForm
  int R4;                // slots per pixel in the interleaved operands: 4 or 8
  int n1p;               // padded pixel count of the interleaved operands
  int accumulate;        // 0: out = result, 1: out += result (later channel chunks of the compression op)
  int out_cf;            // 0: out is (B, pixels, C); 1: out is (B, C, pixels), the layout of the model's feature maps
  float out_scale;       // the result is multiplied by this before it is stored / added (out_cf only)
  int op16;              // G and the feature copies are 16-bit (tcgen05.mma kind::f16) instead of TF32: OP16_BF16 / OP16_FP16
  const float* dev_scale;  // device scalar the result is multiplied by as well (null = 1), see SweepArgs::out_scale
  const float* xu;
  const float* xv;
  float* out;            // gF1 (B,N1,C) or gF2 (B,N2,C)
  int* status;
  unsigned long long wait_limit_ns;  // time limit of one device-side wait; 0 = the default (2 s)
  int whole_tiles, pieces;           // as in SweepArgs, here with pieces of the K sweep (TileSplit)
  int parts, part0;                  // parts of a cut tile in scratch; piece i is part0 + i of them (-1: the output)
  float* part;
  int b0;                            // first sample of the launch, which does d.B of them
  uint8_t* stored;                   // G of those samples (the storing and the stored form), grad_stored_bytes each
};
// Stored G of a sample: [block of 4 image-2 rows x 16 columns, column blocks outermost][n1p image-1 pixels][64 16-bit values], the 16-byte
// chunks of a pixel's 128 bytes in the order of the 128-byte swizzle (chunk index ^ pixel % 8), so that a run of pixels is an operand
// as it lies there.
inline size_t grad_stored_bytes(const Dims& d, int n1p) {
  return (size_t)((d.H2 + GG_UT - 1) / GG_UT) * ((d.W2 + GG_VT - 1) / GG_VT) * n1p * (GG_UT * GG_VT * 2);
}
// Stored G of a launch at most: 4 GiB, a fortieth of the device's memory and enough for launches of several waves (two samples of
// 135 x 240 on itself).  Larger batches take several launches; a sample beyond it generates G twice.
constexpr size_t GRAD_STORED_LIMIT = (size_t)1 << 32;
TileSplit grad_split(const Dims& d, int form);
// The same for the levels of a pyramid that share a launch (same image 1).  Image-1-major: the tiles of all levels but the first go to
// scratch as a whole, to be added up.
void grad_split_levels(const Dims* d, int levels, int form, TileSplit* out);

// Launchers, here and below: the returned error is taken off the runtime, so a caller must pass it on; dropping it does not
// compile (unused results are errors in this build).

// One source of an interleaved slot: dst[b][d][slot/4][p][slot%4] = scale * src[b][p][k][d] (raw copy when scale == 0);
// src is (B, N1, Ksrc, D).  A null src makes the slot the constant `scale` (zero by default) for every valid pixel.
struct SlotSource {
  const void* src;
  int Ksrc, k;
  float scale;
  int dev;   // 0: nothing more; i > 0: the value is multiplied by dev_scales[i - 1] as well (FP16 operands: the
             // power-of-two scales of the gradient and weight tensors, known on the device only)
};
constexpr int MAX_SLOTS = 8;
struct SlotSources {
  SlotSource s[MAX_SLOTS];
  const float* dev_scales;  // may be null when no slot has dev != 0
};
// Same, from channels-first sources: dst[b][d][q][p][j] = scale * src[b][k][d][p], src is (B, Ksrc, D, N1); the groups of four
// slots of several operands in one launch (pack_launches, for very large batches).
struct PackGroup {
  SlotSource s[4];
  float4* dst;    // the operand (B, D, Qtot, n1p, 4)
  int D, Qtot, q; // q: this group
  const float* dev_scales;
};
constexpr int MAX_PACK_GROUPS = 6 * MAX_FUSED_LEVELS;
struct PackGroups {
  PackGroup g[MAX_PACK_GROUPS];
  int count;
  void add(const SlotSources& src, float* dst, int D, int R4, int Qtot, int q0) {
    for (int q = 0; q < R4 / 4; ++q) {
      PackGroup& x = g[count++];
      for (int j = 0; j < 4; ++j) x.s[j] = src.s[4 * q + j];
      x.dst = reinterpret_cast<float4*>(dst);
      x.D = D; x.Qtot = Qtot; x.q = q0 + q;
      x.dev_scales = src.dev_scales;
    }
  }
};
inline int pack_groups_per_launch(int B) { return std::max(1, std::min(MAX_PACK_GROUPS, 65535 / B)); }
inline int pack_launches(int groups, int B) { return (groups + pack_groups_per_launch(B) - 1) / pack_groups_per_launch(B); }
[[nodiscard]] cudaError_t launch_pack_interleaved_cf(const PackGroups& groups, int B, int N1, int n1p, cudaStream_t stream);
// The same from sources (B, N1, Ksrc, D).
[[nodiscard]] cudaError_t launch_pack_interleaved(const PackGroups& groups, int B, int N1, int n1p, cudaStream_t stream);

// Workspace header: the status word, then (64 bytes in) the scale slots of the FP16 operand kind, SCALE_LEVEL for every level of the
// call, all cleared by launch_prepare.  amax slots hold float bits (atomicMax), the others floats; every scale is a power of two.
constexpr size_t WS_HEADER_BYTES = 1024, WS_SCALES_OFFSET = 64;
enum : int {
  SCALE_AMAX_F1 = 0, SCALE_AMAX_F2 = 1, SCALE_AMAX_G = 2, SCALE_AMAX_A = 3,
  SCALE_F1 = 4, SCALE_F2 = 5, SCALE_INV_F1F2 = 6,   // F1h = fp16(s1 F1), F2h = fp16(s2 F2), sweep outputs * 1/(s1 s2)
  SCALE_GA = 7, SCALE_G = 8, SCALE_A = 9,           // gradient slots * sg (* sa when no weight multiplies them), weights * sa
  SCALE_INV_GF1 = 10, SCALE_INV_GF2 = 11,           // gF1 * 1/(sg sa s2), gF2 * 1/(sg sa s1)
  SCALE_TICKET = 12,                                // blocks of a running magnitude search that are done (the first level's)
  SCALE_LEVEL = 16                                  // slots of a level
};
static_assert(WS_SCALES_OFFSET + MAX_FUSED_LEVELS * SCALE_LEVEL * sizeof(float) <= WS_HEADER_BYTES, "scale slots");
// Makes the operand copies of a call's features and clears the workspace header.  TF32 operands (op16 = 0): F1r / F2r,
// rounded to nearest, and the row/column mean rows of F2 in aux.  16-bit operands: F1h / F2h / auxh, from the unrounded
// values (BF16, or FP16 after scaling by the powers of two this call derives from the arrays' largest magnitudes,
// scales[]).  Null arrays are left out.
[[nodiscard]] cudaError_t launch_prepare(const Dims& d, const float* F1, const float* F2, float* F1r, float* F2r, float* aux,
                           int* status, cudaStream_t stream, uint16_t* F1h = nullptr, uint16_t* F2h = nullptr,
                           uint16_t* auxh = nullptr, int op16 = 0, float* scales = nullptr);
// The same from the model's feature maps fmap1 (B, C, H1, W1) and, for every level of the call, fmap2[l] (B, C, H2, W2): F1r =
// round(scale1 * fmap1) transposed to (B, H1, W1, C), F2r = round(fmap2) transposed (core/corr.py:419-422 does this with
// permute().contiguous() and a division).
struct LevelOperands { float *F2r, *aux; uint16_t *F2h, *auxh; };
[[nodiscard]] cudaError_t launch_prepare_cf(const Dims* d, int levels, const float* fmap1, const float* const* fmap2, float scale1,
                              const LevelOperands* out, float* F1r, uint16_t* F1h, int* status, cudaStream_t stream, int op16 = 0,
                              float* scales = nullptr, float* const* pooled = nullptr);
// With `pooled`, the levels from the second on are made here, pooled[l] (= fmap2[l]) from the first.  The same without the rest, from and
// to arrays of any alignment:
[[nodiscard]] cudaError_t launch_pool_levels(const Dims* d, int levels, const float* fmap2, float* const* pooled, cudaStream_t stream);
// Gradients g[l] of the averages, added to the first level's, g0:
[[nodiscard]] cudaError_t launch_unpool_levels(const Dims* d, int levels, float* g0, const float* const* g, cudaStream_t stream);
// Largest |x| * premul of each array, `samples` runs of n values sb apart, combined into its amax slot (SCALE_* of a level), and then the
// multipliers that follow from the slots of every level: those of the features or (gradients) those of the gradient operands.
constexpr int ABSMAX_MAX = 4 * MAX_FUSED_LEVELS;
struct AbsmaxSource { const float* p; size_t n; long long sb; int samples; float premul; int slot; };
inline AbsmaxSource absmax_array(const float* p, size_t n, float premul, int slot) { return AbsmaxSource{p, n, (long long)n, 1, premul, slot}; }
[[nodiscard]] cudaError_t launch_absmax(const AbsmaxSource* src, int count, float* scales, int levels, bool gradients, cudaStream_t stream);
// Channel-major copies from the model's feature maps (B, C, rows*width) times `scale`, as 16-bit operands or (op16 = 0) TF32, padding
// zeroed (layouts below); image 1 and the levels of image 2 in one launch.
constexpr int MAX_MAP_COPIES = 1 + MAX_FUSED_LEVELS;
struct MapCopy {
  const float* src;
  void* dst;
  int rows, width, pitch, blocked;
  float scale;
  const float* scale16;
};
[[nodiscard]] cudaError_t launch_channel_major_cf(const MapCopy* copies, int count, int B, int C, int op16, cudaStream_t stream);
// Channel-major copies of pixel-major feature arrays (B, rows*width, C), as FP32 (of rounded values) or (op16 != 0) as 16-bit operands;
// `scale` is not read.  Padding is zeroed.
//   blocked = 0: dst (B, C, pitch) with pixel index row*width + x (rows = 1)
//   blocked = 1: dst (B, C, ceil(width/16), pitch, 16), element (row, x) at ((x/16)*pitch + row)*16 + x%16
[[nodiscard]] cudaError_t launch_channel_major(const MapCopy& c1, const MapCopy& c2, int B, int C, int op16, cudaStream_t stream);
// Transposes between a tensor of the reference's layout, pixels (B, N1, Kpix, D), of which channels k0 .. k0 + K - 1, and a packed array
// (B, D, R, n1p), of which slots r0 .. (32-bit values as they are).  Pack writes the packed array, zero for N1 <= p < n1p; unpack the
// other.  All tensors of a call in one launch.
constexpr int MAX_PATCH_JOBS = 4;
struct PatchJob {
  const void* pixels;
  float* packed;
  int K, D, Kpix, k0, R, r0;
};
[[nodiscard]] cudaError_t launch_pack(const PatchJob* jobs, int count, int B, int N1, int n1p, cudaStream_t stream);
[[nodiscard]] cudaError_t launch_unpack(const PatchJob* jobs, int count, int B, int N1, int n1p, cudaStream_t stream);
[[nodiscard]] cudaError_t launch_sweep(const SweepArgs& a, const CUtensorMap& tm_f1, const CUtensorMap& tm_f2,
                         const CUtensorMap& tm_aux, cudaStream_t stream);
// The levels of a pyramid in one launch (same image 1, mode, channels and operand type).
[[nodiscard]] cudaError_t launch_sweep_levels(const SweepArgs* a, int levels, const CUtensorMap& tm_f1, const CUtensorMap* tm_f2,
                                const CUtensorMap* tm_aux, cudaStream_t stream);
// Per level: y, channel-major features of the other image (K-major B operand); xu / xv, interleaved operands (xv is only read by the
// image-2-major form; the image-1-major form keeps its (pixel, v) slots in registers).  Several levels: GRAD_FUSED only.
struct GradMaps { CUtensorMap y[MAX_FUSED_LEVELS], xu[MAX_FUSED_LEVELS], xv[MAX_FUSED_LEVELS]; };
[[nodiscard]] cudaError_t launch_grad_gemm(const GradArgs* a, int levels, const GradMaps& maps, cudaStream_t stream);


// Attention weights A = softmax over d of Conv3d(2 -> Kc, 3x3x3, padding 1)(X) on channels-first tensors
// (core/corr.py:437-442): X (B, 2, D, H1, W1) with `x_sb` elements between samples, weight (Kc, 2, 3, 3, 3),
// bias (Kc), A (B, Kc, D, H1, W1).
struct AttentionDims {
  int B, Kc, D, H1, W1;
};
// One tensor that a module is applied to.  A launch takes several: those of a level or of a pyramid's levels, which differ in D alone.
constexpr int MAX_ATTENTION_JOBS = 2 * MAX_FUSED_LEVELS;
struct AttentionModules { const float *weight[2], *bias[2]; };   // null where no job uses the module
struct AttentionJob {
  AttentionDims d;
  int module;
  const float* x;
  long long x_sb;
  float* a;
};
// `status` (optional): a device status word for bounded waits.  With it blocks work on pixel tiles in shared memory (with the
// stencil's halo, zeros outside the image), fetched by TMA when W1 is a multiple of 4 and every x is 16-byte aligned, else
// by copies; without it every thread gathers its own neighbourhood.
[[nodiscard]] cudaError_t launch_attention_forward(const AttentionJob* jobs, int count, const AttentionModules& modules,
                                     cudaStream_t stream, int* status = nullptr);
int attention_forward_launches(const AttentionJob* jobs, int count, const int* status);  // its kernels
// Tiled fp32 tensor map without swizzle, zero fill out of bounds; dims / box innermost first, `strides_bytes` for
// dimensions 1 .. rank-1.  Implemented next to the other tensor maps (c_abi.cu).
[[nodiscard]] cudaError_t encode_plain_map(CUtensorMap* tm, const void* base, int rank, const uint64_t* dims,
                             const uint64_t* strides_bytes, const uint32_t* box);
// Floats of scratch the backward of these jobs needs for its per-block partial sums.
size_t attention_partial_floats(const AttentionDims* d, int count);
// Backward: `g` holds dLoss/dA on entry and the logit gradients on return; gx (B, 2, D, H1, W1) = add + dLoss/dX
// where `add` (same shape, `add_sb` elements between samples) may be null.  The gradients of a module, weight (Kc, 2, 3, 3, 3) and bias
// (Kc), are summed over the jobs that use it.
struct AttentionGradients { float *weight[2], *bias[2]; };
struct AttentionGradJob {
  AttentionDims d;
  int module;
  const float* x;
  long long x_sb;
  const float* a;
  float* g;
  const float* add;
  long long add_sb;
  float* gx;
};
[[nodiscard]] cudaError_t launch_attention_backward(const AttentionGradJob* jobs, int count, const AttentionModules& modules,
                                      const AttentionGradients& grads, float* partial, cudaStream_t stream, int* status = nullptr);
int attention_backward_launches(const AttentionGradJob* jobs, int count);


// Linear resampling along the displacement axis (core/corr.py:459-467: trilinear interpolate with unchanged H1, W1):
// in (B, K, Dl, N1) -> K channels of a larger tensor, out[b] at out + b*out_sb, each (K, D0, N1); Dl <= D0.  A launch takes the
// volumes of several levels.
constexpr int MAX_RESAMPLE_JOBS = 2 * MAX_FUSED_LEVELS;
struct ResampleJob {
  const float* in;
  float* out;
  long long out_sb;
  int Dl, D0;
};
[[nodiscard]] cudaError_t launch_upsample_displacement(const ResampleJob* jobs, int count, int B, int K, int N1, cudaStream_t stream);
// Its adjoint: in (B, K, Dl, N1) is written, from the gradient of those K channels (out is read).
struct ResampleAdjointJob {
  const float* gout;
  long long gout_sb;
  float* gin;
  int Dl, D0;
};
[[nodiscard]] cudaError_t launch_upsample_displacement_adjoint(const ResampleAdjointJob* jobs, int count, int B, int K, int N1,
                                                 cudaStream_t stream);

// Lookup on an aggregated 3D cost volume (the reference's CorrBlock1D, core/corr.py:513-624).
// corr (B, dim, D, H1, W1); pyramid = levels 1 .. levels-1 back to back, level l being (B, dim, D >> l, H1, W1);
// coord: one displacement component per pixel, (B, H1, W1) with `coord_sb` elements between samples;
// out (B, levels*dim*(2*radius+1), H1, W1).
constexpr int LOOKUP_MAX_LEVELS = 8;
struct LookupDims {
  int B, dim, D, H1, W1, levels, radius;
};
size_t lookup_pyramid_floats(const LookupDims& d);
[[nodiscard]] cudaError_t launch_lookup_pyramid(const LookupDims& d, const float* corr, float* pyramid, cudaStream_t stream);
struct LookupCall {
  const float *corr, *pyramid, *coord;
  long long coord_sb;
  float* out;
  int clamp_unit;
};
[[nodiscard]] cudaError_t launch_lookup_forward(const LookupDims& d, const LookupCall& c, cudaStream_t stream);
// The same for two volumes that differ in D alone, in one launch.
[[nodiscard]] cudaError_t launch_lookup_pyramid_pair(const LookupDims (&d)[2], const float* const (&corr)[2], float* const (&pyramid)[2],
                                       cudaStream_t stream);
[[nodiscard]] cudaError_t launch_lookup_forward_pair(const LookupDims (&d)[2], const LookupCall (&c)[2], cudaStream_t stream);
// Gradients of several lookups: each adds the gradients of its windows to the accumulator of its volume (zero before the first),
// for one or two volumes that differ in D alone; the accumulator is then folded into the gradient of the volume.
struct LookupGradient {
  const float *gout, *coord;
  long long coord_sb;
  float* acc;
  int clamp_unit;
};
size_t lookup_accumulator_floats(const LookupDims& d, int clamp_unit);
[[nodiscard]] cudaError_t launch_lookup_accumulate(const LookupDims* d, const LookupGradient* g, int volumes, cudaStream_t stream);
[[nodiscard]] cudaError_t launch_lookup_gradient_fold(const LookupDims& d, const float* acc, float* gcorr, int clamp_unit, cudaStream_t stream);
// gcorr and gpyramid (same sizes as corr / pyramid) are overwritten; gpyramid is scratch.
[[nodiscard]] cudaError_t launch_lookup_backward(const LookupDims& d, const float* gout, const float* coord, long long coord_sb,
                                   float* gcorr, float* gpyramid, int clamp_unit, cudaStream_t stream);

// Lookup on the 4D correlation volume without storing it (the call core/corr.py:491-510 leaves unimplemented; its
// result is the dense block's lookup, core/corr.py:192-247).  F1 (B, H1, W1, C) and the image-2 feature pyramid
// F2[l] (B, H2[l], W2[l], C), channels innermost; coords (B, 2, H1, W1) = (x, y) per pixel;
// out (B, levels*(2*radius+1)^2, H1, W1), every product times `scale`.  C % 4 == 0, C <= 512, radius <= 4.
struct Lookup4dDims {
  int B, H1, W1, C, levels, radius;
  int H2[LOOKUP_MAX_LEVELS], W2[LOOKUP_MAX_LEVELS];
};
[[nodiscard]] cudaError_t launch_lookup4d_forward(const Lookup4dDims& d, const float* F1, const float* const* F2,
                                    const float* coords, float* out, float scale, cudaStream_t stream);
// gF1 (shape of F1) is overwritten; gF2[l] (shape of F2[l]) is zeroed and then accumulated with float reductions.
int lookup4d_backward_launches(const Lookup4dDims& d);
[[nodiscard]] cudaError_t launch_lookup4d_backward(const Lookup4dDims& d, const float* F1, const float* const* F2,
                                     const float* coords, const float* gout, float* gF1, float* const* gF2,
                                     float scale, cudaStream_t stream);

}  // namespace sfb
