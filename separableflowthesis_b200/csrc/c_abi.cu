// C-ABI entry points (include/sepflow_b200.h): argument validation, workspace carving, TMA tensor
// map encoding and the launch sequence of each op.  No torch types, no allocation.
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <algorithm>
#include <atomic>
#include <mutex>
#include <vector>

#include "../../include/sepflow_b200.h"
#include "kernels.h"

namespace {

using namespace sfb;

thread_local char g_err[512] = "";

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

// cuTensorMapEncodeTiled is looked up at run time so the library loads (and its symbols can be
// inspected) on machines without a CUDA driver.
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// cuTensorMapEncodeTiled is a driver call and needs a context that is current to the calling thread.  A thread that
// has made no runtime call yet (an autograd worker whose first node is one of these ops) has none.  Whether one is
// current is asked of the driver (cuCtxGetCurrent, which allocates nothing and is legal at any time); only when
// there is none does the thread bind the device's primary context with cudaFree(0), once.
typedef CUresult (*CtxGetCurrentFn)(CUcontext*);
int bind_context() {
  static thread_local bool bound = false;
  if (bound) return SFB_OK;
  static CtxGetCurrentFn get_current = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return reinterpret_cast<CtxGetCurrentFn>(p);
    return static_cast<CtxGetCurrentFn>(nullptr);
  }();
  CUcontext ctx = nullptr;
  if (get_current == nullptr || get_current(&ctx) != CUDA_SUCCESS || ctx == nullptr) {
    cudaError_t e = cudaFree(nullptr);
    if (e != cudaSuccess) return fail(SFB_ERR_CUDA, "cudaFree(0): %s", cudaGetErrorString(e));
  }
  bound = true;
  return SFB_OK;
}
#define SFB_TRY_BIND_CONTEXT()                 \
  do {                                         \
    int rc_ = bind_context();                  \
    if (rc_ != SFB_OK) return rc_;             \
  } while (0)

// Tiled fp32 tensor map, 128-byte swizzle, innermost box = 32 channels (128 bytes), zero fill out of bounds.
// dims/box are innermost-first; strides are implied by a contiguous tensor.
// `pitch0` (elements, optional): distance between consecutive indices of dimension 1 when the rows are padded.
int make_map(CUtensorMap* tm, const void* base, int rank, const uint64_t* dims, const uint32_t* box,
             CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B, bool bf16 = false, uint64_t pitch0 = 0) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return fail(SFB_ERR_CUDA, "cuTensorMapEncodeTiled is not available (no CUDA driver?)");
  if (base == nullptr) return fail(SFB_ERR_INVALID_ARGUMENT, "internal: tensor map over an array this workspace does not hold");
  SFB_TRY_BIND_CONTEXT();
  cuuint64_t gdim[5], gstride[5];
  cuuint32_t bdim[5], estride[5];
  uint64_t stride = bf16 ? 2 : sizeof(float);
  for (int i = 0; i < rank; ++i) {
    gdim[i] = dims[i];
    bdim[i] = box[i];
    estride[i] = 1;
    stride *= (i == 0 && pitch0 != 0) ? pitch0 : dims[i];
    if (i < rank - 1) gstride[i] = stride;  // byte stride of dimension i+1
  }
  CUresult r = fn(tm, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, (cuuint32_t)rank,
                  const_cast<void*>(base), gdim, gstride,
                  bdim, estride, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(SFB_ERR_CUDA, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
  return SFB_OK;
}

size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

}  // namespace

namespace sfb {
cudaError_t encode_plain_map(CUtensorMap* tm, const void* base, int rank, const uint64_t* dims,
                             const uint64_t* strides_bytes, const uint32_t* box) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr || bind_context() != SFB_OK) return cudaErrorNotSupported;
  cuuint64_t gdim[5], gstride[5];
  cuuint32_t bdim[5], estride[5];
  for (int i = 0; i < rank; ++i) {
    gdim[i] = dims[i];
    bdim[i] = box[i];
    estride[i] = 1;
    if (i < rank - 1) gstride[i] = strides_bytes[i];
  }
  const CUresult r = fn(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, (cuuint32_t)rank, const_cast<void*>(base), gdim, gstride, bdim,
                        estride, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}
}  // namespace sfb

namespace {

// ---- optional per-kernel timing (off by default): CUDA events around each launch on its own stream ----
enum KernelId : int {
  KID_PREPARE = 0, KID_PACK, KID_SWEEP_MAXAVG, KID_SWEEP_COMPRESS, KID_SWEEP_DUMP, KID_GRAD_MAXAVG_IMG1, KID_GRAD_MAXAVG_IMG2,
  KID_GRAD_COMPRESS_IMG1, KID_GRAD_COMPRESS_IMG2, KID_GRAD_FUSED_IMG1, KID_GRAD_FUSED_IMG2, KID_ATTENTION_FWD,
  KID_ATTENTION_BWD, KID_LOOKUP, KID_RESAMPLE, KID_LOOKUP4D, KID_COUNT
};
const char* const kKernelNames[KID_COUNT] = {
    "prepare(round_copy+f2_means)", "pack_kernel/unpack_kernel", "sweep_kernel<maxavg>", "sweep_kernel<compress>", "sweep_kernel<dump>",
    "grad_gemm_kernel<maxavg,image1-major>", "grad_gemm_kernel<maxavg,image2-major>",
    "grad_gemm_kernel<compress,image1-major>", "grad_gemm_kernel<compress,image2-major>",
    "grad_gemm_kernel<fused,image1-major>", "grad_gemm_kernel<fused,image2-major>",
    "attention forward (logits, softmax)", "attention backward (logit, input, weight grads)",
    "lookup kernels (pyramid, forward, backward)", "upsample_displacement kernels",
    "lookup4d kernels (forward, backward)"};
struct TimingRec { cudaEvent_t e0, e1; int id; int launches; };
std::mutex g_timing_mu;
bool g_timing_on = false;
std::vector<TimingRec> g_timing_pending;
std::vector<cudaEvent_t> g_event_pool;
double g_timing_ms[KID_COUNT] = {0};
long long g_timing_launches[KID_COUNT] = {0};

cudaEvent_t take_event() {
  if (!g_event_pool.empty()) { cudaEvent_t e = g_event_pool.back(); g_event_pool.pop_back(); return e; }
  cudaEvent_t e = nullptr;
  cudaEventCreate(&e);
  return e;
}

template <class Launch>
cudaError_t timed(int id, int launches, cudaStream_t st, Launch&& launch) {
  bool on;
  TimingRec rec{nullptr, nullptr, id, launches};
  {
    std::lock_guard<std::mutex> lk(g_timing_mu);
    on = g_timing_on;
    if (on) { rec.e0 = take_event(); rec.e1 = take_event(); }
  }
  if (on) cudaEventRecord(rec.e0, st);
  cudaError_t err = launch();
  if (on) {
    cudaEventRecord(rec.e1, st);
    std::lock_guard<std::mutex> lk(g_timing_mu);
    g_timing_pending.push_back(rec);
  }
  return err;
}

void drain_timing_locked() {
  for (TimingRec& r : g_timing_pending) {
    float ms = 0.f;
    if (cudaEventSynchronize(r.e1) == cudaSuccess && cudaEventElapsedTime(&ms, r.e0, r.e1) == cudaSuccess) {
      g_timing_ms[r.id] += ms;
      g_timing_launches[r.id] += r.launches;
    }
    g_event_pool.push_back(r.e0);
    g_event_pool.push_back(r.e1);
  }
  g_timing_pending.clear();
}

// Operand type of the contractions (sfb_set_sweep_operands): FP16 (default), TF32 or BF16.  Process-wide, because
// a backward runs on an autograd worker thread, not on the thread that chose the precision.
int initial_operands() {  // SFB_OPERANDS=tf32|bf16|fp16 in the environment chooses the initial setting
  const char* e = getenv("SFB_OPERANDS");
  if (e != nullptr) {
    if (strcmp(e, "tf32") == 0) return SFB_OPERANDS_TF32;
    if (strcmp(e, "bf16") == 0) return SFB_OPERANDS_BF16;
  }
  return SFB_OPERANDS_FP16;
}
std::atomic<int> g_sweep_operands{initial_operands()};

// Test hook (sfb_debug_wait_timeout): time limit handed to the kernels' bounded waits and whether the next sweeps
// leave out their last load.  Process-wide; 0 / 0 = normal operation.
std::atomic<unsigned long long> g_wait_limit_ns{0};
std::atomic<int> g_drop_last_load{0};
SweepArgs with_wait_settings(SweepArgs a) {
  a.wait_limit_ns = g_wait_limit_ns.load();
  a.drop_last_load = g_drop_last_load.load();
  return a;
}
GradArgs with_wait_settings(GradArgs a) {
  a.wait_limit_ns = g_wait_limit_ns.load();
  return a;
}

// Operand type of a call's contractions: the process-wide switch (sfb_set_sweep_operands), as OP16_NONE (TF32), OP16_BF16 or OP16_FP16.
// 16-bit rows must be multiples of 16 bytes for TMA: with FP16 operands, which have the precision of TF32, other shapes run with the
// latter; with BF16 operands they are refused (operand_mode).
int op16_of(const Dims& d) {
  const int m = g_sweep_operands.load();
  if (d.C % 8 != 0) return OP16_NONE;
  return m == SFB_OPERANDS_BF16 ? OP16_BF16 : (m == SFB_OPERANDS_FP16 ? OP16_FP16 : OP16_NONE);
}

struct Workspace {
  int* status;
  float* scales;  // scale slots of the FP16 operand kind (kernels.h, SCALE_*), in the header after the status word
  float* F1r;
  float* F2r;
  float* aux;
  uint16_t* F1h;  // the same three as 16-bit copies (FP16 or BF16), in the same memory: operands of the kind::f16 sweeps
  uint16_t* F2h;
  uint16_t* auxh;
  float* xu;   // packed inputs indexed by (u, slot, pixel): (B, H2, Rx, n1p)
  float* xv;   // packed inputs indexed by (v, slot, pixel): (B, W2, Rx, n1p)
  float* ou;   // packed outputs, (B, H2, Ro, n1p)
  float* ov;   // packed outputs, (B, W2, Ro, n1p)
  float* gxu;  // interleaved gradient-GEMM operands, (B, H2, n1p, Rg)
  float* gxv;  // interleaved gradient-GEMM operands, (B, W2, n1p, Rg)
  float* F1t;  // channel-major copies of F1r / F2r for K-major B operands: (B, C, n1p) and, in column blocks of 16
  float* F2t;  // with a multiple of GG_UT rows, (B, C, ceil(W2/16), h2p, 16)
  int h2p;     // H2 rounded up to a multiple of GG_UT
  float* ga_u;  // level backward: attention gradients (B, Kc, W2, N1) / (B, Kc, H2, N1) ...
  float* ga_v;
  float* gm_u;  // ... total gradients of the max/avg channels (B, 2, W2, N1) / (B, 2, H2, N1) ...
  float* gm_v;
  float* at_partial;  // ... and the attention backward's per-block partial sums
  int n1p;
  size_t bytes;        // without the scratch of the tail pieces, which a caller's buffer may lack (the kernels then
  float* part;         // do whole tiles only)
  size_t part_bytes;
  uint8_t* stored;     // G between the gradient GEMMs (16-bit operands), behind the scratch; a buffer may lack it as well (G is then
                       // generated twice)
  size_t stored_bytes;  // the samples that the buffer has room for
};

int padded_pixels(const Dims& d) { return (d.N1() + TILE_M - 1) / TILE_M * TILE_M; }

// (B, D, slots, n1p) workspace array, optionally starting at slot `slot0`
PixView packed_view(float* base, int D, int slots, int n1p, int slot0 = 0) {
  return PixView{base + (size_t)slot0 * n1p, (long long)D * slots * n1p, (uint32_t)(slots * n1p), (uint32_t)n1p};
}
// (B, slots, D, N1) user tensor
PixView cf_view(const void* base, int slots, int D, int N1) {
  return PixView{static_cast<float*>(const_cast<void*>(base)), (long long)slots * D * N1, (uint32_t)N1, (uint32_t)(D * N1)};
}

// What an op keeps in the workspace: the mean rows of F2, Rx packed input slots, Ro packed output slots, Rg interleaved ones;
// whether it has correlation sweeps, whose operands may be 16-bit copies of the features.
struct WsPlan { bool aux; int Rx; int Ro; int Rg; bool level_bwd; bool sweeps; };
constexpr int MAXAVG_SLOTS = 3;  // max, mean, argmax bits
constexpr int MAXAVG_PART_SLOTS = 2;  // of a tail piece: max, argmax bits
int chunk_channels(int Kc) { return Kc < KC_MAX_PER_SWEEP ? Kc : KC_MAX_PER_SWEEP; }
int grad_slots(int kc) { return 2 * kc <= 4 ? 4 : 8; }  // two slots per channel, rounded up to a multiple of 4

WsPlan plan_for(int op, const Dims& d) {
  switch (op) {
    case SFB_OP_MAX_AVG_FORWARD: return {true, 0, MAXAVG_SLOTS, 0, false, true};
    case SFB_OP_COMPRESSION_FORWARD: return {false, d.Kc, d.Kc, 0, false, true};
    case SFB_OP_MAX_ARGMAX_AVG_BACKWARD: return {false, 0, 0, 4, false, false};
    case SFB_OP_COMPRESSION_BACKWARD: return {false, d.Kc, d.Kc, grad_slots(chunk_channels(d.Kc)), false, true};
    case SFB_OP_SEPARATION_BACKWARD: return {false, d.Kc, d.Kc, 4 + grad_slots(chunk_channels(d.Kc)), false, true};
    case SFB_OP_MAX_AVG_FORWARD_CF: return {true, 0, 0, 0, false, true};
    case SFB_OP_COMPRESSION_CF: return {false, 0, 0, 0, false, true};
    case SFB_OP_SEPARATION_FEATURE_BACKWARD_CF: return {false, 0, 0, 4 + grad_slots(chunk_channels(d.Kc)), false, false};
    case SFB_OP_SEPARATION_LEVEL_FORWARD: return {true, 0, 0, 0, false, true};
    case SFB_OP_SEPARATION_LEVEL_BACKWARD: return {false, 0, 0, 4 + grad_slots(chunk_channels(d.Kc)), true, true};
    default: return {false, 0, 0, 0, false, false};
  }
}

// Whether a pair of gradient GEMMs over one or several levels of an image 2 hands G over through memory, or generates it twice.  The storing
// GEMM has one tile per 128 image-1 pixels whose generator waits for its own stores, the reading one tiles of 256 image-2 pixels: less than a
// wave of short tiles gains nothing.  Pairs of one level, C = 256, generated twice / stored (us): 2 x 48 x 64 on itself 70 / 74, 6 x 48 x 64 (144
// tiles) 103 / 114, 4 x 55 x 128 on 13 x 32 64 / 68, 1 x 40 x 100 69 / 72; 8 x 48 x 64 (192 tiles) 161 / 138, 32 x 24 x 32 (192) 81 / 68,
// 4 x 55 x 128 on 27 x 64 136 / 122, 1 x 55 x 128 (55 tiles of 7040 values each) 134 / 121, 1 x 135 x 240 1578 / 1166.
bool grad_hands_over(const Dims& d, int levels) {
  return d.N2() > 4096 || (d.N2() >= 512 && (long long)d.B * ((d.N1() + TILE_M - 1) / TILE_M) * levels > SM_COUNT);
}
// Samples whose G (`bytes` each) is stored at a time: all, as many as fit, or (0) none.  With TF32 operands it is generated twice.
int grad_chunk(const Dims& d, int levels, size_t bytes, int op16) {
  return op16 != OP16_NONE && grad_hands_over(d, levels) ? (int)std::min<size_t>(d.B, GRAD_STORED_LIMIT / bytes) : 0;
}

// stores: with room for G where the gradient GEMMs hand it over (else what they need to generate it twice).
Workspace carve(const Dims& d, void* base, const WsPlan& plan, bool stores = true) {
  Workspace w;
  size_t off = 0;
  char* p = static_cast<char*>(base);
  auto take = [&](size_t floats) {
    float* r = reinterpret_cast<float*>(p + off);
    off += align_up(floats * sizeof(float), 256);
    return r;
  };
  w.status = reinterpret_cast<int*>(p + off);
  w.scales = reinterpret_cast<float*>(p + off + WS_SCALES_OFFSET);
  off += WS_HEADER_BYTES;
  w.n1p = padded_pixels(d);
  w.F1r = take((size_t)d.B * d.N1() * d.C);
  w.F2r = take((size_t)d.B * d.N2() * d.C);
  w.aux = plan.aux ? take((size_t)d.B * d.aux_rows() * d.C) : nullptr;
  // A call makes the copies of one operand type (Features::op16), so the 16-bit ones lie where the FP32 ones would be.
  w.F1h = plan.sweeps ? reinterpret_cast<uint16_t*>(w.F1r) : nullptr;
  w.F2h = plan.sweeps ? reinterpret_cast<uint16_t*>(w.F2r) : nullptr;
  w.auxh = reinterpret_cast<uint16_t*>(w.aux);
  w.xu = plan.Rx ? take((size_t)d.B * d.H2 * plan.Rx * w.n1p) : nullptr;
  w.xv = plan.Rx ? take((size_t)d.B * d.W2 * plan.Rx * w.n1p) : nullptr;
  w.ou = plan.Ro ? take((size_t)d.B * d.H2 * plan.Ro * w.n1p) : nullptr;
  w.ov = plan.Ro ? take((size_t)d.B * d.W2 * plan.Ro * w.n1p) : nullptr;
  w.gxu = plan.Rg ? take((size_t)d.B * d.H2 * plan.Rg * w.n1p) : nullptr;
  w.gxv = plan.Rg ? take((size_t)d.B * d.W2 * plan.Rg * w.n1p) : nullptr;
  w.h2p = (d.H2 + GG_UT - 1) / GG_UT * GG_UT;
  w.F1t = w.F2t = nullptr;
  if (plan.Rg) {
    w.F1t = take((size_t)d.B * d.C * w.n1p);
    w.F2t = take((size_t)d.B * d.C * ((d.W2 + GG_VT - 1) / GG_VT) * w.h2p * GG_VT);
  }
  w.ga_u = w.ga_v = w.gm_u = w.gm_v = w.at_partial = nullptr;
  if (plan.level_bwd) {
    const size_t n1 = (size_t)d.N1();
    w.ga_u = take((size_t)d.B * d.Kc * d.W2 * n1);
    w.ga_v = take((size_t)d.B * d.Kc * d.H2 * n1);
    w.gm_u = take((size_t)d.B * 2 * d.W2 * n1);
    w.gm_v = take((size_t)d.B * 2 * d.H2 * n1);
    const AttentionDims at[2] = {{d.B, d.Kc, d.W2, d.H1, d.W1}, {d.B, d.Kc, d.H2, d.H1, d.W1}};
    w.at_partial = take(attention_partial_floats(at, 2));
  }
  w.bytes = off;
  size_t part = 0;
  if (plan.aux) part = std::max(part, sweep_split(d, MAXAVG_PART_SLOTS, false).part_floats);
  if (d.Kc > 0 && plan.sweeps) part = std::max(part, sweep_split(d, chunk_channels(d.Kc), true).part_floats);
  const int samples = plan.Rg && stores ? grad_chunk(d, 1, grad_stored_bytes(d, w.n1p), op16_of(d)) : 0;
  if (plan.Rg) {
    for (const int form : {GRAD_IMAGE1, GRAD_IMAGE2}) part = std::max(part, grad_split(d, form).part_floats);
    for (const int n : {samples, samples > 0 ? d.B % samples : 0}) {   // full chunks and what is left
      if (n == 0) continue;
      Dims some = d;
      some.B = n;
      for (const int form : {GRAD_IMAGE1_STORING, GRAD_IMAGE2_STORED}) part = std::max(part, grad_split(some, form).part_floats);
    }
  }
  w.part = reinterpret_cast<float*>(p + off);
  w.part_bytes = align_up(part * sizeof(float), 256);
  w.stored = reinterpret_cast<uint8_t*>(p + off + w.part_bytes);
  w.stored_bytes = samples * grad_stored_bytes(d, w.n1p);
  return w;
}

template <class Args> int contraction_launches(const Args& a) { return a.parts > 0 ? 2 : 1; }   // pieces are folded by a kernel of their own

// A sweep's cut into whole tiles and pieces, as far as the workspace has scratch for the pieces.
void set_sweep_split(SweepArgs& a, const Workspace& w, int slots) {
  const TileSplit s = sweep_split(a.d, slots, a.mode == SWEEP_COMPRESS);
  const bool cut = s.pieces > 1 && s.part_floats * sizeof(float) <= w.part_bytes;
  a.whole_tiles = cut ? s.whole_tiles : s.tiles;
  a.pieces = cut ? s.pieces : 1;
  a.parts = cut ? s.parts : 0;
  a.part_slots = slots;
  a.part = w.part;
}

// The same for a gradient GEMM.
void set_grad_split(GradArgs& a, const Workspace& w) {
  const TileSplit s = grad_split(a.d, a.form);
  const bool cut = s.pieces > 1 && s.part_floats * sizeof(float) <= w.part_bytes;
  a.whole_tiles = cut ? s.whole_tiles : s.tiles;
  a.pieces = cut ? s.pieces : 1;
  a.parts = a.pieces - 1;
  a.part0 = -1;
  a.part = w.part;
}

int check_shape(const sfb_shape* s, bool need_kc, Dims* d) {
  if (s == nullptr) return fail(SFB_ERR_INVALID_ARGUMENT, "shape is NULL");
  if (s->B < 1 || s->H1 < 1 || s->W1 < 1 || s->H2 < 1 || s->W2 < 1)
    return fail(SFB_ERR_INVALID_ARGUMENT, "B, H1, W1, H2, W2 must be >= 1 (got %d %d %d %d %d)", s->B, s->H1, s->W1,
                s->H2, s->W2);
  if (s->C < 4 || s->C > MAX_C || (s->C % 4) != 0)
    return fail(SFB_ERR_UNSUPPORTED_SHAPE, "feature dimension C=%d unsupported: need a multiple of 4 in [4, %d]", s->C,
                MAX_C);
  if (need_kc && s->Kc < 1) return fail(SFB_ERR_INVALID_ARGUMENT, "Kc must be >= 1 (got %d)", s->Kc);
  if ((long long)s->H1 * s->W1 > (1ll << 21) || (long long)s->H2 * s->W2 > (1ll << 30))
    return fail(SFB_ERR_UNSUPPORTED_SHAPE, "image 1 has more than 2^21 pixels or image 2 more than 2^30");
  {  // element offsets inside one sample's packed array are 32-bit in the kernels
    const long long n1p = ((long long)s->H1 * s->W1 + TILE_M - 1) / TILE_M * TILE_M;
    const long long kc = need_kc ? s->Kc : 0;  // ops without attention channels ignore (and may not initialise) Kc
    const long long slots = kc + 2 > 8 ? kc + 2 : 8;
    if (n1p * slots * (s->H2 > s->W2 ? s->H2 : s->W2) >= (1ll << 32))
      return fail(SFB_ERR_UNSUPPORTED_SHAPE, "H1*W1*max(H2,W2)*slots exceeds 2^32 elements per sample");
  }
  d->B = s->B; d->H1 = s->H1; d->W1 = s->W1; d->H2 = s->H2; d->W2 = s->W2; d->C = s->C;
  d->Kc = need_kc ? s->Kc : 0;
  return SFB_OK;
}

int check_ptr(const void* p, const char* name) {
  if (p == nullptr) return fail(SFB_ERR_INVALID_ARGUMENT, "%s is NULL", name);
  if ((reinterpret_cast<uintptr_t>(p) & 15u) != 0) return fail(SFB_ERR_INVALID_ARGUMENT, "%s is not 16-byte aligned", name);
  return SFB_OK;
}
#define SFB_CHECK_PTR(p)                       \
  do {                                         \
    int rc_ = check_ptr((p), #p);              \
    if (rc_ != SFB_OK) return rc_;             \
  } while (0)
#define SFB_TRY(expr)                          \
  do {                                         \
    int rc_ = (expr);                          \
    if (rc_ != SFB_OK) return rc_;             \
  } while (0)
#define SFB_CUDA(expr)                                                                           \
  do {                                                                                           \
    cudaError_t e_ = (expr);                                                                     \
    if (e_ != cudaSuccess) return fail(SFB_ERR_CUDA, "%s: %s", #expr, cudaGetErrorString(e_));  \
  } while (0)

// Inside a step of several launches (a function returning cudaError_t): the first one that fails ends it.  A launcher
// takes the error off the runtime when it reports it, so a result that is not passed on is lost.
#define SFB_LAUNCH(expr)                       \
  do {                                         \
    cudaError_t e_ = (expr);                   \
    if (e_ != cudaSuccess) return e_;          \
  } while (0)

int check_workspace(const Dims& d, void* ws, size_t ws_bytes, int op, Workspace* out) {
  if (ws == nullptr) return fail(SFB_ERR_INVALID_ARGUMENT, "workspace is NULL");
  if ((reinterpret_cast<uintptr_t>(ws) & 255u) != 0)
    return fail(SFB_ERR_INVALID_ARGUMENT, "workspace is not 256-byte aligned");
  *out = carve(d, ws, plan_for(op, d));
  if (ws_bytes < out->bytes)
    return fail(SFB_ERR_WORKSPACE_TOO_SMALL, "workspace has %zu bytes, %zu needed", ws_bytes, out->bytes);
  const size_t room = ws_bytes - out->bytes;
  if (out->stored_bytes > 0 && room < out->part_bytes + grad_stored_bytes(d, out->n1p)) *out = carve(d, ws, plan_for(op, d), false);
  out->stored_bytes = room > out->part_bytes ? std::min(out->stored_bytes, room - out->part_bytes) : 0;
  if (room < out->part_bytes) out->part_bytes = 0;
  return SFB_OK;
}

// Tensor maps over the rounded copies.
// `swizzle` is the 16-byte-atom 128B swizzle for K-major operands (rows = pixels of the tile) and the
// 32-byte-atom variant for MN-major TF32 operands (the only layout tcgen05.mma accepts for those).
int map_f1_rows(CUtensorMap* tm, const Dims& d, const void* F1r, uint32_t rows,
                CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B, bool bf16 = false) {  // (C, N1, B)
  const uint64_t dims[3] = {(uint64_t)d.C, (uint64_t)d.N1(), (uint64_t)d.B};
  const uint32_t box[3] = {bf16 ? 2u * KBLK : (uint32_t)KBLK, rows, 1};   // one 128-byte row of channels
  return make_map(tm, F1r, 3, dims, box, swizzle, bf16);
}
int map_f2_tile(CUtensorMap* tm, const Dims& d, const void* F2r, uint32_t ut, uint32_t vt,
                CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B, bool bf16 = false) {  // (C, W2, H2, B)
  const uint64_t dims[4] = {(uint64_t)d.C, (uint64_t)d.W2, (uint64_t)d.H2, (uint64_t)d.B};
  const uint32_t box[4] = {bf16 ? 2u * KBLK : (uint32_t)KBLK, vt, ut, 1};
  return make_map(tm, F2r, 4, dims, box, swizzle, bf16);
}
// Interleaved gradient operands (B, D, Q, n1p, 4), seen by TMA as (4*n1p, Q, D, B) so that the innermost box
// dimension is a long contiguous run (`pixels` * 16 bytes): box = (4*pixels, Q groups, `disps` displacements, 1).
int map_operands(CUtensorMap* tm, const float* x, int B, int D, int Q, int n1p, uint32_t pixels, uint32_t disps) {
  const uint64_t dims[4] = {4ull * (uint64_t)n1p, (uint64_t)Q, (uint64_t)D, (uint64_t)B};
  const uint32_t box[4] = {4 * pixels, (uint32_t)Q, disps, 1};
  return make_map(tm, x, 4, dims, box, CU_TENSOR_MAP_SWIZZLE_NONE);
}
int map_aux(CUtensorMap* tm, const Dims& d, const void* aux, bool bf16 = false) {  // (C, H2+W2, B)
  const uint64_t dims[3] = {(uint64_t)d.C, (uint64_t)d.aux_rows(), (uint64_t)d.B};
  const uint32_t box[3] = {bf16 ? 2u * KBLK : (uint32_t)KBLK, (uint32_t)(SWEEP_UT * SWEEP_VT), 1};
  return make_map(tm, aux, 3, dims, box, CU_TENSOR_MAP_SWIZZLE_128B, bf16);
}

int operand_mode(const Dims& d, int* op16) {
  if (d.C % 8 != 0 && g_sweep_operands.load() == SFB_OPERANDS_BF16)
    return fail(SFB_ERR_UNSUPPORTED_SHAPE, "BF16 operands need a feature dimension that is a multiple of 8 (C=%d)", d.C);
  *op16 = op16_of(d);
  return SFB_OK;
}
// What the sweeps multiply their outputs by: the inverse of the feature scales of FP16 operands, else nothing.
const float* sweep_out_scale(const Workspace& w, int op16) {
  return op16 == OP16_FP16 ? w.scales + SCALE_INV_F1F2 : nullptr;
}

// Tensor maps of the sweeps' operands in a workspace: the rounded FP32 copies or the 16-bit copies.  Image 2 in the tiles of the
// max/avg sweeps (f2) and of the compression (f2_sums); f2, f2_sums and aux may be null.
int map_sweep_operands(const Dims& d, const Workspace& w, int op16, CUtensorMap* f1, CUtensorMap* f2, CUtensorMap* f2_sums,
                       CUtensorMap* aux) {
  SFB_TRY(map_f1_rows(f1, d, op16 ? static_cast<const void*>(w.F1h) : w.F1r, TILE_M, CU_TENSOR_MAP_SWIZZLE_128B, op16 != 0));
  for (const bool sums : {false, true}) {
    CUtensorMap* const f = sums ? f2_sums : f2;
    if (f == nullptr) continue;
    const bool narrow = sweep_narrow(d, sums);
    if (sums && f2 != nullptr && narrow == sweep_narrow(d, false)) {
      *f2_sums = *f2;
      continue;
    }
    SFB_TRY(map_f2_tile(f, d, op16 ? static_cast<const void*>(w.F2h) : w.F2r, narrow ? SWEEP_UT_NARROW : SWEEP_UT,
                        narrow ? SWEEP_VT_NARROW : SWEEP_VT, CU_TENSOR_MAP_SWIZZLE_128B, op16 != 0));
  }
  if (aux != nullptr) SFB_TRY(map_aux(aux, d, op16 ? static_cast<const void*>(w.auxh) : w.aux, op16 != 0));
  return SFB_OK;
}

// The features of a call as the caller holds them: pixel-major (B, pixels, C), or (fmaps) the model's feature maps
// (B, C, pixels) with a factor for image 1; and the operand type of the call (OP16_*).  An entry point reads the
// process-wide switch once, into op16, and every step of the call goes by that: the copies prepare_operands makes are
// those of one type, and another thread may move the switch at any time.
struct Features {
  const float* F1;
  const float* F2;
  bool fmaps;
  float scale1;
  int op16;
};

// Operand copies of a call's features (and of the mean rows of image 2 when with_aux).
cudaError_t prepare_operands(const Dims& d, const Workspace& w, const Features& f, bool with_aux, cudaStream_t st) {
  const int op16 = f.op16;
  // (an op without sweeps has no 16-bit copies in its workspace, but its gradient GEMMs still need the feature scales)
  float* const F1r = op16 ? nullptr : w.F1r;
  float* const F2r = op16 ? nullptr : w.F2r;
  float* const aux = op16 || !with_aux ? nullptr : w.aux;
  uint16_t* const F1h = op16 ? w.F1h : nullptr;
  uint16_t* const F2h = op16 ? w.F2h : nullptr;
  uint16_t* const auxh = op16 && with_aux ? w.auxh : nullptr;
  const LevelOperands out{F2r, aux, F2h, auxh};
  return f.fmaps ? launch_prepare_cf(&d, 1, f.F1, &f.F2, f.scale1, &out, F1r, F1h, w.status, st, op16, w.scales)
                 : launch_prepare(d, f.F1, f.F2, F1r, F2r, aux, w.status, st, F1h, F2h, auxh, op16, w.scales);
}
// Launches of the above: the header is cleared; FP16 operands add the search for the magnitudes; pixel-major features have copies and mean rows in one.
int prepare_launches(const Workspace& w, bool fmaps, bool with_aux, int op16) {
  const bool copies = !op16 || w.F1h != nullptr;
  return 1 + (fmaps ? (copies ? 1 : 0) + (with_aux ? 1 : 0) : (copies || with_aux ? 1 : 0)) + (op16 == OP16_FP16 ? 1 : 0);
}
#define SFB_PREPARE(f, with_aux) \
  SFB_CUDA(timed(KID_PREPARE, prepare_launches(w, (f).fmaps, with_aux, (f).op16), st, [&] { return prepare_operands(d, w, f, with_aux, st); }))

int run_maxavg_forward(const float* F1, const float* F2, float* MA_u, float* MA_v, int32_t* AM_u, int32_t* AM_v,
                       bool with_argmax, const sfb_shape* shape, void* ws, size_t ws_bytes, void* stream) {
  Dims d;
  SFB_TRY(check_shape(shape, false, &d));
  SFB_CHECK_PTR(F1); SFB_CHECK_PTR(F2); SFB_CHECK_PTR(MA_u); SFB_CHECK_PTR(MA_v);
  if (with_argmax) { SFB_CHECK_PTR(AM_u); SFB_CHECK_PTR(AM_v); }
  Workspace w;
  SFB_TRY(check_workspace(d, ws, ws_bytes, SFB_OP_MAX_AVG_FORWARD, &w));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int op16;
  SFB_TRY(operand_mode(d, &op16));
  CUtensorMap tm_f1, tm_f2, tm_aux;
  SFB_TRY(map_sweep_operands(d, w, op16, &tm_f1, &tm_f2, nullptr, &tm_aux));
  const Features feat{F1, F2, false, 1.f, op16};
  SFB_PREPARE(feat, true);
  SweepArgs a;
  memset(&a, 0, sizeof(a));
  a.d = d;
  a.op16 = op16;
  a.out_scale = sweep_out_scale(w, op16);
  a.mode = with_argmax ? SWEEP_MAXARGAVG : SWEEP_MAXAVG;
  a.n_valid = w.n1p;
  a.pu = packed_view(w.ou, d.H2, MAXAVG_SLOTS, w.n1p);
  a.pv = packed_view(w.ov, d.W2, MAXAVG_SLOTS, w.n1p);
  a.pu_arg = packed_view(w.ou, d.H2, MAXAVG_SLOTS, w.n1p, 2);
  a.pv_arg = packed_view(w.ov, d.W2, MAXAVG_SLOTS, w.n1p, 2);
  a.status = w.status;
  set_sweep_split(a, w, MAXAVG_PART_SLOTS);
  SFB_CUDA(timed(KID_SWEEP_MAXAVG, contraction_launches(a), st, [&] { return launch_sweep(with_wait_settings(a), tm_f1, tm_f2, tm_aux, st); }));
  // packed (displacement, slot, pixel) -> the reference's (pixel, channel, displacement) tensors
  const PatchJob out[4] = {{MA_u, w.ou, 2, d.H2, 2, 0, MAXAVG_SLOTS, 0}, {MA_v, w.ov, 2, d.W2, 2, 0, MAXAVG_SLOTS, 0},
                           {AM_u, w.ou, 1, d.H2, 1, 0, MAXAVG_SLOTS, 2}, {AM_v, w.ov, 1, d.W2, 1, 0, MAXAVG_SLOTS, 2}};
  SFB_CUDA(timed(KID_PACK, 1, st, [&] { return launch_unpack(out, with_argmax ? 4 : 2, d.B, d.N1(), w.n1p, st); }));
  return SFB_OK;
}

// ou(b,u,k,p) = sum_v S * w_u[k], ov(b,v,k,p) = sum_u S * w_v[k] for all Kc channels, at most KC_MAX_PER_SWEEP
// channels per sweep.  Weight k is slot (slot0 + k*stride) of the views xu (per u: w_v) / xv (per v: w_u).
int run_compress_sweeps(const Dims& d, const Workspace& w, const CUtensorMap& tm_f1, const CUtensorMap& tm_f2, PixView xu,
                        PixView xv, int wu_slot0, int wv_slot0, int w_stride, PixView ou, PixView ov, int n_valid,
                        cudaStream_t st, int op16 = 0, const float* out_scale = nullptr) {
  for (int k0 = 0; k0 < d.Kc; k0 += KC_MAX_PER_SWEEP) {
    SweepArgs a;
    memset(&a, 0, sizeof(a));
    a.d = d;
    a.mode = SWEEP_COMPRESS;
    a.n_valid = n_valid;
    a.k0 = k0;
    a.kc = chunk_channels(d.Kc - k0);
    a.xu = xu; a.xv = xv;
    a.wu_slot0 = wu_slot0; a.wv_slot0 = wv_slot0; a.w_stride = w_stride;
    a.ou = ou; a.ov = ov;
    a.op16 = op16;
    a.out_scale = out_scale;
    a.status = w.status;
    set_sweep_split(a, w, chunk_channels(d.Kc));
    SFB_CUDA(timed(KID_SWEEP_COMPRESS, contraction_launches(a), st, [&] { return launch_sweep(with_wait_settings(a), tm_f1, tm_f2, tm_f2 /* unused */, st); }));
  }
  return SFB_OK;
}

// Arguments and tensor maps of one level's gradient GEMM, image-1-major or image-2-major, but for its cut.
// gF1 = G * F2 : rows are image-1 pixels, the K sweep streams 4 x 16 blocks of F2 and 4-row blocks of XU.
// gF2 = G^T * F1 : rows are an 8 x 16 block of image-2 pixels, the K sweep streams 32 pixels of F1, XU and XV.
// K-major B operands: channel-major copies of the rounded features (image 2 in column blocks of 16 with a multiple of four
// rows, so that a 4 x 16 block of the image is 64 consecutive values).  Rows and columns of padding must
// read as zero: they meet the G values of cells outside the image.
size_t f2t_per_sample(const Dims& d, const Workspace& w) { return (size_t)d.C * ((d.W2 + GG_VT - 1) / GG_VT) * w.h2p * GG_VT; }
int grad_arguments(const Dims& d, const Workspace& w, int op16, int mode, int R4, int form, float* out, int out_cf, float scale1,
                   GradArgs* a, CUtensorMap* tm_y, CUtensorMap* tm_xu, CUtensorMap* tm_xv) {
  const bool image2_major = grad_is_image2(form);
  memset(a, 0, sizeof(*a));
  a->d = d;
  a->mode = mode;
  a->R4 = R4;
  a->n1p = w.n1p;
  a->xu = w.gxu;
  a->xv = w.gxv;
  a->status = w.status;
  a->op16 = op16;
  a->out_cf = out_cf;
  a->form = form;
  a->out = out;
  a->stored = w.stored;
  a->out_scale = image2_major ? 1.f : scale1;
  a->dev_scale = op16 == OP16_FP16 ? w.scales + (image2_major ? SCALE_INV_GF2 : SCALE_INV_GF1) : nullptr;
  const int Q = R4 / 4;
  const uint32_t crows = (uint32_t)((d.C + KBLK - 1) / KBLK * KBLK);  // channel rows of one feature block
  if (!image2_major) {  // (blocked pixels, C, B); box = 128 bytes of consecutive values (4 rows x 16 columns of a 16-bit type) x all channels
    const uint64_t dims[3] = {(uint64_t)(f2t_per_sample(d, w) / d.C), (uint64_t)d.C, (uint64_t)d.B};
    const uint32_t box[3] = {op16 ? 64u : 32u, crows, 1};
    SFB_TRY(make_map(tm_y, w.F2t, 3, dims, box, CU_TENSOR_MAP_SWIZZLE_128B, op16 != 0));
    SFB_TRY(map_operands(tm_xu, w.gxu, d.B, d.H2, Q, w.n1p, TILE_M / 2, GG_UT));  // two 64-pixel boxes per block
    *tm_xv = *tm_xu;  // unused
    return SFB_OK;
  }
  // (N1, C, B) with rows padded to n1p; box = the pixels of a block x all channels: a row of 32 K-values is 128 bytes of FP32 or 64 bytes of
  // a 16-bit type, one of 64 16-bit values 128 bytes; the swizzle span follows
  const bool stored = form == GRAD_IMAGE2_STORED;
  const uint64_t dims[3] = {(uint64_t)d.N1(), (uint64_t)d.C, (uint64_t)d.B};
  const uint32_t box[3] = {stored ? (uint32_t)GG_SJ : (uint32_t)GG_KJ, crows, 1};
  SFB_TRY(make_map(tm_y, w.F1t, 3, dims, box, op16 && !stored ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, op16 != 0, (uint64_t)w.n1p));
  if (stored) {
    *tm_xu = *tm_xv = *tm_y;  // unused
    return SFB_OK;
  }
  SFB_TRY(map_operands(tm_xu, w.gxu, d.B, d.H2, Q, w.n1p, GG_KJ, GG_ROW_UT));
  return map_operands(tm_xv, w.gxv, d.B, d.W2, Q, w.n1p, GG_KJ, GG_ROW_VT);
}

MapCopy f1_copy(const Dims& d, const Workspace& w, const Features& f) {
  return MapCopy{f.F1, w.F1t, 1, d.N1(), w.n1p, 0, f.scale1, f.op16 == OP16_FP16 ? w.scales + SCALE_F1 : nullptr};
}
MapCopy f2_copy(const Dims& d, const Workspace& w, const float* F2, int op16) {
  return MapCopy{F2, w.F2t, d.H2, d.W2, w.h2p, 1, 1.f, op16 == OP16_FP16 ? w.scales + SCALE_F2 : nullptr};
}

// out_cf: the gradients are written channel-major, (B, C, pixels), gF1 multiplied by scale1.
int run_grad_pair(const Dims& d, const Workspace& w, const Features& feat, int mode, int R4, int accumulate, float* gF1, float* gF2,
                  cudaStream_t st, int out_cf = 0, float scale1 = 1.f) {
  // 16-bit form when the call has 16-bit operands; with FP16 the callers have run grad_operand_scales and packed the
  // operands with those scales
  const int op16 = feat.op16;
  const int kid = mode == GRAD_MAXAVG ? KID_GRAD_MAXAVG_IMG1 : (mode == GRAD_COMPRESS ? KID_GRAD_COMPRESS_IMG1 : KID_GRAD_FUSED_IMG1);
  if (!accumulate) {  // later passes over further channel chunks reuse the copies of the first
    SFB_CUDA(timed(KID_PREPARE, 1, st, [&] {
      MapCopy copies[2] = {f1_copy(d, w, feat), f2_copy(d, w, feat.F2, op16)};
      if (feat.fmaps) return launch_channel_major_cf(copies, 2, d.B, d.C, op16, st);   // already channel-major
      if (!op16) {   // pixel-major features are rounded already
        copies[0].src = w.F1r;
        copies[1].src = w.F2r;
      }
      return launch_channel_major(copies[0], copies[1], d.B, d.C, op16, st);
    }));
  }
  // 16-bit operands: G of as many samples as the workspace takes is generated and stored by one GEMM and read back by the other
  const int samples = op16 != 0 ? (int)(w.stored_bytes / grad_stored_bytes(d, w.n1p)) : 0;
  for (int b0 = 0; b0 < d.B; b0 += samples > 0 ? samples : d.B) {
    for (const int form : {samples > 0 ? GRAD_IMAGE1_STORING : GRAD_IMAGE1, samples > 0 ? GRAD_IMAGE2_STORED : GRAD_IMAGE2}) {
      const bool image2_major = grad_is_image2(form);
      GradArgs a;
      GradMaps maps;
      SFB_TRY(grad_arguments(d, w, op16, mode, R4, form, image2_major ? gF2 : gF1, out_cf, scale1, &a, maps.y, maps.xu, maps.xv));
      a.accumulate = accumulate;
      a.b0 = b0;
      if (samples > 0) a.d.B = std::min(samples, d.B - b0);
      set_grad_split(a, w);
      a = with_wait_settings(a);
      SFB_CUDA(timed(kid + (image2_major ? 1 : 0), contraction_launches(a), st, [&] { return launch_grad_gemm(&a, 1, maps, st); }));
    }
  }
  return SFB_OK;
}

// Interleaved slots of the max/avg backward (kernels.h): XU = (mean-gradient / W2, 1, max-gradient, argmax bits),
// XV = (1, mean-gradient / H2, max-gradient, argmax bits); the two mean-gradients are added, the constants are not read.
// `scales` (FP16 operands, else null): the call's scale slots; the gradient values are then multiplied by sg * sa.
void maxavg_slot_sources(const Dims& d, const int32_t* AM_u, const int32_t* AM_v, const float* gMA_u,
                         const float* gMA_v, SlotSources* su, SlotSources* sv, const float* scales) {
  memset(su, 0, sizeof(*su));
  memset(sv, 0, sizeof(*sv));
  su->s[0] = {gMA_u, 2, 1, 1.f / (float)d.W2};
  su->s[1] = {nullptr, 0, 0, 1.f};
  su->s[2] = {gMA_u, 2, 0, 0.f};
  su->s[3] = {AM_u, 1, 0, 0.f};
  sv->s[0] = {nullptr, 0, 0, 1.f};
  sv->s[1] = {gMA_v, 2, 1, 1.f / (float)d.H2};
  sv->s[2] = {gMA_v, 2, 0, 0.f};
  sv->s[3] = {AM_v, 1, 0, 0.f};
  if (scales != nullptr) {
    su->dev_scales = sv->dev_scales = scales;
    su->s[0].dev = su->s[2].dev = sv->s[1].dev = sv->s[2].dev = SCALE_GA + 1;
  }
}
// Interleaved slots of the compression backward for channels k0 .. k0+kc-1, local channel j:
// XU 2j = gC_u, 2j+1 = A_v;  XV 2j = A_u, 2j+1 = gC_v, so that G[p,u,v] = sum_slots XU[u,p,slot] * XV[v,p,slot].
// The gradients may be channels g0.. of a tensor with gK channels (the concatenated tensors of the call site).
// `scales` (FP16 operands, else null): gradients are multiplied by sg, weights by sa.
void compress_slot_sources(int K, int k0, int kc, const float* A_u, const float* A_v, const float* gC_u,
                           const float* gC_v, SlotSources* su, SlotSources* sv, const float* scales, int gK = 0,
                           int g0 = 0) {
  if (gK == 0) gK = K;
  memset(su, 0, sizeof(*su));
  memset(sv, 0, sizeof(*sv));
  for (int j = 0; j < kc; ++j) {
    su->s[2 * j] = {gC_u, gK, g0 + k0 + j, 0.f};
    su->s[2 * j + 1] = {A_v, K, k0 + j, 0.f};
    sv->s[2 * j] = {A_u, K, k0 + j, 0.f};
    sv->s[2 * j + 1] = {gC_v, gK, g0 + k0 + j, 0.f};
    if (scales != nullptr) {
      su->s[2 * j].dev = sv->s[2 * j + 1].dev = SCALE_G + 1;
      su->s[2 * j + 1].dev = sv->s[2 * j].dev = SCALE_A + 1;
    }
  }
  if (scales != nullptr) su->dev_scales = sv->dev_scales = scales;
}

// FP16 operands: the gradient-operand scales of this call (kernels.h, SCALE_*) from the largest magnitudes of the
// gradient tensors and of the weight tensors that multiply them.  No weight tensors: the weights are softmax outputs,
// known to lie in [0, 1], and their scale stays 1.  Runs after the call's launch_prepare, which cleared the slots and
// found the feature scales.
struct AbsmaxSrc { const float* p; size_t n; };
int grad_operand_scales(const Workspace& w, int op16, std::initializer_list<AbsmaxSrc> grads,
                        std::initializer_list<AbsmaxSrc> weights, cudaStream_t st) {
  if (op16 != OP16_FP16) return SFB_OK;
  AbsmaxSource src[ABSMAX_MAX];
  int n = 0;
  for (const AbsmaxSrc& g : grads) src[n++] = absmax_array(g.p, g.n, 1.f, SCALE_AMAX_G);
  for (const AbsmaxSrc& a : weights) src[n++] = absmax_array(a.p, a.n, 1.f, SCALE_AMAX_A);
  SFB_CUDA(timed(KID_PREPARE, 1, st, [&] { return launch_absmax(src, n, w.scales, 1, true, st); }));
  return SFB_OK;
}
const float* grad_slot_scales(const Workspace& w, int op16) { return op16 == OP16_FP16 ? w.scales : nullptr; }

// Weights w_u (B,N1,K,W2) / w_v (B,N1,K,H2) into the packed inputs, and the packed sums into C_u (B,N1,K,H2) / C_v (B,N1,K,W2).
int pack_weights(const Dims& d, const Workspace& w, const float* w_u, const float* w_v, cudaStream_t st) {
  const int K = d.Kc;
  const PatchJob in[2] = {{w_u, w.xv, K, d.W2, K, 0, K, 0}, {w_v, w.xu, K, d.H2, K, 0, K, 0}};
  SFB_CUDA(timed(KID_PACK, 1, st, [&] { return launch_pack(in, 2, d.B, d.N1(), w.n1p, st); }));
  return SFB_OK;
}
int unpack_sums(const Dims& d, const Workspace& w, float* C_u, float* C_v, cudaStream_t st) {
  const int K = d.Kc;
  const PatchJob out[2] = {{C_u, w.ou, K, d.H2, K, 0, K, 0}, {C_v, w.ov, K, d.W2, K, 0, K, 0}};
  SFB_CUDA(timed(KID_PACK, 1, st, [&] { return launch_unpack(out, 2, d.B, d.N1(), w.n1p, st); }));
  return SFB_OK;
}

// Attention gradients of the compression backward: gA_v[p,k,u] = sum_v S * gC_v[p,k,v] and
// gA_u[p,k,v] = sum_u S * gC_u[p,k,u] -- the forward compression sweep with the upstream gradients in the
// role of the weights (w_u = gC_v, w_v = gC_u).
int run_attention_grads(const Dims& d, const Workspace& w, const float* gC_u, const float* gC_v, float* gA_u,
                        float* gA_v, cudaStream_t st, int op16) {
  CUtensorMap tm_f1, tm_f2;
  SFB_TRY(map_sweep_operands(d, w, op16, &tm_f1, nullptr, &tm_f2, nullptr));
  const int K = d.Kc;
  SFB_TRY(pack_weights(d, w, gC_v, gC_u, st));
  SFB_TRY(run_compress_sweeps(d, w, tm_f1, tm_f2, packed_view(w.xu, d.H2, K, w.n1p), packed_view(w.xv, d.W2, K, w.n1p),
                              0, 0, 1, packed_view(w.ou, d.H2, K, w.n1p), packed_view(w.ov, d.W2, K, w.n1p), w.n1p, st, op16, sweep_out_scale(w, op16)));
  return unpack_sums(d, w, gA_v, gA_u, st);
}

// ---- scratch that lives in the library image, for callers that must not allocate ----
constexpr size_t STATIC_SCRATCH_BYTES = 32u << 20;
// The part of the header past its first 256 bytes comes on top: the shapes that fit stay the ones they were with a header of 256.
constexpr size_t STATIC_ARRAY_BYTES = STATIC_SCRATCH_BYTES + WS_HEADER_BYTES - 256;
static __device__ __align__(256) unsigned char g_static_scratch[STATIC_ARRAY_BYTES];

constexpr int MAX_DEVICES = 64;
std::mutex g_static_mu;
void* g_static_scratch_ptr[MAX_DEVICES] = {nullptr};

// Device address of g_static_scratch on the current device.  In host code the symbol's name is only a
// handle, not an address a kernel could use, so the address is looked up once per device (with that
// device current) and cached.
int static_scratch(void** out) {
  int dev = -1;
  SFB_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= MAX_DEVICES) return fail(SFB_ERR_CUDA, "device ordinal %d outside [0, %d)", dev, MAX_DEVICES);
  std::lock_guard<std::mutex> lk(g_static_mu);
  if (g_static_scratch_ptr[dev] == nullptr) {
    void* p = nullptr;
    SFB_CUDA(cudaGetSymbolAddress(&p, g_static_scratch));
    g_static_scratch_ptr[dev] = p;
  }
  *out = g_static_scratch_ptr[dev];
  return SFB_OK;
}

}  // namespace

extern "C" {

static size_t workspace_bytes_of(int op, const sfb_shape* shape, bool stores) {
  Dims d;
  if (op < SFB_OP_MAX_AVG_FORWARD || op > SFB_OP_SEPARATION_LEVEL_BACKWARD) return 0;
  const bool need_kc = op == SFB_OP_COMPRESSION_FORWARD || op == SFB_OP_COMPRESSION_BACKWARD ||
                       op == SFB_OP_SEPARATION_BACKWARD || op == SFB_OP_COMPRESSION_CF ||
                       op == SFB_OP_SEPARATION_FEATURE_BACKWARD_CF || op == SFB_OP_SEPARATION_LEVEL_FORWARD ||
                       op == SFB_OP_SEPARATION_LEVEL_BACKWARD;
  if (check_shape(shape, need_kc, &d) != SFB_OK) return 0;
  const Workspace w = carve(d, nullptr, plan_for(op, d), stores);
  return w.bytes + w.part_bytes + w.stored_bytes;
}
size_t sfb_workspace_bytes(int op, const sfb_shape* shape) { return workspace_bytes_of(op, shape, true); }
size_t sfb_workspace_least_bytes(int op, const sfb_shape* shape) { return workspace_bytes_of(op, shape, false); }

int sfb_max_avg_forward(const float* F1, const float* F2, float* MA_u, float* MA_v, const sfb_shape* shape,
                        void* workspace, size_t workspace_bytes, void* stream) {
  return run_maxavg_forward(F1, F2, MA_u, MA_v, nullptr, nullptr, false, shape, workspace, workspace_bytes, stream);
}

int sfb_max_avg_forward_static(const float* F1, const float* F2, float* MA_u, float* MA_v, const sfb_shape* shape,
                               void* stream) {
  Dims d;
  SFB_TRY(check_shape(shape, false, &d));
  SFB_CHECK_PTR(F1); SFB_CHECK_PTR(F2); SFB_CHECK_PTR(MA_u); SFB_CHECK_PTR(MA_v);
  const WsPlan plan = plan_for(SFB_OP_MAX_AVG_FORWARD, d);
  const size_t need = carve(d, nullptr, plan).bytes;
  if (need > STATIC_ARRAY_BYTES)
    return fail(SFB_ERR_UNSUPPORTED_SHAPE,
                "this shape needs %zu bytes of scratch but the built-in scratch holds %zu; use sfb_max_avg_forward "
                "with a caller-provided workspace", need, (size_t)STATIC_SCRATCH_BYTES);
  void* scratch = nullptr;
  SFB_TRY(static_scratch(&scratch));
  Workspace w = carve(d, scratch, plan);
  if (need + w.part_bytes > STATIC_ARRAY_BYTES) w.part_bytes = 0;  // no room for the tail pieces: whole tiles only
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  CUtensorMap tm_f1, tm_f2, tm_aux;
  SFB_TRY(map_sweep_operands(d, w, OP16_NONE, &tm_f1, &tm_f2, nullptr, &tm_aux));
  // launch_prepare clears the status word; every other byte of the scratch that is read below is
  // written first by these launches, so nothing depends on what an earlier call left behind
  SFB_CUDA(launch_prepare(d, F1, F2, w.F1r, w.F2r, w.aux, w.status, st));
  SweepArgs a;
  memset(&a, 0, sizeof(a));
  a.d = d;
  a.mode = SWEEP_MAXAVG;
  a.n_valid = w.n1p;
  a.pu = packed_view(w.ou, d.H2, MAXAVG_SLOTS, w.n1p);
  a.pv = packed_view(w.ov, d.W2, MAXAVG_SLOTS, w.n1p);
  a.status = w.status;
  set_sweep_split(a, w, MAXAVG_PART_SLOTS);
  SFB_CUDA(launch_sweep(with_wait_settings(a), tm_f1, tm_f2, tm_aux, st));
  const PatchJob out[2] = {{MA_u, w.ou, 2, d.H2, 2, 0, MAXAVG_SLOTS, 0}, {MA_v, w.ov, 2, d.W2, 2, 0, MAXAVG_SLOTS, 0}};
  SFB_CUDA(launch_unpack(out, 2, d.B, d.N1(), w.n1p, st));
  return SFB_OK;
}

size_t sfb_static_scratch_bytes(void) { return STATIC_SCRATCH_BYTES; }

int sfb_static_device_status(void* stream, int32_t* device_status) {
  void* scratch = nullptr;
  SFB_TRY(static_scratch(&scratch));  // the status word is the first word of the built-in scratch
  return sfb_device_status(scratch, stream, device_status);
}

int sfb_max_argmax_avg_forward(const float* F1, const float* F2, float* MA_u, float* MA_v, int32_t* AM_u,
                               int32_t* AM_v, const sfb_shape* shape, void* workspace, size_t workspace_bytes,
                               void* stream) {
  return run_maxavg_forward(F1, F2, MA_u, MA_v, AM_u, AM_v, true, shape, workspace, workspace_bytes, stream);
}

int sfb_compression_forward(const float* F1, const float* F2, const float* A_u, const float* A_v, float* C_u,
                            float* C_v, const sfb_shape* shape, void* workspace, size_t workspace_bytes,
                            void* stream) {
  Dims d;
  SFB_TRY(check_shape(shape, true, &d));
  SFB_CHECK_PTR(F1); SFB_CHECK_PTR(F2); SFB_CHECK_PTR(A_u); SFB_CHECK_PTR(A_v); SFB_CHECK_PTR(C_u); SFB_CHECK_PTR(C_v);
  Workspace w;
  SFB_TRY(check_workspace(d, workspace, workspace_bytes, SFB_OP_COMPRESSION_FORWARD, &w));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int op16;
  SFB_TRY(operand_mode(d, &op16));
  CUtensorMap tm_f1, tm_f2;
  SFB_TRY(map_sweep_operands(d, w, op16, &tm_f1, nullptr, &tm_f2, nullptr));
  const Features feat{F1, F2, false, 1.f, op16};
  SFB_PREPARE(feat, false);
  const int K = d.Kc;
  SFB_TRY(pack_weights(d, w, A_u, A_v, st));   // w_u[k][v] = XV slot k, w_v[k][u] = XU slot k
  SFB_TRY(run_compress_sweeps(d, w, tm_f1, tm_f2, packed_view(w.xu, d.H2, K, w.n1p), packed_view(w.xv, d.W2, K, w.n1p),
                              0, 0, 1, packed_view(w.ou, d.H2, K, w.n1p), packed_view(w.ov, d.W2, K, w.n1p), w.n1p, st, op16, sweep_out_scale(w, op16)));
  return unpack_sums(d, w, C_u, C_v, st);
}

int sfb_max_argmax_avg_backward(const float* F1, const float* F2, const int32_t* AM_u, const int32_t* AM_v,
                                const float* gMA_u, const float* gMA_v, float* gF1, float* gF2,
                                const sfb_shape* shape, void* workspace, size_t workspace_bytes, void* stream) {
  Dims d;
  SFB_TRY(check_shape(shape, false, &d));
  SFB_CHECK_PTR(F1); SFB_CHECK_PTR(F2); SFB_CHECK_PTR(AM_u); SFB_CHECK_PTR(AM_v);
  SFB_CHECK_PTR(gMA_u); SFB_CHECK_PTR(gMA_v); SFB_CHECK_PTR(gF1); SFB_CHECK_PTR(gF2);
  Workspace w;
  SFB_TRY(check_workspace(d, workspace, workspace_bytes, SFB_OP_MAX_ARGMAX_AVG_BACKWARD, &w));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int op16;
  SFB_TRY(operand_mode(d, &op16));
  const Features feat{F1, F2, false, 1.f, op16};
  SFB_PREPARE(feat, false);
  const size_t pix = (size_t)d.B * d.N1();
  SFB_TRY(grad_operand_scales(w, op16, {{gMA_u, pix * 2 * d.H2}, {gMA_v, pix * 2 * d.W2}}, {}, st));
  SFB_CUDA(timed(KID_PACK, pack_launches(2, d.B), st, [&] {
    SlotSources su, sv;
    PackGroups groups{};
    maxavg_slot_sources(d, AM_u, AM_v, gMA_u, gMA_v, &su, &sv, grad_slot_scales(w, op16));
    groups.add(su, w.gxu, d.H2, 4, 1, 0);
    groups.add(sv, w.gxv, d.W2, 4, 1, 0);
    return launch_pack_interleaved(groups, d.B, d.N1(), w.n1p, st);
  }));
  return run_grad_pair(d, w, feat, GRAD_MAXAVG, 4, 0, gF1, gF2, st);
}

int sfb_compression_backward(const float* F1, const float* F2, const float* A_u, const float* A_v,
                             const float* gC_u, const float* gC_v, float* gF1, float* gF2, float* gA_u,
                             float* gA_v, const sfb_shape* shape, void* workspace, size_t workspace_bytes,
                             void* stream) {
  Dims d;
  SFB_TRY(check_shape(shape, true, &d));
  SFB_CHECK_PTR(F1); SFB_CHECK_PTR(F2); SFB_CHECK_PTR(A_u); SFB_CHECK_PTR(A_v); SFB_CHECK_PTR(gC_u); SFB_CHECK_PTR(gC_v);
  SFB_CHECK_PTR(gF1); SFB_CHECK_PTR(gF2); SFB_CHECK_PTR(gA_u); SFB_CHECK_PTR(gA_v);
  Workspace w;
  SFB_TRY(check_workspace(d, workspace, workspace_bytes, SFB_OP_COMPRESSION_BACKWARD, &w));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int op16;
  SFB_TRY(operand_mode(d, &op16));
  const Features feat{F1, F2, false, 1.f, op16};
  SFB_PREPARE(feat, false);
  const int N1 = d.N1(), K = d.Kc;
  SFB_TRY(run_attention_grads(d, w, gC_u, gC_v, gA_u, gA_v, st, op16));
  {
    const size_t pk = (size_t)d.B * N1 * K;
    SFB_TRY(grad_operand_scales(w, op16, {{gC_u, pk * d.H2}, {gC_v, pk * d.W2}}, {{A_u, pk * d.W2}, {A_v, pk * d.H2}}, st));
  }
  // gradient GEMMs, at most KC_MAX_PER_SWEEP channels per pass; later passes add to gF1 / gF2.
  for (int k0 = 0; k0 < K; k0 += KC_MAX_PER_SWEEP) {
    const int kc = chunk_channels(K - k0), R4 = grad_slots(kc);
    SFB_CUDA(timed(KID_PACK, pack_launches(R4 / 2, d.B), st, [&] {
      SlotSources su, sv;
      PackGroups groups{};
      compress_slot_sources(K, k0, kc, A_u, A_v, gC_u, gC_v, &su, &sv, grad_slot_scales(w, op16));
      groups.add(su, w.gxu, d.H2, R4, R4 / 4, 0);
      groups.add(sv, w.gxv, d.W2, R4, R4 / 4, 0);
      return launch_pack_interleaved(groups, d.B, N1, w.n1p, st);
    }));
    SFB_TRY(run_grad_pair(d, w, feat, GRAD_COMPRESS, R4, k0 > 0 ? 1 : 0, gF1, gF2, st));
  }
  return SFB_OK;
}

int sfb_compression_attention_backward(const float* F1, const float* F2, const float* gC_u, const float* gC_v,
                                       float* gA_u, float* gA_v, const sfb_shape* shape, void* workspace,
                                       size_t workspace_bytes, void* stream) {
  Dims d;
  SFB_TRY(check_shape(shape, true, &d));
  SFB_CHECK_PTR(F1); SFB_CHECK_PTR(F2); SFB_CHECK_PTR(gC_u); SFB_CHECK_PTR(gC_v); SFB_CHECK_PTR(gA_u); SFB_CHECK_PTR(gA_v);
  Workspace w;
  SFB_TRY(check_workspace(d, workspace, workspace_bytes, SFB_OP_COMPRESSION_FORWARD, &w));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int op16;
  SFB_TRY(operand_mode(d, &op16));
  const Features feat{F1, F2, false, 1.f, op16};
  SFB_PREPARE(feat, false);
  return run_attention_grads(d, w, gC_u, gC_v, gA_u, gA_v, st, op16);
}

// Feature gradients of both backward ops from one GEMM pair (plus accumulated passes for channels beyond
// KC_MAX_PER_SWEEP).  The call's prepare_operands has run.
static int run_fused_feature_grads(const Dims& d, const Workspace& w, const Features& feat, const int32_t* AM_u, const int32_t* AM_v,
                                   const float* gMA_u, const float* gMA_v, const float* A_u, const float* A_v,
                                   const float* gC_u, const float* gC_v, float* gF1, float* gF2, cudaStream_t st) {
  const int N1 = d.N1(), K = d.Kc;
  const int op16 = feat.op16;
  {
    const size_t pix = (size_t)d.B * N1;
    SFB_TRY(grad_operand_scales(w, op16,
                                {{gMA_u, pix * 2 * d.H2}, {gMA_v, pix * 2 * d.W2}, {gC_u, pix * K * d.H2}, {gC_v, pix * K * d.W2}},
                                {{A_u, pix * K * d.W2}, {A_v, pix * K * d.H2}}, st));
  }
  const float* const gs = grad_slot_scales(w, op16);
  {  // group 0 = max/avg slots, groups 1.. = the first (up to 4) compression channels; G is their sum
    const int kc = chunk_channels(K), Qc = grad_slots(kc) / 4, Q = 1 + Qc;
    SFB_CUDA(timed(KID_PACK, pack_launches(2 * Q, d.B), st, [&] {
      SlotSources su, sv;
      PackGroups groups{};
      maxavg_slot_sources(d, AM_u, AM_v, gMA_u, gMA_v, &su, &sv, gs);
      groups.add(su, w.gxu, d.H2, 4, Q, 0);
      groups.add(sv, w.gxv, d.W2, 4, Q, 0);
      compress_slot_sources(K, 0, kc, A_u, A_v, gC_u, gC_v, &su, &sv, gs);
      groups.add(su, w.gxu, d.H2, 4 * Qc, Q, 1);
      groups.add(sv, w.gxv, d.W2, 4 * Qc, Q, 1);
      return launch_pack_interleaved(groups, d.B, N1, w.n1p, st);
    }));
    SFB_TRY(run_grad_pair(d, w, feat, GRAD_FUSED, 4 * Q, 0, gF1, gF2, st));
  }
  for (int k0 = KC_MAX_PER_SWEEP; k0 < K; k0 += KC_MAX_PER_SWEEP) {  // remaining channels: compression form, accumulated
    const int kc = chunk_channels(K - k0), R4 = grad_slots(kc);
    SFB_CUDA(timed(KID_PACK, pack_launches(R4 / 2, d.B), st, [&] {
      SlotSources su, sv;
      PackGroups groups{};
      compress_slot_sources(K, k0, kc, A_u, A_v, gC_u, gC_v, &su, &sv, gs);
      groups.add(su, w.gxu, d.H2, R4, R4 / 4, 0);
      groups.add(sv, w.gxv, d.W2, R4, R4 / 4, 0);
      return launch_pack_interleaved(groups, d.B, N1, w.n1p, st);
    }));
    SFB_TRY(run_grad_pair(d, w, feat, GRAD_COMPRESS, R4, 1, gF1, gF2, st));
  }
  return SFB_OK;
}

int sfb_separation_feature_backward(const float* F1, const float* F2, const int32_t* AM_u, const int32_t* AM_v,
                                    const float* gMA_u, const float* gMA_v, const float* A_u, const float* A_v,
                                    const float* gC_u, const float* gC_v, float* gF1, float* gF2,
                                    const sfb_shape* shape, void* workspace, size_t workspace_bytes, void* stream) {
  Dims d;
  SFB_TRY(check_shape(shape, true, &d));
  SFB_CHECK_PTR(F1); SFB_CHECK_PTR(F2); SFB_CHECK_PTR(AM_u); SFB_CHECK_PTR(AM_v); SFB_CHECK_PTR(gMA_u); SFB_CHECK_PTR(gMA_v);
  SFB_CHECK_PTR(A_u); SFB_CHECK_PTR(A_v); SFB_CHECK_PTR(gC_u); SFB_CHECK_PTR(gC_v); SFB_CHECK_PTR(gF1); SFB_CHECK_PTR(gF2);
  Workspace w;
  SFB_TRY(check_workspace(d, workspace, workspace_bytes, SFB_OP_SEPARATION_BACKWARD, &w));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int op16;
  SFB_TRY(operand_mode(d, &op16));
  const Features feat{F1, F2, false, 1.f, op16};
  SFB_PREPARE(feat, false);
  return run_fused_feature_grads(d, w, feat, AM_u, AM_v, gMA_u, gMA_v, A_u, A_v, gC_u, gC_v, gF1, gF2, st);
}

int sfb_separation_backward(const float* F1, const float* F2, const int32_t* AM_u, const int32_t* AM_v,
                            const float* gMA_u, const float* gMA_v, const float* A_u, const float* A_v,
                            const float* gC_u, const float* gC_v, float* gF1, float* gF2, float* gA_u,
                            float* gA_v, const sfb_shape* shape, void* workspace, size_t workspace_bytes,
                            void* stream) {
  Dims d;
  SFB_TRY(check_shape(shape, true, &d));
  SFB_CHECK_PTR(F1); SFB_CHECK_PTR(F2); SFB_CHECK_PTR(AM_u); SFB_CHECK_PTR(AM_v); SFB_CHECK_PTR(gMA_u); SFB_CHECK_PTR(gMA_v);
  SFB_CHECK_PTR(A_u); SFB_CHECK_PTR(A_v); SFB_CHECK_PTR(gC_u); SFB_CHECK_PTR(gC_v);
  SFB_CHECK_PTR(gF1); SFB_CHECK_PTR(gF2); SFB_CHECK_PTR(gA_u); SFB_CHECK_PTR(gA_v);
  Workspace w;
  SFB_TRY(check_workspace(d, workspace, workspace_bytes, SFB_OP_SEPARATION_BACKWARD, &w));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int op16;
  SFB_TRY(operand_mode(d, &op16));
  const Features feat{F1, F2, false, 1.f, op16};
  SFB_PREPARE(feat, false);
  SFB_TRY(run_attention_grads(d, w, gC_u, gC_v, gA_u, gA_v, st, op16));
  return run_fused_feature_grads(d, w, feat, AM_u, AM_v, gMA_u, gMA_v, A_u, A_v, gC_u, gC_v, gF1, gF2, st);
}

int sfb_max_argmax_avg_forward_cf(const float* F1, const float* F2, float* SEP_v, float* SEP_u, int32_t* AM_u,
                                  int32_t* AM_v, const sfb_shape* shape, void* workspace, size_t workspace_bytes,
                                  void* stream) {
  Dims d;
  SFB_TRY(check_shape(shape, false, &d));
  SFB_CHECK_PTR(F1); SFB_CHECK_PTR(F2); SFB_CHECK_PTR(SEP_v); SFB_CHECK_PTR(SEP_u);
  const bool with_argmax = AM_u != nullptr || AM_v != nullptr;
  if (with_argmax) { SFB_CHECK_PTR(AM_u); SFB_CHECK_PTR(AM_v); }
  Workspace w;
  SFB_TRY(check_workspace(d, workspace, workspace_bytes, SFB_OP_MAX_AVG_FORWARD_CF, &w));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int op16;
  SFB_TRY(operand_mode(d, &op16));
  CUtensorMap tm_f1, tm_f2, tm_aux;
  SFB_TRY(map_sweep_operands(d, w, op16, &tm_f1, &tm_f2, nullptr, &tm_aux));
  const Features feat{F1, F2, false, 1.f, op16};
  SFB_PREPARE(feat, true);
  const int N1 = d.N1();
  SweepArgs a;
  memset(&a, 0, sizeof(a));
  a.d = d;
  a.op16 = op16;
  a.out_scale = sweep_out_scale(w, op16);
  a.mode = with_argmax ? SWEEP_MAXARGAVG : SWEEP_MAXAVG;
  a.n_valid = N1;
  a.pu = cf_view(SEP_v, 2, d.H2, N1);       // per-u channels live in the tensor the call site calls sep_v
  a.pv = cf_view(SEP_u, 2, d.W2, N1);
  a.pu_arg = cf_view(AM_u, 1, d.H2, N1);
  a.pv_arg = cf_view(AM_v, 1, d.W2, N1);
  a.status = w.status;
  set_sweep_split(a, w, MAXAVG_PART_SLOTS);
  SFB_CUDA(timed(KID_SWEEP_MAXAVG, contraction_launches(a), st, [&] { return launch_sweep(with_wait_settings(a), tm_f1, tm_f2, tm_aux, st); }));
  return SFB_OK;
}

// compression sweep on channels-first weights / outputs (forward, or attention gradients with the upstream
// gradients as weights)
static int run_compress_cf(const float* F1, const float* F2, const float* W_u, const float* W_v, float* O_u, float* O_v,
                           const sfb_shape* shape, void* workspace, size_t workspace_bytes, void* stream) {
  Dims d;
  SFB_TRY(check_shape(shape, true, &d));
  SFB_CHECK_PTR(F1); SFB_CHECK_PTR(F2); SFB_CHECK_PTR(W_u); SFB_CHECK_PTR(W_v); SFB_CHECK_PTR(O_u); SFB_CHECK_PTR(O_v);
  Workspace w;
  SFB_TRY(check_workspace(d, workspace, workspace_bytes, SFB_OP_COMPRESSION_CF, &w));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int op16;
  SFB_TRY(operand_mode(d, &op16));
  CUtensorMap tm_f1, tm_f2;
  SFB_TRY(map_sweep_operands(d, w, op16, &tm_f1, nullptr, &tm_f2, nullptr));
  const Features feat{F1, F2, false, 1.f, op16};
  SFB_PREPARE(feat, false);
  const int N1 = d.N1(), K = d.Kc;
  // W_u (B,K,W2,N1) weights per v, W_v (B,K,H2,N1) per u; O_u (B,K,H2,N1), O_v (B,K,W2,N1)
  return run_compress_sweeps(d, w, tm_f1, tm_f2, cf_view(W_v, K, d.H2, N1), cf_view(W_u, K, d.W2, N1), 0, 0, 1,
                             cf_view(O_u, K, d.H2, N1), cf_view(O_v, K, d.W2, N1), N1, st, op16, sweep_out_scale(w, op16));
}

int sfb_compression_forward_cf(const float* F1, const float* F2, const float* A_u, const float* A_v, float* C_u,
                               float* C_v, const sfb_shape* shape, void* workspace, size_t workspace_bytes,
                               void* stream) {
  return run_compress_cf(F1, F2, A_u, A_v, C_u, C_v, shape, workspace, workspace_bytes, stream);
}

int sfb_compression_attention_backward_cf(const float* F1, const float* F2, const float* gC_u, const float* gC_v,
                                          float* gA_u, float* gA_v, const sfb_shape* shape, void* workspace,
                                          size_t workspace_bytes, void* stream) {
  // gA_v(b,k,u,p) = sum_v S * gC_v(b,k,v,p), gA_u(b,k,v,p) = sum_u S * gC_u(b,k,u,p)
  return run_compress_cf(F1, F2, gC_v, gC_u, gA_v, gA_u, shape, workspace, workspace_bytes, stream);
}

// Channels-first form of run_fused_feature_grads: gMA sources gM_v (B,2,H2,N1) / gM_u (B,2,W2,N1); the compression
// gradients are channels g0.. of tensors with gK channels.
static int run_fused_feature_grads_cf(const Dims& d, const Workspace& w, const Features& feat, const int32_t* AM_u, const int32_t* AM_v,
                                      const float* gM_v, const float* gM_u, const float* A_u, const float* A_v,
                                      const float* gC_u, const float* gC_v, int gK, int g0, float* gF1, float* gF2,
                                      cudaStream_t st, int out_cf = 0, float scale1 = 1.f, bool unit_weights = false) {
  const int N1 = d.N1(), K = d.Kc;
  const int op16 = feat.op16;
  {  // FP16 operands: scales from the whole gradient tensors (an upper bound when only some channels are this level's);
     // unit_weights: A_u / A_v are softmax outputs
    const size_t bn = (size_t)d.B * N1;
    if (unit_weights)
      SFB_TRY(grad_operand_scales(w, op16, {{gM_v, bn * 2 * d.H2}, {gM_u, bn * 2 * d.W2}, {gC_u, bn * gK * d.H2}, {gC_v, bn * gK * d.W2}}, {}, st));
    else
      SFB_TRY(grad_operand_scales(w, op16, {{gM_v, bn * 2 * d.H2}, {gM_u, bn * 2 * d.W2}, {gC_u, bn * gK * d.H2}, {gC_v, bn * gK * d.W2}},
                                  {{A_u, bn * K * d.W2}, {A_v, bn * K * d.H2}}, st));
  }
  const float* const gs = grad_slot_scales(w, op16);
  {
    const int kc = chunk_channels(K), Qc = grad_slots(kc) / 4, Q = 1 + Qc;
    SFB_CUDA(timed(KID_PACK, pack_launches(2 * Q, d.B), st, [&] {
      SlotSources su, sv;
      PackGroups groups{};
      // channel 0 = max gradient, channel 1 = mean gradient (same slots as the reference layout)
      maxavg_slot_sources(d, AM_u, AM_v, gM_v, gM_u, &su, &sv, gs);
      groups.add(su, w.gxu, d.H2, 4, Q, 0);
      groups.add(sv, w.gxv, d.W2, 4, Q, 0);
      compress_slot_sources(K, 0, kc, A_u, A_v, gC_u, gC_v, &su, &sv, gs, gK, g0);
      groups.add(su, w.gxu, d.H2, 4 * Qc, Q, 1);
      groups.add(sv, w.gxv, d.W2, 4 * Qc, Q, 1);
      return launch_pack_interleaved_cf(groups, d.B, N1, w.n1p, st);
    }));
    SFB_TRY(run_grad_pair(d, w, feat, GRAD_FUSED, 4 * Q, 0, gF1, gF2, st, out_cf, scale1));
  }
  for (int k0 = KC_MAX_PER_SWEEP; k0 < K; k0 += KC_MAX_PER_SWEEP) {
    const int kc = chunk_channels(K - k0), R4 = grad_slots(kc);
    SFB_CUDA(timed(KID_PACK, pack_launches(2 * (R4 / 4), d.B), st, [&] {
      SlotSources su, sv;
      PackGroups groups{};
      compress_slot_sources(K, k0, kc, A_u, A_v, gC_u, gC_v, &su, &sv, gs, gK, g0);
      groups.add(su, w.gxu, d.H2, R4, R4 / 4, 0);
      groups.add(sv, w.gxv, d.W2, R4, R4 / 4, 0);
      return launch_pack_interleaved_cf(groups, d.B, N1, w.n1p, st);
    }));
    SFB_TRY(run_grad_pair(d, w, feat, GRAD_COMPRESS, R4, 1, gF1, gF2, st, out_cf, scale1));
  }
  return SFB_OK;
}

int sfb_separation_feature_backward_cf(const float* F1, const float* F2, const int32_t* AM_u, const int32_t* AM_v,
                                       const float* gSEP_v, const float* gSEP_u, const float* A_u, const float* A_v,
                                       const float* gC_u, const float* gC_v, float* gF1, float* gF2,
                                       const sfb_shape* shape, void* workspace, size_t workspace_bytes,
                                       void* stream) {
  Dims d;
  SFB_TRY(check_shape(shape, true, &d));
  SFB_CHECK_PTR(F1); SFB_CHECK_PTR(F2); SFB_CHECK_PTR(AM_u); SFB_CHECK_PTR(AM_v); SFB_CHECK_PTR(gSEP_v); SFB_CHECK_PTR(gSEP_u);
  SFB_CHECK_PTR(A_u); SFB_CHECK_PTR(A_v); SFB_CHECK_PTR(gC_u); SFB_CHECK_PTR(gC_v); SFB_CHECK_PTR(gF1); SFB_CHECK_PTR(gF2);
  Workspace w;
  SFB_TRY(check_workspace(d, workspace, workspace_bytes, SFB_OP_SEPARATION_FEATURE_BACKWARD_CF, &w));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int op16;
  SFB_TRY(operand_mode(d, &op16));
  const Features feat{F1, F2, false, 1.f, op16};
  SFB_PREPARE(feat, false);
  return run_fused_feature_grads_cf(d, w, feat, AM_u, AM_v, gSEP_v, gSEP_u, A_u, A_v, gC_u, gC_v, d.Kc, 0, gF1, gF2, st);
}

// ---- attention weights: Conv3d(2 -> Kc, 3, padding 1) + softmax over the displacement axis ----
static int check_attention_dims(int B, int Kc, int D, int H1, int W1, AttentionDims* ad) {
  if (B < 1 || Kc < 1 || D < 1 || H1 < 1 || W1 < 1)
    return fail(SFB_ERR_INVALID_ARGUMENT, "B, Kc, D, H1, W1 must be >= 1 (got %d %d %d %d %d)", B, Kc, D, H1, W1);
  if (Kc > 64) return fail(SFB_ERR_UNSUPPORTED_SHAPE, "Kc=%d unsupported: at most 64 attention channels", Kc);
  if ((long long)H1 * W1 > (1ll << 21)) return fail(SFB_ERR_UNSUPPORTED_SHAPE, "image 1 has more than 2^21 pixels");
  *ad = AttentionDims{B, Kc, D, H1, W1};
  return SFB_OK;
}

int sfb_attention_forward(const float* X, int64_t x_batch_stride, const float* weight, const float* bias, float* A,
                          int32_t B, int32_t Kc, int32_t D, int32_t H1, int32_t W1, void* stream) {
  AttentionDims ad;
  SFB_TRY(check_attention_dims(B, Kc, D, H1, W1, &ad));
  if (X == nullptr || weight == nullptr || bias == nullptr || A == nullptr)
    return fail(SFB_ERR_INVALID_ARGUMENT, "X, weight, bias and A must not be NULL");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const AttentionJob job{ad, 0, X, x_batch_stride, A};
  const AttentionModules modules{{weight, nullptr}, {bias, nullptr}};
  SFB_CUDA(timed(KID_ATTENTION_FWD, attention_forward_launches(&job, 1, nullptr), st,
                 [&] { return launch_attention_forward(&job, 1, modules, st); }));
  return SFB_OK;
}

size_t sfb_attention_backward_workspace_bytes(int32_t B, int32_t Kc, int32_t D, int32_t H1, int32_t W1) {
  AttentionDims ad;
  if (check_attention_dims(B, Kc, D, H1, W1, &ad) != SFB_OK) return 0;
  return align_up(attention_partial_floats(&ad, 1) * sizeof(float), 256);
}

int sfb_attention_backward(const float* X, int64_t x_batch_stride, const float* weight, const float* A, float* gA,
                           const float* add, int64_t add_batch_stride, float* gX, float* gweight, float* gbias,
                           int32_t B, int32_t Kc, int32_t D, int32_t H1, int32_t W1, void* workspace,
                           size_t workspace_bytes, void* stream) {
  AttentionDims ad;
  SFB_TRY(check_attention_dims(B, Kc, D, H1, W1, &ad));
  if (X == nullptr || weight == nullptr || A == nullptr || gA == nullptr || gX == nullptr || gweight == nullptr ||
      gbias == nullptr)
    return fail(SFB_ERR_INVALID_ARGUMENT, "X, weight, A, gA, gX, gweight and gbias must not be NULL");
  if (workspace == nullptr) return fail(SFB_ERR_INVALID_ARGUMENT, "workspace is NULL");
  const size_t need = sfb_attention_backward_workspace_bytes(B, Kc, D, H1, W1);
  if (workspace_bytes < need)
    return fail(SFB_ERR_WORKSPACE_TOO_SMALL, "workspace has %zu bytes, %zu needed", workspace_bytes, need);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const AttentionGradJob job{ad, 0, X, x_batch_stride, A, gA, add, add_batch_stride, gX};
  const AttentionModules modules{{weight, nullptr}, {nullptr, nullptr}};
  const AttentionGradients grads{{gweight, nullptr}, {gbias, nullptr}};
  SFB_CUDA(timed(KID_ATTENTION_BWD, attention_backward_launches(&job, 1), st,
                 [&] { return launch_attention_backward(&job, 1, modules, grads, static_cast<float*>(workspace), st); }));
  return SFB_OK;
}

// ---- one pyramid level of the call site ----
// channels c0.. of a concatenated (B, Ktot, D, N1) tensor as a pixel view
static PixView cf_channels(const void* base, int Ktot, int c0, int D, int N1) {
  return PixView{static_cast<float*>(const_cast<void*>(base)) + (size_t)c0 * D * N1, (long long)Ktot * D * N1,
                 (uint32_t)N1, (uint32_t)(D * N1)};
}

// Where a level's (2+Kc)-channel volumes live: channels c0 .. c0+2+Kc-1 of tensors with Ktot channels (the
// concatenated outputs of all pyramid levels); {0, 0} = tensors of their own.
struct Placement { int Ktot, c0; };
static int check_placement(const Dims& d, Placement* pl) {
  const int Kt = 2 + d.Kc;
  if (pl->Ktot == 0 && pl->c0 == 0) pl->Ktot = Kt;
  if (pl->c0 < 0 || pl->c0 + Kt > pl->Ktot)
    return fail(SFB_ERR_INVALID_ARGUMENT, "channels %d..%d do not fit in %d channels", pl->c0, pl->c0 + Kt, pl->Ktot);
  const long long n1p = ((long long)d.N1() + TILE_M - 1) / TILE_M * TILE_M;
  if (n1p * pl->Ktot * (d.H2 > d.W2 ? d.H2 : d.W2) >= (1ll << 32))
    return fail(SFB_ERR_UNSUPPORTED_SHAPE, "H1*W1*max(H2,W2)*channels exceeds 2^32 elements per sample");
  return SFB_OK;
}

// fmaps != 0: F1 / F2 are the model's feature maps (B, C, H, W); F1 is multiplied by scale1 on the way in.
static int level_forward(Placement pl, const float* F1, const float* F2, int fmaps, float scale1, const float* weight_u,
                         const float* bias_u, const float* weight_v, const float* bias_v, float* SEP_u, float* SEP_v,
                         int32_t* AM_u, int32_t* AM_v, float* A_u, float* A_v, const sfb_shape* shape,
                         void* workspace, size_t workspace_bytes, void* stream) {
  Dims d;
  SFB_TRY(check_shape(shape, true, &d));
  AttentionDims ad;
  SFB_TRY(check_attention_dims(d.B, d.Kc, d.H2, d.H1, d.W1, &ad));
  SFB_CHECK_PTR(F1); SFB_CHECK_PTR(F2); SFB_CHECK_PTR(SEP_u); SFB_CHECK_PTR(SEP_v); SFB_CHECK_PTR(A_u); SFB_CHECK_PTR(A_v);
  if (weight_u == nullptr || bias_u == nullptr || weight_v == nullptr || bias_v == nullptr)
    return fail(SFB_ERR_INVALID_ARGUMENT, "attention weights and biases must not be NULL");
  SFB_TRY(check_placement(d, &pl));
  const bool with_argmax = AM_u != nullptr || AM_v != nullptr;
  if (with_argmax) { SFB_CHECK_PTR(AM_u); SFB_CHECK_PTR(AM_v); }
  Workspace w;
  SFB_TRY(check_workspace(d, workspace, workspace_bytes, SFB_OP_SEPARATION_LEVEL_FORWARD, &w));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int op16;
  SFB_TRY(operand_mode(d, &op16));
  CUtensorMap tm_f1, tm_f2, tm_f2_sums, tm_aux;
  SFB_TRY(map_sweep_operands(d, w, op16, &tm_f1, &tm_f2, &tm_f2_sums, &tm_aux));
  const Features feat{F1, F2, fmaps != 0, scale1, op16};
  SFB_PREPARE(feat, true);
  const int N1 = d.N1(), K = d.Kc, Kt = pl.Ktot, c0 = pl.c0;
  SweepArgs a;
  memset(&a, 0, sizeof(a));
  a.d = d;
  a.mode = with_argmax ? SWEEP_MAXARGAVG : SWEEP_MAXAVG;
  a.n_valid = N1;
  a.pu = cf_channels(SEP_v, Kt, c0, d.H2, N1);  // per-u channels live in the tensor the call site calls sep_v
  a.pv = cf_channels(SEP_u, Kt, c0, d.W2, N1);
  a.pu_arg = cf_view(AM_u, 1, d.H2, N1);
  a.pv_arg = cf_view(AM_v, 1, d.W2, N1);
  a.op16 = op16;
  a.out_scale = sweep_out_scale(w, op16);
  a.status = w.status;
  set_sweep_split(a, w, MAXAVG_PART_SLOTS);
  SFB_CUDA(timed(KID_SWEEP_MAXAVG, contraction_launches(a), st, [&] { return launch_sweep(with_wait_settings(a), tm_f1, tm_f2, tm_aux, st); }));
  const long long sb_u = (long long)Kt * d.W2 * N1, sb_v = (long long)Kt * d.H2 * N1;
  const AttentionDims at_u{d.B, K, d.W2, d.H1, d.W1}, at_v{d.B, K, d.H2, d.H1, d.W1};
  const float *const X_u = SEP_u + (size_t)c0 * d.W2 * N1, *const X_v = SEP_v + (size_t)c0 * d.H2 * N1;
  const AttentionJob jobs[2] = {{at_u, 0, X_u, sb_u, A_u}, {at_v, 1, X_v, sb_v, A_v}};
  const AttentionModules modules{{weight_u, weight_v}, {bias_u, bias_v}};
  SFB_CUDA(timed(KID_ATTENTION_FWD, attention_forward_launches(jobs, 2, w.status), st,
                 [&] { return launch_attention_forward(jobs, 2, modules, st, w.status); }));
  // C_u (per u, weights A_u per v) -> SEP_v channels 2.., C_v -> SEP_u channels 2..
  return run_compress_sweeps(d, w, tm_f1, tm_f2_sums, cf_view(A_v, K, d.H2, N1), cf_view(A_u, K, d.W2, N1), 0, 0, 1,
                             cf_channels(SEP_v, Kt, c0 + 2, d.H2, N1), cf_channels(SEP_u, Kt, c0 + 2, d.W2, N1), N1, st,
                             op16, sweep_out_scale(w, op16));
}

int sfb_separation_level_forward(const float* F1, const float* F2, const float* weight_u, const float* bias_u,
                                 const float* weight_v, const float* bias_v, float* SEP_u, float* SEP_v,
                                 int32_t* AM_u, int32_t* AM_v, float* A_u, float* A_v, const sfb_shape* shape,
                                 void* workspace, size_t workspace_bytes, void* stream) {
  return level_forward(Placement{0, 0}, F1, F2, 0, 1.f, weight_u, bias_u, weight_v, bias_v, SEP_u, SEP_v, AM_u, AM_v, A_u,
                       A_v, shape, workspace, workspace_bytes, stream);
}

int sfb_separation_level_forward_fmaps(const float* fmap1, const float* fmap2, float scale1, const float* weight_u,
                                       const float* bias_u, const float* weight_v, const float* bias_v, float* SEP_u,
                                       float* SEP_v, int32_t sep_channels, int32_t sep_channel0, int32_t* AM_u,
                                       int32_t* AM_v, float* A_u, float* A_v, const sfb_shape* shape, void* workspace,
                                       size_t workspace_bytes, void* stream) {
  return level_forward(Placement{sep_channels, sep_channel0}, fmap1, fmap2, 1, scale1, weight_u, bias_u, weight_v, bias_v,
                       SEP_u, SEP_v, AM_u, AM_v, A_u, A_v, shape, workspace, workspace_bytes, stream);
}

static int level_backward(Placement pl, const float* F1, const float* F2, int fmaps, float scale1, const float* weight_u,
                          const float* weight_v, const float* SEP_u, const float* SEP_v, const int32_t* AM_u,
                          const int32_t* AM_v, const float* A_u, const float* A_v, const float* gSEP_u,
                          const float* gSEP_v, float* gF1, float* gF2, float* gweight_u, float* gbias_u,
                          float* gweight_v, float* gbias_v, const sfb_shape* shape, void* workspace,
                          size_t workspace_bytes, void* stream) {
  Dims d;
  SFB_TRY(check_shape(shape, true, &d));
  AttentionDims ad;
  SFB_TRY(check_attention_dims(d.B, d.Kc, d.H2, d.H1, d.W1, &ad));
  SFB_CHECK_PTR(F1); SFB_CHECK_PTR(F2); SFB_CHECK_PTR(SEP_u); SFB_CHECK_PTR(SEP_v); SFB_CHECK_PTR(AM_u); SFB_CHECK_PTR(AM_v);
  SFB_CHECK_PTR(A_u); SFB_CHECK_PTR(A_v); SFB_CHECK_PTR(gSEP_u); SFB_CHECK_PTR(gSEP_v); SFB_CHECK_PTR(gF1); SFB_CHECK_PTR(gF2);
  if (weight_u == nullptr || weight_v == nullptr || gweight_u == nullptr || gbias_u == nullptr || gweight_v == nullptr ||
      gbias_v == nullptr)
    return fail(SFB_ERR_INVALID_ARGUMENT, "attention weights and their gradient buffers must not be NULL");
  SFB_TRY(check_placement(d, &pl));
  Workspace w;
  SFB_TRY(check_workspace(d, workspace, workspace_bytes, SFB_OP_SEPARATION_LEVEL_BACKWARD, &w));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int op16;
  SFB_TRY(operand_mode(d, &op16));
  CUtensorMap tm_f1, tm_f2;
  SFB_TRY(map_sweep_operands(d, w, op16, &tm_f1, nullptr, &tm_f2, nullptr));
  const Features feat{F1, F2, fmaps != 0, fmaps ? scale1 : 1.f, op16};
  SFB_PREPARE(feat, false);
  const int N1 = d.N1(), K = d.Kc, Kt = pl.Ktot, c0 = pl.c0;
  // attention gradients: gA_v(b,k,u,p) = sum_v S * gC_v(b,k,v,p), gA_u(b,k,v,p) = sum_u S * gC_u(b,k,u,p), with
  // gC_u = gSEP_v[:, 2:] (per u) and gC_v = gSEP_u[:, 2:] (per v) in the role of the weights
  SFB_TRY(run_compress_sweeps(d, w, tm_f1, tm_f2, cf_channels(gSEP_v, Kt, c0 + 2, d.H2, N1),
                              cf_channels(gSEP_u, Kt, c0 + 2, d.W2, N1), 0, 0, 1, cf_view(w.ga_v, K, d.H2, N1),
                              cf_view(w.ga_u, K, d.W2, N1), N1, st, op16, sweep_out_scale(w, op16)));
  // through softmax and Conv3d: parameter gradients, and the total gradients of the max/avg channels
  const long long sb_u = (long long)Kt * d.W2 * N1, sb_v = (long long)Kt * d.H2 * N1;
  const size_t ou = (size_t)c0 * d.W2 * N1, ov = (size_t)c0 * d.H2 * N1;  // first channel of this level
  const AttentionGradJob jobs[2] = {
      {AttentionDims{d.B, K, d.W2, d.H1, d.W1}, 0, SEP_u + ou, sb_u, A_u, w.ga_u, gSEP_u + ou, sb_u, w.gm_u},
      {AttentionDims{d.B, K, d.H2, d.H1, d.W1}, 1, SEP_v + ov, sb_v, A_v, w.ga_v, gSEP_v + ov, sb_v, w.gm_v}};
  const AttentionModules modules{{weight_u, weight_v}, {nullptr, nullptr}};
  const AttentionGradients grads{{gweight_u, gweight_v}, {gbias_u, gbias_v}};
  SFB_CUDA(timed(KID_ATTENTION_BWD, attention_backward_launches(jobs, 2), st,
                 [&] { return launch_attention_backward(jobs, 2, modules, grads, w.at_partial, st, w.status); }));
  return run_fused_feature_grads_cf(d, w, feat, AM_u, AM_v, w.gm_v, w.gm_u, A_u, A_v, gSEP_v, gSEP_u, Kt, c0 + 2, gF1, gF2, st,
                                    fmaps, fmaps ? scale1 : 1.f, /*unit_weights=*/true);
}

int sfb_separation_level_backward(const float* F1, const float* F2, const float* weight_u, const float* weight_v,
                                  const float* SEP_u, const float* SEP_v, const int32_t* AM_u, const int32_t* AM_v,
                                  const float* A_u, const float* A_v, const float* gSEP_u, const float* gSEP_v,
                                  float* gF1, float* gF2, float* gweight_u, float* gbias_u, float* gweight_v,
                                  float* gbias_v, const sfb_shape* shape, void* workspace, size_t workspace_bytes,
                                  void* stream) {
  return level_backward(Placement{0, 0}, F1, F2, 0, 1.f, weight_u, weight_v, SEP_u, SEP_v, AM_u, AM_v, A_u, A_v, gSEP_u,
                        gSEP_v, gF1, gF2, gweight_u, gbias_u, gweight_v, gbias_v, shape, workspace, workspace_bytes, stream);
}

int sfb_separation_level_backward_fmaps(const float* fmap1, const float* fmap2, float scale1, const float* weight_u,
                                        const float* weight_v, const float* SEP_u, const float* SEP_v,
                                        int32_t sep_channels, int32_t sep_channel0, const int32_t* AM_u,
                                        const int32_t* AM_v, const float* A_u, const float* A_v, const float* gSEP_u,
                                        const float* gSEP_v, float* gfmap1, float* gfmap2, float* gweight_u,
                                        float* gbias_u, float* gweight_v, float* gbias_v, const sfb_shape* shape,
                                        void* workspace, size_t workspace_bytes, void* stream) {
  return level_backward(Placement{sep_channels, sep_channel0}, fmap1, fmap2, 1, scale1, weight_u, weight_v, SEP_u, SEP_v,
                        AM_u, AM_v, A_u, A_v, gSEP_u, gSEP_v, gfmap1, gfmap2, gweight_u, gbias_u, gweight_v, gbias_v, shape,
                        workspace, workspace_bytes, stream);
}


// ---- placement of a level's volumes into the concatenated level-0-sized outputs ----
static int check_resample(const void* a, const void* b, int B, int K, int Dl, int D0, int H1, int W1) {
  if (a == nullptr || b == nullptr) return fail(SFB_ERR_INVALID_ARGUMENT, "tensor pointers must not be NULL");
  if (B < 1 || K < 1 || Dl < 1 || D0 < 1 || H1 < 1 || W1 < 1)
    return fail(SFB_ERR_INVALID_ARGUMENT, "B, K, Dl, D0, H1, W1 must be >= 1");
  if (Dl > D0) return fail(SFB_ERR_UNSUPPORTED_SHAPE, "Dl=%d > D0=%d: only upsampling is supported", Dl, D0);
  if (B * (long long)K > 65535 || D0 > 65535) return fail(SFB_ERR_UNSUPPORTED_SHAPE, "B*K and D0 must be <= 65535");
  if ((long long)H1 * W1 > (1ll << 24)) return fail(SFB_ERR_UNSUPPORTED_SHAPE, "image 1 has more than 2^24 pixels");
  return SFB_OK;
}

int sfb_upsample_displacement(const float* in, float* out, int64_t out_batch_stride, int32_t B, int32_t K, int32_t Dl,
                              int32_t D0, int32_t H1, int32_t W1, void* stream) {
  SFB_TRY(check_resample(in, out, B, K, Dl, D0, H1, W1));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SFB_CUDA(timed(KID_RESAMPLE, 1, st, [&] {
    const ResampleJob job{in, out, out_batch_stride, Dl, D0};
    return launch_upsample_displacement(&job, 1, B, K, H1 * W1, st);
  }));
  return SFB_OK;
}

int sfb_upsample_displacement_backward(const float* gout, int64_t gout_batch_stride, float* gin, int32_t B, int32_t K,
                                       int32_t Dl, int32_t D0, int32_t H1, int32_t W1, void* stream) {
  SFB_TRY(check_resample(gout, gin, B, K, Dl, D0, H1, W1));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SFB_CUDA(timed(KID_RESAMPLE, 1, st, [&] {
    const ResampleAdjointJob job{gout, gout_batch_stride, gin, Dl, D0};
    return launch_upsample_displacement_adjoint(&job, 1, B, K, H1 * W1, st);
  }));
  return SFB_OK;
}

}  // extern "C"

// ---- all pyramid levels of the call site ----
namespace {
// What the levels of a call share and what each has of its own.  Image 1, C and Kc are the same for all of them.
struct Pyramid {
  int levels;
  Dims d[MAX_FUSED_LEVELS];
  bool in_place[MAX_FUSED_LEVELS];   // the level has the displacement ranges of the outputs: its channels of them are its volumes
};

int check_pyramid(const sfb_shape* shape, const int32_t* H2, const int32_t* W2, int levels, Pyramid* py) {
  if (shape == nullptr || H2 == nullptr || W2 == nullptr) return fail(SFB_ERR_INVALID_ARGUMENT, "shape, H2 and W2 must not be NULL");
  if (levels < 1 || levels > MAX_FUSED_LEVELS)
    return fail(SFB_ERR_UNSUPPORTED_SHAPE, "levels must be in [1, %d] (got %d)", MAX_FUSED_LEVELS, levels);
  py->levels = levels;
  for (int l = 0; l < levels; ++l) {
    sfb_shape s = *shape;
    s.H2 = H2[l];
    s.W2 = W2[l];
    SFB_TRY(check_shape(&s, true, &py->d[l]));
    if (H2[l] > H2[0] || W2[l] > W2[0]) return fail(SFB_ERR_UNSUPPORTED_SHAPE, "level %d of image 2 is larger than level 0", l);
    py->in_place[l] = H2[l] == H2[0] && W2[l] == W2[0];
  }
  const Dims& d = py->d[0];
  if (d.Kc > KC_MAX_PER_SWEEP)
    return fail(SFB_ERR_UNSUPPORTED_SHAPE, "the levels share a launch for at most %d attention channels (got %d)", KC_MAX_PER_SWEEP, d.Kc);
  if ((long long)d.B * (2 + d.Kc) > 65535) return fail(SFB_ERR_UNSUPPORTED_SHAPE, "B * (2 + Kc) must be <= 65535");
  Placement pl{levels * (2 + d.Kc), 0};
  return check_placement(d, &pl);
}

// Tensors a forward leaves for its backward, in one buffer: the volumes of the levels that are not in place, arg-max indices (when
// there is a backward), attention weights.
struct PyramidSaved {
  float *sep_u[MAX_FUSED_LEVELS], *sep_v[MAX_FUSED_LEVELS], *a_u[MAX_FUSED_LEVELS], *a_v[MAX_FUSED_LEVELS];
  int32_t *am_u[MAX_FUSED_LEVELS], *am_v[MAX_FUSED_LEVELS];
  float* fmap2[MAX_FUSED_LEVELS];   // pooled levels
  size_t bytes;
};
PyramidSaved carve_saved(const Pyramid& py, void* base, bool with_argmax, bool pooled) {
  PyramidSaved v;
  size_t off = 0;
  auto take = [&](size_t floats) {
    float* r = reinterpret_cast<float*>(static_cast<char*>(base) + off);
    off += align_up(floats * sizeof(float), 256);
    return r;
  };
  for (int l = 0; l < py.levels; ++l) {
    const Dims& d = py.d[l];
    const size_t bn = (size_t)d.B * d.N1();
    v.sep_u[l] = py.in_place[l] ? nullptr : take(bn * (2 + d.Kc) * d.W2);
    v.sep_v[l] = py.in_place[l] ? nullptr : take(bn * (2 + d.Kc) * d.H2);
    v.am_u[l] = with_argmax ? reinterpret_cast<int32_t*>(take(bn * d.H2)) : nullptr;
    v.am_v[l] = with_argmax ? reinterpret_cast<int32_t*>(take(bn * d.W2)) : nullptr;
    v.a_u[l] = take(bn * d.Kc * d.W2);
    v.a_v[l] = take(bn * d.Kc * d.H2);
  }
  for (int l = 0; l < py.levels; ++l) v.fmap2[l] = pooled && l > 0 ? take((size_t)py.d[l].B * py.d[l].C * py.d[l].N2()) : nullptr;
  v.bytes = off;
  return v;
}

// Workspaces of the levels: every level has what carve() gives it, image 1's copies and the header are level 0's, and the
// scratch of cut tiles follows.
struct PyramidWorkspace {
  Workspace w[MAX_FUSED_LEVELS];
  size_t bytes;
};
// A sweep over all levels is cut as a whole; the parts of its levels lie one behind the other.
size_t pyramid_part_floats(const Pyramid& py, int slots, bool sums, TileSplit* split) {
  sweep_split_levels(py.d, py.levels, slots, sums, split);
  size_t floats = 0;
  for (int l = 0; l < py.levels; ++l) floats += split[l].part_floats;
  return floats;
}
PyramidWorkspace carve_pyramid_forward(const Pyramid& py, void* base) {
  PyramidWorkspace p;
  size_t off = 0;
  auto take = [&](size_t floats) {
    float* r = reinterpret_cast<float*>(static_cast<char*>(base) + off);
    off += align_up(floats * sizeof(float), 256);
    return r;
  };
  const Dims& d0 = py.d[0];
  int* const status = reinterpret_cast<int*>(take(WS_HEADER_BYTES / sizeof(float)));
  float* const F1 = take((size_t)d0.B * d0.N1() * d0.C);
  for (int l = 0; l < py.levels; ++l) {
    const Dims& d = py.d[l];
    Workspace& w = p.w[l];
    w = Workspace{};
    w.status = status;
    w.scales = reinterpret_cast<float*>(reinterpret_cast<char*>(status) + WS_SCALES_OFFSET) + l * SCALE_LEVEL;
    w.n1p = padded_pixels(d);
    w.F1r = F1;
    w.F2r = take((size_t)d.B * d.N2() * d.C);
    w.aux = take((size_t)d.B * d.aux_rows() * d.C);
    w.F1h = reinterpret_cast<uint16_t*>(w.F1r);
    w.F2h = reinterpret_cast<uint16_t*>(w.F2r);
    w.auxh = reinterpret_cast<uint16_t*>(w.aux);
  }
  TileSplit split[MAX_FUSED_LEVELS];
  const size_t part = std::max(pyramid_part_floats(py, MAXAVG_PART_SLOTS, false, split),
                               pyramid_part_floats(py, chunk_channels(d0.Kc), true, split));
  float* const parts = take(part);
  for (int l = 0; l < py.levels; ++l) p.w[l].part = parts;
  p.bytes = off;
  return p;
}

// Cuts of the gradient GEMMs of a pyramid whose G is stored `samples` at a time (0: generated twice), for chunks of the batch and the
// shorter last one, image-1-major and image-2-major; the scratch that the largest takes.
struct PyramidGradPlan {
  int samples;
  TileSplit split[2][2][MAX_FUSED_LEVELS];
  size_t part_bytes;
};
PyramidGradPlan plan_pyramid_grads(const Pyramid& py, int samples) {
  PyramidGradPlan plan;
  plan.samples = samples;
  size_t part = 0;
  const int B = py.d[0].B, chunk = samples > 0 ? samples : B;
  for (const int last : {0, 1}) {
    Dims d[MAX_FUSED_LEVELS];
    for (int l = 0; l < py.levels; ++l) {
      d[l] = py.d[l];
      d[l].B = last ? B % chunk : chunk;
    }
    if (d[0].B == 0) continue;
    for (const int image2 : {0, 1}) {
      TileSplit* const split = plan.split[last][image2];
      grad_split_levels(d, py.levels, samples > 0 ? (image2 ? GRAD_IMAGE2_STORED : GRAD_IMAGE1_STORING) : (image2 ? GRAD_IMAGE2 : GRAD_IMAGE1), split);
      size_t floats = 0;
      for (int l = 0; l < py.levels; ++l) floats += split[l].part_floats;
      part = std::max(part, floats);
    }
  }
  plan.part_bytes = align_up(part * sizeof(float), 256);
  return plan;
}

// The backward's buffer: the header and the gradients of pooled levels of image 2 (gf2), then two regions of which each is used twice.
//   first : the copies of the sweep, the attention gradients and the scratch of both; then, once those are through, the GEMMs' operands
//           and channel-major copies
//   second: the gradients of the max/avg channels and of the volumes that are not in place (gs_u, gs_v), which the operands are packed
//           from; then the GEMMs' scratch and G
// Image 1's copies are shared by the levels.  8 x 135 x 240, C = 256, four channels and levels: 12.9 GB with room for G, 20.2 with all arrays
// side by side; a level alone takes 8.1, 12.3 with room for G.
struct PyramidBackward {
  Workspace w[MAX_FUSED_LEVELS];
  float *gs_u[MAX_FUSED_LEVELS], *gs_v[MAX_FUSED_LEVELS], *gf2[MAX_FUSED_LEVELS];
  size_t second, end;      // where the second region begins, and ends before the GEMMs
  size_t sample_bytes;     // stored G of a sample
  size_t bytes(const PyramidGradPlan& plan) const { return std::max(end, second + plan.part_bytes + plan.samples * sample_bytes); }
};
PyramidBackward carve_pyramid_backward(const Pyramid& py, void* base) {
  PyramidBackward p;
  size_t off = 0;
  auto take = [&](size_t floats) {
    float* r = reinterpret_cast<float*>(static_cast<char*>(base) + off);
    off += align_up(floats * sizeof(float), 256);
    return r;
  };
  const Dims& d0 = py.d[0];
  const size_t bn = (size_t)d0.B * d0.N1();
  const int n1p = padded_pixels(d0), Kt = 2 + d0.Kc, Rg = 4 + grad_slots(d0.Kc);
  int* const status = reinterpret_cast<int*>(take(WS_HEADER_BYTES / sizeof(float)));
  for (int l = 0; l < py.levels; ++l) {
    Workspace& w = p.w[l];
    w = Workspace{};
    w.status = status;
    w.scales = reinterpret_cast<float*>(reinterpret_cast<char*>(status) + WS_SCALES_OFFSET) + l * SCALE_LEVEL;
    w.n1p = n1p;
    p.gf2[l] = l == 0 ? nullptr : take((size_t)py.d[l].B * py.d[l].C * py.d[l].N2());
  }
  const size_t first = off;
  float* const F1 = take(bn * d0.C);
  AttentionDims at[MAX_ATTENTION_JOBS];
  for (int l = 0; l < py.levels; ++l) {
    const Dims& d = py.d[l];
    Workspace& w = p.w[l];
    w.F1r = F1;
    w.F2r = take((size_t)d.B * d.N2() * d.C);
    w.F1h = reinterpret_cast<uint16_t*>(w.F1r);
    w.F2h = reinterpret_cast<uint16_t*>(w.F2r);
    w.ga_u = take(bn * d.Kc * d.W2);
    w.ga_v = take(bn * d.Kc * d.H2);
    at[2 * l] = AttentionDims{d.B, d.Kc, d.W2, d.H1, d.W1};
    at[2 * l + 1] = AttentionDims{d.B, d.Kc, d.H2, d.H1, d.W1};
  }
  TileSplit split[MAX_FUSED_LEVELS];
  float* const parts = take(pyramid_part_floats(py, chunk_channels(d0.Kc), true, split));
  float* const at_partial = take(attention_partial_floats(at, 2 * py.levels));
  const size_t swept = off;
  off = first;
  float* const F1t = take((size_t)d0.B * d0.C * n1p);
  for (int l = 0; l < py.levels; ++l) {
    const Dims& d = py.d[l];
    Workspace& w = p.w[l];
    w.part = parts;
    w.at_partial = at_partial;
    w.F1t = F1t;
    w.h2p = (d.H2 + GG_UT - 1) / GG_UT * GG_UT;
    w.F2t = take((size_t)d.B * f2t_per_sample(d, w));
    w.gxu = take((size_t)d.B * d.H2 * Rg * n1p);
    w.gxv = take((size_t)d.B * d.W2 * Rg * n1p);
  }
  p.second = off = std::max(swept, off);
  p.sample_bytes = 0;
  for (int l = 0; l < py.levels; ++l) {
    const Dims& d = py.d[l];
    Workspace& w = p.w[l];
    w.gm_u = take(bn * 2 * d.W2);
    w.gm_v = take(bn * 2 * d.H2);
    p.gs_u[l] = py.in_place[l] ? nullptr : take(bn * Kt * d.W2);
    p.gs_v[l] = py.in_place[l] ? nullptr : take(bn * Kt * d.H2);
    p.sample_bytes += grad_stored_bytes(d, n1p);
  }
  p.end = off;
  return p;
}
// The most samples of G at a time that a buffer has room for.  Buffers of pyramid_backward_bytes() have it for all that are wanted.
PyramidGradPlan pyramid_grad_plan(const Pyramid& py, const PyramidBackward& pb, int op16, size_t room) {
  for (int n = pb.end <= room ? grad_chunk(py.d[0], py.levels, pb.sample_bytes, op16) : 0; n > 0;) {
    const PyramidGradPlan plan = plan_pyramid_grads(py, n);
    if (pb.bytes(plan) <= room) return plan;
    // the scratch may differ with the cut of a smaller chunk, so that its room is looked at again
    n = std::min<long long>(n - 1, room > pb.second + plan.part_bytes ? (room - pb.second - plan.part_bytes) / pb.sample_bytes : 0);
  }
  return plan_pyramid_grads(py, 0);
}
// least: without room for G beyond what there is anyway.
size_t pyramid_backward_bytes(const Pyramid& py, bool least) {
  const PyramidBackward pb = carve_pyramid_backward(py, nullptr);
  const size_t twice = pb.bytes(plan_pyramid_grads(py, 0));
  return least ? twice : std::max(twice, pb.bytes(pyramid_grad_plan(py, pb, op16_of(py.d[0]), SIZE_MAX)));
}

// The sweeps of all levels: `fill(l, a)` sets a level's views, the rest is common.
template <class Fill>
int run_pyramid_sweeps(const Pyramid& py, const Workspace* w, int op16, int mode, cudaStream_t st, Fill&& fill) {
  const bool sums = mode == SWEEP_COMPRESS;
  const int slots = sums ? chunk_channels(py.d[0].Kc) : MAXAVG_PART_SLOTS;
  CUtensorMap tm_f1, tm_f2[MAX_FUSED_LEVELS], tm_aux[MAX_FUSED_LEVELS];
  SweepArgs a[MAX_FUSED_LEVELS];
  TileSplit split[MAX_FUSED_LEVELS];
  pyramid_part_floats(py, slots, sums, split);
  float* part = w[0].part;
  int launches = 1;
  for (int l = 0; l < py.levels; ++l) {
    SFB_TRY(map_sweep_operands(py.d[l], w[l], op16, &tm_f1, sums ? nullptr : &tm_f2[l], sums ? &tm_f2[l] : nullptr, sums ? nullptr : &tm_aux[l]));
    if (sums) tm_aux[l] = tm_f2[l];   // unused
    memset(&a[l], 0, sizeof(a[l]));
    a[l].d = py.d[l];
    a[l].mode = mode;
    a[l].n_valid = py.d[l].N1();
    a[l].kc = sums ? py.d[l].Kc : 0;
    a[l].w_stride = 1;
    a[l].op16 = op16;
    a[l].out_scale = sweep_out_scale(w[l], op16);
    a[l].status = w[l].status;
    a[l].whole_tiles = split[l].whole_tiles;
    a[l].pieces = split[l].pieces;
    a[l].parts = split[l].parts;
    a[l].part_slots = slots;
    a[l].part = part;
    part += split[l].part_floats;
    if (split[l].pieces > 1) launches = 2;
    fill(l, a[l]);
    a[l] = with_wait_settings(a[l]);
  }
  SFB_CUDA(timed(sums ? KID_SWEEP_COMPRESS : KID_SWEEP_MAXAVG, launches, st,
                 [&] { return launch_sweep_levels(a, py.levels, tm_f1, tm_f2, tm_aux, st); }));
  return SFB_OK;
}

// Operand copies of all levels (and the mean rows of image 2 when with_aux).
int prepare_pyramid(const Pyramid& py, const Workspace* w, const float* fmap1, const float* const* fmap2, float* const* pooled, float scale1,
                    bool with_aux, int op16, cudaStream_t st) {
  LevelOperands out[MAX_FUSED_LEVELS];
  for (int l = 0; l < py.levels; ++l)
    out[l] = op16 ? LevelOperands{nullptr, nullptr, w[l].F2h, with_aux ? w[l].auxh : nullptr}
                  : LevelOperands{w[l].F2r, with_aux ? w[l].aux : nullptr, nullptr, nullptr};
  const int launches = prepare_launches(w[0], true, with_aux, op16) + (pooled != nullptr && op16 != OP16_FP16 ? 1 : 0);
  SFB_CUDA(timed(KID_PREPARE, launches, st, [&] {
    return launch_prepare_cf(py.d, py.levels, fmap1, fmap2, scale1, out, op16 ? nullptr : w[0].F1r, op16 ? w[0].F1h : nullptr, w[0].status,
                             st, op16, w[0].scales, pooled);
  }));
  return SFB_OK;
}

// Image 2's levels as the caller gives them: all, or the first alone (the others NULL), which are then its 2 x 2 averages.
int check_levels(const Pyramid& py, const void* const* fmap2, const char* name, bool* pooled) {
  *pooled = py.levels > 1 && fmap2[1] == nullptr;
  for (int l = 0; l < py.levels; ++l) {
    if (*pooled && l > 0) {
      if (fmap2[l] != nullptr) return fail(SFB_ERR_INVALID_ARGUMENT, "%s: all levels from the second on must be NULL or none", name);
      if (py.d[l].H2 != py.d[l - 1].H2 / 2 || py.d[l].W2 != py.d[l - 1].W2 / 2)
        return fail(SFB_ERR_INVALID_ARGUMENT, "%s: level %d is not half of the level before", name, l);
      continue;
    }
    SFB_TRY(check_ptr(fmap2[l], name));
  }
  return SFB_OK;
}

// Where the volumes of a level are: channels of the outputs, or tensors of their own.
struct LevelVolumes {
  float *u, *v;            // (B, 2 + Kc, W2, N1) / (B, 2 + Kc, H2, N1), first sample
  long long sb_u, sb_v;    // elements between samples
};
LevelVolumes level_volumes(const Pyramid& py, int l, float* SEP_u, float* SEP_v, float* own_u, float* own_v) {
  const Dims& d = py.d[l];
  const int Kt = 2 + d.Kc, N1 = d.N1(), K = py.in_place[l] ? Kt * py.levels : Kt, c0 = py.in_place[l] ? l * Kt : 0;
  return LevelVolumes{(py.in_place[l] ? SEP_u : own_u) + (size_t)c0 * d.W2 * N1, (py.in_place[l] ? SEP_v : own_v) + (size_t)c0 * d.H2 * N1,
                      (long long)K * d.W2 * N1, (long long)K * d.H2 * N1};
}
PixView volume_view(float* base, long long sb, int channel, int D, int N1) {
  return PixView{base + (size_t)channel * D * N1, sb, (uint32_t)N1, (uint32_t)(D * N1)};
}
}  // namespace

extern "C" {

int sfb_pool_levels(const float* fmap2, float* const* pooled, int32_t B, int32_t C, int32_t H, int32_t W, int32_t levels, void* stream) {
  if (levels < 2 || levels > MAX_FUSED_LEVELS)
    return fail(SFB_ERR_UNSUPPORTED_SHAPE, "levels must be in [2, %d] (got %d)", MAX_FUSED_LEVELS, levels);
  if (B < 1 || C < 1 || H < 1 || W < 1 || std::min(H, W) >> (levels - 1) < 1)
    return fail(SFB_ERR_INVALID_ARGUMENT, "%d levels need maps of at least one pixel each (got %d x %d x %d x %d)", levels, B, C, H, W);
  if ((long long)B * C > INT_MAX || (long long)H * W > INT_MAX) return fail(SFB_ERR_UNSUPPORTED_SHAPE, "maps too large");
  Dims d[MAX_FUSED_LEVELS];
  float* out[MAX_FUSED_LEVELS] = {nullptr};
  bool all = fmap2 != nullptr && pooled != nullptr;
  for (int l = 0; l < levels; ++l) {
    d[l] = Dims{B, 1, 1, H >> l, W >> l, C, 0};
    if (l > 0 && all) out[l] = pooled[l - 1];
    all = all && (l == 0 || out[l] != nullptr);
  }
  if (!all) return fail(SFB_ERR_INVALID_ARGUMENT, "fmap2 and pooled must not be NULL");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SFB_CUDA(timed(KID_PREPARE, 1, st, [&] { return launch_pool_levels(d, levels, fmap2, out, st); }));
  return SFB_OK;
}

size_t sfb_separation_pyramid_saved_bytes(const sfb_shape* shape, const int32_t* H2, const int32_t* W2, int32_t levels,
                                          int32_t with_argmax, int32_t pooled) {
  Pyramid py;
  if (check_pyramid(shape, H2, W2, levels, &py) != SFB_OK) return 0;
  return carve_saved(py, nullptr, with_argmax != 0, pooled != 0).bytes;
}

size_t sfb_separation_pyramid_workspace_bytes(const sfb_shape* shape, const int32_t* H2, const int32_t* W2, int32_t levels,
                                              int32_t backward) {
  Pyramid py;
  if (check_pyramid(shape, H2, W2, levels, &py) != SFB_OK) return 0;
  return backward == 0 ? carve_pyramid_forward(py, nullptr).bytes : pyramid_backward_bytes(py, backward == 2);
}

int sfb_separation_pyramid_forward(const float* fmap1, const float* const* fmap2, const int32_t* H2, const int32_t* W2,
                                   int32_t levels, float scale1, const float* weight_u, const float* bias_u,
                                   const float* weight_v, const float* bias_v, float* SEP_u, float* SEP_v, void* saved,
                                   size_t saved_bytes, int32_t with_argmax, const sfb_shape* shape, void* workspace,
                                   size_t workspace_bytes, void* stream) {
  Pyramid py;
  SFB_TRY(check_pyramid(shape, H2, W2, levels, &py));
  SFB_CHECK_PTR(fmap1); SFB_CHECK_PTR(SEP_u); SFB_CHECK_PTR(SEP_v); SFB_CHECK_PTR(saved);
  if (fmap2 == nullptr) return fail(SFB_ERR_INVALID_ARGUMENT, "fmap2 is NULL");
  bool pooled;
  SFB_TRY(check_levels(py, reinterpret_cast<const void* const*>(fmap2), "fmap2", &pooled));
  if (weight_u == nullptr || bias_u == nullptr || weight_v == nullptr || bias_v == nullptr)
    return fail(SFB_ERR_INVALID_ARGUMENT, "attention weights and biases must not be NULL");
  const PyramidSaved sv = carve_saved(py, saved, with_argmax != 0, pooled);
  if (saved_bytes < sv.bytes) return fail(SFB_ERR_WORKSPACE_TOO_SMALL, "saved has %zu bytes, %zu needed", saved_bytes, sv.bytes);
  if (workspace == nullptr || (reinterpret_cast<uintptr_t>(workspace) & 255u) != 0)
    return fail(SFB_ERR_INVALID_ARGUMENT, "workspace is NULL or not 256-byte aligned");
  const PyramidWorkspace pw = carve_pyramid_forward(py, workspace);
  if (workspace_bytes < pw.bytes)
    return fail(SFB_ERR_WORKSPACE_TOO_SMALL, "workspace has %zu bytes, %zu needed", workspace_bytes, pw.bytes);
  const Dims& d0 = py.d[0];
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int op16;
  SFB_TRY(operand_mode(d0, &op16));
  const float* maps2[MAX_FUSED_LEVELS];
  for (int l = 0; l < levels; ++l) maps2[l] = pooled && l > 0 ? sv.fmap2[l] : fmap2[l];
  SFB_TRY(prepare_pyramid(py, pw.w, fmap1, maps2, pooled ? sv.fmap2 : nullptr, scale1, true, op16, st));
  const int N1 = d0.N1(), K = d0.Kc, Kt = 2 + K;
  LevelVolumes vol[MAX_FUSED_LEVELS];
  for (int l = 0; l < levels; ++l) vol[l] = level_volumes(py, l, SEP_u, SEP_v, sv.sep_u[l], sv.sep_v[l]);
  SFB_TRY(run_pyramid_sweeps(py, pw.w, op16, with_argmax != 0 ? SWEEP_MAXARGAVG : SWEEP_MAXAVG, st, [&](int l, SweepArgs& a) {
    a.pu = volume_view(vol[l].v, vol[l].sb_v, 0, py.d[l].H2, N1);   // per-u channels live in the tensor the call site calls sep_v
    a.pv = volume_view(vol[l].u, vol[l].sb_u, 0, py.d[l].W2, N1);
    a.pu_arg = cf_view(sv.am_u[l], 1, py.d[l].H2, N1);
    a.pv_arg = cf_view(sv.am_v[l], 1, py.d[l].W2, N1);
  }));
  AttentionJob jobs[MAX_ATTENTION_JOBS];
  for (int l = 0; l < levels; ++l) {
    const Dims& d = py.d[l];
    jobs[2 * l] = AttentionJob{AttentionDims{d.B, K, d.W2, d.H1, d.W1}, 0, vol[l].u, vol[l].sb_u, sv.a_u[l]};
    jobs[2 * l + 1] = AttentionJob{AttentionDims{d.B, K, d.H2, d.H1, d.W1}, 1, vol[l].v, vol[l].sb_v, sv.a_v[l]};
  }
  const AttentionModules modules{{weight_u, weight_v}, {bias_u, bias_v}};
  int* const status = pw.w[0].status;
  SFB_CUDA(timed(KID_ATTENTION_FWD, attention_forward_launches(jobs, 2 * levels, status), st,
                 [&] { return launch_attention_forward(jobs, 2 * levels, modules, st, status); }));
  // C_u (per u, weights A_u per v) -> the v volume's channels 2.., C_v -> the u volume's
  SFB_TRY(run_pyramid_sweeps(py, pw.w, op16, SWEEP_COMPRESS, st, [&](int l, SweepArgs& a) {
    a.xu = cf_view(sv.a_v[l], K, py.d[l].H2, N1);
    a.xv = cf_view(sv.a_u[l], K, py.d[l].W2, N1);
    a.ou = volume_view(vol[l].v, vol[l].sb_v, 2, py.d[l].H2, N1);
    a.ov = volume_view(vol[l].u, vol[l].sb_u, 2, py.d[l].W2, N1);
  }));
  ResampleJob up[MAX_RESAMPLE_JOBS];
  int n = 0;
  for (int l = 0; l < levels; ++l) {
    if (py.in_place[l]) continue;
    const long long c0 = (long long)l * Kt;
    up[n++] = ResampleJob{vol[l].u, SEP_u + c0 * d0.W2 * N1, (long long)Kt * levels * d0.W2 * N1, py.d[l].W2, d0.W2};
    up[n++] = ResampleJob{vol[l].v, SEP_v + c0 * d0.H2 * N1, (long long)Kt * levels * d0.H2 * N1, py.d[l].H2, d0.H2};
  }
  if (n > 0) SFB_CUDA(timed(KID_RESAMPLE, 1, st, [&] { return launch_upsample_displacement(up, n, d0.B, Kt, N1, st); }));
  return SFB_OK;
}

int sfb_separation_pyramid_backward(const float* fmap1, const float* const* fmap2, const int32_t* H2, const int32_t* W2,
                                    int32_t levels, float scale1, const float* weight_u, const float* weight_v,
                                    const float* SEP_u, const float* SEP_v, const void* saved, size_t saved_bytes,
                                    const float* gSEP_u, const float* gSEP_v, float* gfmap1, float* const* gfmap2,
                                    float* gweight_u, float* gbias_u, float* gweight_v, float* gbias_v,
                                    const sfb_shape* shape, void* workspace, size_t workspace_bytes, void* stream) {
  Pyramid py;
  SFB_TRY(check_pyramid(shape, H2, W2, levels, &py));
  SFB_CHECK_PTR(fmap1); SFB_CHECK_PTR(SEP_u); SFB_CHECK_PTR(SEP_v); SFB_CHECK_PTR(saved);
  SFB_CHECK_PTR(gSEP_u); SFB_CHECK_PTR(gSEP_v); SFB_CHECK_PTR(gfmap1);
  if (fmap2 == nullptr || gfmap2 == nullptr) return fail(SFB_ERR_INVALID_ARGUMENT, "fmap2 and gfmap2 must not be NULL");
  bool pooled, grads_pooled;
  SFB_TRY(check_levels(py, reinterpret_cast<const void* const*>(fmap2), "fmap2", &pooled));
  SFB_TRY(check_levels(py, reinterpret_cast<const void* const*>(gfmap2), "gfmap2", &grads_pooled));
  if (pooled && !grads_pooled) return fail(SFB_ERR_INVALID_ARGUMENT, "gfmap2 must be the first level alone where fmap2 is");
  if (weight_u == nullptr || weight_v == nullptr || gweight_u == nullptr || gbias_u == nullptr || gweight_v == nullptr ||
      gbias_v == nullptr)
    return fail(SFB_ERR_INVALID_ARGUMENT, "attention weights and their gradient buffers must not be NULL");
  const PyramidSaved sv = carve_saved(py, const_cast<void*>(saved), true, pooled);
  if (saved_bytes < sv.bytes) return fail(SFB_ERR_WORKSPACE_TOO_SMALL, "saved has %zu bytes, %zu needed", saved_bytes, sv.bytes);
  if (workspace == nullptr || (reinterpret_cast<uintptr_t>(workspace) & 255u) != 0)
    return fail(SFB_ERR_INVALID_ARGUMENT, "workspace is NULL or not 256-byte aligned");
  const PyramidBackward pb = carve_pyramid_backward(py, workspace);
  int op16;   // read once: it decides the plan, too
  SFB_TRY(operand_mode(py.d[0], &op16));
  const PyramidGradPlan plan = pyramid_grad_plan(py, pb, op16, workspace_bytes);
  if (workspace_bytes < pb.bytes(plan))
    return fail(SFB_ERR_WORKSPACE_TOO_SMALL, "workspace has %zu bytes, %zu needed", workspace_bytes, pb.bytes(plan));
  const Dims& d0 = py.d[0];
  const Workspace* const w = pb.w;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const float* maps2[MAX_FUSED_LEVELS];
  float* grads2[MAX_FUSED_LEVELS];
  for (int l = 0; l < levels; ++l) {
    maps2[l] = pooled && l > 0 ? sv.fmap2[l] : fmap2[l];
    grads2[l] = grads_pooled && l > 0 ? pb.gf2[l] : gfmap2[l];
  }
  SFB_TRY(prepare_pyramid(py, w, fmap1, maps2, nullptr, scale1, false, op16, st));
  const int N1 = d0.N1(), K = d0.Kc, Kt = 2 + K;
  const size_t bn = (size_t)d0.B * N1;
  float *const SU = const_cast<float*>(SEP_u), *const SV = const_cast<float*>(SEP_v);
  float *const GU = const_cast<float*>(gSEP_u), *const GV = const_cast<float*>(gSEP_v);
  LevelVolumes vol[MAX_FUSED_LEVELS], grad[MAX_FUSED_LEVELS];
  ResampleAdjointJob down[MAX_RESAMPLE_JOBS];
  int n = 0;
  for (int l = 0; l < levels; ++l) {
    vol[l] = level_volumes(py, l, SU, SV, sv.sep_u[l], sv.sep_v[l]);
    grad[l] = level_volumes(py, l, GU, GV, pb.gs_u[l], pb.gs_v[l]);
    if (py.in_place[l]) continue;
    const long long c0 = (long long)l * Kt;
    down[n++] = ResampleAdjointJob{gSEP_u + c0 * d0.W2 * N1, (long long)Kt * levels * d0.W2 * N1, pb.gs_u[l], py.d[l].W2, d0.W2};
    down[n++] = ResampleAdjointJob{gSEP_v + c0 * d0.H2 * N1, (long long)Kt * levels * d0.H2 * N1, pb.gs_v[l], py.d[l].H2, d0.H2};
  }
  if (n > 0) SFB_CUDA(timed(KID_RESAMPLE, 1, st, [&] { return launch_upsample_displacement_adjoint(down, n, d0.B, Kt, N1, st); }));
  // attention gradients: the compression sweep with the upstream gradients in the role of the weights (level_backward)
  SFB_TRY(run_pyramid_sweeps(py, w, op16, SWEEP_COMPRESS, st, [&](int l, SweepArgs& a) {
    a.xu = volume_view(grad[l].v, grad[l].sb_v, 2, py.d[l].H2, N1);
    a.xv = volume_view(grad[l].u, grad[l].sb_u, 2, py.d[l].W2, N1);
    a.ou = cf_view(w[l].ga_v, K, py.d[l].H2, N1);
    a.ov = cf_view(w[l].ga_u, K, py.d[l].W2, N1);
  }));
  AttentionGradJob jobs[MAX_ATTENTION_JOBS];
  for (int l = 0; l < levels; ++l) {
    const Dims& d = py.d[l];
    jobs[2 * l] = AttentionGradJob{AttentionDims{d.B, K, d.W2, d.H1, d.W1}, 0, vol[l].u, vol[l].sb_u, sv.a_u[l], w[l].ga_u,
                                   grad[l].u, grad[l].sb_u, w[l].gm_u};
    jobs[2 * l + 1] = AttentionGradJob{AttentionDims{d.B, K, d.H2, d.H1, d.W1}, 1, vol[l].v, vol[l].sb_v, sv.a_v[l], w[l].ga_v,
                                       grad[l].v, grad[l].sb_v, w[l].gm_v};
  }
  const AttentionModules modules{{weight_u, weight_v}, {nullptr, nullptr}};
  const AttentionGradients grads{{gweight_u, gweight_v}, {gbias_u, gbias_v}};
  SFB_CUDA(timed(KID_ATTENTION_BWD, attention_backward_launches(jobs, 2 * levels), st, [&] {
    return launch_attention_backward(jobs, 2 * levels, modules, grads, w[0].at_partial, st, w[0].status);
  }));
  if (op16 == OP16_FP16) {   // scales of the gradient operands, from the level's channels alone; the weights are softmax outputs
    AbsmaxSource src[ABSMAX_MAX];
    int m = 0;
    for (int l = 0; l < levels; ++l) {
      const Dims& d = py.d[l];
      const int slot = l * SCALE_LEVEL + SCALE_AMAX_G;
      auto channels = [&](const float* vols, long long sb, int D) {
        const size_t len = (size_t)K * D * N1;
        // very large batches: the samples with the channels between them, as one array
        return d.B <= 1024 ? AbsmaxSource{vols + (size_t)2 * D * N1, len, sb, d.B, 1.f, slot}
                           : absmax_array(vols + (size_t)2 * D * N1, (size_t)sb * (d.B - 1) + len, 1.f, slot);
      };
      src[m++] = absmax_array(w[l].gm_v, bn * 2 * d.H2, 1.f, slot);
      src[m++] = absmax_array(w[l].gm_u, bn * 2 * d.W2, 1.f, slot);
      src[m++] = channels(grad[l].v, grad[l].sb_v, d.H2);
      src[m++] = channels(grad[l].u, grad[l].sb_u, d.W2);
    }
    SFB_CUDA(timed(KID_PREPARE, 1, st, [&] { return launch_absmax(src, m, w[0].scales, levels, true, st); }));
  }
  // G = max/avg terms + compression terms, as in run_fused_feature_grads_cf
  const int Qc = grad_slots(K) / 4, Q = 1 + Qc;
  PackGroups groups{};
  MapCopy copies[MAX_MAP_COPIES];
  const Features feat{fmap1, nullptr, true, scale1, op16};
  copies[0] = f1_copy(d0, w[0], feat);
  for (int l = 0; l < levels; ++l) {
    const Dims& d = py.d[l];
    const float* const gs = grad_slot_scales(w[l], op16);
    SlotSources su, sv2;
    maxavg_slot_sources(d, sv.am_u[l], sv.am_v[l], w[l].gm_v, w[l].gm_u, &su, &sv2, gs);
    groups.add(su, w[l].gxu, d.H2, 4, Q, 0);
    groups.add(sv2, w[l].gxv, d.W2, 4, Q, 0);
    // (a level that is not in place has its channels in tensors of 2 + Kc)
    const int gK = py.in_place[l] ? Kt * levels : Kt, g0 = py.in_place[l] ? l * Kt + 2 : 2;
    compress_slot_sources(K, 0, K, sv.a_u[l], sv.a_v[l], py.in_place[l] ? gSEP_v : pb.gs_v[l], py.in_place[l] ? gSEP_u : pb.gs_u[l], &su, &sv2,
                          gs, gK, g0);
    groups.add(su, w[l].gxu, d.H2, 4 * Qc, Q, 1);
    groups.add(sv2, w[l].gxv, d.W2, 4 * Qc, Q, 1);
    copies[1 + l] = f2_copy(d, w[l], maps2[l], op16);
  }
  SFB_CUDA(timed(KID_PACK, pack_launches(groups.count, d0.B), st, [&] { return launch_pack_interleaved_cf(groups, d0.B, N1, w[0].n1p, st); }));
  SFB_CUDA(timed(KID_PREPARE, 1, st, [&] { return launch_channel_major_cf(copies, 1 + levels, d0.B, d0.C, op16, st); }));
  // G of as many samples as the workspace takes is generated and stored by one GEMM and read back by the other (run_grad_pair)
  const int samples = plan.samples, chunk = samples > 0 ? samples : d0.B;
  for (int b0 = 0; b0 < d0.B; b0 += chunk) {
    const int here = std::min(chunk, d0.B - b0);
    for (const int form : {samples > 0 ? GRAD_IMAGE1_STORING : GRAD_IMAGE1, samples > 0 ? GRAD_IMAGE2_STORED : GRAD_IMAGE2}) {
      const bool image2_major = grad_is_image2(form);
      const TileSplit* const split = plan.split[here < chunk ? 1 : 0][image2_major ? 1 : 0];
      GradArgs a[MAX_FUSED_LEVELS];
      GradMaps maps;
      float* part = reinterpret_cast<float*>(static_cast<char*>(workspace) + pb.second);
      uint8_t* stored = reinterpret_cast<uint8_t*>(part) + plan.part_bytes;
      int part0 = -1, launches = 1;
      for (int l = 0; l < levels; ++l) {
        SFB_TRY(grad_arguments(py.d[l], w[l], op16, GRAD_FUSED, 4 * Q, form, image2_major ? grads2[l] : gfmap1, 1, scale1, &a[l], &maps.y[l],
                               &maps.xu[l], &maps.xv[l]));
        a[l].d.B = here;
        a[l].b0 = b0;
        a[l].stored = stored;
        stored += samples * grad_stored_bytes(py.d[l], w[l].n1p);
        a[l].whole_tiles = split[l].whole_tiles;
        a[l].pieces = split[l].pieces;
        a[l].parts = split[l].parts;
        a[l].part0 = part0;
        a[l].part = part;
        if (image2_major) part += split[l].part_floats;
        else part0 += split[l].pieces;
        if (a[l].parts > 0) launches = 2;
        a[l] = with_wait_settings(a[l]);
      }
      SFB_CUDA(timed(KID_GRAD_FUSED_IMG1 + (image2_major ? 1 : 0), launches, st, [&] { return launch_grad_gemm(a, levels, maps, st); }));
    }
  }
  if (grads_pooled)
    SFB_CUDA(timed(KID_PREPARE, 1, st, [&] { return launch_unpool_levels(py.d, levels, gfmap2[0], grads2, st); }));
  return SFB_OK;
}

// ---- lookup on the aggregated 3D volumes (CorrBlock1D) ----
static int check_lookup_dims(int B, int dim, int D, int H1, int W1, int levels, int radius, LookupDims* ld) {
  if (B < 1 || dim < 1 || D < 2 || H1 < 1 || W1 < 1)
    return fail(SFB_ERR_INVALID_ARGUMENT, "B, dim, H1, W1 must be >= 1 and D >= 2 (got %d %d %d %d %d)", B, dim, D, H1, W1);
  if (levels < 1 || levels > LOOKUP_MAX_LEVELS || radius < 0 || radius > 64)
    return fail(SFB_ERR_UNSUPPORTED_SHAPE, "levels must be in [1, %d] and radius in [0, 64] (got %d, %d)",
                LOOKUP_MAX_LEVELS, levels, radius);
  if ((D >> (levels - 1)) < 2)
    return fail(SFB_ERR_UNSUPPORTED_SHAPE, "the coarsest level would have fewer than 2 displacements (D=%d, levels=%d)",
                D, levels);
  if ((long long)H1 * W1 > (1ll << 24)) return fail(SFB_ERR_UNSUPPORTED_SHAPE, "image 1 has more than 2^24 pixels");
  *ld = LookupDims{B, dim, D, H1, W1, levels, radius};
  return SFB_OK;
}

static int lookup_pyramid_launches(int levels) { return (levels + 1) / 3; }   // three levels from one

size_t sfb_lookup_pyramid_bytes(int32_t B, int32_t dim, int32_t D, int32_t H1, int32_t W1, int32_t levels) {
  LookupDims ld;
  if (check_lookup_dims(B, dim, D, H1, W1, levels, 0, &ld) != SFB_OK) return 0;
  return lookup_pyramid_floats(ld) * sizeof(float);
}

int sfb_lookup_build_pyramid(const float* corr, float* pyramid, int32_t B, int32_t dim, int32_t D, int32_t H1,
                             int32_t W1, int32_t levels, void* stream) {
  LookupDims ld;
  SFB_TRY(check_lookup_dims(B, dim, D, H1, W1, levels, 0, &ld));
  if (corr == nullptr || (levels > 1 && pyramid == nullptr))
    return fail(SFB_ERR_INVALID_ARGUMENT, "corr and pyramid must not be NULL");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SFB_CUDA(timed(KID_LOOKUP, lookup_pyramid_launches(levels), st, [&] { return launch_lookup_pyramid(ld, corr, pyramid, st); }));
  return SFB_OK;
}

int sfb_lookup_forward(const float* corr, const float* pyramid, const float* coord, int64_t coord_batch_stride,
                       float* out, int32_t B, int32_t dim, int32_t D, int32_t H1, int32_t W1, int32_t levels,
                       int32_t radius, int32_t clamp_unit, void* stream) {
  LookupDims ld;
  SFB_TRY(check_lookup_dims(B, dim, D, H1, W1, levels, radius, &ld));
  if (corr == nullptr || (levels > 1 && pyramid == nullptr) || coord == nullptr || out == nullptr)
    return fail(SFB_ERR_INVALID_ARGUMENT, "corr, pyramid, coord and out must not be NULL");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SFB_CUDA(timed(KID_LOOKUP, 1, st, [&] {
    return launch_lookup_forward(ld, LookupCall{corr, pyramid, coord, coord_batch_stride, out, clamp_unit}, st);
  }));
  return SFB_OK;
}

int sfb_lookup_backward(const float* gout, const float* coord, int64_t coord_batch_stride, float* gcorr,
                        float* gpyramid, int32_t B, int32_t dim, int32_t D, int32_t H1, int32_t W1, int32_t levels,
                        int32_t radius, int32_t clamp_unit, void* stream) {
  LookupDims ld;
  SFB_TRY(check_lookup_dims(B, dim, D, H1, W1, levels, radius, &ld));
  if (gout == nullptr || coord == nullptr || gcorr == nullptr || (levels > 1 && gpyramid == nullptr))
    return fail(SFB_ERR_INVALID_ARGUMENT, "gout, coord, gcorr and gpyramid must not be NULL");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SFB_CUDA(timed(KID_LOOKUP, levels > 1 ? 2 : 1, st, [&] {
    return launch_lookup_backward(ld, gout, coord, coord_batch_stride, gcorr, gpyramid, clamp_unit, st);
  }));
  return SFB_OK;
}

// ---- both aggregated volumes of a model at once ----
static int check_lookup_pair(int B, int dim, int D1, int D2, int H1, int W1, int levels, int radius, LookupDims (&ld)[2]) {
  SFB_TRY(check_lookup_dims(B, dim, D1, H1, W1, levels, radius, &ld[0]));
  return check_lookup_dims(B, dim, D2, H1, W1, levels, radius, &ld[1]);
}

int sfb_lookup_build_pyramid_pair(const float* corr1, float* pyramid1, const float* corr2, float* pyramid2, int32_t B,
                                  int32_t dim, int32_t D1, int32_t D2, int32_t H1, int32_t W1, int32_t levels, void* stream) {
  LookupDims ld[2];
  SFB_TRY(check_lookup_pair(B, dim, D1, D2, H1, W1, levels, 0, ld));
  if (corr1 == nullptr || corr2 == nullptr || (levels > 1 && (pyramid1 == nullptr || pyramid2 == nullptr)))
    return fail(SFB_ERR_INVALID_ARGUMENT, "corr1, corr2, pyramid1 and pyramid2 must not be NULL");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SFB_CUDA(timed(KID_LOOKUP, lookup_pyramid_launches(levels), st,
                 [&] { return launch_lookup_pyramid_pair(ld, {corr1, corr2}, {pyramid1, pyramid2}, st); }));
  return SFB_OK;
}

int sfb_lookup_forward_pair(const float* corr1, const float* pyramid1, const float* corr2, const float* pyramid2,
                            const float* coords, int64_t coords_batch_stride, int64_t coords_component_stride, float* out1,
                            float* out2, int32_t B, int32_t dim, int32_t D1, int32_t D2, int32_t H1, int32_t W1, int32_t levels,
                            int32_t radius, void* stream) {
  LookupDims ld[2];
  SFB_TRY(check_lookup_pair(B, dim, D1, D2, H1, W1, levels, radius, ld));
  if (corr1 == nullptr || corr2 == nullptr || (levels > 1 && (pyramid1 == nullptr || pyramid2 == nullptr)) || coords == nullptr ||
      out1 == nullptr || out2 == nullptr)
    return fail(SFB_ERR_INVALID_ARGUMENT, "corr1, corr2, pyramid1, pyramid2, coords, out1 and out2 must not be NULL");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const LookupCall calls[2] = {{corr1, pyramid1, coords, coords_batch_stride, out1, 1},
                               {corr2, pyramid2, coords + coords_component_stride, coords_batch_stride, out2, 0}};
  SFB_CUDA(timed(KID_LOOKUP, 1, st, [&] { return launch_lookup_forward_pair(ld, calls, st); }));
  return SFB_OK;
}

size_t sfb_lookup_accumulator_bytes(int32_t B, int32_t dim, int32_t D, int32_t H1, int32_t W1, int32_t levels,
                                    int32_t clamp_unit) {
  LookupDims ld;
  if (check_lookup_dims(B, dim, D, H1, W1, levels, 0, &ld) != SFB_OK) return 0;
  return lookup_accumulator_floats(ld, clamp_unit) * sizeof(float);
}

int sfb_lookup_accumulate_pair(const float* gout1, const float* gout2, const float* coords, int64_t coords_batch_stride,
                               int64_t coords_component_stride, float* acc1, float* acc2, int32_t B, int32_t dim, int32_t D1,
                               int32_t D2, int32_t H1, int32_t W1, int32_t levels, int32_t radius, void* stream) {
  LookupDims ld[2];
  SFB_TRY(check_lookup_pair(B, dim, D1, D2, H1, W1, levels, radius, ld));
  if (coords == nullptr || (gout1 == nullptr) != (acc1 == nullptr) || (gout2 == nullptr) != (acc2 == nullptr) ||
      (gout1 == nullptr && gout2 == nullptr))
    return fail(SFB_ERR_INVALID_ARGUMENT, "coords and at least one volume's output gradient and accumulator are needed");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const LookupGradient g[2] = {{gout1, coords, coords_batch_stride, acc1, 1},
                               {gout2, coords + coords_component_stride, coords_batch_stride, acc2, 0}};
  const int first = gout1 != nullptr ? 0 : 1, volumes = gout1 != nullptr && gout2 != nullptr ? 2 : 1;
  SFB_CUDA(timed(KID_LOOKUP, 1, st, [&] { return launch_lookup_accumulate(ld + first, g + first, volumes, st); }));
  return SFB_OK;
}

int sfb_lookup_fold_gradient(const float* acc, float* gcorr, int32_t B, int32_t dim, int32_t D, int32_t H1, int32_t W1,
                             int32_t levels, int32_t clamp_unit, void* stream) {
  LookupDims ld;
  SFB_TRY(check_lookup_dims(B, dim, D, H1, W1, levels, 0, &ld));
  if (acc == nullptr || gcorr == nullptr) return fail(SFB_ERR_INVALID_ARGUMENT, "acc and gcorr must not be NULL");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SFB_CUDA(timed(KID_LOOKUP, 1, st, [&] { return launch_lookup_gradient_fold(ld, acc, gcorr, clamp_unit, st); }));
  return SFB_OK;
}

namespace {
int check_lookup4d(const void* F1, const void* const* F2, const int32_t* H2, const int32_t* W2, int32_t levels,
                   const void* coords, int32_t B, int32_t H1, int32_t W1, int32_t C, int32_t radius,
                   Lookup4dDims* out) {
  if (B < 1 || H1 < 1 || W1 < 1 || C < 1) return fail(SFB_ERR_INVALID_ARGUMENT, "B, H1, W1 and C must be positive");
  if (C % 4 != 0 || C > 512)
    return fail(SFB_ERR_INVALID_ARGUMENT, "the 4D lookup needs C % 4 == 0 and C <= 512");
  if (levels < 1 || levels > LOOKUP_MAX_LEVELS) return fail(SFB_ERR_INVALID_ARGUMENT, "levels must be in [1, 8]");
  if (radius < 0 || radius > 4) return fail(SFB_ERR_INVALID_ARGUMENT, "radius must be in [0, 4]");
  if (F1 == nullptr || F2 == nullptr || H2 == nullptr || W2 == nullptr || coords == nullptr)
    return fail(SFB_ERR_INVALID_ARGUMENT, "F1, F2_levels, H2, W2 and coords must not be NULL");
  if ((long long)H1 * W1 > INT32_MAX / 4) return fail(SFB_ERR_INVALID_ARGUMENT, "H1*W1 too large");
  if (reinterpret_cast<uintptr_t>(F1) % 16 != 0)
    return fail(SFB_ERR_INVALID_ARGUMENT, "feature pointers of the 4D lookup must be 16-byte aligned");
  out->B = B; out->H1 = H1; out->W1 = W1; out->C = C; out->levels = levels; out->radius = radius;
  for (int l = 0; l < levels; ++l) {
    // grid_sample's normalisation divides by size - 1 (core/utils/utils.py:114-115)
    if (H2[l] < 2 || W2[l] < 2)
      return fail(SFB_ERR_INVALID_ARGUMENT, "every pyramid level needs H2 >= 2 and W2 >= 2");
    if (F2[l] == nullptr) return fail(SFB_ERR_INVALID_ARGUMENT, "F2_levels holds a NULL pointer");
    if (reinterpret_cast<uintptr_t>(F2[l]) % 16 != 0)
      return fail(SFB_ERR_INVALID_ARGUMENT, "feature pointers of the 4D lookup must be 16-byte aligned");
    if ((long long)H2[l] * W2[l] > INT32_MAX / 4) return fail(SFB_ERR_INVALID_ARGUMENT, "H2*W2 too large");
    out->H2[l] = H2[l]; out->W2[l] = W2[l];
  }
  return SFB_OK;
}
}  // namespace

int sfb_lookup4d_forward(const float* F1, const float* const* F2_levels, const int32_t* H2, const int32_t* W2,
                         int32_t levels, const float* coords, float* out, int32_t B, int32_t H1, int32_t W1, int32_t C,
                         int32_t radius, float scale, void* stream) {
  Lookup4dDims ld;
  SFB_TRY(check_lookup4d(F1, reinterpret_cast<const void* const*>(F2_levels), H2, W2, levels, coords, B, H1, W1, C,
                         radius, &ld));
  if (out == nullptr) return fail(SFB_ERR_INVALID_ARGUMENT, "out must not be NULL");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SFB_CUDA(timed(KID_LOOKUP4D, 1, st, [&] { return launch_lookup4d_forward(ld, F1, F2_levels, coords, out, scale, st); }));
  return SFB_OK;
}

int sfb_lookup4d_backward(const float* F1, const float* const* F2_levels, const int32_t* H2, const int32_t* W2,
                          int32_t levels, const float* coords, const float* gout, float* gF1,
                          float* const* gF2_levels, int32_t B, int32_t H1, int32_t W1, int32_t C, int32_t radius,
                          float scale, void* stream) {
  Lookup4dDims ld;
  SFB_TRY(check_lookup4d(F1, reinterpret_cast<const void* const*>(F2_levels), H2, W2, levels, coords, B, H1, W1, C,
                         radius, &ld));
  if (gout == nullptr || gF1 == nullptr || gF2_levels == nullptr)
    return fail(SFB_ERR_INVALID_ARGUMENT, "gout, gF1 and gF2_levels must not be NULL");
  for (int l = 0; l < levels; ++l)
    if (gF2_levels[l] == nullptr || reinterpret_cast<uintptr_t>(gF2_levels[l]) % 16 != 0)
      return fail(SFB_ERR_INVALID_ARGUMENT, "gF2_levels holds a NULL or not 16-byte aligned pointer");
  if (reinterpret_cast<uintptr_t>(gF1) % 16 != 0)
    return fail(SFB_ERR_INVALID_ARGUMENT, "gF1 must be 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SFB_CUDA(timed(KID_LOOKUP4D, lookup4d_backward_launches(ld), st, [&] {
    return launch_lookup4d_backward(ld, F1, F2_levels, coords, gout, gF1, gF2_levels, scale, st);
  }));
  return SFB_OK;
}

int sfb_set_sweep_operands(int operands) {
  if (operands != SFB_OPERANDS_TF32 && operands != SFB_OPERANDS_BF16 && operands != SFB_OPERANDS_FP16) return -1;
  return g_sweep_operands.exchange(operands);
}
int sfb_get_sweep_operands(void) { return g_sweep_operands.load(); }

int sfb_corr_volume(const float* F1, const float* F2, float* S, const sfb_shape* shape, void* workspace,
                    size_t workspace_bytes, void* stream) {
  Dims d;
  SFB_TRY(check_shape(shape, false, &d));
  SFB_CHECK_PTR(F1); SFB_CHECK_PTR(F2); SFB_CHECK_PTR(S);
  Workspace w;
  SFB_TRY(check_workspace(d, workspace, workspace_bytes, SFB_OP_CORR_VOLUME, &w));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int op16 = OP16_NONE;  // this test aid always computes with TF32 operands (its workspace has no 16-bit copies)
  CUtensorMap tm_f1, tm_f2;
  SFB_TRY(map_sweep_operands(d, w, op16, &tm_f1, &tm_f2, nullptr, nullptr));
  const Features feat{F1, F2, false, 1.f, op16};
  SFB_PREPARE(feat, false);
  SweepArgs a;
  memset(&a, 0, sizeof(a));
  a.d = d;
  a.mode = SWEEP_DUMP;
  a.n_valid = w.n1p;
  a.dump = S;
  a.status = w.status;
  a.whole_tiles = d.B * ((d.N1() + TILE_M - 1) / TILE_M);
  a.pieces = 1;
  SFB_CUDA(timed(KID_SWEEP_DUMP, 1, st, [&] { return launch_sweep(with_wait_settings(a), tm_f1, tm_f2, tm_f2 /* unused */, st); }));
  return SFB_OK;
}

int sfb_debug_wait_timeout(uint64_t wait_limit_ns, int drop_last_load) {
  g_wait_limit_ns.store(wait_limit_ns);
  g_drop_last_load.store(drop_last_load != 0 ? 1 : 0);
  return SFB_OK;
}

int sfb_device_status(const void* workspace, void* stream, int32_t* device_status) {
  if (workspace == nullptr || device_status == nullptr)
    return fail(SFB_ERR_INVALID_ARGUMENT, "workspace or device_status is NULL");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int32_t v = 0;
  SFB_CUDA(cudaMemcpyAsync(&v, workspace, sizeof(v), cudaMemcpyDeviceToHost, st));
  SFB_CUDA(cudaStreamSynchronize(st));
  *device_status = v;
  if (v != 0) return fail(SFB_ERR_DEVICE_TIMEOUT, "a bounded device-side wait gave up (device status %d)", (int)v);
  return SFB_OK;
}

const char* sfb_status_string(int code) {
  switch (code) {
    case SFB_OK: return "ok";
    case SFB_ERR_INVALID_ARGUMENT: return "invalid argument";
    case SFB_ERR_UNSUPPORTED_SHAPE: return "unsupported shape";
    case SFB_ERR_WORKSPACE_TOO_SMALL: return "workspace too small";
    case SFB_ERR_CUDA: return "CUDA error";
    case SFB_ERR_DEVICE_TIMEOUT: return "device-side wait timed out";
    default: return "unknown status";
  }
}

const char* sfb_last_error(void) { return g_err; }

int sfb_kernel_timing_enable(int on) {
  std::lock_guard<std::mutex> lk(g_timing_mu);
  drain_timing_locked();
  g_timing_on = on != 0;
  for (int i = 0; i < KID_COUNT; ++i) { g_timing_ms[i] = 0; g_timing_launches[i] = 0; }
  return SFB_OK;
}

int sfb_kernel_timing_count(void) { return KID_COUNT; }

int sfb_kernel_timing_read(int kernel, const char** name, double* total_ms, int64_t* launches) {
  if (kernel < 0 || kernel >= KID_COUNT) return fail(SFB_ERR_INVALID_ARGUMENT, "kernel index %d out of range", kernel);
  std::lock_guard<std::mutex> lk(g_timing_mu);
  drain_timing_locked();
  if (name) *name = kKernelNames[kernel];
  if (total_ms) *total_ms = g_timing_ms[kernel];
  if (launches) *launches = g_timing_launches[kernel];
  return SFB_OK;
}

int sfb_version(void) { return 100; }

}  // extern "C"
