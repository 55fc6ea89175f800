// Native Python module `sfb_host`: the host side of the lookups on the two aggregated volumes (ops.lookup_build_pyramid_pair,
// lookup_forward_pair, lookup_accumulate_pair): checks, outputs from torch's allocator, one call of the C ABI on the current stream.
// A refinement makes a dozen of these calls around kernels of some 10 us each; with checks, allocations and the call through ctypes in
// Python a lookup took 15 us of host time, and adding up its gradients 20.  The entry points are handed over by the ctypes layer
// (bind), so both use the same library.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/extension.h>

#include <array>
#include <tuple>

#include "../../include/sepflow_b200.h"

namespace {

struct Abi {
  decltype(&sfb_lookup_pyramid_bytes) pyramid_bytes = nullptr;
  decltype(&sfb_lookup_build_pyramid_pair) build_pyramid_pair = nullptr;
  decltype(&sfb_lookup_forward_pair) forward_pair = nullptr;
  decltype(&sfb_lookup_accumulator_bytes) accumulator_bytes = nullptr;
  decltype(&sfb_lookup_accumulate_pair) accumulate_pair = nullptr;
  decltype(&sfb_status_string) status_string = nullptr;
  decltype(&sfb_last_error) last_error = nullptr;
};
Abi g_abi;

void bind(uintptr_t pyramid_bytes, uintptr_t build_pyramid_pair, uintptr_t forward_pair, uintptr_t accumulator_bytes, uintptr_t accumulate_pair,
          uintptr_t status_string, uintptr_t last_error) {
  g_abi.pyramid_bytes = reinterpret_cast<decltype(g_abi.pyramid_bytes)>(pyramid_bytes);
  g_abi.build_pyramid_pair = reinterpret_cast<decltype(g_abi.build_pyramid_pair)>(build_pyramid_pair);
  g_abi.forward_pair = reinterpret_cast<decltype(g_abi.forward_pair)>(forward_pair);
  g_abi.accumulator_bytes = reinterpret_cast<decltype(g_abi.accumulator_bytes)>(accumulator_bytes);
  g_abi.accumulate_pair = reinterpret_cast<decltype(g_abi.accumulate_pair)>(accumulate_pair);
  g_abi.status_string = reinterpret_cast<decltype(g_abi.status_string)>(status_string);
  g_abi.last_error = reinterpret_cast<decltype(g_abi.last_error)>(last_error);
}

void raise_on(int rc, const char* name) { TORCH_CHECK(rc == SFB_OK, name, ": ", g_abi.status_string(rc), ": ", g_abi.last_error()); }

// ---- checks: those of the Python layer (ops._check, _check_pair_volumes, _check_coords_pair, _check_like) ------
const at::Tensor& tensor(pybind11::handle h, const char* name) {
  TORCH_CHECK(THPVariable_Check(h.ptr()), name, " must be a torch.Tensor");
  return THPVariable_Unpack(h.ptr());
}
void check(const at::Tensor& t, const char* name, int64_t ndim) {
  TORCH_CHECK(t.is_cuda(), name, " must be a CUDA tensor");
  TORCH_CHECK(t.is_contiguous(), name, " must be contiguous");
  TORCH_CHECK(t.scalar_type() == at::kFloat, name, " must have dtype torch.float32, got ", t.scalar_type());
  TORCH_CHECK(t.dim() == ndim, name, " must have ", ndim, " dimensions, got ", t.dim());
}
void check_like(const at::Tensor& t, const char* name, at::IntArrayRef shape, const at::Device& device) {
  check(t, name, static_cast<int64_t>(shape.size()));
  TORCH_CHECK(t.sizes() == shape, name, " must have shape ", shape, ", got ", t.sizes());
  TORCH_CHECK(t.device() == device, name, " is on ", t.device(), ", expected ", device);
}
int32_t int32(int64_t v) {
  TORCH_CHECK(v >= INT32_MIN && v <= INT32_MAX, "a size of ", v, " is out of range");
  return static_cast<int32_t>(v);
}

struct Sizes {
  int32_t B, dim, D1, D2, H1, W1;
};
Sizes pair_sizes(at::IntArrayRef s1, at::IntArrayRef s2) {
  TORCH_CHECK(s1.size() == 5 && s2.size() == 5 && s1[0] == s2[0] && s1[1] == s2[1] && s1[3] == s2[3] && s1[4] == s2[4],
              "the volumes differ in more than their displacements: ", s1, " and ", s2);
  return Sizes{int32(s1[0]), int32(s1[1]), int32(s1[2]), int32(s2[2]), int32(s1[3]), int32(s1[4])};
}
Sizes check_pair_volumes(const at::Tensor& corr1, const at::Tensor& corr2) {
  check(corr1, "corr", 5);
  check(corr2, "corr", 5);
  TORCH_CHECK(corr1.device() == corr2.device(), "corr1 is on ", corr1.device(), ", corr2 on ", corr2.device());
  return pair_sizes(corr1.sizes(), corr2.sizes());
}
// Strides between the samples and the components of coords (B, 2 or more, H1, W1).
std::pair<int64_t, int64_t> check_coords_pair(const at::Tensor& coords, const Sizes& s, const at::Device& dev) {
  TORCH_CHECK(coords.is_cuda() && coords.scalar_type() == at::kFloat && coords.dim() == 4 && coords.device() == dev && coords.size(0) == s.B &&
                  coords.size(1) >= 2 && coords.size(2) == s.H1 && coords.size(3) == s.W1,
              "coords must be a CUDA float32 tensor of shape (", s.B, ", 2, ", s.H1, ", ", s.W1, ") on ", dev);
  TORCH_CHECK((coords.stride(3) == 1 || s.W1 <= 1) && (coords.stride(2) == s.W1 || s.H1 <= 1),
              "coords must be contiguous within a component of a sample");
  return {coords.stride(0), coords.stride(1)};
}

const float* floats(const at::Tensor& t) { return static_cast<const float*>(t.const_data_ptr()); }
float* floats_to_write(const at::Tensor& t) { return static_cast<float*>(t.mutable_data_ptr()); }
at::TensorOptions like(const at::Tensor& t) { return at::TensorOptions().dtype(at::kFloat).device(t.device()); }

// ---- the ops ---------------------------------------------------------------------------------------------
std::pair<at::Tensor, at::Tensor> lookup_build_pyramid_pair(pybind11::handle corr1_, pybind11::handle corr2_, int64_t levels) {
  const at::Tensor &corr1 = tensor(corr1_, "corr"), &corr2 = tensor(corr2_, "corr");
  const Sizes s = check_pair_volumes(corr1, corr2);
  at::Tensor pyramid[2];
  for (int i = 0; i < 2; ++i) {
    const size_t bytes = g_abi.pyramid_bytes(s.B, s.dim, i == 0 ? s.D1 : s.D2, s.H1, s.W1, int32(levels));
    pyramid[i] = at::empty({std::max<int64_t>(static_cast<int64_t>(bytes / 4), 1)}, like(corr1));
  }
  const c10::cuda::CUDAGuard guard(corr1.device());
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream();
  int rc;
  {
    pybind11::gil_scoped_release nogil;
    rc = g_abi.build_pyramid_pair(floats(corr1), floats_to_write(pyramid[0]), floats(corr2), floats_to_write(pyramid[1]), s.B, s.dim, s.D1, s.D2,
                                  s.H1, s.W1, int32(levels), stream);
  }
  raise_on(rc, "sfb_lookup_build_pyramid_pair");
  return {pyramid[0], pyramid[1]};
}

std::pair<at::Tensor, at::Tensor> lookup_forward_pair(pybind11::handle corr1_, pybind11::handle corr2_, pybind11::handle pyramid1_,
                                                      pybind11::handle pyramid2_, pybind11::handle coords_, int64_t levels, int64_t radius) {
  const at::Tensor &corr1 = tensor(corr1_, "corr"), &corr2 = tensor(corr2_, "corr"), &coords = tensor(coords_, "coords");
  const at::Tensor &pyramid1 = tensor(pyramid1_, "pyramid1"), &pyramid2 = tensor(pyramid2_, "pyramid2");
  const Sizes s = check_pair_volumes(corr1, corr2);
  const auto [sb, sc] = check_coords_pair(coords, s, corr1.device());
  const std::array<int64_t, 4> size = {s.B, levels * s.dim * (2 * radius + 1), s.H1, s.W1};
  at::Tensor out1 = at::empty(size, like(corr1)), out2 = at::empty(size, like(corr1));
  const c10::cuda::CUDAGuard guard(corr1.device());
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream();
  int rc;
  {
    pybind11::gil_scoped_release nogil;
    rc = g_abi.forward_pair(floats(corr1), floats(pyramid1), floats(corr2), floats(pyramid2), floats(coords), sb, sc, floats_to_write(out1),
                            floats_to_write(out2), s.B, s.dim, s.D1, s.D2, s.H1, s.W1, int32(levels), int32(radius), stream);
  }
  raise_on(rc, "sfb_lookup_forward_pair");
  return {out1, out2};
}

void lookup_accumulate_pair(const std::vector<int64_t>& shape1, const std::vector<int64_t>& shape2, pybind11::handle coords_, pybind11::handle gout1_,
                            pybind11::handle gout2_, pybind11::handle acc1_, pybind11::handle acc2_, int64_t levels, int64_t radius) {
  const Sizes s = pair_sizes(shape1, shape2);
  const at::Tensor& coords = tensor(coords_, "coords");
  const at::Device dev = coords.device();
  const auto [sb, sc] = check_coords_pair(coords, s, dev);
  const std::array<int64_t, 4> size = {s.B, levels * s.dim * (2 * radius + 1), s.H1, s.W1};
  const float* gout[2] = {nullptr, nullptr};
  float* acc[2] = {nullptr, nullptr};
  for (int i = 0; i < 2; ++i) {
    const pybind11::handle g = i == 0 ? gout1_ : gout2_;
    if (g.is_none()) continue;
    const at::Tensor &grad = tensor(g, "grad_out"), &sum = tensor(i == 0 ? acc1_ : acc2_, "accumulator");
    check_like(grad, "grad_out", size, dev);
    const size_t bytes = g_abi.accumulator_bytes(s.B, s.dim, i == 0 ? s.D1 : s.D2, s.H1, s.W1, int32(levels), i == 0 ? 1 : 0);
    check_like(sum, "accumulator", {static_cast<int64_t>(bytes / 4)}, dev);
    gout[i] = floats(grad);
    acc[i] = floats_to_write(sum);
  }
  const c10::cuda::CUDAGuard guard(dev);
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream();
  int rc;
  {
    pybind11::gil_scoped_release nogil;
    rc = g_abi.accumulate_pair(gout[0], gout[1], floats(coords), sb, sc, acc[0], acc[1], s.B, s.dim, s.D1, s.D2, s.H1, s.W1, int32(levels),
                               int32(radius), stream);
  }
  raise_on(rc, "sfb_lookup_accumulate_pair");
}

}  // namespace

PYBIND11_MODULE(sfb_host, m) {
  m.def("bind", &bind);
  m.def("lookup_build_pyramid_pair", &lookup_build_pyramid_pair);
  m.def("lookup_forward_pair", &lookup_forward_pair);
  m.def("lookup_accumulate_pair", &lookup_accumulate_pair);
}
