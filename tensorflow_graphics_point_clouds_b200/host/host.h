// Host layer over the C ABI: what custom_ops.py, pc.py and mcconv.py call.  Each
// function checks and converts its tensors, allocates the outputs from torch's caching
// allocator and enqueues one or two C-ABI calls on torch's current stream.  In Python
// the same marshalling (ctypes arguments, a dozen tensor allocations per op) took
// longer than the kernels of a small layer: 300 of 345 us per training step on
// 4 x 1024 points.
#pragma once

#include <torch/extension.h>

#include <c10/cuda/CUDAStream.h>

#include <optional>
#include <string>
#include <vector>

#include "tfgpc.h"

namespace tfgpc_host {

using at::Tensor;
using OptTensor = std::optional<Tensor>;
namespace py = pybind11;

// Raises TfgpcError(code, message); cells: its `num_cells` attribute.
[[noreturn]] void raise_error(int code, const std::string& message,
                              const std::vector<int32_t>* cells = nullptr);
[[noreturn]] void raise_value_error(const std::string& message);

inline void check(int code) {
  if (code != 0) raise_error(code, tfgpc_last_error());
}

inline void require(bool ok, const char* message) {
  if (!ok) raise_error(TFGPC_EINVAL, message);
}

inline void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

inline Tensor as(const Tensor& t, at::ScalarType type) {
  if (t.scalar_type() == type && t.is_contiguous()) return t;
  return t.contiguous().to(type);
}
inline Tensor f32(const Tensor& t) { return as(t, at::kFloat); }
inline Tensor i32(const Tensor& t) { return as(t, at::kInt); }

inline void on_gpu(const Tensor& t) {
  if (!t.is_cuda())
    raise_value_error("tfg_custom_ops are registered for the GPU only: got a CPU tensor");
}

inline Tensor empty(at::IntArrayRef shape, at::ScalarType type, const Tensor& like) {
  return at::empty(shape, like.options().dtype(type));
}
inline Tensor bytes(size_t n, const Tensor& like) {
  return empty({(int64_t)n}, at::kByte, like);
}

inline const float* fp(const Tensor& t) { return t.const_data_ptr<float>(); }
inline const int32_t* ip(const Tensor& t) { return t.const_data_ptr<int32_t>(); }
inline float* fpm(const Tensor& t) { return t.mutable_data_ptr<float>(); }
inline int32_t* ipm(const Tensor& t) { return t.mutable_data_ptr<int32_t>(); }
inline const float* fp(const OptTensor& t) { return t ? fp(*t) : nullptr; }
inline const int32_t* ip(const OptTensor& t) { return t ? ip(*t) : nullptr; }

void bind_cells(py::module_& m);    // cells.cpp
void bind_layers(py::module_& m);   // layers.cpp

}  // namespace tfgpc_host
