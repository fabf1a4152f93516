// What the files of the torch layer share: the library's entry points and small helpers.
#pragma once

#include <torch/extension.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>

#include <atomic>
#include <string>

#include "../../include/fields_read.h"

namespace fields_torch {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Variable;
using torch::autograd::variable_list;

// ---------------------------------------------------------------------------------------------
// The library's entry points, looked up in the build that bind() names.
// ---------------------------------------------------------------------------------------------
#define FIELDS_API(X)                                                                             \
    X(fields_status_string) X(fields_last_cuda_error) X(fields_read_workspace_bytes)              \
    X(fields_read_forward) X(fields_read_backward) X(fields_read_state_rows)                      \
    X(fields_read_backward_from_states) X(fields_read_forward_bf16)                               \
    X(fields_read_forward_bf16_stats) X(fields_read_backward_bf16)                                \
    X(fields_read_norm_grad_combine) X(fields_read_step) X(fields_read_step_bf16)                 \
    X(fields_scan_workspace_bytes) X(fields_scan_forward) X(fields_scan_backward)                 \
    X(fields_stack_layout) X(fields_stack_step_norm) X(fields_stack_close_mixer)                  \
    X(fields_stack_swiglu) X(fields_stack_close_ff) X(fields_read_forward_bf16_rows)              \
    X(fields_read_backward_bf16_rows) X(fields_mixer_grad_rows) X(fields_mixer_grad_scratch_bytes) \
    X(fields_mixer_open_grad) X(fields_mixer_close_grad) X(fields_step_w12_rows)                  \
    X(fields_step_layout) X(fields_step_block)

struct Api {
#define X(name) decltype(&::name) name;
    FIELDS_API(X)
#undef X
};
inline std::atomic<const Api*> g_api{nullptr};
inline PyObject* g_error_type = nullptr;  // FieldsLibraryError

inline const Api& api() {
    const Api* a = g_api.load(std::memory_order_acquire);
    TORCH_CHECK(a, "the CUDA library has not been bound");
    return *a;
}

// FieldsLibraryError with the library's own text, from any thread (a backward pass runs on an
// engine thread, which carries the exception to the caller).
inline void check(int rc, const char* what) {
    if (C10_LIKELY(rc == FIELDS_OK)) return;
    std::string text = std::string(what) + ": " + api().fields_status_string(rc);
    if (rc == FIELDS_ERR_LAUNCH) text += std::string(": ") + api().fields_last_cuda_error();
    text += " (status " + std::to_string(rc) + ")";
    pybind11::gil_scoped_acquire gil;
    PyErr_SetString(g_error_type, text.c_str());
    python_error e;
    e.persist();
    throw e;
}

// ---------------------------------------------------------------------------------------------
// Small helpers.
// ---------------------------------------------------------------------------------------------
inline Tensor f32(const Tensor& t) {
    if (t.scalar_type() == at::kFloat && t.is_contiguous()) return t;
    return t.contiguous().to(at::kFloat);
}
inline Tensor dense(const Tensor& t) { return t.is_contiguous() ? t : t.contiguous(); }
inline float* fp(const Tensor& t) { return t.defined() ? static_cast<float*>(t.data_ptr()) : nullptr; }
inline void* vp(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
inline void* stream_of(const Tensor& t) {
    return c10::cuda::getCurrentCUDAStream(t.device().index()).stream();
}
inline Tensor empty(at::IntArrayRef size, at::ScalarType type, c10::Device device) {
    return at::detail::empty_cuda(size, type, device, std::nullopt);
}
inline Tensor workspace(size_t bytes, c10::Device device) {
    return empty({(int64_t)std::max<size_t>(bytes, 256)}, at::kByte, device);
}
inline std::string shape(const Tensor& t) { return c10::str("(", t.sizes(), ")"); }

// Argument unpacking of the Python entry points.
inline void want_args(Py_ssize_t n, Py_ssize_t want) {
    TORCH_CHECK_TYPE(n == want, "expected ", want, " arguments, got ", n);
}
inline const Tensor& tensor_arg(PyObject* o) {
    TORCH_CHECK_TYPE(THPVariable_Check(o), "expected a tensor, got ", Py_TYPE(o)->tp_name);
    return THPVariable_Unpack(o);
}

}  // namespace fields_torch
