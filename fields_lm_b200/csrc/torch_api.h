// What the files of the torch layer share: the library's entry points and small helpers.
#pragma once

#include <torch/extension.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>

#include <c10/cuda/CUDAGraphsC10Utils.h>

#include <algorithm>
#include <atomic>
#include <memory>
#include <mutex>
#include <optional>
#include <string>
#include <thread>
#include <vector>

#include "../../include/fields_read.h"

namespace fields_torch {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Variable;
using torch::autograd::variable_list;

// ---------------------------------------------------------------------------------------------
// The library's entry points, looked up in the build that bind() names.
// ---------------------------------------------------------------------------------------------
#define FIELDS_API(X)                                                                               \
    X(fields_status_string) X(fields_last_cuda_error) X(fields_read_workspace_bytes)                \
    X(fields_read_forward) X(fields_read_backward) X(fields_read_backward_from_states)              \
    X(fields_read_forward_bf16) X(fields_read_forward_bf16_stats) X(fields_read_backward_bf16)      \
    X(fields_read_norm_grad_combine) X(fields_read_step) X(fields_read_step_bf16)                   \
    X(fields_scan_forward) X(fields_scan_backward) X(fields_stack_layout) X(fields_stack_layout_parts) X(fields_product)                                                    \
    X(fields_stack_step_norm) X(fields_stack_close_mixer) X(fields_stack_swiglu)                    \
    X(fields_stack_close_ff) X(fields_read_forward_bf16_rows) X(fields_read_backward_bf16_rows)     \
    X(fields_mixer_grad_rows) X(fields_mixer_grad_scratch_bytes) X(fields_mixer_open_grad)          \
    X(fields_mixer_close_grad) X(fields_step_w12_rows) X(fields_step_layout) X(fields_step_stack)   \
    X(fields_step_block)                                                                            \
    X(fields_read_use_kept) X(fields_read_forward_rows)

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
// ... on the 16 bytes that row kernels and TMA need (a dense view may begin anywhere in its storage)
inline Tensor aligned(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 ? t.clone() : t; }
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
// n elements of `base` from `offset` on, as a tensor of its own on the same storage.
inline Tensor part_of(const Tensor& base, int64_t offset, int64_t n) {
    Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(base.storage()), base.key_set(), base.dtype());
    t.unsafeGetTensorImpl()->set_storage_offset(offset);
    t.unsafeGetTensorImpl()->set_sizes_contiguous({n});
    return t;
}
inline bool all_aligned(std::initializer_list<const void*> ptrs, uintptr_t bytes) {
    uintptr_t any = 0;
    for (const void* p : ptrs) any |= reinterpret_cast<uintptr_t>(p);
    return any % bytes == 0;
}

// The kept workspaces of the torch layer: one per stream (fields_read_use_kept), for the last few streams, up to a
// size. A workspace is 256 bytes and three times a half (two that take turns, and the partial rows), so at most
// 8 x 96 MiB in all. When the allocator runs short on a device (less than an eighth of it left) it takes back
// those that no pass is being issued on; the next pass on such a stream makes its own again.
class KeptWorkspaces {
  public:
    struct Entry {
        int device;
        int64_t stream;
        std::mutex mu;
        std::atomic<bool> busy{false};  // while `ws` must not be taken: by one who holds `mu`, or by release()
        Tensor ws;
        fields_kept state{};
    };
    // An entry held while a pass is issued on it (a pass may be two launches).
    class Hold {
      public:
        Hold(int device, std::optional<int64_t> stream) {
            if (!stream) return;
            e_ = entry(device, *stream);
            lock_ = std::unique_lock<std::mutex>(e_->mu);
            while (e_->busy.exchange(true)) std::this_thread::yield();
        }
        ~Hold() { drop(); }
        Hold(const Hold&) = delete;
        void drop() {
            if (!e_) return;
            e_->busy = false;
            lock_.unlock();
            e_.reset();
        }
        explicit operator bool() const { return e_ != nullptr; }
        Entry* operator->() const { return e_.get(); }

      private:
        std::shared_ptr<Entry> e_;
        std::unique_lock<std::mutex> lock_;  // released before e_
    };

    // Called by the allocator of the current device, with its lock held, when it has no block for a request.
    static bool release() {
        int device = 0;
        size_t left = 0, total = 0;
        if (cudaGetDevice(&device) != cudaSuccess || cudaMemGetInfo(&left, &total) != cudaSuccess) return false;
        const double limit = c10::cuda::CUDACachingAllocator::getMemoryFraction((c10::DeviceIndex)device) * (double)total;
        const auto stats = c10::cuda::CUDACachingAllocator::getDeviceStats((c10::DeviceIndex)device);
        const auto reserved = (double)stats.reserved_bytes[(size_t)c10::CachingAllocator::StatType::AGGREGATE].current;
        if (std::min((double)left, limit - reserved) > (double)total / 8) return false;
        const std::unique_lock<std::mutex> guard(mu(), std::try_to_lock);  // (its holder may wait for the allocator)
        if (!guard) return false;
        bool any = false;
        for (const auto& e : list()) {
            if (e->device != device || e->busy.exchange(true)) continue;
            any = any || e->ws.defined();
            e->ws = Tensor();
            e->busy = false;
        }
        return any;
    }

  private:
    static constexpr size_t kStreams = 8;
    // (never destroyed: the allocator may be gone by the time a process ends)
    static std::vector<std::shared_ptr<Entry>>& list() {
        static auto* all = new std::vector<std::shared_ptr<Entry>>();  // most recently used first
        return *all;
    }
    static std::mutex& mu() {
        static auto* m = new std::mutex();
        return *m;
    }
    static std::shared_ptr<Entry> entry(int device, int64_t stream) {
        const std::lock_guard<std::mutex> guard(mu());
        auto& all = list();
        for (size_t i = 0; i < all.size(); ++i) {
            if (all[i]->device == device && all[i]->stream == stream) {
                if (i) std::rotate(all.begin(), all.begin() + i, all.begin() + i + 1);
                return all.front();
            }
        }
        if (all.size() == kStreams) all.pop_back();
        auto e = std::make_shared<Entry>();
        e->device = device;
        e->stream = stream;
        all.insert(all.begin(), e);
        return e;
    }
};

// The workspace of one forward or backward pass on the current stream: a kept one, which saves an allocation
// and a fill launch per pass, about 4 us of host time and 2 us on the GPU. Passes that are captured into a
// graph and larger ones get one of their own, as does every pass where the library refuses or where there is
// memory for the pass but not for a kept workspace.
class PassWorkspace {
  public:
    PassWorkspace(size_t need, const Tensor& on) : kept_(on.device().index(), keep_for(need, on)) {
        if (kept_ && !ready(need, on)) kept_.drop();
        if (!kept_) {
            own_ = workspace(need, on.device());
            api().fields_read_use_kept(nullptr);  // one that a caller of the library may have left
        }
        ptr_ = kept_ ? kept_->ws.data_ptr() : own_.data_ptr();
    }
    ~PassWorkspace() {
        if (!kept_) return;
        api().fields_read_use_kept(nullptr);  // not left behind by a pass that was refused
        if (!done_) kept_->ws = Tensor();     // the pass threw: start again from the fill
    }
    PassWorkspace(const PassWorkspace&) = delete;
    void* ptr() const { return ptr_; }
    // the status of the pass
    void check(int rc, const char* what) {
        done_ = rc == FIELDS_OK;
        fields_torch::check(rc, what);
    }

  private:
    static constexpr size_t kLeastBytes = 1 << 20, kMostBytes = 32 << 20;  // of a half
    // The current stream, if a pass of this size keeps its workspace there.
    static std::optional<int64_t> keep_for(size_t need, const Tensor& on) {
        const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream(on.device().index());
        // (torch's own streams: another library's may be destroyed while work is pending)
        if (need > kMostBytes || (stream.id() != 0 && !(stream.id() & 1)) ||
            c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None)
            return std::nullopt;
        return stream.id();
    }
    // Whether the entry has a workspace for the pass and the library takes it.
    bool ready(size_t need, const Tensor& on) {
        if (kept_->state.half_bytes < need || !kept_->ws.defined()) {
            size_t half = std::max(kLeastBytes, kept_->state.half_bytes);
            while (half < need) half *= 2;
            Tensor ws;
            try {
                ws = empty({(int64_t)(256 + 3 * half)}, at::kByte, on.device());
            } catch (const c10::OutOfMemoryError&) {
                return false;
            }
            C10_CUDA_CHECK(cudaMemsetAsync(ws.data_ptr(), 0xFF, 256 + 2 * half, static_cast<cudaStream_t>(stream_of(on))));
            // (the entry changes when nothing can fail any more)
            kept_->ws = std::move(ws);
            kept_->state = fields_kept{half, {0, 0}, 0};
        }
        // the last step: a registration without a pass would be taken by the thread's next one
        return api().fields_read_use_kept(&kept_->state) == FIELDS_OK;
    }

    KeptWorkspaces::Hold kept_;
    Tensor own_;
    void* ptr_;
    bool done_ = false;
};
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
