// The package's operators as native torch code: argument checks, allocations, autograd nodes and
// the calls into the C ABI (include/fields_read.h), compiled against the torch headers into
// libfields_torch.so.
//
// Why native: at small and medium sizes a call costs what the host spends on it. Through
// torch.autograd.Function and ctypes one forward + backward of the operator took 145 us of host
// time whatever its size (21 us of kernels at 1 x 256 tokens) and one decode step 15.5 us (1.5 us
// of kernel). Arguments are parsed by hand (METH_FASTCALL) because a signature parser costs as much
// as the rest of a decode step.
//
// The kernels stay in libfields_read.so, which knows nothing of torch; bind() is given the path of
// the build to use, so the tests can point this layer at another build of the library.
#include "torch_api.h"

#include <dlfcn.h>

namespace fields_torch {

void add_stack(PyObject* module);                                                 // torch_stack.cpp
PyObject* py_fused_mixer(PyObject*, PyObject* const* args, Py_ssize_t n);  // torch_mixer.cpp

class ReleaseKept : public c10::FreeMemoryCallback {
  public:
    bool Execute() override { return KeptWorkspaces::release(); }
};
static void register_release() {
    auto* registry = c10::FreeCudaMemoryCallbacksRegistry();
    if (!registry->Has("fields_kept_workspaces"))
        registry->Register(
            "fields_kept_workspaces", [] { return std::unique_ptr<c10::FreeMemoryCallback>(new ReleaseKept()); }, "",
            c10::REGISTRY_DEFAULT);
}

struct Dims {
    int B, L, C;
};

// Checks shared by the forms of the operator (the reference's, same file :923-938).
static Dims check_operator(const Tensor& raw, at::ScalarType type, const char* type_name,
                           const Tensor& tr, const Tensor& ti, const Tensor& gm) {
    TORCH_CHECK(raw.is_cuda(), "Chunked Field kernel requires CUDA");
    TORCH_CHECK_TYPE(raw.scalar_type() == type, "raw must be ", type_name, ", got ",
                     raw.scalar_type());
    TORCH_CHECK_VALUE(raw.dim() == 3 && raw.size(2) % 3 == 0, shape(raw));
    const int64_t C = raw.size(2) / 3;
    TORCH_CHECK_VALUE(tr.numel() == C && ti.numel() == C && gm.numel() == C, shape(raw), " ", shape(tr));
    return Dims{(int)raw.size(0), (int)raw.size(1), (int)C};
}

// ---------------------------------------------------------------------------------------------
// The operator on the fp32 boundary, with an optional carried state.
// ---------------------------------------------------------------------------------------------
struct ForwardArgs {
    Tensor raw, tr, ti, gm, state_in;  // state_in may be undefined
    Dims d;
};

static ForwardArgs forward_args(const Tensor& raw, const Tensor& tr, const Tensor& ti,
                                const Tensor& gm, const Tensor& state_in) {
    const Dims d = check_operator(raw, at::kFloat, "float32", tr, ti, gm);
    if (state_in.defined())
        TORCH_CHECK_VALUE(state_in.dim() == 2 && state_in.size(0) == d.B && state_in.size(1) == 2 * d.C,
                          shape(raw), " ", shape(state_in));
    return ForwardArgs{dense(raw), f32(tr), f32(ti), f32(gm),
                       state_in.defined() ? f32(state_in) : state_in, d};
}

// With `rows` also every eighth state row, written by the kernel where it can (undefined otherwise).
static void run_forward(const ForwardArgs& a, Tensor& read, Tensor& state_out, bool want_state, Tensor* rows = nullptr) {
    const Api& f = api();
    const auto [B, L, C] = a.d;
    const c10::Device dev = a.raw.device();
    const c10::cuda::CUDAGuard guard(dev);
    read = empty({B, L, 4 * C}, at::kFloat, dev);
    if (want_state) state_out = empty({B, 2 * C}, at::kFloat, dev);
    const size_t n = f.fields_read_workspace_bytes(B, L, C, FIELDS_PASS_FORWARD);
    PassWorkspace ws(n, a.raw);
    if (rows && all_aligned({fp(a.raw), fp(a.tr), fp(a.ti), fp(a.gm), fp(a.state_in)}, 16) && B > 0 && L >= 8) {
        *rows = empty({B, L / 8, 2 * C}, at::kFloat, dev);
        ws.check(f.fields_read_forward_rows(fp(a.raw), fp(a.tr), fp(a.ti), fp(a.gm), fp(a.state_in), fp(read), fp(state_out),
                                            fp(*rows), ws.ptr(), n, B, L, C, stream_of(a.raw)),
                 "fields_read_forward");
        return;
    }
    ws.check(f.fields_read_forward(fp(a.raw), fp(a.tr), fp(a.ti), fp(a.gm), fp(a.state_in), fp(read),
                                   fp(state_out), ws.ptr(), n, B, L, C, stream_of(a.raw)),
             "fields_read_forward");
}

struct FieldRead : torch::autograd::Function<FieldRead> {
    static variable_list forward(AutogradContext* ctx, const Tensor& raw_, const Tensor& tr_,
                                 const Tensor& ti_, const Tensor& gm_,
                                 const std::optional<Tensor>& state_, bool lean, bool want_state) {
        const ForwardArgs a = forward_args(raw_, tr_, ti_, gm_, state_.value_or(Tensor()));
        Tensor read, state_out;
        lean = lean && a.d.C % 4 == 0;
        Tensor kept;
        run_forward(a, read, state_out, want_state, lean ? &kept : nullptr);
        if (!lean) kept = read;
        else if (!kept.defined())  // every eighth state row instead of `read`
            kept = read.slice(1, 7, std::nullopt, 8).slice(2, 0, 2 * a.d.C).contiguous();
        ctx->set_materialize_grads(false);
        ctx->save_for_backward({a.raw, a.tr, a.ti, a.gm, kept, a.state_in});
        if (want_state) return {read, state_out};
        return {read};
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const Api& f = api();
        const variable_list saved = ctx->get_saved_variables();
        const Tensor &raw = saved[0], &tr = saved[1], &ti = saved[2], &gm = saved[3], &read = saved[4],
                     &state_in = saved[5];
        const int B = (int)raw.size(0), L = (int)raw.size(1), C = (int)raw.size(2) / 3;
        const bool lean = read.size(2) == 2 * C;  // rows of states, not of `read`
        const c10::Device dev = raw.device();
        const c10::cuda::CUDAGuard guard(dev);
        const Tensor grad_read =
            grads[0].defined() ? f32(grads[0])
                               : at::zeros({B, L, 4 * C}, at::TensorOptions().dtype(at::kFloat).device(dev));
        const Tensor grad_state = grads.size() > 1 && grads[1].defined() ? f32(grads[1]) : Tensor();
        const Tensor grad_raw = empty({B, L, 3 * C}, at::kFloat, dev);
        const Tensor g_par = empty({3, C}, at::kFloat, dev);
        Tensor g_sin;
        if (state_in.defined() && ctx->needs_input_grad(4)) g_sin = empty({B, 2 * C}, at::kFloat, dev);
        const size_t n = f.fields_read_workspace_bytes(B, L, C, FIELDS_PASS_BACKWARD);
        PassWorkspace ws(n, raw);
        auto* entry = lean ? f.fields_read_backward_from_states : f.fields_read_backward;
        // (lean: `read` holds the kept state rows, possibly none for L < 8)
        ws.check(entry(fp(raw), fp(tr), fp(ti), fp(gm), fp(state_in), read.numel() ? fp(read) : nullptr,
                    fp(grad_read), fp(grad_state), fp(grad_raw), fp(g_par), fp(g_par) + C,
                    fp(g_par) + 2 * C, fp(g_sin), ws.ptr(), n, B, L, C, stream_of(raw)),
              "fields_read_backward");
        return {grad_raw, part_of(g_par, 0, C), part_of(g_par, C, C), part_of(g_par, 2 * C, C), g_sin, Tensor(), Tensor()};
    }
};

// ---------------------------------------------------------------------------------------------
// The operator on the bfloat16 boundary; with STATS also the sum of squares of each token's outputs.
// ---------------------------------------------------------------------------------------------
static variable_list run_forward_bf16(const Tensor& raw, const Tensor& tr, const Tensor& ti,
                                      const Tensor& gm, const Dims& d, bool stats) {
    const Api& f = api();
    const auto [B, L, C] = d;
    const c10::Device dev = raw.device();
    const c10::cuda::CUDAGuard guard(dev);
    const Tensor read = empty({B, L, 4 * C}, at::kBFloat16, dev);
    const size_t n = f.fields_read_workspace_bytes(B, L, C, FIELDS_PASS_FORWARD);
    PassWorkspace ws(n, raw);
    if (!stats) {
        ws.check(f.fields_read_forward_bf16(vp(raw), fp(tr), fp(ti), fp(gm), nullptr, vp(read), nullptr,
                                         ws.ptr(), n, B, L, C, stream_of(raw)),
              "fields_read_forward_bf16");
        return {read};
    }
    const Tensor groups = empty({B, L, (C + 127) / 128}, at::kFloat, dev);
    ws.check(f.fields_read_forward_bf16_stats(vp(raw), fp(tr), fp(ti), fp(gm), nullptr, vp(read), fp(groups),
                                           nullptr, ws.ptr(), n, B, L, C, stream_of(raw)),
          "fields_read_forward_bf16_stats");
    return {read, groups.sum(-1)};
}

// grad_raw, d tr, d ti, d gamma from the gradient of `read` (bfloat16, dense).
static variable_list run_backward_bf16(const Tensor& raw, const Tensor& tr, const Tensor& ti,
                                       const Tensor& gm, const Tensor& read, const Tensor& grad_read) {
    const Api& f = api();
    const int B = (int)raw.size(0), L = (int)raw.size(1), C = (int)raw.size(2) / 3;
    const c10::Device dev = raw.device();
    const Tensor grad_raw = empty({B, L, 3 * C}, at::kBFloat16, dev);
    const Tensor g_par = empty({3, C}, at::kFloat, dev);
    const size_t n = f.fields_read_workspace_bytes(B, L, C, FIELDS_PASS_BACKWARD);
    PassWorkspace ws(n, raw);
    ws.check(f.fields_read_backward_bf16(vp(raw), fp(tr), fp(ti), fp(gm), nullptr, vp(read), vp(grad_read),
                                      nullptr, vp(grad_raw), fp(g_par), fp(g_par) + C, fp(g_par) + 2 * C,
                                      nullptr, ws.ptr(), n, B, L, C, stream_of(raw)),
          "fields_read_backward_bf16");
    return {grad_raw, part_of(g_par, 0, C), part_of(g_par, C, C), part_of(g_par, 2 * C, C)};
}

template <bool STATS>
struct FieldReadBf16 : torch::autograd::Function<FieldReadBf16<STATS>> {
    static variable_list forward(AutogradContext* ctx, const Tensor& raw_, const Tensor& tr_,
                                 const Tensor& ti_, const Tensor& gm_) {
        const Dims d = check_operator(raw_, at::kBFloat16, "bfloat16", tr_, ti_, gm_);
        if (STATS) TORCH_CHECK_VALUE(d.B > 0 && d.L > 0, shape(raw_));
        const Tensor raw = dense(raw_), tr = f32(tr_), ti = f32(ti_), gm = f32(gm_);
        const variable_list out = run_forward_bf16(raw, tr, ti, gm, d, STATS);
        if (STATS) ctx->set_materialize_grads(false);
        ctx->save_for_backward({raw, tr, ti, gm, out[0]});
        return out;
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const variable_list saved = ctx->get_saved_variables();
        const Tensor &raw = saved[0], &read = saved[4];
        const c10::cuda::CUDAGuard guard(raw.device());
        Tensor total = grads[0].defined() ? dense(grads[0]).to(at::kBFloat16) : Tensor();
        if (STATS && grads[1].defined()) {
            // d sumsq / d read = 2 read: folded into the gradient the recurrence receives
            const Tensor own = total, sumsq = f32(grads[1]);
            total = empty(read.sizes(), at::kBFloat16, raw.device());
            check(api().fields_read_norm_grad_combine(vp(own), vp(read), fp(sumsq), vp(total),
                                                      read.size(0) * read.size(1), (int)read.size(2),
                                                      stream_of(raw)),
                  "fields_read_norm_grad_combine");
        }
        if (!total.defined()) total = at::zeros_like(read);
        return run_backward_bf16(raw, saved[1], saved[2], saved[3], read, total);
    }
};

// ---------------------------------------------------------------------------------------------
// The real-valued scan.
// ---------------------------------------------------------------------------------------------
// `a` as the library reads it: a dense tensor, or one value per (b, t) broadcast over the channels
// (the expanded view the softpatch mixer passes), read through its own strides.
struct ScanDecay {
    Tensor a;
    long long batch, step;
    int chan;
};

static ScanDecay scan_decay(const Tensor& a) {
    if (a.size(2) > 1 && a.stride(2) == 0) return ScanDecay{a, a.stride(0), a.stride(1), 0};
    const Tensor d = dense(a);
    return ScanDecay{d, d.size(1) * d.size(2), d.size(2), 1};
}

struct LinearScan : torch::autograd::Function<LinearScan> {
    static variable_list forward(AutogradContext* ctx, const Tensor& a_, const Tensor& b_,
                                 const std::optional<Tensor>& state_, bool want_state) {
        const int B = (int)b_.size(0), L = (int)b_.size(1), C = (int)b_.size(2);
        Tensor state_in;
        if (state_ && state_->defined()) {
            TORCH_CHECK_VALUE(state_->dim() == 2 && state_->size(0) == B && state_->size(1) == C,
                              shape(b_), " ", shape(*state_));
            state_in = f32(*state_);
        }
        const Api& f = api();
        const c10::Device dev = b_.device();
        const c10::cuda::CUDAGuard guard(dev);
        const Tensor b = dense(b_);
        const ScanDecay d = scan_decay(a_);
        const Tensor states = empty({B, L, C}, at::kFloat, dev);
        const Tensor state_out = want_state ? empty({B, C}, at::kFloat, dev) : Tensor();
        check(f.fields_scan_forward(fp(d.a), d.batch, d.step, d.chan, fp(b), fp(state_in), fp(states),
                                    fp(state_out), nullptr, 0, B, L, C, stream_of(b)),
              "fields_scan_forward");
        ctx->set_materialize_grads(false);
        ctx->save_for_backward({d.a, states, state_in});
        if (!want_state) return {states};
        return {states, state_out};
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const Api& f = api();
        const variable_list saved = ctx->get_saved_variables();
        const ScanDecay d = scan_decay(saved[0]);
        const Tensor &states = saved[1], &state_in = saved[2];
        const int B = (int)states.size(0), L = (int)states.size(1), C = (int)states.size(2);
        const c10::Device dev = states.device();
        const c10::cuda::CUDAGuard guard(dev);
        const Tensor g = grads[0].defined() ? f32(grads[0]) : at::zeros_like(states);
        const Tensor g_out = grads.size() > 1 && grads[1].defined() ? f32(grads[1]) : Tensor();
        const Tensor grad_a = empty({B, L, C}, at::kFloat, dev), grad_b = empty({B, L, C}, at::kFloat, dev);
        Tensor g_in;
        if (state_in.defined() && ctx->needs_input_grad(2)) g_in = empty({B, C}, at::kFloat, dev);
        check(f.fields_scan_backward(fp(d.a), d.batch, d.step, d.chan, fp(states), fp(state_in), fp(g),
                                     fp(g_out), fp(grad_a), fp(grad_b), fp(g_in), nullptr, 0, B, L, C,
                                     stream_of(states)),
              "fields_scan_backward");
        // dense gradient of `a`; for an expanded `a` autograd sums it over the broadcast channels
        return {grad_a, grad_b, g_in, Tensor()};
    }
};

// ---------------------------------------------------------------------------------------------
// One recurrent step of incremental decoding: `state` advances in place.
// ---------------------------------------------------------------------------------------------
static Tensor step(const Tensor& raw_, const Tensor& tr_, const Tensor& ti_, const Tensor& gm_,
                   const Tensor& state) {
    TORCH_CHECK(raw_.is_cuda(), "Field decode step requires CUDA");
    const at::ScalarType type = raw_.scalar_type();
    TORCH_CHECK_TYPE(type == at::kFloat || type == at::kBFloat16,
                     "raw_row must be float32 or bfloat16, got ", type);
    TORCH_CHECK_TYPE(state.scalar_type() == at::kFloat && state.is_contiguous(),
                     "state must be a contiguous float32 tensor");
    TORCH_CHECK_VALUE(raw_.dim() == 2 && raw_.size(1) % 3 == 0, shape(raw_));
    const int64_t B = raw_.size(0), C = raw_.size(1) / 3;
    TORCH_CHECK_VALUE(state.dim() == 2 && state.size(0) == B && state.size(1) == 2 * C && tr_.numel() == C,
                      shape(raw_), " ", shape(state), " ", shape(tr_));
    const Api& f = api();
    const c10::Device dev = raw_.device();
    const c10::cuda::CUDAGuard guard(dev);
    const Tensor raw = dense(raw_), tr = f32(tr_), ti = f32(ti_), gm = f32(gm_);
    Tensor read = empty({B, 4 * C}, type, dev);
    const int rc = type == at::kFloat
                       ? f.fields_read_step(fp(raw), fp(tr), fp(ti), fp(gm), fp(state), fp(read), (int)B,
                                            (int)C, stream_of(raw))
                       : f.fields_read_step_bf16(vp(raw), fp(tr), fp(ti), fp(gm), fp(state), vp(read), (int)B,
                                                 (int)C, stream_of(raw));
    check(rc, "fields_read_step");
    return read;
}

// ---------------------------------------------------------------------------------------------
// Python entry points.
// ---------------------------------------------------------------------------------------------
static std::optional<Tensor> optional_arg(PyObject* o) {
    if (o == Py_None) return std::nullopt;
    return tensor_arg(o);
}
static PyObject* wrap(const Tensor& t) { return THPVariable_Wrap(t); }
static PyObject* wrap2(const Tensor& a, const Tensor& b) {
    PyObject* out = PyTuple_New(2);
    if (!out) throw python_error();
    PyTuple_SET_ITEM(out, 0, THPVariable_Wrap(a));
    PyTuple_SET_ITEM(out, 1, THPVariable_Wrap(b));
    return out;
}
// Whether the autograd node has to see the call: for a gradient, or to refuse a forward-mode tangent (which
// no_grad does not drop).
static bool wants_grad(std::initializer_list<const Tensor*> ts) {
    for (const Tensor* t : ts)
        if (t->defined() && ((at::GradMode::is_enabled() && t->requires_grad()) || t->_fw_grad(0).defined())) return true;
    return false;
}

// field_read(raw, tr, ti, gamma, state_in or None, lean, want_state) -> read, or (read, state_out)
static PyObject* py_field_read(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    want_args(n, 7);
    const Tensor &raw = tensor_arg(args[0]), &tr = tensor_arg(args[1]), &ti = tensor_arg(args[2]),
                 &gm = tensor_arg(args[3]);
    const std::optional<Tensor> state_in = optional_arg(args[4]);
    const bool lean = PyObject_IsTrue(args[5]) == 1, want_state = PyObject_IsTrue(args[6]) == 1;
    Tensor read, state_out;
    {
        pybind11::gil_scoped_release no_gil;
        const Tensor s = state_in.value_or(Tensor());
        if (wants_grad({&raw, &tr, &ti, &gm, &s})) {
            const variable_list out = FieldRead::apply(raw, tr, ti, gm, state_in, lean, want_state);
            read = out[0];
            if (want_state) state_out = out[1];
        } else {
            run_forward(forward_args(raw, tr, ti, gm, s), read, state_out, want_state);
        }
    }
    return want_state ? wrap2(read, state_out) : wrap(read);
    END_HANDLE_TH_ERRORS
}

// field_read_bf16(raw, tr, ti, gamma, stats) -> read, or (read, sumsq)
static PyObject* py_field_read_bf16(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    want_args(n, 5);
    const Tensor &raw = tensor_arg(args[0]), &tr = tensor_arg(args[1]), &ti = tensor_arg(args[2]),
                 &gm = tensor_arg(args[3]);
    const bool stats = PyObject_IsTrue(args[4]) == 1;
    variable_list out;
    {
        pybind11::gil_scoped_release no_gil;
        out = stats ? FieldReadBf16<true>::apply(raw, tr, ti, gm) : FieldReadBf16<false>::apply(raw, tr, ti, gm);
    }
    return stats ? wrap2(out[0], out[1]) : wrap(out[0]);
    END_HANDLE_TH_ERRORS
}

// linear_scan(a, b, state_in or None, want_state) -> states, or (states, state_out)
static PyObject* py_linear_scan(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    want_args(n, 4);
    const Tensor &a = tensor_arg(args[0]), &b = tensor_arg(args[1]);
    const std::optional<Tensor> state_in = optional_arg(args[2]);
    const bool want_state = PyObject_IsTrue(args[3]) == 1;
    TORCH_CHECK(a.is_cuda() && b.is_cuda(), "linear_scan requires CUDA tensors");
    TORCH_CHECK_TYPE(a.scalar_type() == at::kFloat && b.scalar_type() == at::kFloat, "a and b must be float32, got ",
                     a.scalar_type(), " and ", b.scalar_type());
    TORCH_CHECK_VALUE(a.dim() == 3 && a.sizes() == b.sizes(), shape(a), " ", shape(b));
    variable_list out;
    {
        pybind11::gil_scoped_release no_gil;
        out = LinearScan::apply(a, b, state_in, want_state);
    }
    return want_state ? wrap2(out[0], out[1]) : wrap(out[0]);
    END_HANDLE_TH_ERRORS
}

// step(raw_row, tr, ti, gamma, state) -> read
static PyObject* py_step(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    want_args(n, 5);
    const Tensor &raw = tensor_arg(args[0]), &tr = tensor_arg(args[1]), &ti = tensor_arg(args[2]),
                 &gm = tensor_arg(args[3]), &state = tensor_arg(args[4]);
    Tensor read;
    {
        pybind11::gil_scoped_release no_gil;
        read = step(raw, tr, ti, gm, state);
    }
    return wrap(read);
    END_HANDLE_TH_ERRORS
}

// bind(path, error_type): use the build of the library at `path` from now on.
static PyObject* py_bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    want_args(n, 2);
    const char* path = PyUnicode_AsUTF8(args[0]);
    if (!path) throw python_error();
    void* handle = dlopen(path, RTLD_NOW | RTLD_LOCAL);
    TORCH_CHECK(handle, "cannot open ", path, ": ", dlerror());
    auto table = std::make_unique<Api>();
#define X(name)                                                                   \
    table->name = reinterpret_cast<decltype(&::name)>(dlsym(handle, #name));      \
    TORCH_CHECK(table->name, path, " has no symbol " #name);
    FIELDS_API(X)
#undef X
    Py_INCREF(args[1]);
    g_error_type = args[1];
    // (a backward pass may still hold the old table: one small struct per bound build stays alive)
    g_api.store(table.release(), std::memory_order_release);
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

#define FAST(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
static PyMethodDef g_methods[] = {
    FAST("bind", py_bind),
    FAST("field_read", py_field_read),
    FAST("field_read_bf16", py_field_read_bf16),
    FAST("fused_mixer", py_fused_mixer),
    FAST("linear_scan", py_linear_scan),
    FAST("step", py_step),
    {nullptr, nullptr, 0, nullptr},
};
static PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "libfields_torch", nullptr, -1, g_methods,
                               nullptr, nullptr, nullptr, nullptr};

}  // namespace fields_torch

PyMODINIT_FUNC PyInit_libfields_torch(void) {
    PyObject* m = PyModule_Create(&fields_torch::g_module);
    if (!m) return nullptr;
    try {
        fields_torch::register_release();
        fields_torch::add_stack(m);
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_ImportError, e.what());
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}
