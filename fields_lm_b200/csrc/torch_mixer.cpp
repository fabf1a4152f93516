// The fused Field mixer (bfloat16 boundary, norm behind the output projection) as one autograd node.
//
// As a composition of torch operations the mixer's forward + backward made 76 launches and was bound
// by the host (1.2 - 1.3 ms at 8 x 2,048 x 1,024 against 0.9 ms of kernels). Here it is two matrix
// products forward and four backward (the two projections of x are one product over
// [write_w | gate_w], and so are their two gradients) and the kernels of field_rows.cuh and
// field_mixer_grad.cuh between them. Where kMixerProducts (torch_gemm.h) says so the products of the forward pass and the gradients
// of read and x have fused epilogues (field_product.cuh); the others are library calls. Weight gradients come out of the products in fp32.
#include "torch_gemm.h"

#include <ATen/ops/addmm_cuda_dispatch.h>

namespace fields_torch {

enum { kX, kWriteW, kWriteB, kRadius, kTheta, kNormW, kOutW, kOutB, kGateW, kGateB, kMixerInputs };

// Whether every input is what the node works on: fp32 on one GPU, sizes that fit, parameters dense and aligned (x and the incoming
// gradient, which may be any views, are copied where they are not).
static bool mixer_applies(const std::vector<Tensor>& in) {
    const Tensor& x = in[kX];
    if (x.dim() != 3 || x.numel() == 0 || !x.is_cuda()) return false;
    const int64_t D = x.size(2), C = D / 2;
    if (D % 8 || D > 4096 || x.size(0) > INT_MAX || x.size(1) > INT_MAX) return false;
    const std::vector<int64_t> shapes[kMixerInputs] = {{},     {3 * C, D},     {3 * C}, {C},    {C},
                                                       {2 * D}, {D, 2 * D},     {D},     {D, D}, {D}};
    for (int i = 0; i < kMixerInputs; ++i) {
        const Tensor& t = in[i];
        if (t.scalar_type() != at::kFloat || t.device() != x.device() || t.layout() != at::kStrided) return false;
        if (i == kX) continue;
        if (t.sizes() != at::IntArrayRef(shapes[i]) || !t.is_contiguous() ||
            reinterpret_cast<uintptr_t>(t.data_ptr()) % 16)
            return false;
    }
    return true;
}

struct FusedMixer : torch::autograd::Function<FusedMixer> {
    static variable_list forward(AutogradContext* ctx, const Tensor& x_, const Tensor& write_w, const Tensor& write_b,
                                 const Tensor& radius, const Tensor& theta, const Tensor& norm_w, const Tensor& out_w,
                                 const Tensor& out_b, const Tensor& gate_w, const Tensor& gate_b, double eps) {
        const Api& f = api();
        const Tensor x = aligned(dense(x_));
        const int64_t B = x.size(0), L = x.size(1), D = x.size(2), N = B * L, C = D / 2, W = 3 * C + D, G = (C + 127) / 128;
        const c10::Device dev = x.device();
        const c10::cuda::CUDAGuard guard(dev);
        void* st = stream_of(x);
        const Tensor in_w = empty({W, D}, at::kBFloat16, dev), in_b = empty({W}, at::kBFloat16, dev),
                     out16 = empty({D, 2 * D}, at::kBFloat16, dev), par = empty({3, C}, at::kFloat, dev);
        fields_stack_weights w{};
        w.write_w = fp(write_w); w.write_b = fp(write_b); w.gate_w = fp(gate_w); w.out_w = fp(out_w);
        w.read_norm_w = fp(norm_w); w.radius_logit = fp(radius); w.theta = fp(theta);
        w.in_w = vp(in_w); w.in_b = vp(in_b); w.out_w16 = vp(out16); w.par = fp(par);
        w.dim = (int)D; w.hidden = 0;
        check(f.fields_stack_layout(&w, 1, st), "fields_stack_layout");
        const Tensor xb = empty({N, D}, at::kBFloat16, dev);
        check(f.fields_stack_close_ff(fp(x), nullptr, nullptr, nullptr, vp(xb), 0.0f, N, (int)D, st),
              "fields_stack_close_ff");
        Tensor u = empty({N, W}, at::kBFloat16, dev);
        const bool fused = fused_products(N, D);
        if (fused) {
            fields_product_args q{};
            q.a = vp(xb); q.b = vp(in_w); q.rows = N; q.cols = (int)W; q.depth = (int)D;
            q.bias16 = vp(in_b); q.h = vp(u); q.h_pitch = W;
            check(f.fields_product(&q, FIELDS_PRODUCT_BIAS, st), "fields_product");
        } else {
            at::cuda::addmm_out(u, in_b, xb, in_w.t(), 1, 1);
        }
        const Tensor read = empty({N, 4 * C}, at::kBFloat16, dev), groups = empty({N, G}, at::kFloat, dev);
        {
            const size_t n = f.fields_read_workspace_bytes((int)B, (int)L, (int)C, FIELDS_PASS_FORWARD);
            PassWorkspace ws(n, u);
            float* p = fp(par);
            ws.check(f.fields_read_forward_bf16_rows(vp(u), W, p, p + C, p + 2 * C, nullptr, vp(read), fp(groups), nullptr,
                                                  ws.ptr(), n, (int)B, (int)L, (int)C, st),
                  "fields_read_forward_bf16_rows");
        }
        Tensor acc = empty({N, D}, at::kBFloat16, dev);
        const Tensor y = empty({B, L, D}, at::kFloat, dev);
        if (fused) {  // (74 us at 16,384 rows of 1,024; the library's product and the row kernel 51 + 41)
            fields_product_args q{};
            q.a = vp(read); q.b = vp(out16); q.rows = N; q.cols = (int)D; q.depth = (int)(2 * D);
            q.x = fp(x); q.bias = fp(out_b); q.gate_bias = fp(gate_b); q.gate = gate_of(u, C); q.gate_pitch = W;
            q.sums = fp(groups); q.entries = (int)G; q.features = (int)(2 * D); q.eps = (float)eps;
            q.y = fp(y); q.acc = vp(acc);
            check(f.fields_product(&q, FIELDS_PRODUCT_GATE, st), "fields_product");
        } else {
            product(acc, plain(read), transposed(out16), N, D, 2 * D);
            check(f.fields_stack_close_mixer(fp(x), vp(acc), gate_of(u, C), W, fp(groups), (int)G, fp(out_b), fp(gate_b),
                                             nullptr, fp(y), nullptr, (float)eps, (int)(2 * D), 0.0f, N, (int)D, st),
                  "fields_stack_close_mixer");
        }
        ctx->save_for_backward({xb, u, read, groups, acc, in_w, out16, par, radius, theta, norm_w, out_w, out_b, gate_b});
        ctx->saved_data["eps"] = eps;
        ctx->saved_data["length"] = L;
        return {y};
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const Api& f = api();
        const variable_list s = ctx->get_saved_variables();
        const Tensor &xb = s[0], &u = s[1], &read = s[2], &groups = s[3], &acc = s[4], &in_w = s[5], &out16 = s[6],
                     &par = s[7], &radius = s[8], &theta = s[9], &norm_w = s[10], &out_w = s[11], &out_b = s[12],
                     &gate_b = s[13];
        const Tensor gy = aligned(f32(grads[0]));
        const int64_t N = xb.size(0), D = xb.size(1), C = D / 2, W = 3 * C + D, G = groups.size(1);
        const int64_t L = ctx->saved_data["length"].toInt(), B = N / L;
        const float eps = (float)ctx->saved_data["eps"].toDouble();
        const c10::Device dev = xb.device();
        const c10::cuda::CUDAGuard guard(dev);
        void* st = stream_of(xb);
        auto f32s = [&](at::IntArrayRef size) { return empty(size, at::kFloat, dev); };

        const int64_t n_rows = (int64_t)f.fields_mixer_grad_rows(N),
                      n_scratch = (int64_t)(f.fields_mixer_grad_scratch_bytes((int)D) / 4);
        const Tensor grad_acc = empty({N, D}, at::kBFloat16, dev), grad_u = empty({N, W}, at::kBFloat16, dev),
                     // scratch: partial rows of open_grad, of close_grad, grad_sumsq, gradients of the transition
                     temp = f32s({2 * n_rows * D + n_scratch + 3 * C + N});
        float *rows = fp(temp), *scratch = rows + 2 * n_rows * D, *g = scratch + n_scratch, *grad_sumsq = g + 3 * C;
        check(f.fields_mixer_open_grad(fp(gy), vp(acc), gate_of(u, C), W, fp(groups), (int)G, fp(out_b), fp(gate_b),
                                       vp(grad_acc), gate_of(grad_u, C), W, grad_sumsq, rows, eps, (int)(2 * D),
                                       N, (int)D, st),
              "fields_mixer_open_grad");
        // What a frozen parameter leaves out; the recurrence runs backward for x and what lies before it.
        auto need = [&](int i) { return ctx->needs_input_grad(i); };
        const bool recurrence = need(kX) || need(kWriteW) || need(kWriteB) || need(kRadius) || need(kTheta);
        float* p = fp(par);
        // The products of the gradients of read and x have epilogues where those of the forward pass have.
        const bool fused = fused_products(N, D);
        if (recurrence) {
            const Tensor grad_read = empty({N, 4 * C}, at::kBFloat16, dev);
            if (fused) {
                fields_product_args q{};
                q.a = vp(grad_acc); q.b = vp(out16); q.rows = N; q.cols = (int)(2 * D); q.depth = (int)D;
                q.read = vp(read); q.row = grad_sumsq; q.h = vp(grad_read); q.h_pitch = 2 * D;
                check(f.fields_product(&q, FIELDS_PRODUCT_NORM_GRAD + FIELDS_PRODUCT_BY_DEPTH, st), "fields_product");
            } else {
                product(grad_read, plain(grad_acc), plain(out16), N, 2 * D, D);
                check(f.fields_read_norm_grad_combine(vp(grad_read), vp(read), grad_sumsq, vp(grad_read), N, (int)(4 * C), st),
                      "fields_read_norm_grad_combine");
            }
            const size_t n = f.fields_read_workspace_bytes((int)B, (int)L, (int)C, FIELDS_PASS_BACKWARD);
            PassWorkspace ws(n, u);
            ws.check(f.fields_read_backward_bf16_rows(vp(u), W, p, p + C, p + 2 * C, vp(read), vp(grad_read), vp(grad_u), W,
                                                   g, g + C, g + 2 * C, ws.ptr(), n, (int)B, (int)L, (int)C, st),
                  "fields_read_backward_bf16_rows");
        }
        Tensor grad_out;
        if (need(kOutW) || need(kNormW)) {
            grad_out = f32s({D, 2 * D});
            product(grad_out, transposed(grad_acc), plain(read), D, 2 * D, N);
        }
        Tensor grad_x;
        if (need(kX)) {
            grad_x = f32s({B, L, D});
            if (fused) {
                fields_product_args q{};
                q.a = vp(grad_u); q.b = vp(in_w); q.rows = N; q.cols = (int)D; q.depth = (int)W;
                q.x = fp(gy); q.y = fp(grad_x);
                check(f.fields_product(&q, FIELDS_PRODUCT_RESIDUAL + FIELDS_PRODUCT_BY_DEPTH, st), "fields_product");
            } else {
                Tensor back = empty({N, D}, at::kBFloat16, dev);
                product(back, plain(grad_u), plain(in_w), N, D, W);
                check(f.fields_stack_close_ff(fp(gy), vp(back), nullptr, fp(grad_x), nullptr, 0.0f, N, (int)D, st),
                      "fields_stack_close_ff");
            }
        }
        Tensor grad_write_w, grad_gate_w;  // (one product over both where both are wanted)
        if (need(kWriteW) || need(kGateW)) {
            const int64_t first = need(kWriteW) ? 0 : 3 * C, rows_in = (need(kGateW) ? W : 3 * C) - first;
            const Tensor grad_in = f32s({rows_in, D});
            product(grad_in, Operand{static_cast<at::BFloat16*>(vp(grad_u)) + first, true, W}, plain(xb), rows_in, D, N);
            if (need(kWriteW)) grad_write_w = grad_in.narrow(0, 0, 3 * C);
            if (need(kGateW)) grad_gate_w = grad_in.narrow(0, 3 * C - first, D);
        }

        // the small gradients share an allocation
        const Tensor small = f32s({4 * D + 5 * C});
        int64_t at = 0;
        auto part = [&](int i, int64_t n) {
            at += n;
            return need(i) ? part_of(small, at - n, n) : Tensor();
        };
        const Tensor g_out_b = part(kOutB, D), g_gate_b = part(kGateB, D), g_norm = part(kNormW, 2 * D),
                     g_write_b = part(kWriteB, 3 * C), g_radius = part(kRadius, C), g_theta = part(kTheta, C);
        fields_mixer_grads q{};
        q.rows = rows; q.grad_raw = vp(grad_u); q.grad_pitch = W; q.grad_out = fp(grad_out); q.out_w = fp(out_w);
        q.norm_w = fp(norm_w); q.radius_logit = fp(radius); q.theta = fp(theta);
        q.grad_tr = g; q.grad_ti = g + C; q.grad_gamma = g + 2 * C;
        q.grad_out_b = fp(g_out_b); q.grad_gate_b = fp(g_gate_b); q.grad_write_b = fp(g_write_b);
        q.grad_norm_w = fp(g_norm); q.grad_radius = fp(g_radius); q.grad_theta = fp(g_theta); q.scratch = scratch;
        check(f.fields_mixer_close_grad(&q, N, (int)D, st), "fields_mixer_close_grad");
        return {grad_x,   grad_write_w, g_write_b,   g_radius, g_theta, g_norm, need(kOutW) ? grad_out : Tensor(),
                g_out_b, grad_gate_w,  g_gate_b,  Tensor()};
    }

  private:
    // (widths whose rows TMA can address)
    static bool fused_products(int64_t N, int64_t D) { return D % 16 == 0 && fields_torch::fused_products(N, D, kMixerProducts); }
    // the gate columns of [raw | gate]
    static void* gate_of(const Tensor& u, int64_t C) { return static_cast<at::BFloat16*>(vp(u)) + 3 * C; }
};

// fused_mixer(x, write_w, write_b, radius_logit, theta, norm_w, out_w, out_b, gate_w, gate_b, eps) -> y, or None
// where the node does not apply
PyObject* py_fused_mixer(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    want_args(n, kMixerInputs + 1);
    std::vector<Tensor> in;
    in.reserve(kMixerInputs);
    for (int i = 0; i < kMixerInputs; ++i) in.push_back(tensor_arg(args[i]));
    const double eps = PyFloat_AsDouble(args[kMixerInputs]);
    if (PyErr_Occurred()) throw python_error();
    Tensor y;
    {
        pybind11::gil_scoped_release no_gil;
        if (mixer_applies(in))
            y = FusedMixer::apply(in[kX], in[kWriteW], in[kWriteB], in[kRadius], in[kTheta], in[kNormW], in[kOutW],
                                  in[kOutB], in[kGateW], in[kGateB], eps)[0];
    }
    if (!y.defined()) Py_RETURN_NONE;
    return THPVariable_Wrap(y);
    END_HANDLE_TH_ERRORS
}

}  // namespace fields_torch
