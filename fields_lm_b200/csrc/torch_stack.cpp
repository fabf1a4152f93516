// A stack of Field blocks at inference under bfloat16 autocast: the prefill of a batch of prompts and the
// single-token step, block by block in native code.
//
// Per block of a prefill the recurrence and four products with fused epilogues (field_product.cuh), or, for few rows of a
// wide model, library products and row kernels (field_rows.cuh); a step is one launch (field_step_gemm.cuh).
// A block's modules make some 48 launches. The bfloat16 copies of the weights that autocast makes on
// every call are laid out once per prefill and kept for the steps
// that follow it. The owner (FieldStackDecoder) asks current() before a step: the copies are used
// only while every module, parameter and hook is what it was and no parameter has been written to, as far as
// torch counts it (a write through `.data` or by another library is not counted; the next prefill sees
// it). Parameters without a count (inference tensors) are laid out for every step.
#include "torch_gemm.h"

#include <ATen/cuda/CUDAEvent.h>
#include <ATen/ops/addmm_cuda_dispatch.h>
#include <ATen/ops/mm_cuda_dispatch.h>
#include <torch/csrc/utils/pybind.h>

#include <array>

namespace fields_torch {

namespace py = pybind11;

// A parameter (the module's own tensor), where its data lay when the plan was made and its version
// when its copy was made. Inference tensors have no version: their copies are never up to date.
struct Source {
    explicit Source(const Tensor& p) : t(p), data(p.data_ptr()) {}
    void copied() { version = t.is_inference() ? 0 : t._version(); }
    bool current() const { return !t.is_inference() && t._version() == version; }
    Tensor t;
    const void* data;
    uint64_t version = 0;
};

struct Block {
    // write_w, write_b, gate_w, gate_b, out_w, out_b, read_norm_w, ff_norm_w, w12, w3, radius_logit, theta
    enum { kWriteW, kWriteB, kGateW, kGateB, kOutW, kOutB, kReadNorm, kFfNorm, kW12, kW3, kRadius, kTheta, kCount };
    std::vector<Source> src;
    double read_eps = 0, ff_eps = 0;
    // bfloat16, transposed views for the products; `in` = write over gate, scaled `out`
    Tensor in_w, in_b, in_t, out_t, w12_t, w3_t, par;
    // rows of `in` and w12 in the order of the fused step, its biases (made by the first step after a layout)
    Tensor step_in, step_w12, step_b;
    float* f(int i) const { return fp(src[i].t); }
};

// Copies that are allocated together lie in memory of the stream that first laid them out (home), and every later call
// may be on another: a call waits for the layout, a layout for the calls on other streams, and the memory goes back
// only behind all of them. On one stream this costs an event per layout. One thread issues at a time. Copies that calls
// lay out on the way have a home of their own each: the stream of the call that first needed them.
class CopyUses {
  public:
    using Stream = c10::cuda::CUDAStream;

    // One call that uses (or, `writes`, lays out and may then use) the copies on the current stream of `device`.
    class Call {
      public:
        Call(CopyUses& u, c10::Device device, bool writes)
            : u_(u), lock_(u.mu_), stream_(c10::cuda::getCurrentCUDAStream(device.index())), writes_(writes) {
            if (!u.home_) u.home_ = stream_;
            if (u.laid_on_ && *u.laid_on_ != stream_) u.laid_.block(stream_);
            if (writes) u.wait_for_uses(stream_);
        }
        // (not on the way out of an exception alone: what was issued before it is a use as well)
        ~Call() {
            try {
                if (writes_) laid_out();
                if (stream_ != *u_.home_ || external(stream_)) u_.used_on(stream_);
            } catch (...) {
            }
        }
        Call(const Call&) = delete;
        // The layout has been issued: calls on other streams wait for nothing behind it.
        void laid_out() {
            writes_ = false;
            if (captured(stream_)) return;  // (a plan of its own, used on this stream only)
            u_.laid_.record(stream_);
            u_.laid_on_ = stream_;
        }

      private:
        CopyUses& u_;
        std::lock_guard<std::recursive_mutex> lock_;
        Stream stream_;
        bool writes_;
    };

    CopyUses() = default;
    CopyUses(const CopyUses&) = delete;
    ~CopyUses() {
        try {
            if (home_ && !captured(*home_)) {
                if (laid_on_ && *laid_on_ != *home_) laid_.block(*home_);
                wait_for_uses(*home_);
            }
        } catch (...) {
        }
    }

  private:
    struct Use {
        Stream stream;
        at::cuda::CUDAEvent last;
    };
    static bool captured(Stream s) {
        cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
        return cudaStreamIsCapturing(s.stream(), &status) != cudaSuccess || status != cudaStreamCaptureStatusNone;
    }
    // another library's stream, which may be gone when a later call would record on it
    static bool external(Stream s) { return s.id() != 0 && !(s.id() & 1); }
    void used_on(Stream s) {
        if (captured(s)) return;
        for (Use& u : uses_)
            if (u.stream == s) return u.last.record(s);
        uses_.push_back(Use{s, at::cuda::CUDAEvent()});
        uses_.back().last.record(s);
    }
    void wait_for_uses(Stream s) {
        if (captured(s)) return;
        if (*home_ != s && !external(*home_) && !captured(*home_)) used_on(*home_);
        for (Use& u : uses_)
            if (u.stream != s) u.last.block(s);
        uses_.clear();
    }

    std::recursive_mutex mu_;
    std::optional<Stream> home_, laid_on_;
    at::cuda::CUDAEvent laid_;
    std::vector<Use> uses_;  // last uses on streams other than home since all of them were waited for
};

class FieldStack {
  public:
    FieldStack(const std::vector<std::vector<Tensor>>& params, const std::vector<std::pair<double, double>>& eps,
               std::vector<std::tuple<py::object, py::object, py::object>> slots,
               std::vector<std::pair<py::object, int64_t>> sizes,
               std::vector<std::pair<py::object, py::object>> classes, std::vector<Tensor> tail, double tail_eps,
               bool usable)
        : slots_(std::move(slots)), sizes_(std::move(sizes)), classes_(std::move(classes)), tail_eps_(tail_eps),
          usable_(usable) {
        for (size_t i = 0; i < params.size(); ++i) {
            Block b;
            TORCH_CHECK_VALUE(params[i].size() == Block::kCount, "a block has ", (int)Block::kCount, " parameters");
            for (const Tensor& t : params[i]) b.src.emplace_back(t);
            b.read_eps = eps[i].first;
            b.ff_eps = eps[i].second;
            blocks_.push_back(std::move(b));
        }
        for (const Tensor& t : tail) tail_.emplace_back(t);
        D_ = (int)blocks_[0].src[Block::kGateW].t.size(0);
        H_ = (int)blocks_[0].src[Block::kW3].t.size(1);
    }

    // Whether the model still consists of the same modules, attributes and parameters where they were, with
    // the same code and no hooks on them.
    bool same_model() const {
        for (const auto& [dict, key, want] : slots_)
            if (PyDict_GetItem(dict.ptr(), key.ptr()) != want.ptr()) return false;
        for (const auto& [dict, size] : sizes_)
            if (PyDict_Size(dict.ptr()) != size) return false;
        for (const auto& [cls, forward] : classes_)
            if (py::object(cls.attr("forward")).ptr() != forward.ptr()) return false;
        return every_source([](const Source& s) { return s.t.data_ptr() == s.data; });
    }

    // ... and whether the copies of the parameters are up to date.
    bool current() const {
        return copies_[kBase].laid_out && same_model() && every_source([](const Source& s) { return s.current(); });
    }

    // The same plan without copies, for a graph that is being captured: its copies are laid out by the graph
    // itself, from the weights of the moment it runs, into memory of its own.
    std::unique_ptr<FieldStack> fresh() const {
        auto other = std::make_unique<FieldStack>(*this);
        for (Copies& c : other->copies_) c = Copies();
        for (Block& b : other->blocks_) b.in_w = b.in_b = b.in_t = b.out_t = b.w12_t = b.w3_t = b.par = b.step_in = b.step_w12 = b.step_b = Tensor();
        other->head_ = other->head_w_ = other->head_b_ = Tensor();
        return other;
    }

    // Whether the model's modules compute what this class does; if not, the plan only stands for the refusal.
    bool usable() const { return usable_; }

    // Whether step() goes on to the logits.
    bool has_head() const { return !tail_.empty(); }

    // Makes the bfloat16 copies for a prefill of `prefill_rows` rows and the steps of `step_rows` rows that may follow it, or
    // (0 rows of prefill) for a step. Once per prefill: 0.21 ms for 18 blocks of d_model 1,024, 0.45 GB. What only
    // a fused step reads is made by the first one: 0.09 GB, and 0.19 GB of w12 in its order where the prefill took
    // library products.
    void layout(int64_t prefill_rows, int64_t step_rows) {
        const c10::Device dev = blocks_[0].src[0].t.device();
        const c10::cuda::CUDAGuard guard(dev);
        const CopyUses::Call call(*copies_[kBase].uses, dev, true);
        const int64_t D = D_, C = D / 2, H = H_;
        for (Copies& c : copies_) c.laid_out = false;
        for (Block& b : blocks_) {
            for (Source& s : b.src) s.copied();
            if (!b.in_w.defined()) {
                b.in_w = empty({3 * C + D, D}, at::kBFloat16, dev);
                b.in_b = empty({3 * C + D}, at::kBFloat16, dev);
                b.in_t = b.in_w.t();
                b.out_t = empty({D, 2 * D}, at::kBFloat16, dev).t();
                b.w3_t = empty({D, H}, at::kBFloat16, dev).t();
                b.par = empty({3, C}, at::kFloat, dev);
            }
        }
        void* st = stream_of(blocks_[0].in_w);
        bool need[kCopies] = {};  // the orders of w12
        if (prefill_rows > 0) need[fused_products(prefill_rows, D_, kPrefillProducts) ? kOrdered : kPlain] = true;
        if (prefill_rows == 0 || !fused_step(step_rows)) need[fused_step(step_rows) ? kOrdered : kPlain] = true;
        int parts = FIELDS_LAYOUT_REST;
        for (int which : {kOrdered, kPlain}) {
            if (!need[which]) continue;
            std::optional<CopyUses::Call> w12_call;
            use(which, w12_call);
            lay_out(parts | part_of_w12(which), st);
            laid_out(which, *w12_call);
            parts = 0;
        }
        if (!tail_.empty()) {
            for (Source& s : tail_) s.copied();
            const at::NoGradGuard no_grad;
            auto copy = [&](Tensor& to, const Tensor& from) {
                if (!to.defined()) {
                    const c10::InferenceMode off(false);  // written again in whatever mode the next layout has
                    to = empty(from.sizes(), at::kBFloat16, dev);
                }
                to.copy_(from);
            };
            copy(head_, tail_[1].t);
            head_w_ = head_.t();
            if (tail_.size() > 2) copy(head_b_, tail_[2].t);
        }
        copies_[kBase].laid_out = true;
    }

    // x [B, L, D] fp32 -> the stack's output [B, L, D] and every block's end state [B, D].
    std::pair<Tensor, std::vector<Tensor>> prefill(const Tensor& x_) {
        const Api& f = api();
        const Tensor x = activations(x_, 3);
        const int64_t B = x.size(0), L = x.size(1), N = B * L, D = D_, C = D / 2, W = 3 * C + D, G = (C + 127) / 128;
        const c10::Device dev = x.device();
        const c10::cuda::CUDAGuard guard(dev);
        const CopyUses::Call call(*copies_[kBase].uses, dev, false);
        void* st = stream_of(x);
        const bool products = fused_products(N, D, kPrefillProducts);
        std::optional<CopyUses::Call> w12_call;
        need_w12(products, w12_call, st);
        const Tensor xb = empty({N, D}, at::kBFloat16, dev), y = empty({B, L, D}, at::kFloat, dev),
                     read = empty({N, 4 * C}, at::kBFloat16, dev), groups = empty({N, G}, at::kFloat, dev);
        const size_t ws_bytes = f.fields_read_workspace_bytes((int)B, (int)L, (int)C, FIELDS_PASS_FORWARD);
        Tensor u = empty({N, W}, at::kBFloat16, dev), act = empty({N, H_}, at::kBFloat16, dev), acc, uv, y_sq;
        if (products) {
            y_sq = empty({N, (D + 31) / 32}, at::kFloat, dev);
        } else {
            acc = empty({N, D}, at::kBFloat16, dev);
            uv = empty({N, 2 * (int64_t)H_}, at::kBFloat16, dev);
        }
        std::vector<Tensor> states;
        check(f.fields_stack_close_ff(fp(x), nullptr, nullptr, nullptr, vp(xb), 0.0f, N, D_, st),
              "fields_stack_close_ff");
        const float* in = fp(x);
        for (const Block& b : blocks_) {
            fields_product_args q{};
            q.rows = N;
            if (products) {
                q.a = vp(xb); q.b = vp(b.in_w); q.cols = (int)W; q.depth = D_;
                q.bias16 = vp(b.in_b); q.h = vp(u); q.h_pitch = W;
                check(f.fields_product(&q, FIELDS_PRODUCT_BIAS, st), "fields_product");
            } else {
                at::cuda::addmm_out(u, b.in_b, xb, b.in_t, 1, 1);
            }
            const Tensor state = empty({B, D}, at::kFloat, dev);
            PassWorkspace ws(ws_bytes, u);
            float* par = fp(b.par);
            ws.check(f.fields_read_forward_bf16_rows(vp(u), W, par, par + C, par + 2 * C, nullptr, vp(read), fp(groups),
                                                  fp(state), ws.ptr(), ws_bytes, (int)B, (int)L, (int)C, st),
                  "fields_read_forward_bf16_rows");
            const void* gate = static_cast<at::BFloat16*>(vp(u)) + 3 * C;
            if (products) {
                q.a = vp(read); q.b = vp(b.out_t); q.cols = D_; q.depth = 2 * D_;
                q.x = in; q.bias = b.f(Block::kOutB); q.gate_bias = b.f(Block::kGateB); q.gate = gate; q.gate_pitch = W;
                q.sums = fp(groups); q.entries = (int)G; q.features = 2 * D_; q.eps = (float)b.read_eps;
                q.y = fp(y); q.h = vp(xb); q.h_pitch = D; q.sums_out = fp(y_sq);
                check(f.fields_product(&q, FIELDS_PRODUCT_GATE, st), "fields_product");
                q.a = vp(xb); q.b = vp(b.step_w12); q.cols = 2 * H_; q.depth = D_;
                q.sums = fp(y_sq); q.entries = (int)((D + 31) / 32); q.features = D_; q.eps = (float)b.ff_eps;
                q.h = vp(act); q.h_pitch = H_;
                check(f.fields_product(&q, FIELDS_PRODUCT_SWIGLU, st), "fields_product");
                q.a = vp(act); q.b = vp(b.w3_t); q.cols = D_; q.depth = H_;
                q.x = fp(y); q.h = vp(xb); q.h_pitch = D;
                check(f.fields_product(&q, FIELDS_PRODUCT_RESIDUAL, st), "fields_product");
            } else {
                product(acc, plain(read), transposed(b.out_t), N, D, 2 * D);
                check(f.fields_stack_close_mixer(in, vp(acc), gate, W, fp(groups), (int)G,
                                                 b.f(Block::kOutB), b.f(Block::kGateB), b.f(Block::kFfNorm), fp(y),
                                                 vp(xb), (float)b.read_eps, 2 * D_, (float)b.ff_eps, N, D_, st),
                      "fields_stack_close_mixer");
                feed_forward(b, xb, uv, act, acc, N, st);
                check(f.fields_stack_close_ff(fp(y), vp(acc), nullptr, fp(y), vp(xb), 0.0f, N, D_, st),
                      "fields_stack_close_ff");
            }
            in = fp(y);
            states.push_back(state);
        }
        return {y, states};
    }

    // One token per row: x [B, D] fp32; states advance in place. Returns the logits where the tail (final
    // norm and head) is part of the plan, else the stack's output.
    Tensor step(const Tensor& x_, const std::vector<Tensor>& states) {
        const Tensor x = activations(x_, 2);
        const int64_t N = x.size(0), D = D_;
        TORCH_CHECK_VALUE(states.size() == blocks_.size(), "one state per block is needed");
        std::vector<Tensor> own = states;  // 16-byte aligned: a caller's may be any view
        bool aligned = true;
        for (const Tensor& s : states) {
            TORCH_CHECK_VALUE(s.device() == x.device() && s.scalar_type() == at::kFloat && s.is_contiguous() && s.dim() == 2 &&
                                  s.size(0) == N && s.size(1) == D,
                              shape(s));
            aligned = aligned && reinterpret_cast<uintptr_t>(s.data_ptr()) % 16 == 0;
        }
        const c10::cuda::CUDAGuard guard(x.device());
        const CopyUses::Call call(*copies_[kBase].uses, x.device(), false);
        std::optional<CopyUses::Call> w12_call, in_call;
        if (!aligned)
            for (Tensor& s : own) s = s.clone();
        const bool fused = fused_step(N);
        if (fused) step_layout(w12_call, in_call, stream_of(x));
        else need_w12(false, w12_call, stream_of(x));
        const Tensor xb = empty({N, D}, at::kBFloat16, x.device()), y = empty({N, D}, at::kFloat, x.device());
        check(api().fields_stack_close_ff(fp(x), nullptr, nullptr, nullptr, vp(xb), 0.0f, N, D_, stream_of(x)),
              "fields_stack_close_ff");
        if (fused) step_fused(x, own, xb, y);
        else step_products(x, own, xb, y);
        if (!aligned)
            for (size_t i = 0; i < states.size(); ++i) states[i].copy_(own[i]);
        if (tail_.empty()) return y;
        check(api().fields_stack_close_ff(fp(y), nullptr, fp(tail_[0].t), nullptr, vp(xb), (float)tail_eps_, N, D_,
                                          stream_of(x)),
              "fields_stack_close_ff");
        Tensor logits = empty({N, head_w_.size(1)}, at::kBFloat16, x.device());
        if (head_b_.defined()) at::cuda::addmm_out(logits, head_b_, xb, head_w_, 1, 1);
        else at::cuda::mm_out(logits, xb, head_w_);
        return logits;
    }

  private:
    // Fused products instead of the library's while those of the step have tiles (128 rows x 64 features) few enough. us per step
    // against library products: eight blocks of d_model 576 264 and 355 at 512 rows, 1,024 250 and 350 at 256 rows, 316 and 358 at 257,
    // 322 and 355 at 512 (64 tiles), 1,280 360 and 395 at 384, but 604 and 441 at 400 (80); four blocks of 2,048 258 and 260 at
    // 256 rows. Wider ones while there are up to 64 rows: 2,560 255 and 284 at 1 row, 269 and 276 at 64, 297 and 289 at 128; 3,072 293
    // and 366, 311 and 323, 340 and 332; 4,096 389 and 512, 412 and 449.
    bool fused_step(int64_t rows) const {
        return D_ % 16 == 0 && H_ % 8 == 0 && rows <= 512 && (rows + 127) / 128 * ((D_ + 63) / 64) <= 64 &&
               (D_ <= 2048 || rows <= 64);
    }

    // Whether its blocks are one launch or four launches each. Eight blocks, us as one and as four each: d_model 64 113 and 147 at one
    // row, 130 and 151 at 64, 148 and 150 at 65, but 173 and 162 at 128 and 174 and 170 at 256, where a phase is one tile of which
    // a thread block finishes 128 rows by itself; 176 and 177 at 512. Wider ones always: 128 117 and 164 at one row, 165 and 175 at 128,
    // 168 and 196 at 512; 256 130 and 165, 156 and 175, 159 and 187; 512 142 and 211, 164 and 216, 210 and 239; 768 158 and 235,
    // 187 and 242 and, at 256 rows, 226 and 262.
    bool step_in_one_launch(int64_t rows) const { return D_ > 64 || rows <= 64 || rows > 256; }

    // The embedding's output as the kernels take it: a width of another model is refused, as nn.Linear does.
    Tensor activations(const Tensor& x, int64_t dims) const {
        const c10::Device dev = blocks_[0].src[0].t.device();
        TORCH_CHECK(x.dim() == dims && x.size(dims - 1) == D_ && x.scalar_type() == at::kFloat && x.device() == dev,
                    "activations of shape ", shape(x), " on ", x.device(), " do not fit blocks of width ", D_, " on ", dev);
        return aligned(dense(x));
    }

    template <class F>
    bool every_source(F ok) const {
        for (const Block& b : blocks_)
            for (const Source& s : b.src)
                if (!ok(s)) return false;
        for (const Source& s : tail_)
            if (!ok(s)) return false;
        return true;
    }

    // Weights in the order of the fused step. (w12 may be there already, from a prefill with fused products. The rows that its
    // buffer has beyond those of w12 reach no column that is stored.)
    void step_layout(std::optional<CopyUses::Call>& w12_call, std::optional<CopyUses::Call>& in_call, void* st) {
        const Api& f = api();
        need_w12(true, w12_call, st);
        if (use(kStepIn, in_call)) return;
        const int64_t D = D_, C = D / 2;
        const c10::Device dev = blocks_[0].in_w.device();
        for (Block& b : blocks_) {
            if (!b.step_in.defined()) {
                b.step_in = empty({5 * C, D}, at::kBFloat16, dev);
                b.step_b = empty({5 * C}, at::kFloat, dev);
            }
            fields_step_weights w{};
            w.write_w = b.f(Block::kWriteW); w.write_b = b.f(Block::kWriteB); w.gate_w = b.f(Block::kGateW);
            w.gate_b = b.f(Block::kGateB);
            w.in_w = vp(b.step_in); w.in_b = fp(b.step_b);
            w.dim = D_; w.hidden = H_;
            check(f.fields_step_layout(&w, st), "fields_step_layout");
        }
        laid_out(kStepIn, *in_call);
    }

    fields_stack_weights weights_of(const Block& b) const {
        fields_stack_weights w{};
        w.write_w = b.f(Block::kWriteW); w.write_b = b.f(Block::kWriteB); w.gate_w = b.f(Block::kGateW);
        w.out_w = b.f(Block::kOutW); w.read_norm_w = b.f(Block::kReadNorm); w.w12 = b.f(Block::kW12);
        w.w3 = b.f(Block::kW3); w.radius_logit = b.f(Block::kRadius); w.theta = b.f(Block::kTheta);
        w.in_w = vp(b.in_w); w.in_b = vp(b.in_b); w.out_w16 = vp(b.out_t); w.w3_16 = vp(b.w3_t); w.par = fp(b.par);
        w.dim = D_; w.hidden = H_;
        return w;
    }

    // Opens a call on copies that may have to be laid out first; whether they need not be.
    bool use(int which, std::optional<CopyUses::Call>& call) {
        call.emplace(*copies_[which].uses, blocks_[0].in_w.device(), !copies_[which].laid_out);
        return copies_[which].laid_out;
    }
    void laid_out(int which, CopyUses::Call& call) {
        call.laid_out();
        copies_[which].laid_out = true;
    }

    static int part_of_w12(int which) { return which == kOrdered ? FIELDS_LAYOUT_W12_STEP : FIELDS_LAYOUT_W12; }
    // `parts` of all blocks, w12 among them in one of its orders.
    void lay_out(int parts, void* st) {
        const c10::Device dev = blocks_[0].in_w.device();
        std::vector<fields_stack_weights> all;
        std::vector<const float*> norms;
        for (Block& b : blocks_) {
            const bool ordered = parts & FIELDS_LAYOUT_W12_STEP;
            Tensor& to = ordered ? b.step_w12 : b.w12_t;
            if (!to.defined())
                to = ordered ? empty({api().fields_step_w12_rows(H_), D_}, at::kBFloat16, dev)
                             : empty({2 * (int64_t)H_, D_}, at::kBFloat16, dev).t();
            all.push_back(weights_of(b));
            all.back().w12_16 = vp(to);
            norms.push_back(b.f(Block::kFfNorm));
        }
        check(api().fields_stack_layout_parts(all.data(), norms.data(), (int)all.size(), parts, st), "fields_stack_layout_parts");
    }

    // w12 as the library's products take it, or in the order of the fused products and of the step: whichever a call
    // needs first lays it out.
    void need_w12(bool step, std::optional<CopyUses::Call>& call, void* st) {
        const int which = step ? kOrdered : kPlain;
        if (use(which, call)) return;
        lay_out(part_of_w12(which), st);
        laid_out(which, *call);
    }

    // The blocks of a step in one launch, each a chain of four products with fused epilogues (field_step_gemm.cuh).
    void step_fused(const Tensor& x, const std::vector<Tensor>& states, const Tensor& xb, const Tensor& y) {
        const Api& f = api();
        const int64_t N = x.size(0), D = D_, C = D / 2, H = H_;
        const c10::Device dev = x.device();
        void* st = stream_of(x);
        const Tensor yb = empty({N, D}, at::kBFloat16, dev), read = empty({N, 4 * C}, at::kBFloat16, dev),
                     gate = empty({N, D}, at::kBFloat16, dev), act = empty({N, H}, at::kBFloat16, dev),
                     read_sq = empty({C / 8, N}, at::kFloat, dev), y_sq = empty({D / 8, N}, at::kFloat, dev),
                     sync = empty({512}, at::kByte, dev);
        std::vector<fields_step_args> all;
        fields_step_args g{};
        g.x = fp(x); g.y = fp(y); g.xb = vp(xb); g.yb = vp(yb); g.read = vp(read); g.gate = vp(gate); g.act = vp(act);
        g.read_sq = fp(read_sq); g.y_sq = fp(y_sq);
        g.rows = (int)N; g.dim = D_; g.hidden = H_;
        g.settled = 1;  // step()'s copy of x stands between a layout and the first block, and waits for it
        for (size_t i = 0; i < blocks_.size(); ++i) {
            const Block& b = blocks_[i];
            g.state = fp(states[i]);
            g.in_w = vp(b.step_in); g.out_w16 = vp(b.out_t); g.w12_w = vp(b.step_w12); g.w3_16 = vp(b.w3_t);
            g.in_b = fp(b.step_b); g.par = fp(b.par); g.out_b = b.f(Block::kOutB);
            g.read_eps = (float)b.read_eps; g.ff_eps = (float)b.ff_eps;
            all.push_back(g);
            g.x = g.y;
        }
        if (!step_in_one_launch(N)) {
            for (const fields_step_args& block : all) check(f.fields_step_block(&block, st), "fields_step_block");
            return;
        }
        check(f.fields_step_stack(all.data(), (int)all.size(), vp(sync), st), "fields_step_stack");
    }

    // The same with library products, for what the fused step does not take.
    void step_products(const Tensor& x, const std::vector<Tensor>& states, const Tensor& xb, const Tensor& y) {
        const Api& f = api();
        const int64_t N = x.size(0), D = D_, C = D / 2, W = 3 * C + D;
        const c10::Device dev = x.device();
        void* st = stream_of(x);
        const Tensor read = empty({N, 4 * C}, at::kBFloat16, dev);
        Tensor acc = empty({N, D}, at::kBFloat16, dev), in = empty({N, W}, at::kBFloat16, dev),
               uv = empty({N, 2 * (int64_t)H_}, at::kBFloat16, dev), act = empty({N, H_}, at::kBFloat16, dev);
        const float* from = fp(x);
        for (size_t i = 0; i < blocks_.size(); ++i) {
            const Block& b = blocks_[i];
            at::cuda::addmm_out(in, b.in_b, xb, b.in_t, 1, 1);
            check(f.fields_stack_step_norm(vp(in), W, fp(b.par), fp(states[i]), vp(read), (float)b.read_eps, N,
                                           (int)C, st),
                  "fields_stack_step_norm");
            product(acc, plain(read), transposed(b.out_t), N, D, 2 * D);
            const void* gate = static_cast<at::BFloat16*>(vp(in)) + 3 * C;
            check(f.fields_stack_close_mixer(from, vp(acc), gate, W, nullptr, 0, b.f(Block::kOutB),
                                             b.f(Block::kGateB), b.f(Block::kFfNorm), fp(y), vp(xb), 0.0f, 1,
                                             (float)b.ff_eps, N, D_, st),
                  "fields_stack_close_mixer");
            feed_forward(b, xb, uv, act, acc, N, st);
            check(f.fields_stack_close_ff(fp(y), vp(acc), nullptr, fp(y), vp(xb), 0.0f, N, D_, st),
                  "fields_stack_close_ff");
            from = fp(y);
        }
    }

    void feed_forward(const Block& b, const Tensor& h, Tensor& uv, Tensor& act, Tensor& out, int64_t N, void* st) {
        product(uv, plain(h), transposed(b.w12_t), N, 2 * (int64_t)H_, D_);
        check(api().fields_stack_swiglu(vp(uv), vp(act), N, H_, st), "fields_stack_swiglu");
        product(out, plain(act), transposed(b.w3_t), N, D_, H_);
    }

    std::vector<Block> blocks_;
    std::vector<std::tuple<py::object, py::object, py::object>> slots_;  // (dict, key, the object there)
    std::vector<std::pair<py::object, int64_t>> sizes_;                  // dicts and the sizes they have to have
    std::vector<std::pair<py::object, py::object>> classes_;             // and the `forward` they have to have
    std::vector<Source> tail_;  // final norm weight, head weight[, head bias]; may be empty
    Tensor head_, head_w_, head_b_;
    double tail_eps_;
    bool usable_;
    int D_ = 0, H_ = 0;
    // in_w, in_b, out_t, w3_t, par and the head; w12_t; step_w12; step_in and step_b. A call takes kBase first.
    enum { kBase, kPlain, kOrdered, kStepIn, kCopies };
    struct Copies {
        std::shared_ptr<CopyUses> uses = std::make_shared<CopyUses>();
        bool laid_out = false;
    };
    std::array<Copies, kCopies> copies_;  // destroyed before the copies above
};

void add_stack(PyObject* module) {
    py::module_ m = py::reinterpret_borrow<py::module_>(module);
    py::class_<FieldStack>(m, "FieldStack")
        .def(py::init<const std::vector<std::vector<Tensor>>&, const std::vector<std::pair<double, double>>&,
                      std::vector<std::tuple<py::object, py::object, py::object>>,
                      std::vector<std::pair<py::object, int64_t>>, std::vector<std::pair<py::object, py::object>>,
                      std::vector<Tensor>, double, bool>())
        .def_property_readonly("usable", &FieldStack::usable)
        .def_property_readonly("has_head", &FieldStack::has_head)
        .def("same_model", &FieldStack::same_model)
        .def("current", &FieldStack::current)
        .def("fresh", &FieldStack::fresh)
        .def("layout", torch::wrap_pybind_function_no_gil([](FieldStack& s, int64_t prefill_rows, int64_t step_rows) {
                           s.layout(prefill_rows, step_rows);
                       }))
        .def("prefill", torch::wrap_pybind_function_no_gil([](FieldStack& s, const Tensor& x) { return s.prefill(x); }))
        .def("step", torch::wrap_pybind_function_no_gil(
                         [](FieldStack& s, const Tensor& x, const std::vector<Tensor>& st) { return s.step(x, st); }));
}

}  // namespace fields_torch
