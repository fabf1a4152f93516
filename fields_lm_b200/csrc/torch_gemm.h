// The library's matrix products of the torch layer, called directly: the same cuBLAS routine that at::mm
// calls for these types, without its checks, wrappers and tensor views (8 us of host time per product
// against 3; a block's prefill of a few hundred tokens was bound by them).
#pragma once

#include <ATen/cuda/CUDAContextLight.h>
#include <ATen/cuda/Exceptions.h>

#include "torch_api.h"

namespace fields_torch {

// Whether products with fused epilogues (field_product.cuh) take the place of the library's with row kernels between
// them, us against the library's. Prefill of eight blocks, 128 to 8,192 rows: d_model 512 397 to 847 and 256 337 to 507
// against 490 to 938 and 491 to 548 (the host's launches bound the library's). Wider models from `least` rows on: their
// tiles of 256 rows leave much of the GPU idle when there are few; d_model 1,024, 1,024 rows 693 against 622, 2,048 793 against
// 812, 4,096 1,151 against 1,207, 8,192 1,993 against 2,179; 600 at 2,048 rows 608 and 734, 768 611 and 627, 1,536 1,341 and
// 1,364. Up to `widest`: all column tiles follow one another for each 256 rows, and beyond it the weights of a product no
// longer stay in L2 meanwhile. Two blocks, 2,048 and 8,192 rows: d_model 2,048 535 and 1,536 against 541 and 1,631, 2,560 874 and
// 2,649 against 747 and 2,552, 4,096 2,178 and 6,924 against 1,827 and 6,080.
struct ProductRule {
    int64_t least, widest;
};
constexpr ProductRule kPrefillProducts{2048, 2048};
// The mixer's backward pass has two weights to transpose (12 us at d_model 1,024) for 18 us at 4,096 rows, some 50 at 16,384:
// d_model 1,024 at 6,144 rows 285 against 295, 640 219 against 240, 2,048 750 against 763; at 6,144 and 8,192 rows 3,072 1,641 and
// 2,127 against 1,617 and 2,149, 4,096 2,927 and 3,728 against 2,785 and 3,580.
constexpr ProductRule kMixerProducts{6144, 3072};
inline bool fused_products(int64_t rows, int64_t dim, ProductRule rule) {
    return dim <= 512 || (rows >= rule.least && dim <= rule.widest);
}

// A bfloat16 matrix as a product takes it: `rows x cols` after the transposition, if any; rows as stored are
// `pitch` elements apart (0: dense).
struct Operand {
    const void* p;
    bool transposed;  // stored [cols, rows]
    int64_t pitch = 0;
};
inline Operand plain(const Tensor& t) { return Operand{vp(t), false}; }
inline Operand transposed(const Tensor& t) { return Operand{vp(t), true}; }

// torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False, as at::mm heeds it: partial sums
// of a product that is split along K are added in fp32.
class ReductionMode {
  public:
    explicit ReductionMode(cublasHandle_t handle) : handle_(handle) {
        if (at::globalContext().allowBF16ReductionCuBLAS() == at::CuBLASReductionOption::AllowReducedPrecisionWithSplitK)
            return;
        TORCH_CUDABLAS_CHECK(cublasGetMathMode(handle_, &before_));
        TORCH_CUDABLAS_CHECK(cublasSetMathMode(
            handle_, static_cast<cublasMath_t>(before_ | CUBLAS_MATH_DISALLOW_REDUCED_PRECISION_REDUCTION)));
        set_ = true;
    }
    ~ReductionMode() {
        if (set_) cublasSetMathMode(handle_, before_);
    }
    ReductionMode(const ReductionMode&) = delete;

  private:
    cublasHandle_t handle_;
    cublasMath_t before_ = CUBLAS_DEFAULT_MATH;
    bool set_ = false;
};

// out [M, N] = a [M, K] b [K, N], row-major, fp32 accumulation; out is bfloat16 or fp32. On the current stream.
inline void product(const Tensor& out, Operand a, Operand b, int64_t M, int64_t N, int64_t K) {
    const float one = 1.0f, zero = 0.0f;
    const cublasHandle_t handle = at::cuda::getCurrentCUDABlasHandle();
    const ReductionMode mode(handle);
    // cuBLAS is column-major: out^T = b^T a^T
    TORCH_CUDABLAS_CHECK(cublasGemmEx(
        handle, b.transposed ? CUBLAS_OP_T : CUBLAS_OP_N,
        a.transposed ? CUBLAS_OP_T : CUBLAS_OP_N, (int)N, (int)M, (int)K, &one, b.p, CUDA_R_16BF,
        (int)(b.pitch ? b.pitch : b.transposed ? K : N), a.p, CUDA_R_16BF,
        (int)(a.pitch ? a.pitch : a.transposed ? M : K), &zero, out.data_ptr(),
        out.scalar_type() == at::kFloat ? CUDA_R_32F : CUDA_R_16BF, (int)N, CUBLAS_COMPUTE_32F,
        CUBLAS_GEMM_DEFAULT_TENSOR_OP));
}

}  // namespace fields_torch
