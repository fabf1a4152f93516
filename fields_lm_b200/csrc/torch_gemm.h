// The library's matrix products of the torch layer, called directly: the same cuBLAS routine that at::mm
// calls for these types, without its checks, wrappers and tensor views (8 us of host time per product
// against 3; a block's prefill of a few hundred tokens was bound by them).
#pragma once

#include <ATen/cuda/CUDAContextLight.h>
#include <ATen/cuda/Exceptions.h>

#include "torch_api.h"

namespace fields_torch {

// Whether products with fused epilogues (field_product.cuh) take the place of the library's with row kernels between
// them: up to `narrow` always, where the host's launches bound the library's; up to `widest` from `least` rows on, as their
// tiles of 256 rows leave much of the GPU idle when there are few.
struct ProductRule {
    int64_t narrow, least, widest;
};
// Prefill, us against the library's. Eight blocks: d_model 256 438 to 355 against 524 and 512 374 to 461 against 527 (128 to
// 2,048 rows); 640 424 at 256 rows, 453 at 1,024 and 506 at 2,048 against 506, 510 and 545; 768 469, 497 and 561 against 512, 514
// and 607 (544 and 531 at 1,536); 1,024 562, 585 and 648 at 256, 512 and 1,024 rows against 514, 520 and 601, but 673 against 703 at
// 1,536 and 752 against 792 at 2,048. Two blocks: 1,536 304 against 318 at 1,536 rows, 2,048 511 and 1,512 against 534 and 1,646 at 2,048
// and 8,192. Wider: all column tiles follow one another for each 256 rows, and the weights of a product no
// longer stay in L2 meanwhile: 2,560 854 and 1,354 against 741 and 1,343 at 2,048 and 4,096 rows, 3,072 3,697 against 3,474 at 8,192,
// 4,096 6,460 against 6,003.
constexpr ProductRule kPrefillProducts{768, 1536, 2048};
// Mixer, forward and backward: 640 to 2,048 wide 202 to 297 against 244 to 337 from 512 to 2,048 rows, 2,048 869 against 936 at 8,192; 2,560
// 495 against 479 at 2,048 rows, but 726 against 753 at 4,096, 3,072 968 and 1,931 against 1,048 and 2,018 at 4,096 and 8,192, 4,096 1,750 and
// 3,378 against 1,813 and 3,398.
constexpr ProductRule kMixerProducts{2048, 4096, 4096};
inline bool fused_products(int64_t rows, int64_t dim, ProductRule rule) {
    return dim <= rule.narrow || (rows >= rule.least && dim <= rule.widest);
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
