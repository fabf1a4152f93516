// The library's matrix products of the torch layer, called directly: the same cuBLAS routine that at::mm
// calls for these types, without its checks, wrappers and tensor views (8 us of host time per product
// against 3; a block's prefill of a few hundred tokens was bound by them).
#pragma once

#include <ATen/cuda/CUDAContextLight.h>
#include <ATen/cuda/Exceptions.h>

#include "torch_api.h"

namespace fields_torch {

// Whether products with fused epilogues (field_product.cuh) take the place of the library's with row kernels between
// them: in narrow models, where the host's launches bound the library's, and in wider ones where there are rows enough, as their
// tiles of 256 rows leave much of the GPU idle when there are few. The lines lie where calls are as fast. (A captured graph, where
// the host's launches do not count, takes the same products, as its results are those of the call: there the library's would be
// faster below 2,048 rows, prefill of eight blocks of d_model 512 256, 293 and 379 us against 323, 359 and 402 at 64, 512 and 1,536
// rows, 768 355 and 396 against 424 and 449, mixers as below.)
struct ProductRule {
    int64_t narrow;            // up to this width always
    int64_t less_narrow, few;  // up to this one for so few rows
    int64_t widest, least;     // up to this one from so many rows on
};
// Prefill, us against the library's. Eight blocks: d_model 256 432, 335 and 357 against 543, 560 and 549 at 128, 512 and 2,048 rows; 576
// 401, 435 and 486 against 487, 498 and 507 at 256, 1,024 and 2,048; 640 428, 455 and 508 against 486, 499 and 543, 704 453, 480 and 544 against
// 492, 504 and 585 (at 1,408 rows, the least gain, 493 and 496, 523 and 525); 768 452, 472 and 494 against 531, 501 and 502 at 64, 512 and 768
// rows, but 496 against 495 at 896 and 534 against 512 at 1,028 (75 tiles where 74 pairs run), 553 against 545 at 1,536 and 577 against
// 635 at 2,048; 896 596 against 560 at 1,280, 612 against 633 at 1,536; 1,024 662 against 641 at 1,280, 679 against 704 at 1,536, 754
// against 797 at 2,044. Two blocks: 1,536 305 against 320 and 359 against 374 at 1,536 and 2,044 rows (340 and 338 at 1,792), 2,048 435
// against 418 at 1,280, 468 and 465 at 1,536, 486 and 507 at 1,792, 1,583 and 1,741 at 8,192. Wider: all column tiles follow one another for
// each 256 rows, and the weights of a product no longer stay in L2 meanwhile: 2,560 850 against 785 at 2,048 rows, 1,426 and 1,428
// at 4,096, 2,611 and 2,616 at 8,192 (2,473 and 2,555 in another run), 3,072 3,673 and 3,546.
constexpr ProductRule kPrefillProducts{704, 768, 768, 2048, 1536};
// Mixer, forward and backward. As calls 200 to 290 us against 240 to 380 for 256 to 2,048 wide ones of 64 to 1,024 rows (1,024 wide: 213 and
// 261, 215 and 302, 207 and 341 at 64, 128 and 256 rows; 2,048: 246 and 347, 242 and 344, 234 and 349). In a graph
// 1,024 wide 90 and 86, 93 and 88, 98 and 92, 103 and 100, 118 and 117 us at 64, 128, 256, 512 and 1,024 rows, 133 and 137 at 1,536; 2,048
// 160 and 155, 165 and 158, 171 and 168, 186 and 180, 220 and 228. Wider ones, calls: 2,560 496 and 492 at 2,048 rows, 759 and 807 at
// 4,096, 1,480 and 1,522 at 8,192; 3,072 632 and 629, 1,084 and 1,120, 2,080 and 2,108; 3,584 1,517 and 1,541 at 4,096, 5,456 and 5,464 at
// 16,384; 3,840 1,738 and 1,723, 6,230 and 6,045; 4,096 1,938 and 1,911, 3,668 and 3,501 at 8,192, 7,186 and 6,796.
constexpr ProductRule kMixerProducts{2048, 0, 0, 3072, 4096};
inline bool fused_products(int64_t rows, int64_t dim, ProductRule rule) {
    return dim <= rule.narrow || (dim <= rule.less_narrow && rows <= rule.few) || (dim <= rule.widest && rows >= rule.least);
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
