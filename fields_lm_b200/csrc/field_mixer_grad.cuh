// Row-wise glue of the fused Field mixer's backward pass: what lies around its matrix products.
//
// With u = [raw | gate] = xb @ in_w^T + in_b, read and its sums of squares from the recurrence and
// acc = read @ out_w^T, the mixer is y = x + (acc rstd + b) sigmoid(gate + b_g) (close_mixer in
// field_rows.cuh). As library calls its backward made about 45 launches besides the products: casts
// of every weight gradient, the gradient sums of five parameters, elementwise passes. Here:
//   open_grad        one pass over grad_y, acc and gate: gradients of acc and gate, of the sum of
//                    squares, partial rows of the gradients of the two biases
//   column_sums      gradient of the write projection's bias, as partial rows
//   out_weight_grad  from the gradient of out_proj diag(norm) to those of its two factors
//   finish_grad      adds every set of partial rows; gradients of radius and angle
// All are bound by HBM; rows are taken several at a time so that enough loads are in flight (the
// one-row form of open_grad ran at 3.5 TB/s: 55 us at 16,384 x 1,024; now 5.3). Sums run in a fixed order.
// Device only.
#pragma once

#include "field_rows.cuh"

#ifndef FIELDS_HOST_EMU

namespace fields {

constexpr int kGradRowsMax = 64;    // rows of one block of open_grad
constexpr int kGradBlocks = 3 * 148;  // blocks to aim at: one round at three per SM

struct OpenGradParams {
    const float* grad_y;    // [N, D]
    const uint16_t* acc;    // [N, D] bf16
    const uint16_t* gate;   // rows of gate_stride, bf16
    const float* groups;    // [N, G]
    const float* bias;      // [D]
    const float* gate_bias; // [D]
    uint16_t* grad_acc;     // [N, D] bf16
    uint16_t* grad_gate;    // rows of grad_gate_stride, bf16
    float* grad_sumsq;      // [N]
    float* rows;            // [2][blocks][D]: sums of grad_y sigmoid, of grad_gate
    long long N, gate_stride, grad_gate_stride;
    int D, G, per_block;
    float eps, inv_features;
};

// OWN groups of four columns per thread; R rows are loaded together, under the rows before them (without that, four rows at a time and
// three blocks per SM: 48.5 us at 16,384 rows of 1,024, 38.8 now; one row at a time, four groups and three blocks per SM: 87.3 us
// of 2,048 columns and 128 of 3,072). Up to 2,048 columns two groups and three blocks per SM, 69.4 us: with four groups, whose
// registers hold two rows for two blocks, 95.5 (4,096 rows 20.4 and 30.0; two groups, two rows and two blocks 88.3). Above that four and two
// blocks, 121 us of 3,072 and 147 of 4,096 (168 before).
template <int OWN, int R>
__global__ void __launch_bounds__(kRowThreads, OWN > 2 ? 2 : 3) open_grad(const OpenGradParams p) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ float dots[kGradRowsMax][kRowThreads / 32];
    __shared__ float rstds[kGradRowsMax];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const long long row0 = (long long)blockIdx.x * p.per_block;
    const int rows = (int)(p.N - row0 < p.per_block ? p.N - row0 : p.per_block);
    struct Rows {
        Vec<4> gy[OWN][R];
        Bits4 a[OWN][R], g[OWN][R];
    };
    auto load = [&](int r, Rows& to) {
#pragma unroll
        for (int j = 0; j < OWN; ++j) {
            const int c = (int)threadIdx.x * 4 + j * kRowThreads * 4;
#pragma unroll
            for (int q = 0; q < R; ++q) {
                if (r + q < rows && c < p.D) {
                    const long long n = row0 + r + q;
                    to.gy[j][q] = vec_load_stream<4>(p.grad_y + n * p.D + c);
                    to.a[j][q] = load_bits4(p.acc + n * p.D + c);
                    to.g[j][q] = load_bits4(p.gate + n * p.gate_stride + c);
                }
            }
        }
    };
    Rows now;
    load(0, now);
    if ((int)threadIdx.x < rows) {
        float s = 0.0f;
        for (int k = 0; k < p.G; ++k) s += p.groups[(row0 + threadIdx.x) * p.G + k];
        rstds[threadIdx.x] = rsqrtf(s * p.inv_features + p.eps);
    }
    __syncthreads();
    Vec<4> sum_b[OWN], sum_g[OWN];
#pragma unroll
    for (int j = 0; j < OWN; ++j) sum_b[j] = sum_g[j] = vec_fill<4>(0.0f);
    for (int r = 0; r < rows; r += R) {
        Rows next;
        load(r + R, next);
        float dot[R];
#pragma unroll
        for (int q = 0; q < R; ++q) dot[q] = 0.0f;
#pragma unroll
        for (int j = 0; j < OWN; ++j) {
            const int c = (int)threadIdx.x * 4 + j * kRowThreads * 4;
            if (c >= p.D) continue;
            const Vec<4> b = load4(p.bias + c), gb = load4(p.gate_bias + c);
#pragma unroll
            for (int q = 0; q < R; ++q) {
                if (r + q < rows) {
                    const long long n = row0 + r + q;
                    const Vec<4> gy = now.gy[j][q], a = bf16x4_unpack(now.a[j][q].lo, now.a[j][q].hi),
                                 g = bf16x4_unpack(now.g[j][q].lo, now.g[j][q].hi);
                    const float rstd = rstds[r + q];
                    Vec<4> ga, gg;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const float s = sigmoidf_fast(g.v[k] + gb.v[k]);
                        const float go = gy.v[k] * s;
                        ga.v[k] = go * rstd;
                        gg.v[k] = gy.v[k] * (a.v[k] * rstd + b.v[k]) * (s - s * s);
                        dot[q] += go * a.v[k];
                        sum_b[j].v[k] += go;
                        sum_g[j].v[k] += gg.v[k];
                    }
                    store_bf16x4(p.grad_acc + n * p.D + c, ga);
                    store_bf16x4(p.grad_gate + n * p.grad_gate_stride + c, gg);
                }
            }
        }
        now = next;
#pragma unroll
        for (int q = 0; q < R; ++q) {
            float v = dot[q];
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
            if (lane == 0 && r + q < rows) dots[r + q][warp] = v;
        }
    }
    __syncthreads();
    if ((int)threadIdx.x < rows) {
        const long long n = row0 + threadIdx.x;
        float total = 0.0f;
        const float rstd = rstds[threadIdx.x];
        for (int w = 0; w < warps; ++w) total += dots[threadIdx.x][w];
        p.grad_sumsq[n] = -0.5f * rstd * rstd * rstd * p.inv_features * total;
    }
#pragma unroll
    for (int j = 0; j < OWN; ++j) {
        const int c = (int)threadIdx.x * 4 + j * kRowThreads * 4;
        if (c < p.D) {
            vec_store<4>(p.rows + (size_t)blockIdx.x * p.D + c, sum_b[j]);
            vec_store<4>(p.rows + ((size_t)gridDim.x + blockIdx.x) * p.D + c, sum_g[j]);
        }
    }
}

struct ColumnSumParams {
    const uint16_t* x;  // rows of stride, bf16
    float* rows;        // [gridDim.y][cols]
    long long N, stride;
    int cols, per_block;
};

// blockIdx.x: 1,024 columns, four per thread; blockIdx.y: per_block rows, sixteen in flight (eight: 15.4 us at 16,384 rows of
// 1,536 columns, 14.2 now).
__global__ void __launch_bounds__(kRowThreads) column_sums(const ColumnSumParams p) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int c = ((int)blockIdx.x * kRowThreads + (int)threadIdx.x) * 4;
    if (c >= p.cols) return;
    const long long row0 = (long long)blockIdx.y * p.per_block;
    const int rows = (int)(p.N - row0 < p.per_block ? p.N - row0 : p.per_block);
    Vec<4> sum = vec_fill<4>(0.0f);
    const uint16_t* x = p.x + row0 * p.stride + c;
    constexpr int kFlight = 16;
    for (int r = 0; r < rows; r += kFlight) {
        Bits4 w[kFlight];
#pragma unroll
        for (int q = 0; q < kFlight; ++q)
            if (r + q < rows) w[q] = load_bits4(x + (r + q) * p.stride);
#pragma unroll
        for (int q = 0; q < kFlight; ++q) {
            if (r + q < rows) {
                const Vec<4> v = bf16x4_unpack(w[q].lo, w[q].hi);
#pragma unroll
                for (int k = 0; k < 4; ++k) sum.v[k] += v.v[k];
            }
        }
    }
    vec_store<4>(p.rows + (size_t)blockIdx.y * p.cols + c, sum);
}

struct OutWeightGradParams {
    float* grad;          // [D, cols] in: gradient of out_w diag(norm_w); out: that of out_w
    const float* out_w;   // [D, cols]
    const float* norm_w;  // [cols]
    float* rows;          // [gridDim.y][cols]: sums of grad * out_w
    int D, cols, per_block;
};

__global__ void __launch_bounds__(kRowThreads) out_weight_grad(const OutWeightGradParams p) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int c = ((int)blockIdx.x * kRowThreads + (int)threadIdx.x) * 4;
    if (c >= p.cols) return;
    const int row0 = (int)blockIdx.y * p.per_block;
    const int rows = p.D - row0 < p.per_block ? p.D - row0 : p.per_block;
    const Vec<4> w = load4(p.norm_w + c);
    Vec<4> sum = vec_fill<4>(0.0f);
    for (int r = 0; r < rows; r += 4) {
        Vec<4> g[4], o[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (r + q < rows) {
                const size_t at = (size_t)(row0 + r + q) * p.cols + c;
                g[q] = load4(p.grad + at);
                o[q] = load4(p.out_w + at);
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (r + q < rows) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    sum.v[k] += g[q].v[k] * o[q].v[k];
                    g[q].v[k] *= w.v[k];
                }
                vec_store<4>(p.grad + (size_t)(row0 + r + q) * p.cols + c, g[q]);
            }
        }
    }
    vec_store<4>(p.rows + (size_t)blockIdx.y * p.cols + c, sum);
}

struct PartialRows {
    const float* rows;  // [count][cols]
    float* out;         // [cols]
    int count, cols, first_block;
};
constexpr int kPartialSets = 4;

struct FinishGradParams {
    PartialRows set[kPartialSets];
    int transition_block;  // first of the blocks that compute the gradients of radius and angle
    const float* radius_logit;  // [C]
    const float* theta;
    const float* g_tr;
    const float* g_ti;
    const float* g_gm;
    float* g_radius;  // or null
    float* g_theta;   // or null
    int C;
};

// A block of 256 threads adds 32 columns: eight warps take every eighth row, then are added in order.
__global__ void __launch_bounds__(kRowThreads) finish_grad(const FinishGradParams p) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ float part[kRowThreads / 32][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if ((int)blockIdx.x >= p.transition_block) {
        // lambda = r e^{i theta}, r = clamp(sigmoid(logit), 0.5, 0.99995), gamma = sqrt(max(1 - r^2, 1e-4))
        const int c = ((int)blockIdx.x - p.transition_block) * kRowThreads + (int)threadIdx.x;
        if (c >= p.C) return;
        const float sig = 1.0f / (1.0f + expf(-p.radius_logit[c]));
        const float r = clamp_nan(sig, 0.50f, 0.99995f);
        const float co = cosf(p.theta[c]), si = sinf(p.theta[c]);
        const float q = 1.0f - r * r, gm = sqrtf(clamp_nan(q, 1e-4f, 1.0f));
        const float gtr = p.g_tr[c], gti = p.g_ti[c];
        float gr = gtr * co + gti * si;
        if (q >= 1e-4f) gr -= p.g_gm[c] * r / gm;
        if (p.g_theta) p.g_theta[c] = r * (gti * co - gtr * si);
        if (p.g_radius) p.g_radius[c] = (sig >= 0.50f && sig <= 0.99995f ? gr : 0.0f) * sig * (1.0f - sig);
        return;
    }
    int k = 0;
    while (k + 1 < kPartialSets && (int)blockIdx.x >= p.set[k + 1].first_block) ++k;
    const PartialRows s = p.set[k];
    const int c = ((int)blockIdx.x - s.first_block) * 32 + lane;
    float sum = 0.0f;
    if (c < s.cols) {
        // (16 loads in flight: with four this kernel took 17 us for 6 MB)
        for (int r = warp; r < s.count; r += 8 * 16) {
            float v[16];
#pragma unroll
            for (int q = 0; q < 16; ++q) v[q] = r + 8 * q < s.count ? s.rows[(size_t)(r + 8 * q) * s.cols + c] : 0.0f;
#pragma unroll
            for (int q = 0; q < 16; ++q) sum += v[q];
        }
    }
    part[warp][lane] = sum;
    __syncthreads();
    if (warp == 0 && c < s.cols) {
        float total = 0.0f;
#pragma unroll
        for (int w = 0; w < kRowThreads / 32; ++w) total += part[w][lane];
        s.out[c] = total;
    }
}

}  // namespace fields

#endif  // FIELDS_HOST_EMU
