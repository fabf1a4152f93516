// Row-wise glue of a Field block's inference path: everything between its matrix products.
//
// A block of the reference (field_only_v4_chunked_triton_wiki100.py:1198-1221) is, per token,
//   y = x + out_proj(read_norm(read)) * sigmoid(gate_proj(x));   x' = y + w3(silu(u) * v),
//   (u, v) = w12(ff_norm(y)).
// Run as library calls that is about 35 elementwise and reduction kernels per block, each of them a
// pass over [tokens, dim] (12 ms of a 13.3 ms prefill of 8 x 1,024 tokens through 18 blocks, 2.0 of
// 2.5 ms of the kernels of a 256-row decode step). Here it is four kernels, each of which reads its
// inputs once and leaves what the next matrix product wants, in bfloat16:
//   layout_block   bfloat16 copies of a block's weights and its transition parameters
//   step_norm      the decode recurrence of a row and its RMS norm      -> operand of out_proj
//   close_mixer    residual and gate, then ff_norm                      -> operand of w12
//   swiglu         silu(u) * v                                          -> operand of w3
//   close_ff       residual, then a cast or the next norm               -> operand of what follows
// The read_norm weight is folded into the out_proj copy (W diag(w)), so the norm is a per-token
// scale: step_norm applies it to the row, close_mixer applies it to the product when the row's sum of
// squares comes from the recurrence kernel (`groups`).
//
// All of it is bound by HBM for thousands of rows (close_mixer 14 B, swiglu 6 B per hidden unit,
// close_ff 12 B per element) and by latency for a few hundred: a row is owned by one warp when there
// are rows enough to fill the GPU that way, by four warps otherwise. Arithmetic is fp32 throughout.
// Device only.
#pragma once

#include "field_math.cuh"

#ifndef FIELDS_HOST_EMU

namespace fields {

constexpr int kRowThreads = 256;

// clamp as torch has it: a NaN stays one.
__device__ __forceinline__ float clamp_nan(float x, float lo, float hi) { return x < lo ? lo : x > hi ? hi : x; }

__device__ __forceinline__ Vec<4> load4(const float* p) { return vec_load<4>(p); }
__device__ __forceinline__ Vec<4> load4(const uint16_t* p) { return io_load4(p); }

// Ordinary (not streaming) store of four bfloat16: the next kernel reads them from L2.
__device__ __forceinline__ void store_bf16x4(uint16_t* p, const Vec<4>& x) {
    uint32_t lo, hi;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(x.v[1]), "f"(x.v[0]));
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(x.v[3]), "f"(x.v[2]));
    *reinterpret_cast<uint2*>(p) = make_uint2(lo, hi);
}

// Sum over the W warps that own a row (W = 1: one warp; otherwise all warps of the block in groups of W).
template <int W>
__device__ __forceinline__ float row_sum(float v, float* scratch) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if constexpr (W > 1) {
        const int warp = threadIdx.x >> 5;
        if ((threadIdx.x & 31) == 0) scratch[warp] = v;
        __syncthreads();
        v = 0.0f;
#pragma unroll
        for (int w = 0; w < W; ++w) v += scratch[warp / W * W + w];
    }
    return v;
}

struct CloseMixerParams {
    const float* x;          // [N, D]
    const uint16_t* acc;     // [N, D] bf16: output projection of the (scaled or unscaled) read rows
    const uint16_t* gate;    // rows of gate_stride, bf16
    const float* groups;     // [N, G] sums of squares of the read row, or null: acc is already scaled
    const float* bias;       // [D] of the output projection
    const float* gate_bias;  // [D] or null
    const float* norm_w;     // [D] of ff_norm
    float* y;                // [N, D] (may be x)
    uint16_t* h;             // [N, D] bf16, or null (with norm_w): y only
    long long N, gate_stride;
    int D, G;
    float eps, inv_features, norm_eps;
};

// W warps per row, V groups of four columns per lane: D <= 128 * W * V.
template <int W, int V>
__global__ void __launch_bounds__(kRowThreads) close_mixer(const CloseMixerParams p) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ float scratch[kRowThreads / 32];
    constexpr int kRows = kRowThreads / 32 / W;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long n = (long long)blockIdx.x * kRows + warp / W;
    const bool row_ok = n < p.N;
    const int col = ((warp % W) * 32 + lane) * 4;
    float rstd = 1.0f;
    if (row_ok && p.groups) {
        float s = 0.0f;
        for (int g = 0; g < p.G; ++g) s += p.groups[n * p.G + g];
        rstd = rsqrtf(s * p.inv_features + p.eps);
    }
    Vec<4> y[V];
    float sq = 0.0f;
#pragma unroll
    for (int j = 0; j < V; ++j) {
        const int c = col + j * 128 * W;
        if (row_ok && c < p.D) {
            const Vec<4> xv = load4(p.x + n * p.D + c);
            const Vec<4> a = load4(p.acc + n * p.D + c);
            const Vec<4> g = load4(p.gate + n * p.gate_stride + c);
            const Vec<4> b = load4(p.bias + c);
            const Vec<4> gb = p.gate_bias ? load4(p.gate_bias + c) : vec_fill<4>(0.0f);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                y[j].v[k] = xv.v[k] + (a.v[k] * rstd + b.v[k]) * sigmoidf_fast(g.v[k] + gb.v[k]);
                sq += y[j].v[k] * y[j].v[k];
            }
            vec_store<4>(p.y + n * p.D + c, y[j]);
        }
    }
    if (!p.h) return;
    const float inv = rsqrtf(row_sum<W>(sq, scratch) / (float)p.D + p.norm_eps);
#pragma unroll
    for (int j = 0; j < V; ++j) {
        const int c = col + j * 128 * W;
        if (row_ok && c < p.D) {
            const Vec<4> w = load4(p.norm_w + c);
#pragma unroll
            for (int k = 0; k < 4; ++k) y[j].v[k] = y[j].v[k] * inv * w.v[k];
            store_bf16x4(p.h + n * p.D + c, y[j]);
        }
    }
}

struct CloseFfParams {
    const float* x;        // [N, D]
    const uint16_t* f;     // [N, D] bf16: output of the feed-forward, or null
    const float* norm_w;   // [D] of the norm that follows, or null: plain cast
    float* y;              // [N, D] x + f (may be x), or null
    uint16_t* h;           // [N, D] bf16, or null
    long long N;
    int D;
    float norm_eps;
};

template <int W, int V>
__global__ void __launch_bounds__(kRowThreads) close_ff(const CloseFfParams p) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ float scratch[kRowThreads / 32];
    constexpr int kRows = kRowThreads / 32 / W;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long n = (long long)blockIdx.x * kRows + warp / W;
    const bool row_ok = n < p.N;
    const int col = ((warp % W) * 32 + lane) * 4;
    Vec<4> y[V];
    float sq = 0.0f;
#pragma unroll
    for (int j = 0; j < V; ++j) {
        const int c = col + j * 128 * W;
        if (row_ok && c < p.D) {
            y[j] = load4(p.x + n * p.D + c);
            if (p.f) {
                const Vec<4> f = load4(p.f + n * p.D + c);
#pragma unroll
                for (int k = 0; k < 4; ++k) y[j].v[k] += f.v[k];
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) sq += y[j].v[k] * y[j].v[k];
            if (p.y) vec_store<4>(p.y + n * p.D + c, y[j]);
        }
    }
    if (!p.h) return;
    float inv = 1.0f;
    if (p.norm_w) inv = rsqrtf(row_sum<W>(sq, scratch) / (float)p.D + p.norm_eps);  // (uniform branch)
#pragma unroll
    for (int j = 0; j < V; ++j) {
        const int c = col + j * 128 * W;
        if (row_ok && c < p.D) {
            if (p.norm_w) {
                const Vec<4> w = load4(p.norm_w + c);
#pragma unroll
                for (int k = 0; k < 4; ++k) y[j].v[k] = y[j].v[k] * inv * w.v[k];
            }
            store_bf16x4(p.h + n * p.D + c, y[j]);
        }
    }
}

// close_ff without a norm: nothing couples the elements of a row, so threads take four float4 each,
// a block's width apart (29.7 -> 17.3 us against the row form at 16,384 x 1,024).
struct AddCastParams {
    const float* x;
    const uint16_t* f;  // or null
    float* y;           // or null (may be x)
    uint16_t* h;        // or null
    long long n;        // elements, a multiple of 4
};

__global__ void __launch_bounds__(kRowThreads) add_cast(const AddCastParams p) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const long long i0 = ((long long)blockIdx.x * 4 * kRowThreads + threadIdx.x) * 4;
    constexpr int kStep = kRowThreads * 4;
    Vec<4> v[4];
    Bits4 f[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (i0 + j * kStep < p.n) {
            v[j] = load4(p.x + i0 + j * kStep);
            if (p.f) f[j] = load_bits4(p.f + i0 + j * kStep);
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const long long i = i0 + j * kStep;
        if (i < p.n) {
            if (p.f) {
                const F2 a = add2(lo2(v[j]), f[j].pair(0)), b = add2(hi2(v[j]), f[j].pair(1));
                v[j] = join2(a, b);
            }
            if (p.y) vec_store<4>(p.y + i, v[j]);
            if (p.h) store_bf16x4(p.h + i, v[j]);
        }
    }
}

struct SwigluParams {
    const uint16_t* uv;  // [N, 2H] bf16: u | v
    uint16_t* out;       // [N, H] bf16
    long long N;
    int H;
};

// One 16-byte access of each half and one of the result per thread and item; H % 8 == 0.
__global__ void __launch_bounds__(kRowThreads) swiglu(const SwigluParams p) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int per_row = p.H / 8;
    const long long items = p.N * per_row;
    const long long i = (long long)blockIdx.x * kRowThreads + threadIdx.x;
    if (i >= items) return;
    const long long n = i / per_row;
    const int c = (int)(i - n * per_row) * 8;
    const uint4 u = *reinterpret_cast<const uint4*>(p.uv + n * 2 * p.H + c);
    const uint4 v = *reinterpret_cast<const uint4*>(p.uv + n * 2 * p.H + p.H + c);
    const Vec<4> u0 = bf16x4_unpack(u.x, u.y), u1 = bf16x4_unpack(u.z, u.w);
    const Vec<4> v0 = bf16x4_unpack(v.x, v.y), v1 = bf16x4_unpack(v.z, v.w);
    Vec<4> a, b;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        a.v[k] = u0.v[k] * sigmoidf_fast(u0.v[k]) * v0.v[k];
        b.v[k] = u1.v[k] * sigmoidf_fast(u1.v[k]) * v1.v[k];
    }
    uint32_t o[4];
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(o[0]) : "f"(a.v[1]), "f"(a.v[0]));
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(o[1]) : "f"(a.v[3]), "f"(a.v[2]));
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(o[2]) : "f"(b.v[1]), "f"(b.v[0]));
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(o[3]) : "f"(b.v[3]), "f"(b.v[2]));
    *reinterpret_cast<uint4*>(p.out + n * p.H + c) = make_uint4(o[0], o[1], o[2], o[3]);
}

struct StepNormParams {
    const uint16_t* raw;  // rows of raw_stride, bf16: z_r | z_i | z_v
    const float* par;     // [3, C] Re lambda | Im lambda | gamma
    float* state;         // [N, 2C] in and out
    uint16_t* out;        // [N, 4C] bf16: read / rms(read)
    long long N, raw_stride;
    int C;
    float eps;
};

// One recurrence step of a row (the arithmetic of DecodeStep) and its RMS norm; 128 threads per row,
// four channels per thread and group: C <= 512 * V, C % 4 == 0.
template <int V>
__global__ void __launch_bounds__(128) step_norm(const StepNormParams p) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ float scratch[4];
    const long long n = blockIdx.x;
    const int C = p.C;
    Vec<4> sr[V], si[V], dr[V], di[V];
    float sq = 0.0f;
#pragma unroll
    for (int j = 0; j < V; ++j) {
        const int c = (int)threadIdx.x * 4 + j * 512;
        if (c < C) {
            const uint16_t* raw = p.raw + n * p.raw_stride + c;
            const Vec<4> zr = load4(raw), zi = load4(raw + C), zv = load4(raw + 2 * C);
            const Vec<4> lr = load4(p.par + c), li = load4(p.par + C + c), gm = load4(p.par + 2 * C + c);
            float* st = p.state + n * 2 * C + c;
            sr[j] = load4(st);
            si[j] = load4(st + C);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const Gate g = make_gate(zr.v[k], zi.v[k], zv.v[k]);
                float mr, mi;
                cmul(lr.v[k], li.v[k], sr[j].v[k], si[j].v[k], mr, mi);
                const float bs = gm.v[k] * g.vac;
                sr[j].v[k] = (1.0f - g.vac) * mr + bs * g.inj_r;
                si[j].v[k] = (1.0f - g.vac) * mi + bs * g.inj_i;
                dr[j].v[k] = g.vac * mr;
                di[j].v[k] = g.vac * mi;
                sq += sr[j].v[k] * sr[j].v[k] + si[j].v[k] * si[j].v[k] + dr[j].v[k] * dr[j].v[k] +
                      di[j].v[k] * di[j].v[k];
            }
            vec_store<4>(st, sr[j]);
            vec_store<4>(st + C, si[j]);
        }
    }
    const float inv = rsqrtf(row_sum<4>(sq, scratch) / (float)(4 * C) + p.eps);
#pragma unroll
    for (int j = 0; j < V; ++j) {
        const int c = (int)threadIdx.x * 4 + j * 512;
        if (c < C) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                sr[j].v[k] *= inv; si[j].v[k] *= inv; dr[j].v[k] *= inv; di[j].v[k] *= inv;
            }
            uint16_t* o = p.out + n * 4 * C + c;
            store_bf16x4(o, sr[j]);
            store_bf16x4(o + C, si[j]);
            store_bf16x4(o + 2 * C, dr[j]);
            store_bf16x4(o + 3 * C, di[j]);
        }
    }
}

// One contiguous piece of a block's weights on its way to bfloat16: n elements (a multiple of 4),
// column j of a row of `cols` scaled by scale[j] if given; zeros where src is null. radius / theta pieces: see layout_block.
struct LayoutPiece {
    const float* src;
    uint16_t* dst;
    const float* scale;
    long long n;
    int cols;
    int hidden;  // w12 in the order of the fused step and product: rows 16 j ... are u of eight features, then v of the same
};
constexpr int kLayoutPieces = 8;
constexpr int kLayoutChunk = kRowThreads * 4 * 4;  // elements per block: four loads of four per thread

struct LayoutParams {
    LayoutPiece piece[kLayoutPieces];
    long long first[kLayoutPieces + 1];  // first block of each piece, and of the transition parameters
    const float* radius_logit;  // [C]
    const float* theta;         // [C]
    float* par;                 // [3, C]
    int C;
};

// A block takes one chunk of one piece, with four loads in flight per thread (a fixed number of blocks per
// piece, one load each, ran at 2.2 TB/s: 25 us for a block of d_model 1,024); the blocks after the
// last piece compute the transition parameters (reference :1169-1173):
// lambda = r e^{i theta}, r = clamp(sigmoid(logit), 0.5, 0.99995), gamma = sqrt(max(1 - r^2, 1e-4)).
// Up to kLayoutBlocks blocks of a stack in one launch (blockIdx.y): 18 launches of 13.6 us became three.
constexpr int kLayoutBlocks = 8;
struct LayoutBatch {
    LayoutParams block[kLayoutBlocks];
};
static_assert(sizeof(LayoutBatch) <= 4000, "kernel parameters");

__global__ void __launch_bounds__(kRowThreads) layout_block(const __grid_constant__ LayoutBatch batch) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const LayoutParams& p = batch.block[blockIdx.y];
    const long long block = blockIdx.x;
    if (block >= p.first[kLayoutPieces]) {
        const int c = (int)(block - p.first[kLayoutPieces]) * kRowThreads + (int)threadIdx.x;
        if (c >= p.C) return;
        const float r = clamp_nan(1.0f / (1.0f + expf(-p.radius_logit[c])), 0.50f, 0.99995f);
        const float t = p.theta[c];
        p.par[c] = r * cosf(t);
        p.par[p.C + c] = r * sinf(t);
        p.par[2 * p.C + c] = sqrtf(clamp_nan(1.0f - r * r, 1e-4f, 1.0f));
        return;
    }
    int k = 0;
    while (block >= p.first[k + 1]) ++k;
    const LayoutPiece q = p.piece[k];
    const long long i0 = (block - p.first[k]) * kLayoutChunk + (long long)threadIdx.x * 4;
    Vec<4> v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        long long i = i0 + j * kRowThreads * 4;
        const bool inside = i < q.n && q.src;
        if (q.hidden) {
            const int r = (int)(i / q.cols), h = r / 16 * 8 + r % 8;
            i += (long long)((r % 16 < 8 ? h : q.hidden + h) - r) * q.cols;
        }
        v[j] = inside ? vec_load_stream<4>(q.src + i) : vec_fill<4>(0.0f);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const long long i = i0 + j * kRowThreads * 4;
        if (i >= q.n) continue;
        if (q.scale) {
            const Vec<4> s = load4(q.scale + i % q.cols);
#pragma unroll
            for (int e = 0; e < 4; ++e) v[j].v[e] *= s.v[e];
        }
        store_bf16x4(q.dst + i, v[j]);
    }
}

// out [cols, rows] = in [rows, cols] transposed, bfloat16: 64 x 64 through shared memory, two matrices in a launch.
struct TransposePart {
    const uint16_t* in;
    uint16_t* out;
    int rows, cols, tiles_c, tiles;
};
struct TransposeParams {
    TransposePart part[2];
};
__global__ void __launch_bounds__(kRowThreads) transpose_bf16(const TransposeParams p) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ uint16_t tile[64][66];
    const int second = (int)blockIdx.x >= p.part[0].tiles;
    const TransposePart& q = p.part[second];
    const int t = (int)blockIdx.x - (second ? p.part[0].tiles : 0);
    const int r0 = t / q.tiles_c * 64, c0 = t % q.tiles_c * 64, x = threadIdx.x % 32 * 2;
    for (int y = threadIdx.x / 32; y < 64; y += kRowThreads / 32) {
        if (r0 + y >= q.rows || c0 + x >= q.cols) continue;  // (an even number of columns)
        const uint32_t w = *reinterpret_cast<const uint32_t*>(q.in + (size_t)(r0 + y) * q.cols + c0 + x);
        tile[y][x] = (uint16_t)w;
        tile[y][x + 1] = (uint16_t)(w >> 16);
    }
    __syncthreads();
    for (int y = threadIdx.x / 32; y < 64; y += kRowThreads / 32) {
        if (c0 + y >= q.cols || r0 + x >= q.rows) continue;  // (and of rows)
        *reinterpret_cast<uint32_t*>(q.out + (size_t)(c0 + y) * q.rows + r0 + x) =
            (uint32_t)tile[x][y] | (uint32_t)tile[x + 1][y] << 16;
    }
}

}  // namespace fields

#endif  // FIELDS_HOST_EMU
