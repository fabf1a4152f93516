// Matrix products of thousands of rows with everything that follows them elementwise as their epilogue:
//   out = a @ b^T, a [M, K] activations, b [N, K] weights, both bfloat16 with K contiguous, fp32 accumulation (or out = a @ b,
//   b [K, N]).
//
//   ProductBias      u = out + bias                                      in bfloat16
//   ProductGate      y = x + (out rstd + b) sigmoid(gate + b_g)          fp32, and what the caller asks for of: its
//                    bfloat16 copy, its sums of squares per row, out itself in bfloat16
//   ProductSwiglu    act = silu(u rstd) (v rstd), u and v interleaved columns of out, in bfloat16
//   ProductResidual  y = x + out                                         fp32, and its bfloat16 copy if asked for
//   ProductNormGrad  g = out + 2 c read, c per row                       in bfloat16
//
// As library products with row kernels between them a Field block wrote and read every product's result once
// more: of a prefill of 8 x 1,024 tokens through 18 blocks of d_model 1,024 (4.93 ms) 3.05 ms were products and
// 1.0 ms the row kernels. Then 4.45, and now 4.20. Alone, 8,192 rows, products of the library and, with what follows, these
// (us): bias, 2,560 columns of depth 1,024, 33 and 35; SwiGLU, 5,056 of 1,024, 66 (+ 19 for the row kernel) and 61; residual,
// 1,024 of 2,528, 33 (+ 14) and 43; gate, 1,024 of 2,048, 27 (+ 21) and 42; 16,384 rows: gate 51 (+ 37) and 74, gradient of the
// norm, 2,048 of 1,024, 59 (+ 36) and 56.
//
// What bounds them. Products of many tiles the tensor cores, at the clock that power leaves (1.4 to 1.5 GHz in a prefill).
// Those of two tiles a pair (1,024 columns, 8,192 rows) one tile's products, the other's, of which the epilogue of the first is
// in the shadow, and the epilogue of the second: in cycles for the gate 22,500, 23,000 and 13,500, for the residual 24,500, 26,000
// and 7,500. What the epilogue's own cycles go to, gate, per tile: arithmetic 7,000 (4,000 of them special functions), waiting
// for the inputs 8,000 (2,000 in the last tile), for the buffer to be read and the stores to be issued 5,500.
// With every access to global memory by the epilogue's lanes (rows of 64 or 128 bytes, through shared memory to turn
// them) the gate took 24,000 and 20,000 cycles, the residual 15,000 and 11,500, SwiGLU 8,700 of a tile's 8,200 of products
// (50, 45 and 65 us): the loads and stores were issued at the rate of the addresses that they touch, not waited for.
//
// A pair of thread blocks (cluster of two, cta_group::2) computes tiles of 256 x NT: each block holds 128 rows of a
// and NT / 2 rows of b, so that an operand byte fetched from L2 serves twice the products of a single block.
// Roles: one elected thread per block issues the TMA loads (a ring of k-blocks of 64, 128-byte swizzle), one of the
// pair the products (tcgen05.mma into tensor memory), eight warps are the epilogue. Tensor memory holds two
// tiles' accumulators: the epilogue of one runs under the products of the next. Persistent: a pair takes
// every pairs-th tile.
// Waits are bounded; after one that ran out the results are NaN. Device only.
#pragma once

#include "field_step_gemm.cuh"

#ifndef FIELDS_HOST_EMU

namespace fields {

constexpr int kProductWarps = 8;     // of the epilogue; loads and products: a warp each
constexpr int kProductRows = 128;     // of a block; a tile is twice as high
constexpr int kProductColumns = 128;  // of a tile that a warp of the epilogue does, at the most

struct ProductParams {
    long long M;
    int N, k_blocks;
    int tiles_n, pairs;
    long long tiles;
    // (what an epilogue does not use is null)
    const uint16_t* bias16;  // [N]
    const float *bias, *gate_bias;  // [N]
    const float* sums;       // [M, entries] sums of squares behind rstd = rsqrt(sum * inv_features + eps)
    int entries;
    float inv_features, eps;
    const float* row;        // [M] factor of a row
    float* sums_out;         // [M, ceil(N / 32)]: a warp's columns in the first of their entries, zero in the other
    // The bfloat16 tensors beside the matrix, for rows that TMA does not address (`direct_in`, `direct_out`), and h and acc where
    // both are wanted: in16 is gate or read, h the output.
    int direct_in, direct_out;
    const uint16_t* in16;
    long long in_pitch;
    uint16_t* h;
    long long h_pitch;
    uint16_t* acc;           // [M, N]
    int has_h, has_acc;      // whether h, and whether acc, is wanted at all
};
// Operands, and the tensors of the epilogue in boxes of 32 rows: x and y fp32, in16 gate or read, out16 h (or acc where no h is
// wanted).
struct alignas(64) ProductMaps {
    CUtensorMap a, b, x, y, in16, out16;
};

// A row's part of a 16-byte unit in a box of 32 rows as TMA writes it with the swizzle of that row length: eight neighbouring
// rows' units of one column lie in different banks, so a lane per row reads and writes them at full rate.
template <int ROW_BYTES>
__device__ __forceinline__ unsigned product_unit(int row, int u) {
    static_assert(ROW_BYTES == 128 || ROW_BYTES == 64, "swizzles");
    return (unsigned)(row * ROW_BYTES + ((u ^ (ROW_BYTES == 128 ? row & 7 : row >> 1 & 3)) << 4));
}
__device__ __forceinline__ uint4 lds16(unsigned addr) {
    uint4 r;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(addr) : "memory");
    return r;
}
__device__ __forceinline__ void sts16(unsigned addr, const uint4& v) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint2 lds8(unsigned addr) {
    uint2 r;
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(r.x), "=r"(r.y) : "r"(addr) : "memory");
    return r;
}
__device__ __forceinline__ void sts8(unsigned addr, const uint2& v) {
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(v.x), "r"(v.y) : "memory");
}
// Eight bfloat16 values of a row in global memory that may lie on 8 bytes only, the second four where they exist.
__device__ __forceinline__ void store_halves(uint16_t* p, const uint4& v, bool second) {
    *reinterpret_cast<uint2*>(p) = make_uint2(v.x, v.y);
    if (second) *reinterpret_cast<uint2*>(p + 4) = make_uint2(v.z, v.w);
}
__device__ __forceinline__ uint4 pack8(const float* v) {
    uint4 r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r.x) : "f"(v[1]), "f"(v[0]));
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r.y) : "f"(v[3]), "f"(v[2]));
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r.z) : "f"(v[5]), "f"(v[4]));
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r.w) : "f"(v[7]), "f"(v[6]));
    return r;
}
__device__ __forceinline__ void unpack8(const uint4& w, float* v) {
    const Vec<4> a = bf16x4_unpack(w.x, w.y), b = bf16x4_unpack(w.z, w.w);
#pragma unroll
    for (int k = 0; k < 4; ++k) { v[k] = a.v[k]; v[4 + k] = b.v[k]; }
}
__device__ __forceinline__ uint4 float_bits(const float* v) {
    return make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
}
__device__ __forceinline__ void bits_float(const uint4& w, float* v) {
    v[0] = __uint_as_float(w.x); v[1] = __uint_as_float(w.y); v[2] = __uint_as_float(w.z); v[3] = __uint_as_float(w.w);
}

// An epilogue. run() does eight columns of a row, `at` counted in the warp's: of the product in v, of fp32 input in x (then
// output), of bfloat16 input in `in`. Leaves fp32 output in x, bfloat16 output in v.
//   kF32     fp32 input and output      kIn   bfloat16 input      kChunk   columns between two exchanges with memory
//   keep     constants of four columns of a tile, by the lane of those columns, `to` its place in shared memory
struct ProductBias {
    static constexpr bool kDependents = false;
    static constexpr int kChunk = 64;
    static constexpr bool kF32 = false, kIn = false, kSums = false, kSwiglu = false, kAcc = false;
    __device__ static float factor(const ProductParams&, long long) { return 1.0f; }
    // A lane keeps four columns' biases, and all take them from there: a load of the same address by all lanes is as slow as
    // any (5,000 cycles of a tile's epilogue against 3,300).
    using Kept = uint2;
    static constexpr int kConstants = 0;
    __device__ static Kept keep(const ProductParams& p, int col, bool here, float*) {
        return here ? *reinterpret_cast<const uint2*>(p.bias16 + col) : make_uint2(0u, 0u);
    }
    __device__ static void run(const Kept& kept, const float*, int at, float* v, float*, const float*, float, F2&) {
        uint4 w;
        w.x = __shfl_sync(0xffffffffu, kept.x, at / 4);
        w.y = __shfl_sync(0xffffffffu, kept.y, at / 4);
        w.z = __shfl_sync(0xffffffffu, kept.x, at / 4 + 1);
        w.w = __shfl_sync(0xffffffffu, kept.y, at / 4 + 1);
        float b[8];
        unpack8(w, b);
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] += b[k];
    }
};
// rsqrt of the mean of a row's squares. (The loads of a row go out together: one by one, 32 entries took longer than the
// products of a tile of depth 1,024, 90 us instead of 56 for 8,192 x 5,056.)
__device__ __forceinline__ float product_rstd(const ProductParams& p, long long row) {
    const float* s = p.sums + row * p.entries;
    float sum = 0.0f;
    if (p.entries % 4 == 0 && reinterpret_cast<unsigned long long>(p.sums) % 16 == 0) {
        for (int i = 0; i < p.entries; i += 32) {
            float4 v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j)
                v[j] = i + 4 * j < p.entries ? *reinterpret_cast<const float4*>(s + i + 4 * j) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for (int j = 0; j < 8; ++j) sum += v[j].x + v[j].y + v[j].z + v[j].w;
        }
    } else {
        for (int i = 0; i < p.entries; ++i) sum += s[i];
    }
    return rsqrtf(sum * p.inv_features + p.eps);
}
struct ProductGate {
    static constexpr bool kDependents = true;
    static constexpr int kChunk = 32;
    static constexpr bool kF32 = true, kIn = true, kSums = true, kSwiglu = false, kAcc = true;
    __device__ static float factor(const ProductParams& p, long long row) { return product_rstd(p, row); }
    // Both biases of a warp's columns wait in shared memory (loaded by all lanes from the same address where they are needed,
    // arithmetic took 11,500 cycles of a tile instead of 7,700).
    struct Kept {};
    static constexpr int kConstants = 2;  // floats per column
    __device__ static Kept keep(const ProductParams& p, int col, bool here, float* to) {
        const Vec<4> b = here ? load4(p.bias + col) : vec_fill<4>(0.0f), gb = here ? load4(p.gate_bias + col) : vec_fill<4>(0.0f);
        vec_store<4>(to, b);
        vec_store<4>(to + kProductColumns, gb);
        return {};
    }
    __device__ static void run(const Kept&, const float* constants, int at, float* v, float* x, const float* in, float rstd, F2& sq) {
        const F2* b = reinterpret_cast<const F2*>(constants + at);
        const F2* gb = reinterpret_cast<const F2*>(constants + kProductColumns + at);
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
            const F2 g = sigmoid2(add2(F2{in[k], in[k + 1]}, gb[k / 2]));
            const F2 y = fma2(fma2(F2{v[k], v[k + 1]}, splat2(rstd), b[k / 2]), g, F2{x[k], x[k + 1]});
            sq = fma2(y, y, sq);
            x[k] = v[k] = y.x;
            x[k + 1] = v[k + 1] = y.y;
        }
    }
};
struct ProductSwiglu {
    static constexpr bool kDependents = true;
    static constexpr int kChunk = 64;
    static constexpr bool kF32 = false, kIn = false, kSums = false, kSwiglu = true, kAcc = false;
    struct Kept {};
    static constexpr int kConstants = 0;
    __device__ static Kept keep(const ProductParams&, int, bool, float*) { return {}; }
    __device__ static float factor(const ProductParams& p, long long row) { return product_rstd(p, row); }
    // (sixteen columns: u of eight features, then v of the same)
    __device__ static void run(float* v, float rstd) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float us = v[k] * rstd;
            v[k] = us * sigmoidf_fast(us) * (v[8 + k] * rstd);
        }
    }
};
struct ProductResidual {
    static constexpr bool kDependents = true;
    static constexpr int kChunk = 32;
    static constexpr bool kF32 = true, kIn = false, kSums = false, kSwiglu = false, kAcc = false;
    struct Kept {};
    static constexpr int kConstants = 0;
    __device__ static Kept keep(const ProductParams&, int, bool, float*) { return {}; }
    __device__ static float factor(const ProductParams&, long long) { return 1.0f; }
    __device__ static void run(const Kept&, const float*, int, float* v, float* x, const float*, float, F2&) {
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = x[k] += v[k];
    }
};
struct ProductNormGrad {
    static constexpr bool kDependents = false;
    static constexpr int kChunk = 64;
    static constexpr bool kF32 = false, kIn = true, kSums = false, kSwiglu = false, kAcc = false;
    struct Kept {};
    static constexpr int kConstants = 0;
    __device__ static Kept keep(const ProductParams&, int, bool, float*) { return {}; }
    __device__ static float factor(const ProductParams& p, long long row) { return 2.0f * p.row[row]; }
    __device__ static void run(const Kept&, const float*, int, float* v, float*, const float* in, float c, F2&) {
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] += c * in[k];
    }
};

template <class Epi, int NT>
struct ProductShape {
    static constexpr int kBox = 64;  // of K
    static constexpr int kABytes = kProductRows * kBox * 2, kBBytes = NT / 2 * kBox * 2, kStageBytes = kABytes + kBBytes;
    // A warp's share of a tile: 32 rows x kColumns, in chunks that pass through a buffer of its own: fp32 rows of 128 bytes and
    // behind them bfloat16 rows of kHalfRow bytes.
    static constexpr int kColumns = NT / (kProductWarps / 4), kChunk = Epi::kChunk, kChunks = kColumns / kChunk;
    static constexpr int kHalfColumns = Epi::kSwiglu ? kChunk / 2 : kChunk, kHalfRow = kHalfColumns * 2;
    static constexpr int kF32Bytes = Epi::kF32 ? 32 * 128 : 0, kBufferBytes = kF32Bytes + 32 * kHalfRow;
    // As many stages as there is space for beside the buffers. (The loop of products alone, 8,192 x 1,024: depth 2,048 28.4 us
    // with six stages, 29.1 with five, 32.4 with four; depth 2,528 35.2, 36.5 and 41.9. Five stages beside buffers for h as well or
    // six with h through the buffer of y, after it, are the same, 47 us.)
    static constexpr int kConstBytes = Epi::kConstants * kProductColumns * 4;  // of a warp
    static constexpr int kStages = (227 * 1024 - 1024 - 512 - kProductWarps * (kBufferBytes + kConstBytes)) / kStageBytes;
    static constexpr int kLoads = Epi::kF32 || Epi::kIn ? kProductWarps * kChunks : 0;  // barriers of the inputs
    static constexpr int kBars = 2 * kStages + 4 + kLoads;
    static constexpr size_t kSmemBytes = 1024 + (size_t)kStages * kStageBytes + kProductWarps * (kBufferBytes + kConstBytes) + kBars * 8 + 16;
    static constexpr unsigned kTmem = 2 * NT;  // columns of tensor memory
    static_assert(kSmemBytes <= 227 * 1024, "shared memory of an SM");
    static_assert(NT == 256 || NT == 128, "tiles the tensor cores and the epilogue's warps take");
    static_assert((kChunks - 1) * kProductWarps * kBufferBytes <= kStages * kStageBytes, "the last tile's inputs go where operands were");
};

// A load whose bytes count on a barrier of either block of the pair.
__device__ __forceinline__ void tma_load2_pair(unsigned dst, const CUtensorMap* map, int x, int y, unsigned cluster_bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            dst),
        "l"(map), "r"(x), "r"(y), "r"(cluster_bar)
        : "memory");
}
__device__ __forceinline__ void pair_mma(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc,
                                         unsigned accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrives on the barrier at this offset in both blocks once the products issued so far are done.
__device__ __forceinline__ void pair_commit(unsigned bar) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
        "h"((unsigned short)3)
        : "memory");
}
__device__ __forceinline__ void tmem_load32(unsigned addr, unsigned* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(addr)
        : "memory");
}

__device__ __forceinline__ void tma_store2(const CUtensorMap* map, unsigned src, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(x), "r"(y),
                 "r"(src)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// An epilogue warp: 32 rows x kColumns of every tile of its block. A lane has a row, as tensor memory gives it; what the row
// needs from global memory comes, and what it leaves goes, by TMA through the warp's buffer in shared memory, the outputs in the
// place of the inputs.
template <class Epi, int NT>
struct ProductWarp {
    using T = ProductShape<Epi, NT>;
    static constexpr int kChunks = T::kChunks;
    static constexpr bool kLoads = Epi::kF32 || Epi::kIn;
    const ProductParams& p;
    const ProductMaps& maps;
    unsigned own, ring, bars;  // the buffer; where the last tile's other chunks go; this warp's barriers, one per chunk
    float* constants;          // of the tile's columns
    int warp, lane;
    bool leader, dead = false;
    unsigned parity = 0;       // of the first barrier

    __device__ unsigned buffer(int c, bool last) const {
        return last && c > 0 ? ring + (unsigned)(((c - 1) * kProductWarps + warp) * T::kBufferBytes) : own;
    }
    // Inputs of the 32 rows from row0 on and the chunk's columns from col on.
    __device__ void load(unsigned buf, unsigned bar, long long row0, int col) const {
        if (!leader || dead) return;
        const bool in = Epi::kIn && !p.direct_in;
        const int bytes = T::kF32Bytes + (in ? 32 * T::kHalfRow : 0);
        if (bytes == 0) return;
        mbar_expect(bar, (unsigned)bytes);
        if constexpr (Epi::kF32) tma_load2(buf, &maps.x, col, (int)row0, bar);
        if (in) tma_load2(buf + T::kF32Bytes, &maps.in16, col, (int)row0, bar);
    }
    __device__ void buffer_read() const {  // what was sent from the buffer has left it
        if (leader) bulk_wait_read();
        __syncwarp();
    }
    // Bfloat16 rows that lie on 8 bytes only, from row0 and hcol on: lanes along the rows, between global memory and where TMA would
    // have them. (With a lane per row, which touches 32 rows at once, the bias product of 16,384 rows of 1,300 columns and depth 520
    // took 64.6 us, of 8,192 32.2, the gate of 520 columns 53.3 and 36.0; now 37.8, 21.6, 41.1 and 27.4.)
    static constexpr int kAcross = T::kHalfRow / 8;  // lanes of a row, and accesses of a lane
    struct Halves {
        uint2 w[kAcross];
    };
    template <class F>
    __device__ void along_rows(unsigned buf, int left, int hcol, int cols, F f) const {
        const int q = lane % kAcross;
#pragma unroll
        for (int i = 0; i < kAcross; ++i) {
            const int r = (i * 32 + lane) / kAcross;
            f(i, r, hcol + 4 * q, buf + T::kF32Bytes + product_unit<T::kHalfRow>(r, q / 2) + (unsigned)(q & 1) * 8,
              r < left && hcol + 4 * q < cols);
        }
    }
    __device__ void fetch_halves(Halves& to, long long row0, int left, int hcol) const {
        along_rows(0, left, hcol, p.N, [&](int i, int r, int c, unsigned, bool in) {
            to.w[i] = in ? *reinterpret_cast<const uint2*>(p.in16 + (row0 + r) * p.in_pitch + c) : make_uint2(0u, 0u);
        });
    }
    __device__ void put_halves(const Halves& from, unsigned buf) const {
        along_rows(buf, 0, 0, 0, [&](int i, int, int, unsigned at, bool) { sts8(at, from.w[i]); });
    }
    __device__ void send_halves(unsigned buf, uint16_t* to, long long pitch, long long row0, int left, int hcol, int cols) const {
        along_rows(buf, left, hcol, cols, [&](int, int r, int c, unsigned at, bool in) {
            if (in) *reinterpret_cast<uint2*>(to + (row0 + r) * pitch + c) = lds8(at);
        });
    }
    // 32 columns of the row, `k` of the chunk on, which begins at the warp's column `c0` and the matrix's column `col0`. (Loads,
    // arithmetic and stores one after the other: in turns for eight columns the loads' latency was waited for four times,
    // 7,700 cycles of a tile's gate against 6,700.)
    __device__ void part(const typename Epi::Kept& kept, int k, unsigned buf, float* v, int row, bool in_rows, int c0, int col0,
                         float factor, F2& sq) const {
        constexpr int kUnits = Epi::kSwiglu ? 2 : 4, kWide = Epi::kSwiglu ? 16 : 8;  // units of eight bfloat16 columns
        const int cols = Epi::kSwiglu ? p.N / 2 : p.N, hk = Epi::kSwiglu ? k / 2 : k, hcol = Epi::kSwiglu ? (col0 + k) / 2 : col0 + k;
        auto half_at = [&](int j) { return buf + T::kF32Bytes + product_unit<T::kHalfRow>(lane, hk / 8 + j); };
        auto inside = [&](int j) { return in_rows && hcol + 8 * j < cols; };
        auto second = [&](int j) { return hcol + 8 * j + 4 < cols; };
        float x[Epi::kF32 ? 32 : 1];
        uint4 in[Epi::kIn ? kUnits : 1], acc[Epi::kAcc ? kUnits : 1];
        if constexpr (Epi::kF32) {
#pragma unroll
            for (int j = 0; j < 8; ++j) bits_float(lds16(buf + product_unit<128>(lane, k / 4 + j)), x + 4 * j);
        }
        if constexpr (Epi::kIn) {
#pragma unroll
            for (int j = 0; j < kUnits; ++j) in[j] = lds16(half_at(j));
        }
#pragma unroll
        for (int j = 0; j < kUnits; ++j) {
            float* w = v + j * kWide;
            if constexpr (Epi::kSwiglu) {
                Epi::run(w, factor);
            } else {
                float u[8];
                if constexpr (Epi::kIn) unpack8(in[j], u);
                if constexpr (Epi::kAcc) acc[j] = pack8(w);
                Epi::run(kept, constants, c0 + k + 8 * j, w, x + (Epi::kF32 ? 8 * j : 0), u, factor, sq);
            }
        }
        if constexpr (Epi::kF32) {
#pragma unroll
            for (int j = 0; j < 8; ++j) sts16(buf + product_unit<128>(lane, k / 4 + j), float_bits(x + 4 * j));
        }
        if constexpr (Epi::kAcc) {
            if (p.has_acc) {
#pragma unroll
                for (int j = 0; j < kUnits; ++j) {
                    if (!p.has_h) sts16(half_at(j), acc[j]);
                    else if (inside(j)) store_halves(p.acc + (long long)row * p.N + hcol + 8 * j, acc[j], second(j));
                }
            }
        }
        if (p.has_h) {
#pragma unroll
            for (int j = 0; j < kUnits; ++j) sts16(half_at(j), pack8(v + j * kWide));
        }
    }
    // A tile: tmem is the warp's lanes and first column, acc_full is done where the product is, released where to say that
    // it has been read.
    __device__ void tile(long long row0, int col0, bool last, unsigned tmem, unsigned acc_full, unsigned acc_parity, unsigned released) {
        const int left = p.M - row0 < 32 ? (int)(p.M - row0) : 32, row = (int)row0 + lane;
        const bool in_rows = lane < left, any = left > 0 && col0 < p.N;
        if (kLoads) {
            buffer_read();
            if (any) load(own, bars, row0, col0);
        }
        Halves in16;
        constexpr bool kAhead = Epi::kIn && kAcross == 8;  // (sixteen accesses ahead do not fit the registers)
        if (kAhead && p.direct_in && any) fetch_halves(in16, row0, left, col0);
        const float factor = in_rows ? Epi::factor(p, row) : 1.0f;
        const typename Epi::Kept kept =
            Epi::keep(p, col0 + lane * 4, lane * 4 < T::kColumns && col0 + lane * 4 < p.N, constants + lane * 4);
        F2 sq = splat2(0.0f);
        mbar_wait_local(acc_full, acc_parity, dead);
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // (all operands of the last tile have been read: there is space for the inputs of its other chunks)
        last = last && !__any_sync(0xffffffffu, dead);
        if (kLoads && last)
#pragma unroll
            for (int c = 1; c < kChunks; ++c)
                if (any && col0 + c * T::kChunk < p.N) load(buffer(c, true), bars + c * 8, row0, col0 + c * T::kChunk);
#pragma unroll 1
        for (int c = 0; c < kChunks; ++c) {
            const int col = col0 + c * T::kChunk;
            const bool here = any && col < p.N;
            const unsigned buf = buffer(c, last);
            if (!kLoads) {
                if (here) buffer_read();
            } else if (c > 0 && !last && here) {
                buffer_read();
                load(own, bars, row0, col);
            }
            if (Epi::kIn && p.direct_in && here) {
                if (!kAhead) fetch_halves(in16, row0, left, col);
                put_halves(in16, buf);
                if (kAhead && c + 1 < kChunks) fetch_halves(in16, row0, left, col + T::kChunk);
            }
            if (here && kLoads && (Epi::kF32 || !p.direct_in)) {
                if (last && c > 0) {
                    mbar_wait_local(bars + c * 8, 0, dead);
                } else {
                    mbar_wait_local(bars, parity, dead);
                    parity ^= 1;
                }
            }
            __syncwarp();
#pragma unroll
            for (int k = 0; k < T::kChunk; k += 32) {
                unsigned v[32];
                tmem_load32(tmem + (unsigned)(c * T::kChunk + k), v);
                tmem_wait();
                if (c + 1 == kChunks && k + 32 == T::kChunk) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    // (at block scope: at cluster scope it waits for the warp's stores, 2,500 cycles, and orders nothing but
                    // tensor memory)
                    if (lane == 0) asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(released) : "memory");
                }
                float f[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) f[i] = dead ? nanf("") : __uint_as_float(v[i]);
                if (here) part(kept, k, buf, f, row, in_rows, c * T::kChunk, col, factor, sq);
                __syncwarp();
            }
            if (here) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (leader) {
                    if constexpr (Epi::kF32) tma_store2(&maps.y, buf, col, (int)row0);
                    if (!p.direct_out && (p.has_h || p.has_acc))
                        tma_store2(&maps.out16, buf + T::kF32Bytes, Epi::kSwiglu ? col / 2 : col, (int)row0);
                    bulk_commit();
                }
                const int hcol = Epi::kSwiglu ? col / 2 : col, cols = Epi::kSwiglu ? p.N / 2 : p.N;
                if (p.direct_out && p.has_h) send_halves(buf, p.h, p.h_pitch, row0, left, hcol, cols);
                else if (p.direct_out && p.has_acc) send_halves(buf, p.acc, p.N, row0, left, hcol, cols);
            }
        }
        if constexpr (Epi::kSums) {
            const int entries = (p.N + 31) / 32;
            if (p.sums_out && in_rows)
#pragma unroll
                for (int i = 0; i < T::kColumns / 32; ++i)
                    if (col0 / 32 + i < entries) p.sums_out[(long long)row * entries + col0 / 32 + i] = i ? 0.0f : sq.x + sq.y;
        }
    }
};

// Shared-memory descriptor of b as it lies in memory with K as its rows: 64 columns of N are 128 bytes of a row of K, with the
// 128-byte swizzle; groups of eight rows 1,024 bytes apart, the next 64 columns behind the k-block's rows.
__device__ __forceinline__ unsigned long long depth_desc(unsigned addr) {
    constexpr unsigned long long kNext64 = 64 * 128 >> 4;
    return (unsigned long long)((addr & 0x3FFFFu) >> 4) | (kNext64 << 16) | ((unsigned long long)(1024 >> 4) << 32) | (1ull << 46) |
           (2ull << 61);
}

// BY_DEPTH: b is [K, N], N contiguous, a weight as the forward pass has it. (The mixer's two had been transposed by a launch of
// their own, 11 us: 558 -> 549 us at 8 x 2,048 x 1,024. The products are as fast either way.)
template <class Epi, int NT, bool BY_DEPTH>
__global__ void __launch_bounds__(32 * (kProductWarps + 2), 1)
    pair_product(const __grid_constant__ ProductMaps maps, const __grid_constant__ ProductParams p) {
    using T = ProductShape<Epi, NT>;
    extern __shared__ __align__(1024) char product_smem[];
    char* ring = product_smem + (1024 - (smem_addr(product_smem) & 1023)) % 1024;
    char* buffers = ring + T::kStages * T::kStageBytes;
    char* constants = buffers + kProductWarps * T::kBufferBytes;
    char* tail = constants + kProductWarps * T::kConstBytes;
    // loads have landed (both blocks', on the first block's barriers); stage free, accumulator full (each block's own);
    // accumulator free (the first block's); inputs of the epilogue have landed
    const unsigned full = smem_addr(tail), empty = full + T::kStages * 8, acc_full = empty + T::kStages * 8,
                   acc_free = acc_full + 16, loaded = acc_free + 16;
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(tail + T::kBars * 8);
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), rank = (int)cluster_rank();

    if (threadIdx.x == 0) {
        for (int i = 0; i < 2 * T::kStages + 2; ++i) mbar_init(full + i * 8, 1);
        for (int i = 0; i < 2; ++i) mbar_init(acc_free + i * 8, 2 * kProductWarps);
        for (int i = 0; i < T::kLoads; ++i) mbar_init(loaded + i * 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kProductWarps) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(T::kTmem)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();  // the other block's barriers are ready
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = *tmem_slot;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // Every block runs from the start: those of the next kernel take the places of the first that end, and set themselves up
    // (prefill of 4 x 500 tokens through 8 blocks of d_model 512 494 -> 472 us, of 8 x 1,024 through 18 of 1,024 4,258 -> 4,219).
    // Where the next kernel is a product, that is where it reads h: the blocks of a recurrence or of a row kernel then lie on
    // few SMs (mixer of 8 x 2,048 567 -> 584 us with all products, 546 -> 551 with those two).
    if (Epi::kDependents && p.has_h) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    const long long first = blockIdx.x / 2;
    bool dead = false;
    if (warp < kProductWarps) {
        ProductWarp<Epi, NT> w{p, maps, smem_addr(buffers + warp * T::kBufferBytes), smem_addr(ring),
                               loaded + (unsigned)(T::kLoads ? warp * T::kChunks * 8 : 0),
                               reinterpret_cast<float*>(constants + warp * T::kConstBytes), warp, (int)threadIdx.x & 31, elect_one()};
        const unsigned lanes = tmem + ((unsigned)(warp % 4 * 32) << 16) + (unsigned)(warp / 4 * T::kColumns);
        unsigned n = 0;
        for (long long t = first; t < p.tiles; t += p.pairs, ++n) {
            const unsigned buf = n & 1;
            w.tile(t / p.tiles_n * (2 * kProductRows) + rank * kProductRows + warp % 4 * 32,
                   (int)(t % p.tiles_n) * NT + warp / 4 * T::kColumns, t + p.pairs >= p.tiles, lanes + buf * NT, acc_full + buf * 8,
                   n / 2 & 1, peer_addr(acc_free + buf * 8, 0));
        }
        if (w.leader) bulk_wait_all();
        dead = w.dead;
    } else if (warp == kProductWarps) {
        if (elect_one()) {
            StepRing<T::kStages> r;
            for (long long t = first; t < p.tiles; t += p.pairs) {
                const int m0 = (int)(t / p.tiles_n) * (2 * kProductRows) + rank * kProductRows,
                          n0 = (int)(t % p.tiles_n) * NT + rank * (NT / 2);
                for (int i = 0; i < p.k_blocks; ++i) {
                    if (!r.fresh()) mbar_wait_local(empty + r.slot * 8, r.parity ^ 1, dead);
                    if (dead) break;
                    if (rank == 0) mbar_expect(full + r.slot * 8, 2 * T::kStageBytes);
                    const unsigned bar = peer_addr(full + r.slot * 8, 0), at = smem_addr(ring + r.slot * T::kStageBytes);
                    tma_load2_pair(at, &maps.a, i * T::kBox, m0, bar);
                    if constexpr (BY_DEPTH) {
#pragma unroll
                        for (int g = 0; g < NT / 128; ++g)
                            tma_load2_pair(at + T::kABytes + g * (T::kBox * 128), &maps.b, n0 + g * 64, i * T::kBox, bar);
                    } else {
                        tma_load2_pair(at + T::kABytes, &maps.b, i * T::kBox, n0, bar);
                    }
                    r.next();
                }
            }
        }
    } else if (rank == 0) {
        if (elect_one()) {
            StepRing<T::kStages> r;
            const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)BY_DEPTH << 16) | ((unsigned)(NT >> 3) << 17) |
                                   ((unsigned)(2 * kProductRows >> 4) << 24);
            constexpr unsigned kNextK = BY_DEPTH ? 16 * 128 >> 4 : 16 * 2 >> 4;  // 16 of K further in b
            unsigned n = 0;
            for (long long t = first; t < p.tiles; t += p.pairs, ++n) {
                const unsigned buf = n & 1;
                if (n > 1) mbar_wait(acc_free + buf * 8, n / 2 - 1 & 1, dead);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                bool here = false;  // (tried ahead, as in step_feed)
                for (int i = 0; i < p.k_blocks; ++i) {
                    const unsigned slot = r.slot;
                    if (!here) mbar_wait_local(full + slot * 8, r.parity, dead);
                    if (dead) break;
                    r.next();
                    here = i + 1 < p.k_blocks && mbar_try<false>(full + r.slot * 8, r.parity);
                    const unsigned at = smem_addr(ring + slot * T::kStageBytes);
                    const unsigned long long a = step_desc(at),
                                             b = BY_DEPTH ? depth_desc(at + T::kABytes) : step_desc(at + T::kABytes);
#pragma unroll
                    for (int k = 0; k < T::kBox / 16; ++k)
                        pair_mma(tmem + buf * NT, a + 2 * k, b + kNextK * k, idesc, i > 0 || k > 0);
                    pair_commit(empty + slot * 8);
                }
                if (dead) break;
                pair_commit(acc_full + buf * 8);
            }
        }
    }
    // (after a wait that ran out: what is still on its way arrives before the block leaves)
    if (dead)
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();  // no arrivals at a block that has left
    if (warp == kProductWarps) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(T::kTmem) : "memory");
    }
}

}  // namespace fields

#endif  // FIELDS_HOST_EMU
