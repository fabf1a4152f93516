// Matrix products of thousands of rows with everything that follows them elementwise as their epilogue:
//   out = a @ b^T, a [M, K] activations, b [N, K] weights, both bfloat16 with K contiguous, fp32 accumulation.
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
// 1.0 ms the row kernels. Now 4.57. Alone, 8,192 rows, products of the library and, with what follows, these (us): bias,
// 2,560 columns of depth 1,024, 33 and 32; SwiGLU, 5,056 of 1,024, 66 (+ 19 for the row kernel) and 56; residual,
// 1,024 of 2,528, 33 (+ 14) and 42; gate, 1,024 of 2,048, 27 (+ 21) and 46; gradient of the norm, 2,048 of 1,024, 30 (+ 18)
// and 35. Products run at 1.3 to 1.5 PFLOP/s; the epilogues with fp32 inputs and outputs are bound by the latency
// of HBM under load (3,000 cycles) and the 24 to 32 KB that a block's registers keep in flight.
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

struct ProductParams {
    long long M;
    int N, k_blocks;
    int tiles_n, pairs;
    long long tiles;
    // (what an epilogue does not use is null)
    const float* x;          // [M, N]
    const uint16_t* bias16;  // [N]
    const float *bias, *gate_bias;  // [N]
    const uint16_t* gate;    // rows of gate_pitch
    long long gate_pitch;
    const float* sums;       // [M, entries] sums of squares behind rstd = rsqrt(sum * inv_features + eps)
    int entries;
    float inv_features, eps;
    const float* row;        // [M] factor of a row
    const uint16_t* read;    // [M, N]
    float* y;                // [M, N] (may be x)
    uint16_t* h;             // [M, N], or rows of h_pitch
    long long h_pitch;
    float* sums_out;         // [M, ceil(N / 32)]: a warp's columns in the first of their entries, zero in the other
    uint16_t* acc;           // [M, N]
};

// Tensors from the first row and column of a warp's part of a tile on.
struct ProductBase {
    const float* x;
    float* y;
    uint16_t *h, *acc;
    const uint16_t *gate, *read;
};

// A lane's four columns of a row. Column holds what they need whatever the row (`col` counts in the matrix), Loaded what
// they need of the row, `factor` is a value of the row; run() does the rest and returns their sum of squares. Offsets
// count from the ProductBase: `at` in [M, N], `gate_at` and `h_at` in the tensors with a pitch. A piece is kPiece columns.
struct ProductBias {
    static constexpr int kPiece = 32;
    static constexpr bool kSums = false, kSwiglu = false;
    using Column = Vec<4>;
    struct Loaded {};
    __device__ static Column column(const ProductParams& p, int col) { return load4(p.bias16 + col); }
    __device__ static float factor(const ProductParams&, long long) { return 1.0f; }
    __device__ static void load(const ProductBase&, int, int, Loaded&) {}
    __device__ static float run(const ProductBase& b, int, int h_at, Vec<4> v, float, const Column& bias, const Loaded&) {
#pragma unroll
        for (int k = 0; k < 4; ++k) v.v[k] += bias.v[k];
        store_bf16x4(b.h + h_at, v);
        return 0.0f;
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
    static constexpr int kPiece = 16;  // (two pieces' inputs are in registers)
    static constexpr bool kSums = true, kSwiglu = false;
    struct Column {
        Vec<4> b, gb;
    };
    struct Loaded {
        Vec<4> x;
        uint2 gate;
    };
    __device__ static Column column(const ProductParams& p, int col) { return Column{load4(p.bias + col), load4(p.gate_bias + col)}; }
    __device__ static float factor(const ProductParams& p, long long row) { return product_rstd(p, row); }
    __device__ static void load(const ProductBase& b, int at, int gate_at, Loaded& l) {
        l.x = load4(b.x + at);
        l.gate = *reinterpret_cast<const uint2*>(b.gate + gate_at);
    }
    __device__ static float run(const ProductBase& b, int at, int h_at, Vec<4> v, float rstd, const Column& c, const Loaded& l) {
        if (b.acc) store_bf16x4(b.acc + at, v);
        const Vec<4> gate = bf16x4_unpack(l.gate.x, l.gate.y);
        float sq = 0.0f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v.v[k] = l.x.v[k] + (v.v[k] * rstd + c.b.v[k]) * sigmoidf_fast(gate.v[k] + c.gb.v[k]);
            sq += v.v[k] * v.v[k];
        }
        vec_store<4>(b.y + at, v);
        if (b.h) store_bf16x4(b.h + h_at, v);
        return sq;
    }
};
struct ProductSwiglu {
    static constexpr int kPiece = 32;
    static constexpr bool kSums = false, kSwiglu = true;
    struct Column {};
    struct Loaded {};
    __device__ static float factor(const ProductParams& p, long long row) { return product_rstd(p, row); }
};
struct ProductResidual {
    static constexpr int kPiece = 32;
    static constexpr bool kSums = false, kSwiglu = false;
    struct Column {};
    struct Loaded {
        Vec<4> x;
    };
    __device__ static Column column(const ProductParams&, int) { return {}; }
    __device__ static float factor(const ProductParams&, long long) { return 1.0f; }
    __device__ static void load(const ProductBase& b, int at, int, Loaded& l) { l.x = load4(b.x + at); }
    __device__ static float run(const ProductBase& b, int at, int h_at, Vec<4> v, float, const Column&, const Loaded& l) {
#pragma unroll
        for (int k = 0; k < 4; ++k) v.v[k] += l.x.v[k];
        vec_store<4>(b.y + at, v);
        if (b.h) store_bf16x4(b.h + h_at, v);
        return 0.0f;
    }
};
struct ProductNormGrad {
    static constexpr int kPiece = 32;
    static constexpr bool kSums = false, kSwiglu = false;
    struct Column {};
    struct Loaded {
        uint2 r;
    };
    __device__ static Column column(const ProductParams&, int) { return {}; }
    __device__ static float factor(const ProductParams& p, long long row) { return 2.0f * p.row[row]; }
    __device__ static void load(const ProductBase& b, int at, int, Loaded& l) { l.r = *reinterpret_cast<const uint2*>(b.read + at); }
    __device__ static float run(const ProductBase& b, int, int h_at, Vec<4> v, float c, const Column&, const Loaded& l) {
        const Vec<4> r = bf16x4_unpack(l.r.x, l.r.y);
#pragma unroll
        for (int k = 0; k < 4; ++k) v.v[k] += c * r.v[k];
        store_bf16x4(b.h + h_at, v);
        return 0.0f;
    }
};

template <int NT>
struct ProductShape {
    static constexpr int kBox = 64;  // of K
    static constexpr int kABytes = kProductRows * kBox * 2, kBBytes = NT / 2 * kBox * 2, kStageBytes = kABytes + kBBytes;
    // As many stages as there is space for beside 32 rows x 256 columns of pieces: under load a copy takes some 3,000
    // cycles to arrive, the products of a stage 512. With five stages instead of six the products of a tile of depth
    // 2,528 took 26,000 cycles instead of 20,900, with four those of depth 2,048 29,000 instead of 17,000.
    static constexpr int kPiecesBytes = 32 * 1024;
    static constexpr int kStages = (227 * 1024 - 1024 - 256 - kPiecesBytes) / kStageBytes;
    static constexpr int kBars = 2 * kStages + 4;
    static constexpr size_t kSmemBytes = 1024 + (size_t)kStages * kStageBytes + kPiecesBytes + kBars * 8 + 16;
    static constexpr unsigned kColumns = 2 * NT;  // of tensor memory
    static_assert(kSmemBytes <= 227 * 1024, "shared memory of an SM");
    static_assert(NT == 256 || NT == 128, "tiles the tensor cores and the epilogue's warps take");
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

__device__ __forceinline__ Vec<4> vec_of(const float4& a) { return Vec<4>{{a.x, a.y, a.z, a.w}}; }

// A tile's share of one warp: 32 rows x NT / 2 columns of its block, a piece at a time. A lane has a row of
// the product, and accesses to global memory want lanes along the rows, so a piece passes through shared memory.
// What it needs besides is loaded into registers under the piece before it, that of the first under the product. (The
// pieces are a loop, two at a time for the registers' sake: unrolled they are up to 77 KB of code, run at the rate at
// which it is fetched. Loads of the next piece between the stores of this one made every row wait for all of them:
// their scoreboards are shared.)
template <class Epi, int NT>
struct ProductTile {
    using T = ProductShape<NT>;
    static constexpr int kPiece = Epi::kPiece, kColumns = NT / (kProductWarps / 4), kPieces = kColumns / kPiece;
    static constexpr int kUnits = kPiece / 4, kRows = 32 / kUnits;  // units of four columns; rows of a warp-wide access
    static_assert(kPieces % 2 == 0, "pieces go in pairs");
    struct Inputs {  // of a lane: its unit of kUnits rows
        typename Epi::Column column;
        typename Epi::Loaded row[kUnits];
    };
    const ProductParams& p;
    char* piece;
    long long row0;
    int col0, lane, rows;
    ProductBase base;
    float factor = 1.0f;  // of row0 + lane
    float sq[kUnits];
    Inputs even, odd;

    __device__ ProductTile(const ProductParams& p, char* piece, long long row0, int col0)
        : p(p), piece(piece), row0(row0), col0(col0), lane(threadIdx.x & 31),
          rows(p.M - row0 < 32 ? (int)(p.M - row0) : 32) {
        const long long at = row0 * p.N + col0;
        base.x = p.x + at;
        base.y = p.y + at;
        base.read = p.read + at;
        base.acc = p.acc ? p.acc + at : nullptr;
        base.h = p.h ? p.h + row0 * p.h_pitch + (Epi::kSwiglu ? col0 / 2 : col0) : nullptr;
        base.gate = p.gate + row0 * p.gate_pitch + col0;
        load(0, even);
        if (lane < rows) factor = Epi::factor(p, row0 + lane);
    }
    __device__ int row_of(int i) const { return i * kRows + lane / kUnits; }
    __device__ int col_of(int k) const { return k * kPiece + lane % kUnits * 4; }
    __device__ void load(int k, Inputs& to) const {
        if constexpr (!Epi::kSwiglu) {
            const int col = col_of(k);
            if (k >= kPieces || col0 + col >= p.N) return;
            to.column = Epi::column(p, col0 + col);
#pragma unroll
            for (int i = 0; i < kUnits; ++i)
                if (row_of(i) < rows) Epi::load(base, row_of(i) * p.N + col, row_of(i) * (int)p.gate_pitch + col, to.row[i]);
        }
    }
    // 16 bytes of a row of the piece, permuted so that neither a lane per row nor lanes along the rows meet in a bank
    __device__ float4* unit(int row, int u) const {
        const int turn = kUnits == 8 ? row & 7 : row >> 1 & 3;
        return reinterpret_cast<float4*>(piece + row * (kPiece * 4) + (u ^ turn) * 16);
    }
    // tmem: the warp's lanes and first column; released: where to say that they have been read
    __device__ void one(int k, unsigned tmem, unsigned released, bool dead, const Inputs& use, Inputs& next) {
        load(k + 1, next);
        unsigned v[kPiece];
        __syncwarp();
        if constexpr (kPiece == 32) tmem_load32(tmem + (unsigned)(k * kPiece), v);
        else tmem_load<kPiece>(tmem + (unsigned)(k * kPiece), v);
        tmem_wait();
        if (k + 1 == kPieces) {
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            // (at block scope: at cluster scope it waits for the warp's stores, 2,500 cycles, and orders nothing but
            // tensor memory)
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(released) : "memory");
        }
        if (dead) {
#pragma unroll
            for (int i = 0; i < kPiece; ++i) v[i] = ~0u;  // NaN
        }
#pragma unroll
        for (int i = 0; i < kUnits; ++i)
            *unit(lane, i) = make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]),
                                         __uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3]));
        __syncwarp();
        if constexpr (Epi::kSwiglu) {
            // columns: u of eight features, v of the same; a lane takes four features of a row
            const int j = lane % 4, at = j / 2 * 4 + j % 2, f = k * (kPiece / 2) + j * 4;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int rl = i * 8 + lane / 4;
                const float rs = __shfl_sync(0xffffffffu, factor, rl);
                const Vec<4> u = vec_of(*unit(rl, at)), w = vec_of(*unit(rl, at + 2));
                Vec<4> a;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float us = u.v[e] * rs;
                    a.v[e] = us * sigmoidf_fast(us) * (w.v[e] * rs);
                }
                if (rl < rows && col0 / 2 + f < p.N / 2) store_bf16x4(base.h + rl * (int)p.h_pitch + f, a);
            }
        } else {
            const int col = col_of(k);
            Vec<4> a[kUnits];
#pragma unroll
            for (int i = 0; i < kUnits; ++i) a[i] = vec_of(*unit(row_of(i), lane % kUnits));
#pragma unroll
            for (int i = 0; i < kUnits; ++i) {
                const float f = __shfl_sync(0xffffffffu, factor, row_of(i));
                if (row_of(i) < rows && col0 + col < p.N)
                    sq[i] += Epi::run(base, row_of(i) * p.N + col, row_of(i) * (int)p.h_pitch + col, a[i], f, use.column, use.row[i]);
            }
        }
    }
    __device__ void finish(unsigned tmem, unsigned released, bool dead) {
#pragma unroll
        for (int i = 0; i < kUnits; ++i) sq[i] = 0.0f;
#pragma unroll 1
        for (int k = 0; k < kPieces; k += 2) {
            one(k, tmem, released, dead, even, odd);
            one(k + 1, tmem, released, dead, odd, even);
        }
        if constexpr (Epi::kSums) {
            if (!p.sums_out) return;
            const int entries = (p.N + 31) / 32, at = col0 / 32 + lane % kUnits;
#pragma unroll
            for (int i = 0; i < kUnits; ++i) {
#pragma unroll
                for (int off = kUnits / 2; off > 0; off >>= 1) sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], off);
                if (lane % kUnits < kColumns / 32 && row_of(i) < rows && at < entries)
                    p.sums_out[(row0 + row_of(i)) * entries + at] = lane % kUnits ? 0.0f : sq[i];
            }
        }
    }
};

template <class Epi, int NT>
__global__ void __launch_bounds__(32 * (kProductWarps + 2), 1)
    pair_product(const __grid_constant__ CUtensorMap a_map, const __grid_constant__ CUtensorMap b_map,
                 const __grid_constant__ ProductParams p) {
    using T = ProductShape<NT>;
    extern __shared__ __align__(1024) char product_smem[];
    char* ring = product_smem + (1024 - (smem_addr(product_smem) & 1023)) % 1024;
    char* pieces = ring + T::kStages * T::kStageBytes;
    char* tail = pieces + T::kPiecesBytes;
    // loads have landed (both blocks', on the first block's barriers); stage free, accumulator full (each block's own);
    // accumulator free (the first block's)
    const unsigned full = smem_addr(tail), empty = full + T::kStages * 8, acc_full = empty + T::kStages * 8,
                   acc_free = acc_full + 16;
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(tail + T::kBars * 8);
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), rank = (int)cluster_rank();

    if (threadIdx.x == 0) {
        for (int i = 0; i < 2 * T::kStages + 2; ++i) mbar_init(full + i * 8, 1);
        for (int i = 0; i < 2; ++i) mbar_init(acc_free + i * 8, 2 * kProductWarps);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kProductWarps) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(T::kColumns)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();  // the other block's barriers are ready
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = *tmem_slot;
    asm volatile("griddepcontrol.wait;" ::: "memory");

    const long long first = blockIdx.x / 2;
    bool dead = false;
    static_assert(kProductWarps * 32 * Epi::kPiece * 4 <= T::kPiecesBytes, "space for the pieces");
    if (warp < kProductWarps) {
        const unsigned lanes = tmem + ((unsigned)(warp % 4 * 32) << 16) + (unsigned)(warp / 4 * ProductTile<Epi, NT>::kColumns);
        unsigned n = 0;
        for (long long t = first; t < p.tiles; t += p.pairs, ++n) {
            const unsigned buf = n & 1;
            ProductTile<Epi, NT> tile(p, pieces + warp * (32 * Epi::kPiece * 4), t / p.tiles_n * (2 * kProductRows) + rank * kProductRows + warp % 4 * 32,
                                      (int)(t % p.tiles_n) * NT + warp / 4 * ProductTile<Epi, NT>::kColumns);
            mbar_wait_local(acc_full + buf * 8, n / 2 & 1, dead);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            tile.finish(lanes + buf * NT, peer_addr(acc_free + buf * 8, 0), dead);
        }
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
                    tma_load2_pair(at, &a_map, i * T::kBox, m0, bar);
                    tma_load2_pair(at + T::kABytes, &b_map, i * T::kBox, n0, bar);
                    r.next();
                }
            }
        }
    } else if (rank == 0) {
        if (elect_one()) {
            StepRing<T::kStages> r;
            const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(NT >> 3) << 17) |
                                   ((unsigned)(2 * kProductRows >> 4) << 24);
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
                    const unsigned long long a = step_desc(smem_addr(ring + slot * T::kStageBytes)), b = a + (T::kABytes >> 4);
#pragma unroll
                    for (int k = 0; k < T::kBox / 16; ++k)
                        pair_mma(tmem + buf * NT, a + 2 * k, b + 2 * k, idesc, i > 0 || k > 0);
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
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(T::kColumns) : "memory");
    }
}

}  // namespace fields

#endif  // FIELDS_HOST_EMU
