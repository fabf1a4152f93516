// Single-token step of a Field block as four kernels: each is a matrix product on the tensor cores
// (tcgen05.mma, operands by TMA, accumulator in tensor memory) whose epilogue does everything
// that follows it elementwise, down to the operand of the next product.
//
//   EpiIn   u = xb @ [write | gate]^T      -> the recurrence step: state, read row, its sums of squares; gate
//   EpiOut  acc = read @ (out diag(norm))^T -> y = x + (acc rstd + b) sigmoid(gate), bf16 copy, sums of squares
//   EpiUv   uv = yb @ (w12 diag(norm))^T    -> act = silu(u rstd) (v rstd)
//   EpiFf   f = act @ w3^T                  -> x' = y + f, bf16 copy
//
// A step of a few hundred rows is bound by the 25 MB of weights per block of d_model 1,024 (3.9 us at the
// copy bandwidth) and, far above that, by latency: as library products with elementwise kernels between
// them a block took nine launches. Here it is four, of about 9.4 us each in a row of them (10.8 to 12.3 alone
// and on a cold cache): 256 rows through 18 blocks 763 -> 680 us, 16 rows 745 -> 620. What is done about it:
//   - the RMS norms become a per-row scale of the product that follows (their weights are folded into the
//     bfloat16 copies), so a norm needs only partial sums of squares per row, which the
//     producing epilogue leaves in a small table;
//   - the rows of [write | gate] and w12 are laid out so that what an epilogue combines (the three
//     planes of a channel and two gate features; u and v of a feature) are columns of one tile;
//   - K is split over a cluster of S blocks, so that about 128 blocks share the loads of a product; each
//     then owns 1/S of the tile's columns, to which the others send their partial sums through
//     distributed shared memory (field_dsmem.cuh);
//   - the next kernel is let in at the start (dependent launch) and loads its weights before it waits for
//     this one, as far as SMs are free for it. (Blocks small enough that the next kernel's fit beside them
//     were slower, 797 us: blocks of one kernel then share SMs, and received sums have to wait for the
//     operands' space.)
//
// Tile: 128 rows (batch) x NT columns; TMEM lane = row, so an epilogue thread owns one row.
// Operands are K-major with the 128-byte swizzle: a k-block is 64 bf16 = 128 bytes per row.
// Device only; rows past the batch and columns past the matrix are zero-filled by TMA and not stored.
#pragma once

#include "field_dsmem.cuh"
#include "field_rows.cuh"

#ifndef FIELDS_HOST_EMU

#include <cuda.h>

namespace fields {

constexpr int kStepThreads = 160;  // four epilogue warps and one that issues loads and products
constexpr int kStepRows = 128;
constexpr int kStepKBlock = 64;    // bf16 per k-block

__device__ __forceinline__ void tma_load2(unsigned dst, const CUtensorMap* map, int x, int y, unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void send4(unsigned dst, float x, float y, float z, float w, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
                 "f"(x), "f"(y), "f"(z), "f"(w), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void send1(unsigned dst, float x, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(dst), "f"(x), "r"(bar)
                 : "memory");
}
// Shared-memory descriptor of a K-major operand with the 128-byte swizzle: rows of 128 bytes, groups
// of eight rows 1,024 bytes apart, descriptor version 1.
__device__ __forceinline__ unsigned long long step_desc(unsigned addr) {
    return (unsigned long long)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((unsigned long long)(1024 >> 4) << 32) |
           (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void step_mma(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc,
                                         unsigned accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void step_commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// Eight columns of the thread's lane; the values are there after tmem_wait().
__device__ __forceinline__ void tmem_load8(unsigned addr, unsigned* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ void tmem_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// Everything the four epilogues touch.
struct StepBlockParams {
    // activations
    const float* x;         // [M, D] the block's input
    uint16_t* gate;         // [M, D] bf16
    uint16_t* read;         // [M, 4C] bf16
    float* state;           // [M, 2C]
    float* y;               // [M, D] after the mixer
    uint16_t* yb;           // [M, D] bf16
    uint16_t* act;          // [M, H] bf16
    float* out;             // [M, D] the block's output (may be x)
    uint16_t* xb;           // [M, D] bf16 of the input, then of the output
    float* read_sq;         // [C / 8][M] partial sums of squares of the read row
    float* y_sq;            // [D / 8][M] of y
    // parameters
    const float* in_b;      // [5C] in the column order of the first product
    const float* par;       // [3, C]
    const float* out_b;     // [D]
    float read_eps, ff_eps;
    int M, D, C, H;
    // tiling
    int tiles_n, S, k_blocks;
    int wait_first;         // non-zero: parameters are read, and the next kernel let in, after the kernels before this one
};

__device__ __forceinline__ void store8(float* p, const float* v) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ void load8(const float* p, float* v) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void store8(uint16_t* p, const float* v) {
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(o[i]) : "f"(v[2 * i + 1]), "f"(v[2 * i]));
    *reinterpret_cast<uint4*>(p) = make_uint4(o[0], o[1], o[2], o[3]);
}
__device__ __forceinline__ void load8(const uint16_t* p, float* v) {
    const uint4 w = *reinterpret_cast<const uint4*>(p);
    const Vec<4> a = bf16x4_unpack(w.x, w.y), b = bf16x4_unpack(w.z, w.w);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        v[i] = a.v[i];
        v[4 + i] = b.v[i];
    }
}
// Sum of a row's partial sums of squares, block `rank` of S taking its share of the table ([count][M], so that
// a warp's rows are adjacent); the loads are issued together.
__device__ __forceinline__ float table_share(const float* table, int count, int M, int row, int rank, int S) {
    const int per = (count + S - 1) / S, lo = rank * per, hi = lo + per < count ? lo + per : count;
    float s = 0.0f;
    for (int i = lo; i < hi; i += 32) {
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = i + j < hi ? table[(size_t)(i + j) * M + row] : 0.0f;
#pragma unroll
        for (int j = 0; j < 32; ++j) s += v[j];
    }
    return s;
}

// An epilogue: kSlice columns at a time of row `row`; slice index g counts over the whole matrix.
//   constants  parameters of a slice into shared memory, before the wait for the previous kernel
//   share      this block's share of the sums of squares of the row (kScaled; exchanged like the products)
//   fetch      what slice g needs from global memory, while the product still runs
//   run        the rest
struct EpiIn {  // slice: eight channels' z_r | z_i | z_v, then sixteen gate features
    static constexpr int kSlice = 40, kSlices = 2, kStages = 7, kConst = 64;
    static constexpr bool kScaled = false;
    struct Fetched {
        float sr[8], si[8];
    };
    __device__ static float constant(const StepBlockParams& p, int g, int i) {  // 40 biases, 3 x 8 transition values
        if (g * 8 >= p.C) return 0.0f;
        return i < 40 ? p.in_b[g * 40 + i] : p.par[(i - 40) / 8 * p.C + g * 8 + (i - 40) % 8];
    }
    __device__ static float share(const StepBlockParams&, int, int, int) { return 0.0f; }
    __device__ void scale(const StepBlockParams&, float) {}
    __device__ void fetch(const StepBlockParams& p, int row, int g, Fetched& f) {
        if (g * 8 >= p.C) return;
        const float* st = p.state + (size_t)row * 2 * p.C + g * 8;
        load8(st, f.sr);
        load8(st + p.C, f.si);
    }
    __device__ void run(const StepBlockParams& p, int row, int g, const float* acc, const float* konst, Fetched& f) {
        const int c0 = g * 8, C = p.C;
        if (c0 >= C) return;
        float dr[8], di[8], sq = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const Gate gt = make_gate(acc[k] + konst[k], acc[8 + k] + konst[8 + k], acc[16 + k] + konst[16 + k]);
            float mr, mi;
            cmul(konst[40 + k], konst[48 + k], f.sr[k], f.si[k], mr, mi);
            const float bs = konst[56 + k] * gt.vac;
            f.sr[k] = (1.0f - gt.vac) * mr + bs * gt.inj_r;
            f.si[k] = (1.0f - gt.vac) * mi + bs * gt.inj_i;
            dr[k] = gt.vac * mr;
            di[k] = gt.vac * mi;
            sq += f.sr[k] * f.sr[k] + f.si[k] * f.si[k] + dr[k] * dr[k] + di[k] * di[k];
        }
        float* st = p.state + (size_t)row * 2 * C + c0;
        store8(st, f.sr);
        store8(st + C, f.si);
        uint16_t* o = p.read + (size_t)row * 4 * C + c0;
        store8(o, f.sr);
        store8(o + C, f.si);
        store8(o + 2 * C, dr);
        store8(o + 3 * C, di);
        p.read_sq[(size_t)g * p.M + row] = sq;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = acc[24 + h * 8 + k] + konst[24 + h * 8 + k];
            store8(p.gate + (size_t)row * p.D + g * 16 + h * 8, v);
        }
    }
};

// EpiOut and EpiFf come with tiles of 64 and of 32 features (and EpiUv with two of its slices for the same row
// counts). Where 64 leave so few tiles that K would be split
// over clusters of eight (up to 128 rows at d_model 1,024), 32 with clusters of four are faster: a kernel's
// clusters of eight took up to 14 us to get started (18 blocks, 16 rows: 736 -> 620 us; 128 rows: 730 -> 589).
template <int SLICES>
struct EpiOut {  // slice: eight features
    static constexpr int kSlice = 8, kSlices = SLICES, kStages = 7, kConst = 8;
    static constexpr bool kScaled = true;
    struct Fetched {
        float x[8], gate[8];
    };
    float rstd;
    __device__ static float constant(const StepBlockParams& p, int g, int i) { return g * 8 < p.D ? p.out_b[g * 8 + i] : 0.0f; }
    __device__ static float share(const StepBlockParams& p, int row, int rank, int S) {
        return table_share(p.read_sq, p.C / 8, p.M, row, rank, S);
    }
    __device__ void scale(const StepBlockParams& p, float sum) { rstd = rsqrtf(sum / (float)(4 * p.C) + p.read_eps); }
    __device__ void fetch(const StepBlockParams& p, int row, int g, Fetched& f) {
        if (g * 8 >= p.D) return;
        load8(p.x + (size_t)row * p.D + g * 8, f.x);
        load8(p.gate + (size_t)row * p.D + g * 8, f.gate);
    }
    __device__ void run(const StepBlockParams& p, int row, int g, const float* acc, const float* konst, Fetched& f) {
        if (g * 8 >= p.D) return;
        const size_t at = (size_t)row * p.D + g * 8;
        float sq = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            f.x[k] += (acc[k] * rstd + konst[k]) * sigmoidf_fast(f.gate[k]);
            sq += f.x[k] * f.x[k];
        }
        store8(p.y + at, f.x);
        store8(p.yb + at, f.x);
        p.y_sq[(size_t)g * p.M + row] = sq;
    }
};

template <int SLICES>
struct EpiUv {  // slice: u of twenty features, then v of the same
    static constexpr int kSlice = 40, kSlices = SLICES, kStages = SLICES == 4 ? 4 : 7, kConst = 0;
    static constexpr bool kScaled = true;
    struct Fetched {};
    float rstd;
    __device__ static float constant(const StepBlockParams&, int, int) { return 0.0f; }
    __device__ static float share(const StepBlockParams& p, int row, int rank, int S) {
        return table_share(p.y_sq, p.D / 8, p.M, row, rank, S);
    }
    __device__ void scale(const StepBlockParams& p, float sum) { rstd = rsqrtf(sum / (float)p.D + p.ff_eps); }
    __device__ void fetch(const StepBlockParams&, int, int, Fetched&) {}
    __device__ void run(const StepBlockParams& p, int row, int g, const float* acc, const float*, Fetched&) {
        const int h0 = g * 20;
        uint16_t* o = p.act + (size_t)row * p.H + h0;
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            if (h0 + q * 4 < p.H) {  // H % 8 == 0: four at a time are inside or outside
                Vec<4> a;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float u = acc[q * 4 + k] * rstd, v = acc[20 + q * 4 + k] * rstd;
                    a.v[k] = u * sigmoidf_fast(u) * v;
                }
                store_bf16x4(o + q * 4, a);
            }
        }
    }
};

template <int SLICES>
struct EpiFf {  // slice: eight features
    static constexpr int kSlice = 8, kSlices = SLICES, kStages = 7, kConst = 0;
    static constexpr bool kScaled = false;
    struct Fetched {
        float y[8];
    };
    __device__ static float constant(const StepBlockParams&, int, int) { return 0.0f; }
    __device__ static float share(const StepBlockParams&, int, int, int) { return 0.0f; }
    __device__ void scale(const StepBlockParams&, float) {}
    __device__ void fetch(const StepBlockParams& p, int row, int g, Fetched& f) {
        if (g * 8 < p.D) load8(p.y + (size_t)row * p.D + g * 8, f.y);
    }
    __device__ void run(const StepBlockParams& p, int row, int g, const float* acc, const float*, Fetched& f) {
        if (g * 8 >= p.D) return;
        const size_t at = (size_t)row * p.D + g * 8;
#pragma unroll
        for (int k = 0; k < 8; ++k) f.y[k] += acc[k];
        store8(p.out + at, f.y);
        store8(p.xb + at, f.y);
    }
};

template <class Epi>
struct StepTile {
    static constexpr int kNT = Epi::kSlice * Epi::kSlices;
    static constexpr int kABytes = kStepRows * 128, kBBytes = kNT * 128, kStageBytes = kABytes + kBBytes;
    static constexpr unsigned kColumns = kNT <= 64 ? 64 : kNT <= 128 ? 128 : 256;  // of tensor memory
    static constexpr int kOperandBytes = Epi::kStages * kStageBytes;
    // what S - 1 blocks send, [src][column / 4][row] float4; most for S = kSlices
    static constexpr int kRecvBytes = (Epi::kSlices - 1) * Epi::kSlice * kStepRows * 4;
    static constexpr int kShareBytes = Epi::kScaled ? Epi::kSlices * kStepRows * 4 : 0;
    static constexpr int kConstBytes = Epi::kSlices * Epi::kConst * 4;
    static constexpr size_t kSmemBytes =
        1024 + (size_t)kOperandBytes + kRecvBytes + kShareBytes + kConstBytes + (2 * Epi::kStages + 2) * 8 + 16;
    static_assert(kSmemBytes <= 227 * 1024, "shared memory of an SM");
    static_assert(kNT % 16 == 0 && kNT <= 256 && kBBytes % 1024 == 0, "a tile the tensor cores take");
};

template <class Epi>
__global__ void __launch_bounds__(kStepThreads, 1)
    step_gemm(const __grid_constant__ CUtensorMap a_map, const __grid_constant__ CUtensorMap b_map,
              const StepBlockParams p) {
    using T = StepTile<Epi>;
    constexpr int kStages = Epi::kStages, kSlice = Epi::kSlice;
    extern __shared__ __align__(1024) char step_smem[];
    char* base = step_smem + (1024 - (smem_addr(step_smem) & 1023)) % 1024;
    char* recv = base + T::kOperandBytes;
    float* shares = reinterpret_cast<float*>(recv + T::kRecvBytes);  // [block of the cluster][row]
    float* konst = shares + T::kShareBytes / 4;
    char* tail = reinterpret_cast<char*>(konst) + T::kConstBytes;
    const unsigned full = smem_addr(tail), empty = full + kStages * 8, done = empty + kStages * 8, got = done + 8;
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(tail + (2 * kStages + 2) * 8);
    const int tid = threadIdx.x, warp = tid >> 5, S = p.S;
    const int rank = S > 1 ? (int)cluster_rank() : 0;
    const int tile = blockIdx.x / S, n_tile = tile % p.tiles_n, m0 = tile / p.tiles_n * kStepRows;
    const int per = (p.k_blocks + S - 1) / S, kb0 = rank * per;
    const int count = (p.k_blocks - kb0 < per ? p.k_blocks - kb0 : per);  // > 0: the host chose S so
    const int own = Epi::kSlices / S;                                    // slices this block finishes
    const int g0 = n_tile * Epi::kSlices + rank * own;                   // the first of them
    const bool control = tid == 4 * 32;
    bool dead = false;

    auto stage_a = [&](int i) { return smem_addr(base + (i % kStages) * T::kStageBytes); };
    auto load_b = [&](int i) {
        mbar_expect(full + (i % kStages) * 8, T::kStageBytes);
        tma_load2(stage_a(i) + T::kABytes, &b_map, (kb0 + i) * kStepKBlock, n_tile * T::kNT, full + (i % kStages) * 8);
    };
    auto load_a = [&](int i) {
        tma_load2(stage_a(i), &a_map, (kb0 + i) * kStepKBlock, m0, full + (i % kStages) * 8);
    };
    if (p.wait_first) asm volatile("griddepcontrol.wait;" ::: "memory");
    if (control) {
        for (int i = 0; i < kStages; ++i) {
            mbar_init(full + i * 8, 1);
            mbar_init(empty + i * 8, 1);
        }
        mbar_init(done, 1);
        mbar_init(got, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (S > 1) mbar_expect(got, (unsigned)((S - 1) * (own * kSlice + (Epi::kScaled ? 1 : 0)) * kStepRows * 4));
        // weights do not depend on the kernels before this one (or those have been waited for)
        for (int i = 0; i < kStages && i < count; ++i) load_b(i);
    }
    __syncwarp();
    if (warp == 4) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(T::kColumns)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if constexpr (Epi::kConst > 0) {
        for (int i = tid; i < own * Epi::kConst; i += kStepThreads)
            konst[i] = Epi::constant(p, g0 + i / Epi::kConst, i % Epi::kConst);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (S > 1) asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
    const unsigned tmem = *tmem_slot;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    constexpr int kAhead = 2;  // slices whose inputs are fetched while the product runs
    Epi epi;
    typename Epi::Fetched fetched[kAhead];
    float share = 0.0f;
    const int row = m0 + tid;
    const bool row_ok = tid < kStepRows && row < p.M;
    if (control) {
        for (int i = 0; i < kStages && i < count; ++i) load_a(i);
        const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(T::kNT >> 3) << 17) |
                               ((unsigned)(kStepRows >> 4) << 24);
        for (int i = 0; i < count; ++i) {
            mbar_wait(full + (i % kStages) * 8, (i / kStages) & 1, dead);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned long long a = step_desc(stage_a(i)), b = step_desc(stage_a(i) + T::kABytes);
#pragma unroll
            for (int k = 0; k < kStepKBlock / 16; ++k)  // 16 of K: 32 bytes further in the swizzle atom
                step_mma(tmem, a + 2 * k, b + 2 * k, idesc, i > 0 || k > 0);
            step_commit(empty + (i % kStages) * 8);
            // refill the stage of the product before this one
            const int j = i - 1 + kStages;
            if (i > 0 && j < count) {
                mbar_wait(empty + ((i - 1) % kStages) * 8, ((i - 1) / kStages) & 1, dead);
                load_b(j);
                load_a(j);
            }
        }
        step_commit(done);
    } else if (row_ok) {
#pragma unroll
        for (int q = 0; q < kAhead; ++q)
            if (q < own) epi.fetch(p, row, g0 + q, fetched[q]);
        if constexpr (Epi::kScaled) share = epi.share(p, row, rank, S);
    }
    __syncwarp();  // (the control thread's warp)
    if (S > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");  // the peers' barriers are ready
    mbar_wait(done, 0, dead);
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp < 4) {
        const unsigned lane_addr = tmem + ((unsigned)(warp * 32) << 16);
        if constexpr (Epi::kScaled) shares[rank * kStepRows + tid] = share;
        for (int d = 1; d < S; ++d) {  // the other blocks' columns, each block starting with its neighbour
            const int j = (rank + d) % S, src = rank > j ? rank - 1 : rank;
            const unsigned bar = peer_addr(got, j);
            const unsigned at = peer_addr(smem_addr(recv) + (unsigned)((src * own * kSlice / 4 * kStepRows + tid) * 16), j);
            if constexpr (Epi::kScaled) send1(peer_addr(smem_addr(shares + rank * kStepRows + tid), j), share, bar);
            for (int q = 0; q < own; ++q) {
                unsigned v[kSlice];
#pragma unroll
                for (int c = 0; c < kSlice; c += 8) tmem_load8(lane_addr + (j * own + q) * kSlice + c, v + c);
                tmem_wait();
#pragma unroll
                for (int c = 0; c < kSlice; c += 4)
                    send4(at + (unsigned)((q * kSlice + c) / 4 * kStepRows * 16), __uint_as_float(v[c]),
                          __uint_as_float(v[c + 1]), __uint_as_float(v[c + 2]), __uint_as_float(v[c + 3]), bar);
            }
        }
        auto finish = [&](int q, typename Epi::Fetched& f) {
            unsigned v[kSlice];
            float acc[kSlice];
#pragma unroll
            for (int c = 0; c < kSlice; c += 8) tmem_load8(lane_addr + (rank * own + q) * kSlice + c, v + c);
            tmem_wait();
#pragma unroll
            for (int c = 0; c < kSlice; ++c) acc[c] = dead ? nanf("") : __uint_as_float(v[c]);
            for (int src = 0; src < S - 1; ++src) {
                const float4* r = reinterpret_cast<const float4*>(recv) + (src * own + q) * (kSlice / 4) * kStepRows + tid;
#pragma unroll
                for (int c = 0; c < kSlice / 4; ++c) {
                    const float4 w = r[c * kStepRows];
                    acc[4 * c] += w.x; acc[4 * c + 1] += w.y; acc[4 * c + 2] += w.z; acc[4 * c + 3] += w.w;
                }
            }
            if (row_ok) epi.run(p, row, g0 + q, acc, konst + q * Epi::kConst, f);
        };
        if (S > 1) mbar_wait(got, 0, dead);
        __syncwarp();
        if constexpr (Epi::kScaled) {
            float sum = 0.0f;
            for (int r = 0; r < S; ++r) sum += shares[r * kStepRows + tid];
            epi.scale(p, sum);
        }
#pragma unroll
        for (int q = 0; q < kAhead; ++q)
            if (q < own) finish(q, fetched[q]);
        for (int q = kAhead; q < own; ++q) {
            if (row_ok) epi.fetch(p, row, g0 + q, fetched[0]);
            finish(q, fetched[0]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 4) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(T::kColumns) : "memory");
    }
}

// Rows of [write | gate] and of w12 diag(norm) in the order the epilogues want, in bfloat16, and the biases of
// the first product: one block per row.
struct StepLayoutParams {
    const float *write_w, *write_b, *gate_w, *gate_b, *w12, *norm_w;
    uint16_t *in_w, *w12_w;  // [5C, D], [40 ceil(H / 20), D]
    float* in_b;             // [5C]
    int D, C, H;
};

__global__ void __launch_bounds__(kRowThreads) step_layout(const StepLayoutParams p) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int C = p.C, D = p.D;
    int r = (int)blockIdx.x;
    const float *src, *scale = nullptr;
    uint16_t* dst;
    if (r < 5 * C) {
        const int g = r / 40, q = r % 40;
        const int from = q < 24 ? q / 8 * C + g * 8 + q % 8 : g * 16 + q - 24;
        src = (q < 24 ? p.write_w : p.gate_w) + (size_t)from * D;
        dst = p.in_w + (size_t)r * D;
        if (threadIdx.x == 0) p.in_b[r] = (q < 24 ? p.write_b : p.gate_b)[from];
    } else {
        r -= 5 * C;
        const int h = r / 40 * 20 + r % 20;
        src = h < p.H ? p.w12 + (size_t)(r % 40 < 20 ? h : p.H + h) * D : nullptr;
        dst = p.w12_w + (size_t)r * D;
        scale = p.norm_w;
    }
    for (int c = (int)threadIdx.x * 4; c < D; c += kRowThreads * 4) {
        Vec<4> v = src ? vec_load_stream<4>(src + c) : vec_fill<4>(0.0f);
        if (scale) {
            const Vec<4> w = load4(scale + c);
#pragma unroll
            for (int k = 0; k < 4; ++k) v.v[k] *= w.v[k];
        }
        store_bf16x4(dst + c, v);
    }
}

}  // namespace fields

#endif  // FIELDS_HOST_EMU
