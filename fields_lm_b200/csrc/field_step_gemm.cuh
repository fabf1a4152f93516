// Single-token step of a stack of Field blocks as one kernel. Per block it is four phases, each a matrix
// product on the tensor cores (tcgen05.mma, operands by TMA, accumulator in tensor memory) whose epilogue
// does everything that follows it elementwise, down to the operand of the next product.
//
//   EpiIn   u = xb @ [write | gate]^T      -> the recurrence step: state, read row, its sums of squares; gate
//   EpiOut  acc = read @ (out diag(norm))^T -> y = x + (acc rstd + b) sigmoid(gate), bf16 copy, sums of squares
//   EpiUv   uv = yb @ (w12 diag(norm))^T    -> act = silu(u rstd) (v rstd)
//   EpiFf   f = act @ w3^T                  -> x' = y + f, bf16 copy
//
// A step of a few hundred rows is bound by latency: the 25 MB of weights of a block of d_model 1,024 take
// 3.9 us at the copy bandwidth, its products 4 us. A phase takes 7,100 to 7,800 cycles at 1 row and 9,900 to 14,300 at 256: there
// 1,200 from a block's publication to the count that lets the next phase's loads go (800 for the last block to publish, and the
// others wait for it), 1,400 until its operands are there, 3,200 to 3,900 until the product is done, 5,700 in the 160-column product,
// 1,400 to 2,600 for the exchange of partial sums, 700 to 2,600 for the epilogue, 1,100 until it is published. 18 blocks of d_model
// 1,024 take 312 us at 1 row and 471 at 256; the first form of this launch 429 and 602, four launches per block
// (field_step_phase.cuh, where that is still the faster way) 589 and 682. What is done about it:
//   - all blocks of the stack in one cooperative launch. A row tile (128 rows) is a chain of its own: its
//     thread blocks count the finished tiles of a phase in global memory, and the loads of the next phase's
//     activations wait for that count;
//   - weights do not wait for anything: one warp streams them into a ring of their own, across phases and
//     blocks of the stack, so they are there when the activations arrive;
//   - the RMS norms become a per-row scale of the product that follows (their weights are folded into the
//     bfloat16 copies), so a norm needs only sums of squares per row and tile, which the producing
//     epilogue leaves in a small table;
//   - the rows of [write | gate] and w12 are laid out so that what an epilogue combines (the three
//     planes of a channel and two gate features; u and v of a feature) are columns of one tile;
//   - K is split over S thread blocks of a cluster, so that about 128 of them share the loads of a product; each
//     then finishes 1/S of the tile's rows, to which the others send their partial sums through distributed
//     shared memory (field_dsmem.cuh). All sums pass through shared memory, so that the epilogue's lanes lie along
//     a row: with TMEM's one lane per row every access touched 32 rows (256 rows: 628 us).
//
// Tile: 128 rows (batch) x NT columns. Operands are K-major with the 128-byte swizzle: boxes of 64 bf16 = 128 bytes
// per row, two to a k-block.
// Device only; rows past the batch and columns past the matrix are zero-filled by TMA (or, where the batch is
// shorter than a tile, left as they are in lanes that nothing reads) and not stored.
#pragma once

#include "field_dsmem.cuh"
#include "field_rows.cuh"

#ifndef FIELDS_HOST_EMU

#include <cuda.h>

namespace fields {

constexpr int kStepThreads = 352;  // eight epilogue warps; weights, activations, products: a warp each
constexpr int kStepRows = 128;
constexpr int kStepKBox = 64;      // bf16 of K in a TMA box: the swizzle's 128 bytes
constexpr int kStepKBoxes = 2;     // boxes of a k-block
constexpr int kStepKBlock = kStepKBox * kStepKBoxes;

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
// Eight columns of the thread's lane, or a multiple of eight; the values are there after tmem_wait().
__device__ __forceinline__ void tmem_load8(unsigned addr, unsigned* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(addr)
                 : "memory");
}
template <int N>
__device__ __forceinline__ void tmem_load(unsigned addr, unsigned* r) {
    static_assert(N % 8 == 0, "columns");
#pragma unroll
    for (int k = 0; k < N; k += 8) tmem_load8(addr + k, r + k);
}
__device__ __forceinline__ void tmem_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// Everything the four epilogues touch.
struct StepBlockParams {
    // activations
    const float* x;         // [M, D] the block's input
    uint16_t* gate;         // [M, D] bf16
    uint16_t* read;         // [M, 4C] bf16
    float* state;           // [M, 2C]
    float* y;               // [M, D] after the mixer, then the block's output (may be x)
    uint16_t* yb;           // [M, D] bf16
    uint16_t* act;          // [M, H] bf16
    uint16_t* xb;           // [M, D] bf16 of the input, then of the output
    float* read_sq;         // [M][tiles of the first product] partial sums of squares of the read row
    float* y_sq;            // [M][tiles of the second] of y
    // parameters
    const float* in_b;      // [5C] in the column order of the first product
    const float* par;       // [3, C]
    const float* out_b;     // [D]
    float read_eps, ff_eps;
    int M, D, C, H;
};

// (what other SMs wrote during this kernel is read from L2)
__device__ __forceinline__ Vec<4> load4_l2(const float* p) {
    const float4 a = __ldcg(reinterpret_cast<const float4*>(p));
    return Vec<4>{{a.x, a.y, a.z, a.w}};
}
__device__ __forceinline__ Vec<4> load4_l2(const uint16_t* p) {
    const uint2 w = __ldcg(reinterpret_cast<const uint2*>(p));
    return bf16x4_unpack(w.x, w.y);
}

// An epilogue: a unit is one slice (kSlice columns) of a row; the slices of a row are neighbouring lanes, so that
// what they read and write in global memory is contiguous. Slice index g counts over the whole matrix.
//   constants  parameters of a slice, into shared memory before the wait for the phase before it
//   fetch      what a unit needs from global memory, while the product still runs (kEarly: before that wait); for the
//              first kAhead units of a thread, which is all of them where K is split as far as it can be
//   run        the rest; returns the unit's sum of squares for the norm that follows
//   sum_table  where a row's sums of squares go, one per tile (kSums), and
//   table      where those of the norm before this product come from, `entries` a row (kScaled): the scale of the
//              row is rsqrt(their sum / features + eps)
struct EpiIn {  // slice: four channels' z_r | z_i | z_v, then eight gate features
    static constexpr int kSlice = 20, kSlices = 4, kConst = 32, kMaxSplit = 2;
    static constexpr int kAhead = 1;
    static constexpr bool kScaled = false, kEarly = true, kSums = true;
    struct Fetched {
        Vec<4> sr, si;
    };
    __device__ static float constant(const StepBlockParams& p, int g, int i) {  // 20 biases, 3 x 4 transition values
        if (g * 4 >= p.C) return 0.0f;
        return i < 20 ? p.in_b[g * 20 + i] : p.par[(i - 20) / 4 * p.C + g * 4 + (i - 20) % 4];
    }
    __device__ static float* sum_table(const StepBlockParams& p) { return p.read_sq; }
    __device__ static void fetch(const StepBlockParams& p, int row, int g, Fetched& f) {
        if (g * 4 >= p.C) return;
        const float* st = p.state + (size_t)row * 2 * p.C + g * 4;
        f.sr = load4_l2(st);
        f.si = load4_l2(st + p.C);
    }
    __device__ static float run(const StepBlockParams& p, int row, int g, const float* acc, float, const float* konst, Fetched& f) {
        const int c0 = g * 4, C = p.C;
        if (c0 >= C) return 0.0f;
        Vec<4> dr, di;
        float sq = 0.0f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const Gate gt = make_gate(acc[k] + konst[k], acc[4 + k] + konst[4 + k], acc[8 + k] + konst[8 + k]);
            float mr, mi;
            cmul(konst[20 + k], konst[24 + k], f.sr.v[k], f.si.v[k], mr, mi);
            const float bs = konst[28 + k] * gt.vac;
            f.sr.v[k] = (1.0f - gt.vac) * mr + bs * gt.inj_r;
            f.si.v[k] = (1.0f - gt.vac) * mi + bs * gt.inj_i;
            dr.v[k] = gt.vac * mr;
            di.v[k] = gt.vac * mi;
            sq += f.sr.v[k] * f.sr.v[k] + f.si.v[k] * f.si.v[k] + dr.v[k] * dr.v[k] + di.v[k] * di.v[k];
        }
        float* st = p.state + (size_t)row * 2 * C + c0;
        vec_store<4>(st, f.sr);
        vec_store<4>(st + C, f.si);
        uint16_t* o = p.read + (size_t)row * 4 * C + c0;
        store_bf16x4(o, f.sr);
        store_bf16x4(o + C, f.si);
        store_bf16x4(o + 2 * C, dr);
        store_bf16x4(o + 3 * C, di);
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            asm("cvt.rn.bf16x2.f32 %0, %1, %2;"
                : "=r"(w[k])
                : "f"(acc[13 + 2 * k] + konst[13 + 2 * k]), "f"(acc[12 + 2 * k] + konst[12 + 2 * k]));
        *reinterpret_cast<uint4*>(p.gate + (size_t)row * p.D + g * 8) = make_uint4(w[0], w[1], w[2], w[3]);
        return sq;
    }
};

// EpiOut and EpiFf come with tiles of 64 and of 32 features, and EpiUv with ten and five slices: the narrow ones
// where the wide ones would leave most of the GPU without a tile (up to 128 rows at d_model 1,024).
template <int SLICES>
struct EpiOut {  // slice: four features
    static constexpr int kSlice = 4, kSlices = SLICES, kConst = 4, kMaxSplit = 4;
    static constexpr int kAhead = SLICES > 8 ? 2 : 1;
    static constexpr bool kScaled = true, kEarly = false, kSums = true;
    struct Fetched {
        Vec<4> x, gate;
    };
    __device__ static float constant(const StepBlockParams& p, int g, int i) { return g * 4 < p.D ? p.out_b[g * 4 + i] : 0.0f; }
    __device__ static const float* table(const StepBlockParams& p) { return p.read_sq; }
    __device__ static float rstd(const StepBlockParams& p, float sum) { return rsqrtf(sum / (float)(4 * p.C) + p.read_eps); }
    __device__ static float* sum_table(const StepBlockParams& p) { return p.y_sq; }
    __device__ static void fetch(const StepBlockParams& p, int row, int g, Fetched& f) {
        if (g * 4 >= p.D) return;
        f.x = load4_l2(p.x + (size_t)row * p.D + g * 4);
        f.gate = load4_l2(p.gate + (size_t)row * p.D + g * 4);
    }
    __device__ static float run(const StepBlockParams& p, int row, int g, const float* acc, float rstd, const float* konst,
                                Fetched& f) {
        if (g * 4 >= p.D) return 0.0f;
        const size_t at = (size_t)row * p.D + g * 4;
        float sq = 0.0f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            f.x.v[k] += (acc[k] * rstd + konst[k]) * sigmoidf_fast(f.gate.v[k]);
            sq += f.x.v[k] * f.x.v[k];
        }
        vec_store<4>(p.y + at, f.x);
        store_bf16x4(p.yb + at, f.x);
        return sq;
    }
};

template <int SLICES>
struct EpiUv {  // slice: u of eight features, then v of the same
    static constexpr int kSlice = 16, kSlices = SLICES, kConst = 0, kMaxSplit = 2;
    static constexpr int kAhead = 0;
    static constexpr bool kScaled = true, kEarly = false, kSums = false;
    struct Fetched {};
    __device__ static const float* table(const StepBlockParams& p) { return p.y_sq; }
    __device__ static float rstd(const StepBlockParams& p, float sum) { return rsqrtf(sum / (float)p.D + p.ff_eps); }
    __device__ static void fetch(const StepBlockParams&, int, int, Fetched&) {}
    __device__ static float run(const StepBlockParams& p, int row, int g, const float* acc, float rstd, const float*, Fetched&) {
        if (g * 8 >= p.H) return 0.0f;
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            float a[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const float u = acc[q * 2 + k] * rstd, v = acc[8 + q * 2 + k] * rstd;
                a[k] = u * sigmoidf_fast(u) * v;
            }
            asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w[q]) : "f"(a[1]), "f"(a[0]));
        }
        *reinterpret_cast<uint4*>(p.act + (size_t)row * p.H + g * 8) = make_uint4(w[0], w[1], w[2], w[3]);
        return 0.0f;
    }
};

template <int SLICES>
struct EpiFf {  // slice: four features
    static constexpr int kSlice = 4, kSlices = SLICES, kConst = 0, kMaxSplit = 4;
    static constexpr int kAhead = SLICES > 8 ? 2 : 1;
    static constexpr bool kScaled = false, kEarly = false, kSums = false;
    struct Fetched {
        Vec<4> y;
    };
    __device__ static void fetch(const StepBlockParams& p, int row, int g, Fetched& f) {
        if (g * 4 < p.D) f.y = load4_l2(p.y + (size_t)row * p.D + g * 4);
    }
    __device__ static float run(const StepBlockParams& p, int row, int g, const float* acc, float, const float*, Fetched& f) {
        if (g * 4 >= p.D) return 0.0f;
        const size_t at = (size_t)row * p.D + g * 4;
#pragma unroll
        for (int k = 0; k < 4; ++k) f.y.v[k] += acc[k];
        vec_store<4>(p.y + at, f.y);
        store_bf16x4(p.xb + at, f.y);
        return 0.0f;
    }
};

constexpr int kStepPhases = 4, kStepCluster = 4;
constexpr int kStepMaxBlocks = 24;  // of the stack in one launch (kernel parameters)
constexpr int kStepSlotRows = 80;   // weight rows of a slot of their ring
constexpr size_t kStepSyncBytes = 512;  // four row tiles

// Column tiles of the four products, and how many slots their weights take per k-block.
template <bool NARROW>
struct StepShape {
    using In = EpiIn;
    using Out = EpiOut<NARROW ? 8 : 16>;
    using Uv = EpiUv<NARROW ? 5 : 10>;
    using Ff = EpiFf<NARROW ? 8 : 16>;
    template <class Epi>
    __host__ __device__ static constexpr int columns() { return Epi::kSlice * Epi::kSlices; }
    __host__ __device__ static constexpr int nt(int ph) {
        return ph == 0 ? columns<In>() : ph == 1 ? columns<Out>() : ph == 2 ? columns<Uv>() : columns<Ff>();
    }
    __host__ __device__ static constexpr int parts(int ph) { return (nt(ph) + kStepSlotRows - 1) / kStepSlotRows; }
    __host__ __device__ static constexpr int box(int ph) { return nt(ph) / parts(ph); }
    static constexpr int kAStages = 3, kBSlots = NARROW ? 5 : 4;
    static constexpr int kABox = kStepRows * 128, kBBox = kStepSlotRows * 128;
    static constexpr int kABytes = kABox * kStepKBoxes, kBBytes = kBBox * kStepKBoxes;
    // Partial sums of the rows that a block finishes, [source][column / 4][row] float4, rows padded to an odd number. Those of
    // the S - 1 other blocks have space of their own; the block's own go where its activations were.
    __host__ __device__ static constexpr int sums_bytes(int nt, int rows) { return nt / 4 * (rows + 1) * 16; }
    template <class Epi>
    static constexpr int recv() {
        return (Epi::kMaxSplit - 1) * sums_bytes(columns<Epi>(), kStepRows / Epi::kMaxSplit);
    }
    static constexpr int max2(int a, int b) { return a > b ? a : b; }
    static constexpr int kRecvBytes = max2(max2(max2(recv<In>(), recv<Out>()), max2(recv<Uv>(), recv<Ff>())),
                                           max2(sums_bytes(columns<Out>(), kStepRows / 2), sums_bytes(columns<Ff>(), kStepRows / 2)));
    static_assert(sums_bytes(columns<Uv>(), kStepRows) <= kAStages * kABytes && columns<Uv>() >= columns<In>() &&
                      columns<Uv>() >= columns<Out>(), "own sums");
    static constexpr int kConsts = 128;  // In: four slices of 32; Out: up to sixteen of 4
    static constexpr int kScaleBytes = kStepRows * 4;
    static constexpr int kBars = 2 * kAStages + 2 * kBSlots + 2 + 2 * kStepCluster + 3;
    static constexpr size_t kSmemBytes = 1024 + (size_t)kAStages * kABytes + (size_t)kBSlots * kBBytes + kRecvBytes +
                                         kScaleBytes + kConsts * 4 + kBars * 8 + 16;
    static_assert(kSmemBytes <= 227 * 1024, "shared memory of an SM");
    static_assert(In::kSlices * In::kConst <= kConsts && Out::kSlices * Out::kConst <= kConsts, "constants");
};
constexpr unsigned kStepColumns = 256;  // of tensor memory

struct StepPhase {
    int tiles_n, S, k_blocks, per;  // column tiles; K in S parts of `per` k-blocks
    int iters;                      // tiles that a block of a cluster takes, one after the other
};
struct alignas(64) StepWeights {
    CUtensorMap b[kStepPhases];
    const float *x, *in_b, *par, *out_b;
    float* state;
    float read_eps, ff_eps;
};
struct StepStackParams {
    CUtensorMap a[kStepPhases];
    StepWeights block[kStepMaxBlocks];
    StepPhase phase[kStepPhases];
    uint16_t *gate, *read, *yb, *act, *xb;
    float *y, *read_sq, *y_sq;
    unsigned* sync;  // finished parts of tiles (a block's) of each row tile, 32 words apart, or null: one phase alone
    int M, D, C, H;
    int a_rows;                            // rows of a box of activations
    int row_tiles, groups, group_clusters; // clusters of a group serve the same row tiles
    int first, last;                       // phases of this launch, counted over the blocks of the stack
};

// Waits until `count` parts of tiles are finished, with a bound (2^22 polls are seconds).
__device__ __forceinline__ void wait_for_tiles(const unsigned* p, unsigned count, bool& dead) {
    for (unsigned tries = 0; !dead; ++tries) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
        if (v >= count) return;
        dead = tries >= (1u << 22);
    }
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_at(unsigned peer_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(peer_bar) : "memory");
}
// One thread of a converged warp, in a way that the compiler knows to be one.
__device__ __forceinline__ bool elect_one() {
    unsigned one;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(one));
    return one != 0;
}
__device__ __forceinline__ void epilogue_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

// A block of a cluster and its shared memory.
struct StepCta {
    char *a, *b, *recv;
    float *scale, *konst;  // of a row that this block finishes; constants of the tile's slices
    // barriers: rings of activations and weights (full, empty); product done; partial sums here; receiving
    // buffer of each peer free again after an even and after an odd iteration (a peer may be an iteration
    // ahead of this block's wait, and a parity tells no more than two states apart); phase ready, phase
    // left, tensor memory free
    unsigned a_full, a_empty, b_full, b_empty, done, got, freed, ready, left, tmem_free;
    volatile int* dead;  // the wait for a phase has run out
    unsigned tmem;
    int rank, cluster_of_group;
};
// The tile of this block in iteration `it` of a phase, or -1.
__device__ __forceinline__ int step_tile(const StepStackParams& p, const StepPhase& h, const StepCta& c, int it) {
    const int tile = (it * p.group_clusters + c.cluster_of_group) * (kStepCluster / h.S) + c.rank / h.S;
    return tile < h.tiles_n ? tile : -1;
}
__device__ __forceinline__ int step_k(const StepPhase& h, int r) {  // k-blocks of part r: > 0, the host chose S so
    const int left = h.k_blocks - r * h.per;
    return left < h.per ? left : h.per;
}

// Counts of an epilogue thread over the whole launch; their parities are those of the barriers.
struct StepCounts {
    unsigned phases = 0, iters = 0, items = 0, sums = 0;
    bool dead = false;
};

// Place of four columns among the partial sums: the first four of all slices, then the next, so that neighbouring
// lanes (the slices of a row) read neighbouring banks (rows are an odd number of 16 bytes apart).
template <class Epi>
__device__ __forceinline__ int step_line(int four) {
    constexpr int kFours = Epi::kSlice / 4;
    return four % kFours * Epi::kSlices + four / kFours;
}
template <class Epi>
__device__ __forceinline__ void step_epilogue(const StepStackParams& p, const StepBlockParams& bp, const StepPhase& h,
                                              const StepCta& c, int row_tile, int entries, StepCounts& n) {
    constexpr int kSlice = Epi::kSlice, kSlices = Epi::kSlices, kColumns = kSlice * kSlices;
    constexpr int kThreads = 2 * kStepRows, kAhead = Epi::kAhead;  // units of a thread whose inputs are fetched ahead
    const int tid = threadIdx.x, S = h.S, r = c.rank % S, first = c.rank - r;
    const int m0 = row_tile * kStepRows, rows = p.M - m0 < kStepRows ? p.M - m0 : kStepRows;
    // each of the S blocks finishes `per` rows of the tile (the last ones perhaps fewer, or none)
    const int per = (rows + S - 1) / S, row0 = r * per, mine = rows - row0 < per ? (rows > row0 ? rows - row0 : 0) : per;
    const int units = mine * kSlices, pitch = per | 1;
    for (int it = 0; it < h.iters; ++it, ++n.iters) {
        const int tile = step_tile(p, h, c, it), g0 = tile * kSlices;
        typename Epi::Fetched fetched[kAhead > 0 ? kAhead : 1];
        auto fetch = [&] {
#pragma unroll
            for (int i = 0; i < kAhead; ++i) {
                const int u = i * kThreads + tid;
                if (u < units) Epi::fetch(bp, m0 + row0 + u / kSlices, g0 + u % kSlices, fetched[i]);
            }
        };
        if (tile >= 0) {
            if constexpr (Epi::kConst > 0) {
                for (int i = tid; i < kSlices * Epi::kConst; i += kThreads)
                    c.konst[i] = Epi::constant(bp, g0 + i / Epi::kConst, i % Epi::kConst);
            }
            if constexpr (Epi::kEarly) fetch();
        }
        if (n.iters > 0) {  // the peers have read what was sent to them in the iteration before
            const unsigned last = n.iters - 1;
            const int j = tid & 31;
            bool late = n.dead;
            if (j < kStepCluster && j != c.rank) mbar_wait(c.freed + (last % 2 * kStepCluster + j) * 8, last / 2 & 1, late);
            n.dead = __any_sync(0xffffffffu, late);
        }
        if (it == 0) {
            mbar_wait_local(c.ready, n.phases++ & 1, n.dead);
            n.dead = n.dead || *c.dead;
        }
        if (tile >= 0) {
            if constexpr (!Epi::kEarly) fetch();
            if constexpr (Epi::kScaled) {  // kThreads / per threads add a row's sums of squares
                constexpr int kLanes = 8;
                for (int at = 0; at < mine; at += kThreads / kLanes) {
                    const int rl = at + tid / kLanes;
                    float sum = 0.0f;
                    if (rl < mine) {
                        const float* t = Epi::table(bp) + (size_t)(m0 + row0 + rl) * entries;
#pragma unroll 4
                        for (int i = tid % kLanes; i < entries; i += kLanes) sum += __ldcg(t + i);
                    }
#pragma unroll
                    for (int off = kLanes / 2; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
                    if (rl < mine && tid % kLanes == 0) c.scale[rl] = Epi::rstd(bp, sum);
                }
            }
            if (tid == 0 && S > 1 && !n.dead) mbar_expect(c.got, (unsigned)((S - 1) * mine * kColumns * 4));
            // (where the sums go is worked out under the product: 476 -> 471 us for 18 blocks of d_model 1,024 at 256 rows, 318 ->
            // 312 at 1)
            constexpr int kHalf = kColumns / 2;
            const int row = tid % kStepRows, to = row / per, rl = row - to * per, col0 = tid / kStepRows * kHalf;
            const int src = r > to ? r - 1 : r;
            float4* own = reinterpret_cast<float4*>(c.a) + rl;
            const unsigned peer = first + (row < rows ? to : r), bar = peer_addr(c.got, peer);
            const unsigned at = peer_addr(smem_addr(c.recv) + (unsigned)((src * (kColumns / 4) * pitch + rl) * 16), peer);
            const unsigned lane_addr = c.tmem + ((unsigned)(row & ~31) << 16) + (unsigned)col0;
            mbar_wait_local(c.done, n.items & 1, n.dead);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            {   // the product's rows to the blocks that finish them; two warps share a quarter of the lanes
                const bool send = row < rows && to != r && !n.dead;  // (nothing after a wait that ran out)
                constexpr int kStep = kHalf % 16 == 0 ? 16 : 8;
#pragma unroll
                for (int k0 = 0; k0 < kHalf; k0 += kStep) {
                    unsigned v[kStep];
                    __syncwarp();
                    tmem_load<kStep>(lane_addr + k0, v);
                    tmem_wait();
#pragma unroll
                    for (int k = 0; k < kStep; k += 4) {
                        const int line = step_line<Epi>((col0 + k0 + k) / 4) * pitch;
                        const float4 w = make_float4(__uint_as_float(v[k]), __uint_as_float(v[k + 1]),
                                                     __uint_as_float(v[k + 2]), __uint_as_float(v[k + 3]));
                        if (send) send4(at + (unsigned)line * 16, w.x, w.y, w.z, w.w, bar);
                        else if (row < rows) own[line] = w;
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            epilogue_sync();
            if (S > 1) mbar_wait(c.got, n.sums++ & 1, n.dead);
            __syncwarp();
            auto finish = [&](int u, typename Epi::Fetched& f) {
                const int rl = u / kSlices, s = u % kSlices;
                float sq = 0.0f;
                if (u < units) {
                    float acc[kSlice];
#pragma unroll
                    for (int k = 0; k < kSlice; k += 4) {
                        const int line = (k / 4 * kSlices + s) * pitch + rl;
                        float4 w = reinterpret_cast<const float4*>(c.a)[line];
                        // (of constant length: as a loop over S - 1 every source was waited for before the next one's load
                        // went out; 18 blocks of d_model 1,024 525 us instead of 486 at 256 rows, 367 and 328 at 1)
#pragma unroll
                        for (int src = 0; src < Epi::kMaxSplit - 1; ++src) {
                            if (src >= S - 1) continue;
                            const float4 o = reinterpret_cast<const float4*>(c.recv)[src * (kColumns / 4) * pitch + line];
                            w.x += o.x; w.y += o.y; w.z += o.z; w.w += o.w;
                        }
                        acc[k] = n.dead ? nanf("") : w.x;
                        acc[k + 1] = n.dead ? nanf("") : w.y;
                        acc[k + 2] = n.dead ? nanf("") : w.z;
                        acc[k + 3] = n.dead ? nanf("") : w.w;
                    }
                    sq = Epi::run(bp, m0 + row0 + rl, g0 + s, acc, Epi::kScaled ? c.scale[rl] : 1.0f,
                                  c.konst + s * Epi::kConst, f);
                }
                if constexpr (Epi::kSums) {  // over the lanes of the row
#pragma unroll
                    for (int off = kSlices / 2; off > 0; off >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, off);
                    if (u < units && s == 0) Epi::sum_table(bp)[(size_t)(m0 + row0 + rl) * h.tiles_n + tile] = sq;
                }
            };
#pragma unroll
            for (int i = 0; i < kAhead; ++i)
                if (i * kThreads < units) finish(i * kThreads + tid, fetched[i]);
#pragma unroll 1
            for (int i = kAhead; i * kThreads < units; ++i) {
                const int u = i * kThreads + tid;
                if (u < units) Epi::fetch(bp, m0 + row0 + u / kSlices, g0 + u % kSlices, fetched[0]);
                finish(u, fetched[0]);
            }
            ++n.items;
            // (the space of the block's own sums is written by its next loads)
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        epilogue_sync();
        if (tid == 0) {
            if (tile >= 0) mbar_arrive(c.tmem_free);
            // One addition per block: with one per warp, up to 1,152 to the same word and as many waits for the stores before
            // them, 18 blocks of d_model 1,024 took 426 us at 1 row, 491 at 100 and 596 at 256; 404, 467 and 578 with one, and 363,
            // 409 and 525 with the arrivals at the peers, 300 cycles each behind the addition's 1,000, by other warps and the proxy
            // fence for what is stored by the reader. (Polls without acquire and a fence behind the last: 33 us more; two polls in
            // flight: 35; polls that begin 800 to 2,400 cycles later: the same; two warps that do nothing but this: 15 at 1 row.)
            if (p.sync && tile >= 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p.sync + row_tile * 32) : "memory");
        }
        if (tid >= 32 && tid % 32 == 0 && tid < 32 * (1 + kStepCluster)) {  // a warp per peer
            const int j = tid / 32 - 1;
            if (j != c.rank) mbar_arrive_at(peer_addr(c.freed + (n.iters % 2 * kStepCluster + c.rank) * 8, j));
        }
        if (tid == 32 * 5 && it + 1 == h.iters) mbar_arrive(c.left);
    }
}

// The three single threads that feed the tensor cores walk the same phases, tiles and k-blocks. They are elected
// (elect.sync): of a thread picked by its index the compiler does not know that it is alone, and a product or a
// load took 200 to 480 cycles to issue.
enum { kStepWeights, kStepActivations, kStepProducts };
// A place in a ring of barriers: the parity is that of its present use.
template <int N>
struct StepRing {
    unsigned slot = 0, parity = 0, used = 0;
    __device__ void next() {
        ++used;
        if (++slot == N) {
            slot = 0;
            parity ^= 1;
        }
    }
    // (a producer waits for the use before this one)
    __device__ bool fresh() const { return used < N; }
};
template <bool NARROW, int ROLE>
__device__ __forceinline__ void step_feed(const StepStackParams& p, const StepCta& c, int group) {
    using T = StepShape<NARROW>;
    bool dead = false;
    StepRing<T::kAStages> ar;
    StepRing<T::kBSlots> br;
    unsigned items = 0, phases = 0;
    for (int m = group; m < p.row_tiles; m += p.groups) {
        unsigned target = 0;
        for (int q = p.first; q < p.last; ++q) {
            const int ph = q % kStepPhases, parts = T::parts(ph), box = T::box(ph);
            const StepPhase& h = p.phase[ph];
            const int r = c.rank % h.S, count = step_k(h, r), k0 = r * h.per, iters = h.iters;
            const int first_tile = step_tile(p, h, c, 0);
            if constexpr (ROLE == kStepActivations) {
                if (phases > 0) mbar_wait_local(c.left, (phases - 1) & 1, dead);
                ++phases;
                // What does not depend on the phase before is done ahead of the wait for it (with the products' wait for weights
                // ahead of that for activations 487 -> 476 us for 18 blocks of d_model 1,024 at 256 rows, 327 -> 319 at 1).
                if (first_tile >= 0 && !dead)
                    for (int i = 0; i < count && i < T::kAStages; ++i)
                        mbar_expect(c.a_full + (ar.slot + i) % T::kAStages * 8, (unsigned)p.a_rows * 128 * kStepKBoxes);
                if (p.sync && q > p.first) {
                    wait_for_tiles(p.sync + m * 32, target, dead);
                    if (dead) *c.dead = 1;
                    asm volatile("fence.proxy.async.global;" ::: "memory");  // (stored by lanes, read by TMA)
                }
                target += (unsigned)(h.tiles_n * h.S);
                mbar_arrive(c.ready);
            }
            for (int it = 0; it < iters; ++it) {
                const int tile = it == 0 ? first_tile : step_tile(p, h, c, it);
                if (tile < 0) continue;
                if constexpr (ROLE == kStepWeights) {
                    const CUtensorMap* map = &p.block[q / kStepPhases].b[ph];
                    const int n0 = tile * T::nt(ph);
                    for (int i = 0; i < count; ++i)
                        for (int part = 0; part < parts; ++part) {
                            if (!br.fresh()) mbar_wait_local(c.b_empty + br.slot * 8, br.parity ^ 1, dead);
                            if (dead) continue;
                            mbar_expect(c.b_full + br.slot * 8, (unsigned)box * 128 * kStepKBoxes);
#pragma unroll
                            for (int x = 0; x < kStepKBoxes; ++x)
                                tma_load2(smem_addr(c.b + br.slot * T::kBBytes + x * T::kBBox), map,
                                          (k0 + i) * kStepKBlock + x * kStepKBox, n0 + part * box, c.b_full + br.slot * 8);
                            br.next();
                        }
                } else if constexpr (ROLE == kStepActivations) {
                    const CUtensorMap* map = &p.a[ph];
                    const unsigned bytes = (unsigned)p.a_rows * 128 * kStepKBoxes;
                    // the epilogue has done with the tile before, and with it the products: all stages are free
                    // (c.left says so for the first tile of a phase)
                    if (it > 0 && items > 0) mbar_wait_local(c.tmem_free, (items - 1) & 1, dead);
                    ++items;
                    for (int i = 0; i < count; ++i) {
                        if (i >= T::kAStages) mbar_wait_local(c.a_empty + ar.slot * 8, ar.parity ^ 1, dead);
                        if (dead) continue;
                        if (it > 0 || i >= T::kAStages) mbar_expect(c.a_full + ar.slot * 8, bytes);
#pragma unroll
                        for (int x = 0; x < kStepKBoxes; ++x)
                            tma_load2(smem_addr(c.a + ar.slot * T::kABytes + x * T::kABox), map,
                                      (k0 + i) * kStepKBlock + x * kStepKBox, m * kStepRows, c.a_full + ar.slot * 8);
                        ar.next();
                    }
                } else {
                    const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(box >> 3) << 17) |
                                           ((unsigned)(kStepRows >> 4) << 24);
                    if (items > 0) mbar_wait_local(c.tmem_free, (items - 1) & 1, dead);
                    if (dead) continue;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    ++items;
                    // A wait takes 165 cycles even where there is nothing to wait for, about as long as the eight
                    // products between two of them, so it is tried ahead: operands of the next part before the products
                    // of this one.
                    bool here = false;
                    for (int i = 0; i < count; ++i) {
                        for (int part = 0; part < parts; ++part) {
                            const unsigned as = ar.slot, bs = br.slot;
                            if (!here) {
                                mbar_wait_local(c.b_full + bs * 8, br.parity, dead);  // (there long before)
                                if (part == 0) mbar_wait_local(c.a_full + as * 8, ar.parity, dead);
                            }
                            if (dead) continue;
                            const bool last_part = part + 1 == parts;
                            br.next();
                            if (last_part) ar.next();
                            here = false;
                            if (!last_part || i + 1 < count) {
                                here = mbar_try<false>(c.b_full + br.slot * 8, br.parity);
                                if (last_part) here = mbar_try<false>(c.a_full + ar.slot * 8, ar.parity) && here;
                            }
                            const unsigned long long a = step_desc(smem_addr(c.a + as * T::kABytes)),
                                                     b = step_desc(smem_addr(c.b + bs * T::kBBytes));
#pragma unroll
                            for (int x = 0; x < kStepKBoxes; ++x)
#pragma unroll
                                for (int k = 0; k < kStepKBox / 16; ++k)  // 16 of K: 32 bytes further in the swizzle atom
                                    step_mma(c.tmem + (unsigned)(part * box), a + x * (T::kABox >> 4) + 2 * k,
                                             b + x * (T::kBBox >> 4) + 2 * k, idesc, i > 0 || x > 0 || k > 0);
                            step_commit(c.b_empty + bs * 8);
                            if (last_part) step_commit(c.a_empty + as * 8);
                        }
                    }
                    if (!dead) step_commit(c.done);
                }
            }
        }
    }
    if (dead && ROLE != kStepProducts) {  // a wait has run out: what is still on its way arrives before the block leaves
        const unsigned full = ROLE == kStepWeights ? c.b_full : c.a_full,
                       slots = ROLE == kStepWeights ? T::kBSlots : T::kAStages,
                       issued = ROLE == kStepWeights ? br.used : ar.used;
        bool late = false;
        for (unsigned i = issued > slots ? issued - slots : 0; i < issued; ++i)
            mbar_wait_local(full + i % slots * 8, i / slots & 1, late);
    }
}

template <bool NARROW>
__global__ void __launch_bounds__(kStepThreads, 1) step_stack(const __grid_constant__ StepStackParams p) {
    using T = StepShape<NARROW>;
    extern __shared__ __align__(1024) char step_smem[];
    StepCta c;
    c.a = step_smem + (1024 - (smem_addr(step_smem) & 1023)) % 1024;
    c.b = c.a + T::kAStages * T::kABytes;
    c.recv = c.b + T::kBSlots * T::kBBytes;
    c.scale = reinterpret_cast<float*>(c.recv + T::kRecvBytes);
    c.konst = c.scale + T::kScaleBytes / 4;
    char* tail = reinterpret_cast<char*>(c.konst + T::kConsts);
    c.a_full = smem_addr(tail);
    c.a_empty = c.a_full + T::kAStages * 8;
    c.b_full = c.a_empty + T::kAStages * 8;
    c.b_empty = c.b_full + T::kBSlots * 8;
    c.done = c.b_empty + T::kBSlots * 8;
    c.got = c.done + 8;
    c.freed = c.got + 8;
    c.ready = c.freed + 2 * kStepCluster * 8;
    c.left = c.ready + 8;
    c.tmem_free = c.left + 8;
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(tail + T::kBars * 8);
    c.dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
    c.rank = (int)cluster_rank();
    const int cluster = (int)blockIdx.x / kStepCluster, group = cluster % p.groups;
    c.cluster_of_group = cluster / p.groups;
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);

    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2 * T::kAStages + 2 * T::kBSlots; ++i) mbar_init(c.a_full + i * 8, 1);
        mbar_init(c.done, 1);
        mbar_init(c.got, 1);
        for (int j = 0; j < 2 * kStepCluster; ++j) mbar_init(c.freed + j * 8, 1);
        mbar_init(c.ready, 1);
        mbar_init(c.left, 1);
        mbar_init(c.tmem_free, 1);
        *c.dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(kStepColumns)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();  // the peers' barriers are ready
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    c.tmem = *tmem_slot;

    if (warp < 8) {
        StepCounts n;
        for (int m = group; m < p.row_tiles; m += p.groups) {
            for (int q = p.first; q < p.last; ++q) {
                const int ph = q % kStepPhases;
                const StepWeights& w = p.block[q / kStepPhases];
                const StepBlockParams bp{w.x, p.gate, p.read, w.state, p.y, p.yb, p.act, p.xb, p.read_sq, p.y_sq,
                                         w.in_b, w.par, w.out_b, w.read_eps, w.ff_eps, p.M, p.D, p.C, p.H};
                if (ph == 0) step_epilogue<typename T::In>(p, bp, p.phase[0], c, m, 0, n);
                else if (ph == 1) step_epilogue<typename T::Out>(p, bp, p.phase[1], c, m, p.phase[0].tiles_n, n);
                else if (ph == 2) step_epilogue<typename T::Uv>(p, bp, p.phase[2], c, m, p.phase[1].tiles_n, n);
                else step_epilogue<typename T::Ff>(p, bp, p.phase[3], c, m, 0, n);
            }
        }
    } else if (warp == 8) {
        if (elect_one()) step_feed<NARROW, kStepWeights>(p, c, group);
    } else if (warp == 9) {
        if (elect_one()) step_feed<NARROW, kStepActivations>(p, c, group);
    } else {
        if (elect_one()) step_feed<NARROW, kStepProducts>(p, c, group);
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();  // nothing is sent to a block that has left
    if (warp == 8) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(c.tmem), "r"(kStepColumns) : "memory");
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
        const int g = r / 20, q = r % 20;
        const int from = q < 12 ? q / 4 * C + g * 4 + q % 4 : g * 8 + q - 12;
        src = (q < 12 ? p.write_w : p.gate_w) + (size_t)from * D;
        dst = p.in_w + (size_t)r * D;
        if (threadIdx.x == 0) p.in_b[r] = (q < 12 ? p.write_b : p.gate_b)[from];
    } else {
        r -= 5 * C;
        const int h = r / 16 * 8 + r % 8;
        src = h < p.H ? p.w12 + (size_t)(r % 16 < 8 ? h : p.H + h) * D : nullptr;
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
