// Single-token step of a Field block as four kernels, one per phase of field_step_gemm.cuh with its weights in the same
// order: each is a matrix product on the tensor cores (tcgen05.mma, operands by TMA, accumulator in tensor memory)
// whose epilogue goes on to the operand of the next.
//
// For single blocks, for devices that do not hold the cooperative launch of a stack, and for stacks of d_model 64 at 65 to 256
// rows: there a phase is one tile, whose K cannot be split, so that a thread block finishes 128 rows by itself, and that and the
// hand-over through global memory cost more than a launch that was let in ahead. Eight blocks: d_model 64 at 128 rows 162 us,
// as one launch 173; 128 175 and 165, 256 at 16 and 512 rows 173 and 149, 187 and 159. What is done about a launch:
//   - the next kernel is let in at the start (dependent launch) and loads its weights before it waits for
//     this one, as far as SMs are free for it;
//   - K is split over a cluster of S blocks; each then owns 1/S of the tile's columns, to which the others send
//     their partial sums through distributed shared memory (field_dsmem.cuh);
//   - a thread has a row, straight from tensor memory.
//
// Tile: 128 rows (batch) x NT columns. Operands are K-major with the 128-byte swizzle: a k-block is 64 bf16 = 128 bytes per
// row. Waits are bounded; after one that ran out the results are NaN. Device only; rows past the batch and columns past the
// matrix are zero-filled by TMA and not stored.
#pragma once

#include "field_step_gemm.cuh"

#ifndef FIELDS_HOST_EMU

namespace fields {

constexpr int kPhaseThreads = 160;  // four epilogue warps and one that issues loads and products

__device__ __forceinline__ void send1(unsigned dst, float x, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(dst), "f"(x), "r"(bar)
                 : "memory");
}
// (read_sq is [C / 8][M] and y_sq [D / 8][M] here: a slice's sums of squares of all rows are adjacent)
struct PhaseParams : StepBlockParams {
    int tiles_n, S, k_blocks;
    int wait_first;  // non-zero: parameters are read, and the next kernel let in, after the kernels before this one
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
struct PhaseIn {  // slice: twice four channels' z_r | z_i | z_v and then eight gate features
    static constexpr int kSlice = 40, kSlices = 2, kMaxSplit = 2, kStages = 7, kConst = 64;
    static constexpr bool kScaled = false;
    struct Fetched {
        float sr[8], si[8];
    };
    __device__ static float constant(const PhaseParams& p, int g, int i) {  // 40 biases, 3 x 8 transition values
        if (g * 8 >= p.C) return 0.0f;
        return i < 40 ? p.in_b[g * 40 + i] : p.par[(i - 40) / 8 * p.C + g * 8 + (i - 40) % 8];
    }
    __device__ static float share(const PhaseParams&, int, int, int) { return 0.0f; }
    __device__ void scale(const PhaseParams&, float) {}
    __device__ void fetch(const PhaseParams& p, int row, int g, Fetched& f) {
        if (g * 8 >= p.C) return;
        const float* st = p.state + (size_t)row * 2 * p.C + g * 8;
        load8(st, f.sr);
        load8(st + p.C, f.si);
    }
    __device__ void run(const PhaseParams& p, int row, int g, const float* acc, const float* konst, Fetched& f) {
        const int c0 = g * 8, C = p.C;
        if (c0 >= C) return;
        float dr[8], di[8], sq = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int at = k / 4 * 20 + k % 4;
            const Gate gt = make_gate(acc[at] + konst[at], acc[at + 4] + konst[at + 4], acc[at + 8] + konst[at + 8]);
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
            for (int k = 0; k < 8; ++k) v[k] = acc[12 + h * 20 + k] + konst[12 + h * 20 + k];
            store8(p.gate + (size_t)row * p.D + g * 16 + h * 8, v);
        }
    }
};

// PhaseOut and PhaseFf come with tiles of 64 and of 32 features (and PhaseUv with ten and five slices). Where 64 leave so
// few tiles that K would be split over clusters of eight, 32 with clusters of four are faster: a kernel's clusters of
// eight took up to 14 us to get started.
template <int SLICES>
struct PhaseOut {  // slice: eight features
    static constexpr int kSlice = 8, kSlices = SLICES, kMaxSplit = SLICES, kStages = 7, kConst = 8;
    static constexpr bool kScaled = true;
    struct Fetched {
        float x[8], gate[8];
    };
    float rstd;
    __device__ static float constant(const PhaseParams& p, int g, int i) { return g * 8 < p.D ? p.out_b[g * 8 + i] : 0.0f; }
    __device__ static float share(const PhaseParams& p, int row, int rank, int S) {
        return table_share(p.read_sq, p.C / 8, p.M, row, rank, S);
    }
    __device__ void scale(const PhaseParams& p, float sum) { rstd = rsqrtf(sum / (float)(4 * p.C) + p.read_eps); }
    __device__ void fetch(const PhaseParams& p, int row, int g, Fetched& f) {
        if (g * 8 >= p.D) return;
        load8(p.x + (size_t)row * p.D + g * 8, f.x);
        load8(p.gate + (size_t)row * p.D + g * 8, f.gate);
    }
    __device__ void run(const PhaseParams& p, int row, int g, const float* acc, const float* konst, Fetched& f) {
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
struct PhaseUv {  // slice: u of eight features, then v of the same
    static constexpr int kSlice = 16, kSlices = SLICES, kMaxSplit = SLICES == 10 ? 4 : 2, kStages = SLICES == 10 ? 4 : 7, kConst = 0;
    static constexpr bool kScaled = true;
    struct Fetched {};
    float rstd;
    __device__ static float constant(const PhaseParams&, int, int) { return 0.0f; }
    __device__ static float share(const PhaseParams& p, int row, int rank, int S) {
        return table_share(p.y_sq, p.D / 8, p.M, row, rank, S);
    }
    __device__ void scale(const PhaseParams& p, float sum) { rstd = rsqrtf(sum / (float)p.D + p.ff_eps); }
    __device__ void fetch(const PhaseParams&, int, int, Fetched&) {}
    __device__ void run(const PhaseParams& p, int row, int g, const float* acc, const float*, Fetched&) {
        if (g * 8 >= p.H) return;
        float a[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float u = acc[k] * rstd, v = acc[8 + k] * rstd;
            a[k] = u * sigmoidf_fast(u) * v;
        }
        store8(p.act + (size_t)row * p.H + g * 8, a);
    }
};

template <int SLICES>
struct PhaseFf {  // slice: eight features
    static constexpr int kSlice = 8, kSlices = SLICES, kMaxSplit = SLICES, kStages = 7, kConst = 0;
    static constexpr bool kScaled = false;
    struct Fetched {
        float y[8];
    };
    __device__ static float constant(const PhaseParams&, int, int) { return 0.0f; }
    __device__ static float share(const PhaseParams&, int, int, int) { return 0.0f; }
    __device__ void scale(const PhaseParams&, float) {}
    __device__ void fetch(const PhaseParams& p, int row, int g, Fetched& f) {
        if (g * 8 < p.D) load8(p.y + (size_t)row * p.D + g * 8, f.y);
    }
    __device__ void run(const PhaseParams& p, int row, int g, const float* acc, const float*, Fetched& f) {
        if (g * 8 >= p.D) return;
        const size_t at = (size_t)row * p.D + g * 8;
#pragma unroll
        for (int k = 0; k < 8; ++k) f.y[k] += acc[k];
        store8(p.y + at, f.y);
        store8(p.xb + at, f.y);
    }
};

template <class Epi>
struct PhaseTile {
    static constexpr int kNT = Epi::kSlice * Epi::kSlices;
    static constexpr int kABytes = kStepRows * 128, kBBytes = kNT * 128, kStageBytes = kABytes + kBBytes;
    static constexpr unsigned kColumns = kNT <= 64 ? 64 : kNT <= 128 ? 128 : 256;  // of tensor memory
    static constexpr int kOperandBytes = Epi::kStages * kStageBytes;
    // what S - 1 blocks send, [src][column / 4][row] float4; most for the largest S
    static constexpr int kRecvBytes =
        (Epi::kMaxSplit - 1) * ((Epi::kSlices + Epi::kMaxSplit - 1) / Epi::kMaxSplit) * Epi::kSlice * kStepRows * 4;
    static constexpr int kShareBytes = Epi::kScaled ? Epi::kMaxSplit * kStepRows * 4 : 0;
    static constexpr int kConstBytes = Epi::kSlices * Epi::kConst * 4;
    static constexpr size_t kSmemBytes =
        1024 + (size_t)kOperandBytes + kRecvBytes + kShareBytes + kConstBytes + (2 * Epi::kStages + 2) * 8 + 16;
    static_assert(kSmemBytes <= 227 * 1024, "shared memory of an SM");
    static_assert(kNT % 16 == 0 && kNT <= 256 && kBBytes % 1024 == 0, "a tile the tensor cores take");
};

template <class Epi>
__global__ void __launch_bounds__(kPhaseThreads, 1)
    step_phase(const __grid_constant__ CUtensorMap a_map, const __grid_constant__ CUtensorMap b_map,
              const PhaseParams p) {
    using T = PhaseTile<Epi>;
    constexpr int kStages = Epi::kStages, kSlice = Epi::kSlice;
    extern __shared__ __align__(1024) char phase_smem[];
    char* base = phase_smem + (1024 - (smem_addr(phase_smem) & 1023)) % 1024;
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
    const int own = (Epi::kSlices + S - 1) / S;                          // slices a block finishes, the last perhaps fewer
    auto owned = [&](int j) { return Epi::kSlices - j * own < own ? Epi::kSlices - j * own : own; };
    const int mine = owned(rank), g0 = n_tile * Epi::kSlices + rank * own;
    const bool control = tid == 4 * 32;
    bool dead = false;

    auto stage_a = [&](int i) { return smem_addr(base + (i % kStages) * T::kStageBytes); };
    auto load_b = [&](int i) {
        mbar_expect(full + (i % kStages) * 8, T::kStageBytes);
        tma_load2(stage_a(i) + T::kABytes, &b_map, (kb0 + i) * kStepKBox, n_tile * T::kNT, full + (i % kStages) * 8);
    };
    auto load_a = [&](int i) {
        tma_load2(stage_a(i), &a_map, (kb0 + i) * kStepKBox, m0, full + (i % kStages) * 8);
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
        if (S > 1) mbar_expect(got, (unsigned)((S - 1) * (mine * kSlice + (Epi::kScaled ? 1 : 0)) * kStepRows * 4));
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
        for (int i = tid; i < mine * Epi::kConst; i += kPhaseThreads)
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
        int issued = kStages < count ? kStages : count;
        for (int i = 0; i < count; ++i) {
            mbar_wait(full + (i % kStages) * 8, (i / kStages) & 1, dead);
            if (dead) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned long long a = step_desc(stage_a(i)), b = step_desc(stage_a(i) + T::kABytes);
#pragma unroll
            for (int k = 0; k < kStepKBox / 16; ++k)  // 16 of K: 32 bytes further in the swizzle atom
                step_mma(tmem, a + 2 * k, b + 2 * k, idesc, i > 0 || k > 0);
            step_commit(empty + (i % kStages) * 8);
            // refill the stage of the product before this one
            const int j = i - 1 + kStages;
            if (i > 0 && j < count) {
                mbar_wait(empty + ((i - 1) % kStages) * 8, ((i - 1) / kStages) & 1, dead);
                if (dead) break;
                load_b(j);
                load_a(j);
                ++issued;
            }
        }
        if (!dead) {
            step_commit(done);
        } else {  // what is still on its way arrives before the block leaves
            bool late = false;
            for (int i = issued > kStages ? issued - kStages : 0; i < issued; ++i)
                mbar_wait(full + (i % kStages) * 8, (i / kStages) & 1, late);
        }
    } else if (row_ok) {
#pragma unroll
        for (int q = 0; q < kAhead; ++q)
            if (q < mine) epi.fetch(p, row, g0 + q, fetched[q]);
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
        // the other blocks' columns, each block starting with its neighbour (after a wait that ran out nothing is sent: theirs
        // run out as well)
        for (int d = 1; d < S && !__any_sync(0xffffffffu, dead); ++d) {
            const int j = (rank + d) % S, src = rank > j ? rank - 1 : rank;
            const unsigned bar = peer_addr(got, j);
            const unsigned at = peer_addr(smem_addr(recv) + (unsigned)((src * own * kSlice / 4 * kStepRows + tid) * 16), j);
            if constexpr (Epi::kScaled) send1(peer_addr(smem_addr(shares + rank * kStepRows + tid), j), share, bar);
            for (int q = 0; q < owned(j); ++q) {
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
            if (q < mine) finish(q, fetched[q]);
        for (int q = kAhead; q < mine; ++q) {
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
    // (a block that has given up stays until the others have left: they may still send to it)
    if (S > 1 && dead) asm volatile("barrier.cluster.arrive;\n\tbarrier.cluster.wait;" ::: "memory");
}

}  // namespace fields

#endif  // FIELDS_HOST_EMU
