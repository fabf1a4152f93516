// Real-valued first-order scan  s_t = a_t s_{t-1} + x_t  over [B, L, C], forward and backward.
//
// The second call site of the reference's scan primitive: `hierarchical_scan(a, drive, block=32)`
// (field_only_v4_chunked_triton_wiki100.py:347-391) as the softpatch mixer calls it on a rank-64
// state (official_source/field_hybrid_speed_optimization_v6.py:333-335), where `a` is one decay per
// token broadcast over the channels. The reference computes it with a log-depth doubling scan
// inside blocks of 32 and a second doubling scan over the blocks.
//
// The tensors of this call site are a few MB, so a launch and a round trip through memory count: the
// earlier form (chunk maps, carries, states: three launches, the carries by one thread per channel)
// took 16 us forward and 21 us backward at 8 x 2,048 x 64, most of it the serial carries. Here each
// direction is ONE launch: a cluster of Q blocks owns a chain (a batch row of 32 channels, a lane per
// channel, so that a row is one 128-byte line per warp) and walks it in super-tiles of Q x 128 steps.
// A thread keeps its 16 steps in registers between the two halves; the maps of the warps are
// composed in shared memory, those of the blocks exchanged through distributed shared memory
// (field_dsmem.cuh), and the next super-tile's loads are in flight meanwhile.
//
// Backward (g = grad of the states, c = carry from the later steps, c_{L-1} = grad_state_out):
//   lambda_t = g_t + c_t,  grad_x_t = lambda_t,  grad_a_t = lambda_t s_{t-1},  c_{t-1} = a_t lambda_t;
// the same walk from the last tile to the first.
//
// The host emulation runs the same phases with one super-tile (as many "blocks" as tiles) and the
// exchange through the workspace.
#pragma once

#include "field_dsmem.cuh"

namespace fields {

constexpr int kScanSteps = 16;   // steps per thread
constexpr int kScanWarps = 8;
constexpr int kScanTile = kScanSteps * kScanWarps;
constexpr int kScanMaxCluster = 16;

// `a` may be a broadcast view: element (b, t, c) is a[b * a_batch + t * a_step + c * a_chan].
struct ScanShape {
    int B, L, C;
    int NT;   // tiles per sequence
    int CG;   // groups of 32 channels
    int Q, K; // blocks per cluster, super-tiles
    long long a_batch, a_step;
    int a_chan;
};

struct ScanParams {
    const float* a;
    const float* x;      // forward: drive; backward: gradient of the states       [B, L, C]
    const float* states; // backward: the forward's output                         [B, L, C]
    const float* first;  // state before the first step, or null (zero)            [B, C]
    const float* last;   // backward: gradient of the state after the last step    [B, C] or null
    float* out;          // forward: states; backward: gradient of the drive       [B, L, C]
    float* grad_a;       // backward (dense, also for a broadcast `a`)             [B, L, C]
    float* end;          // forward: state after the last step; backward: gradient of the first  [B, C] or null
    float* maps;         // host emulation only: exchanged maps [2][B][NT][C]
    ScanShape s;
};

template <bool BWD>
struct ScanWalk {
    using Params = ScanParams;
    static constexpr int kThreads = 32 * kScanWarps;
    static constexpr int kPhases = 3;
    static constexpr int kSplitPhase = 2;  // host emulation: phases < 2 of all blocks run first
    // warp maps [W][2][32], then the value entering each warp [W][32]
    static constexpr int kSmemFloats = kScanWarps * 3 * 32;

    struct State {
        float a[kScanSteps], x[kScanSteps], prev[BWD ? kScanSteps : 1];
        float carry;  // first warp: the value entering the super-tile
    };

    // Where a thread of block `rank` of a chain works in super-tile k.
    struct At {
        int b, c, tile, t0;  // t0: first of the thread's steps
        bool chan_ok;
    };
    FL_HD static At where(const ScanShape& s, int chain, int rank, int k, int thread) {
        At at;
        at.b = chain / s.CG;
        at.c = chain % s.CG * 32 + (thread & 31);
        at.chan_ok = at.c < s.C;
        const int pos = k * s.Q + rank;  // in walking order; tiles past the end have no steps
        at.tile = BWD ? s.NT - 1 - pos : pos;
        at.t0 = (int)((unsigned)at.tile * kScanTile + (unsigned)(thread >> 5) * kScanSteps);
        return at;
    }
    // (a step outside the sequence is the identity in either direction; unsigned, because the tiles that fill the
    // last super-tile may lie beyond 2^31 steps)
    FL_HD static bool inside(const ScanShape& s, const At& at, int j) {
        return at.chan_ok && (unsigned)at.t0 + (unsigned)j < (unsigned)s.L;
    }
    FL_HD static int warp_at(int pos) { return BWD ? kScanWarps - 1 - pos : pos; }

    FL_HD static void load(const Params& p, const At& at, State& st) {
        const ScanShape& s = p.s;
        const float* ap = p.a + at.b * s.a_batch + at.t0 * s.a_step + (long long)at.c * s.a_chan;
        const size_t row = ((size_t)at.b * s.L + at.t0) * s.C + at.c;
#pragma unroll
        for (int j = 0; j < kScanSteps; ++j) {
            const bool in = inside(s, at, j);
            st.a[j] = in ? ap[j * s.a_step] : 1.0f;
            st.x[j] = in ? p.x[row + (size_t)j * s.C] : 0.0f;
            if constexpr (BWD) {
                if ((unsigned)at.t0 + (unsigned)j > 0) st.prev[j] = in ? p.states[row + (size_t)j * s.C - s.C] : 0.0f;
                else st.prev[j] = in && p.first ? p.first[(size_t)at.b * s.C + at.c] : 0.0f;
            }
        }
    }

    // the map of the thread's steps
    FL_HD static void warp_map(int thread, const State& st, float* smem) {
        float A = 1.0f, Bv = 0.0f;
#pragma unroll
        for (int i = 0; i < kScanSteps; ++i) {
            const int j = BWD ? kScanSteps - 1 - i : i;
            A *= st.a[j];
            Bv = BWD ? st.a[j] * (Bv + st.x[j]) : st.a[j] * Bv + st.x[j];
        }
        float* m = smem + (thread >> 5) * 64 + (thread & 31);
        m[0] = A;
        m[32] = Bv;
    }

    // the block's map from its warps', first warp only
    FL_HD static void block_map(int lane, const float* smem, float& A, float& Bv) {
        A = 1.0f;
        Bv = 0.0f;
#pragma unroll
        for (int i = 0; i < kScanWarps; ++i) {
            const float* m = smem + warp_at(i) * 64 + lane;
            A *= m[0];
            Bv = m[0] * Bv + m[32];
        }
    }

    // the value entering each warp, first warp only
    FL_HD static void enter(int lane, float v, float* smem) {
#pragma unroll
        for (int i = 0; i < kScanWarps; ++i) {
            const int w = warp_at(i);
            const float* m = smem + w * 64 + lane;
            smem[kScanWarps * 64 + w * 32 + lane] = v;
            v = m[0] * v + m[32];
        }
    }

    FL_HD static float begin(const Params& p, const At& at) {
        const float* src = BWD ? p.last : p.first;
        return at.chan_ok && src ? src[(size_t)at.b * p.s.C + at.c] : 0.0f;
    }

    FL_HD static void emit(const Params& p, const At& at, int thread, const State& st, const float* smem) {
        const ScanShape& s = p.s;
        float v = smem[kScanWarps * 64 + thread];
        const size_t row = ((size_t)at.b * s.L + at.t0) * s.C + at.c;
#pragma unroll
        for (int i = 0; i < kScanSteps; ++i) {
            const int j = BWD ? kScanSteps - 1 - i : i;
            if (!inside(s, at, j)) continue;
            if constexpr (BWD) {
                const float lam = st.x[j] + v;
                p.out[row + (size_t)j * s.C] = lam;
                p.grad_a[row + (size_t)j * s.C] = lam * st.prev[j];
                v = st.a[j] * lam;
            } else {
                v = st.a[j] * v + st.x[j];
                p.out[row + (size_t)j * s.C] = v;
            }
            // the outgoing value is the last emitted one, bit for bit
            if (p.end && at.t0 + j == (BWD ? 0 : s.L - 1)) p.end[(size_t)at.b * s.C + at.c] = v;
        }
    }

#ifdef FIELDS_HOST_EMU
    // One super-tile: block = chain * NT + rank.
    FL_HD static float* slot(const Params& p, const At& at, int plane) {
        return p.maps + (((size_t)plane * p.s.B + at.b) * p.s.NT + at.tile) * p.s.C + at.c;
    }
    template <int PH>
    FL_HD static void phase(const Params& p, int block, int thread, float* smem, State& st) {
        const int chain = block / p.s.Q, rank = block % p.s.Q, lane = thread & 31;
        const At at = where(p.s, chain, rank, 0, thread);
        if constexpr (PH == 0) {
            load(p, at, st);
            warp_map(thread, st, smem);
        } else if constexpr (PH == 1) {
            if (thread < 32 && at.chan_ok) block_map(lane, smem, *slot(p, at, 0), *slot(p, at, 1));
        } else {
            if (thread == 0)  // (threads run one after another: the first warp's part comes first)
                for (int l = 0; l < 32; ++l) {
                    At a = where(p.s, chain, 0, 0, l);
                    float v = begin(p, a);
                    for (int r = 0; a.chan_ok && r < rank; ++r) {
                        a = where(p.s, chain, r, 0, l);
                        v = *slot(p, a, 0) * v + *slot(p, a, 1);
                    }
                    enter(l, v, smem);
                }
            emit(p, at, thread, st, smem);
        }
    }
#endif
};

#ifndef FIELDS_HOST_EMU
template <bool BWD>
__global__ void __launch_bounds__(ScanWalk<BWD>::kThreads) scan_walk(const ScanParams p) {
    using W = ScanWalk<BWD>;
    __shared__ float smem[W::kSmemFloats];
    __shared__ __align__(8) float2 exch[2][kScanMaxCluster][32];
    __shared__ __align__(8) unsigned long long bars[2];
    const ScanShape& s = p.s;
    const int tid = threadIdx.x, Q = s.Q, rank = Q > 1 ? (int)cluster_rank() : 0, chain = blockIdx.x / Q;
    if (tid == 0) {
        mbar_init(smem_addr(&bars[0]), 1);
        mbar_init(smem_addr(&bars[1]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (Q > 1) cluster_sync_all();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    bool dead = false;
    typename W::State st, next;
    float carry = 0.0f;
    typename W::At at = W::where(s, chain, rank, 0, tid);
    if (tid < 32) carry = W::begin(p, at);
    W::load(p, at, st);
    for (int k = 0; k < s.K; ++k) {
        W::warp_map(tid, st, smem);
        const typename W::At ahead = W::where(s, chain, rank, k + 1, tid);
        if (k + 1 < s.K) W::load(p, ahead, next);
        __syncthreads();
        if (tid < 32) {
            float A, Bv, v = carry;
            W::block_map(tid, smem, A, Bv);
            if (Q > 1) {
                const unsigned bar = smem_addr(&bars[k & 1]), mine = smem_addr(&exch[k & 1][rank][tid]);
                if (tid == 0) mbar_expect(bar, Q * 32 * 8);
                for (int r = 0; r < Q; ++r) send2(peer_addr(mine, r), A, Bv, peer_addr(bar, r));
                mbar_wait(bar, (k >> 1) & 1, dead);
                for (int r = 0; r < Q; ++r) {
                    const float2 m = exch[k & 1][r][tid];
                    if (r == rank) v = carry;
                    carry = m.x * carry + m.y;
                }
                if (dead) v = nanf("");
            } else {
                carry = A * carry + Bv;
            }
            W::enter(tid, v, smem);
        }
        __syncthreads();
        W::emit(p, at, tid, st, smem);
        st = next;
        at = ahead;
    }
    if (Q > 1) cluster_sync_all();  // no block leaves while a peer may still store into it
}
#endif

}  // namespace fields
