// C ABI of the Field-recurrence library: argument checks, the launch plan and
// the kernel launches. Declarations and the contract of every entry point are
// in include/fields_read.h.
//
// Compiled by nvcc for sm_100a into libfields_read.so. The CPU tests compile
// this same file with g++ and FIELDS_HOST_EMU defined: launches then become
// nested loops over (block, phase, thread) on host memory, so the plan, the
// index arithmetic and the formulas are checked without a GPU. That build is
// test infrastructure; it is never loaded by the package.
#include "field_kernels.cuh"
#include "field_singlepass.cuh"
#ifdef FIELDS_ALL_VARIANTS
#include "field_walk.cuh"
#endif
#include "field_span.cuh"
#include "field_tensor.cuh"
#include "field_scan.cuh"
#include "field_epilogue.cuh"
#include "field_rows.cuh"
#include "field_mixer_grad.cuh"
#include "field_step_gemm.cuh"
#include "field_step_phase.cuh"
#include "field_product.cuh"

#include "../../include/fields_read.h"

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

namespace fields {

// ---------------------------------------------------------------------------
// Launch machinery
// ---------------------------------------------------------------------------
#ifdef FIELDS_HOST_EMU

using Stream = void*;
static thread_local const char* g_last_error = "no error";

template <class K>
static int launch(const typename K::Params& p, long long grid, Stream) {
    std::vector<double> smem_store((K::kSmemFloats + 1) / 2 + 1);  // double-aligned
    float* smem = reinterpret_cast<float*>(smem_store.data());
    for (long long block = 0; block < grid; ++block) {
        for (int thread = 0; thread < K::kThreads; ++thread) K::phase0(p, (int)block, thread, smem);
        if constexpr (K::kPhases > 1) {
            for (int thread = 0; thread < K::kThreads; ++thread)
                K::phase1(p, (int)block, thread, smem);
        }
    }
    return FIELDS_OK;
}

static int fill_zero(float* p, size_t n, Stream) {
    for (size_t i = 0; i < n; ++i) p[i] = 0.0f;
    return FIELDS_OK;
}

template <class K, int PH>
static void emu_phase_range(const typename K::Params& p, int block, float* smem,
                            typename K::State* st, int lo, int hi) {
    if constexpr (PH < K::kPhases) {
        if (PH >= lo && PH < hi)
            for (int thread = 0; thread < K::kThreads; ++thread)
                K::template phase<PH>(p, block, thread, smem, st[thread]);
        emu_phase_range<K, PH + 1>(p, block, smem, st, lo, hi);
    }
}

// Kernels whose blocks wait for one another: every block first runs up to the point
// where it has published its aggregate, then the blocks finish one at a time. With
// FIELDS_EMU_ORDER=reverse the later tiles finish first (after the first tile of each
// chain), which drives the look-back through whole chains of aggregates; the default
// order meets an inclusive state at the first step back.
template <class K>
static int launch_stateful(const typename K::Params& p, long long grid, long long first_wave,
                           Stream, bool = false) {
    std::vector<double> smem_store((size_t)grid * (K::kSmemFloats / 2 + 1));
    std::vector<typename K::State> states((size_t)grid * K::kThreads);
    auto smem_of = [&](long long b) {
        return reinterpret_cast<float*>(smem_store.data() + (size_t)b * (K::kSmemFloats / 2 + 1));
    };
    for (long long b = 0; b < grid; ++b)
        emu_phase_range<K, 0>(p, (int)b, smem_of(b), &states[(size_t)b * K::kThreads], 0,
                              K::kSplitPhase);
    const char* order = std::getenv("FIELDS_EMU_ORDER");
    const bool reverse = order && std::string(order) == "reverse";
    std::vector<long long> seq;
    for (long long b = 0; b < first_wave && b < grid; ++b) seq.push_back(b);
    if (reverse) for (long long b = grid - 1; b >= first_wave; --b) seq.push_back(b);
    else for (long long b = first_wave; b < grid; ++b) seq.push_back(b);
    for (long long b : seq)
        emu_phase_range<K, 0>(p, (int)b, smem_of(b), &states[(size_t)b * K::kThreads],
                              K::kSplitPhase, K::kPhases);
    return FIELDS_OK;
}

static int fill_unset(void* p, size_t bytes, Stream) {
    std::memset(p, kUnsetByte, bytes);
    return FIELDS_OK;
}

template <class K>
static int resident_blocks() { return 4; }  // any positive distance exercises the prefetch path

// Persistent kernels written as one block program over an executor (field_span.cuh): the
// blocks run one after another, every phase as a loop over the block's threads.
template <class K>
struct EmuExec {
    typename K::State* states;
    int nblocks;
    template <class F> void all(F f) { for (int t = 0; t < K::kThreads; ++t) f(t, states[t]); }
    template <class F> void run(F f) { all(f); }
    int blocks() const { return nblocks; }
};

template <class K>
static int launch_span(const typename K::Params& p, int grid, Stream) {
    std::vector<double> smem_store(K::kSmemFloats / 2 + 1);
    float* smem = reinterpret_cast<float*>(smem_store.data());
    std::vector<typename K::State> states(K::kThreads);
    for (int block = 0; block < grid; ++block) {
        EmuExec<K> ex{states.data(), grid};
        typename K::Params q = p;
        q.stages = p.stages & 1;  // every block's first sweep (and the scans) before any wait
        K::run_block(q, block, smem, ex);
    }
    // second part item by item in index order (a block's later items may need maps that blocks
    // with a higher index produce in an earlier round; on the GPU those run concurrently)
    const int rounds = (p.s.items + grid - 1) / grid;
    for (int round = 0; round < rounds; ++round) {
        for (int block = 0; block < grid; ++block) {
            EmuExec<K> ex{states.data(), grid};
            typename K::Params q = p;
            q.stages = p.stages & 6;
            q.emu_round = round;
            K::run_block(q, block, smem, ex);
        }
    }
    return FIELDS_OK;
}

static int g_emu_span_stages = 3;

template <class K>
static int span_grid() { return 6; }  // a handful of blocks: several runs per chain, several items per block

// Kernels whose number of barrier-separated phases depends on the extents.
template <class K>
static int launch_walk(const typename K::Params& p, long long grid, Stream) {
    std::vector<double> smem_store(K::kSmemFloats / 2 + 1);
    float* smem = reinterpret_cast<float*>(smem_store.data());
    std::vector<typename K::State> states(K::kThreads);
    const int n = K::phases(p);
    for (long long block = 0; block < grid; ++block)
        for (int ph = 0; ph < n; ++ph)
            for (int thread = 0; thread < K::kThreads; ++thread)
                K::phase(ph, p, (int)block, thread, smem, states[thread]);
    return FIELDS_OK;
}

#else  // real CUDA build

using Stream = cudaStream_t;
static thread_local const char* g_last_error = "no error";

// Programmatic dependent launch. Every kernel of this library is launched with the
// programmatic-serialization attribute and waits until the kernel before it on the stream has
// completed and its writes are visible. The launch itself (grid set-up, block scheduling) then
// overlaps the end of the previous kernel instead of following it. Because every kernel waits, the
// completion order of the stream is kept along the whole chain. All but one wait before they
// touch any memory and do not signal early: letting the next grid take SM slots while this one
// still ran its last blocks was measured and was slower for the recurrence. step_phase does both: it lets the next kernel
// in at its start and reads parameters ahead of its own wait, which its caller has to allow (settled, in
// fields_step_args). The instruction does nothing in a kernel launched
// without the attribute (FIELDS_READ_PDL=0).
__device__ __forceinline__ void wait_for_previous_kernel() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

static bool dependent_launch_from_env() {
    const char* e = std::getenv("FIELDS_READ_PDL");
    return !(e && e[0] == '0');
}
#ifdef FIELDS_ALL_VARIANTS
static bool dependent_launch_enabled() { return dependent_launch_from_env(); }  // test build: per call
#else
// (the environment is read once, at the first launch)
static bool dependent_launch_enabled() {
    static const bool enabled = dependent_launch_from_env();
    return enabled;
}
#endif

template <class K>
__global__ void __launch_bounds__(K::kThreads) kernel_entry(const typename K::Params p) {
    extern __shared__ __align__(16) float smem[];
    wait_for_previous_kernel();
    K::phase0(p, (int)blockIdx.x, (int)threadIdx.x, smem);
    if constexpr (K::kPhases > 1) {
        __syncthreads();
        K::phase1(p, (int)blockIdx.x, (int)threadIdx.x, smem);
    }
}

static int check_cuda(cudaError_t e) {
    if (e == cudaSuccess) return FIELDS_OK;
    g_last_error = cudaGetErrorString(e);
    return FIELDS_ERR_LAUNCH;
}

// One launch, with the programmatic-serialization attribute unless FIELDS_READ_PDL=0.
template <class P>
static int launch_grid(void (*fn)(const P), dim3 grid, unsigned threads, Stream st, const P& params,
                       size_t bytes = 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = dependent_launch_enabled() ? 1 : 0;
    return check_cuda(cudaLaunchKernelEx(&cfg, fn, params));
}

template <class P>
static int launch_on(void (*fn)(const P), unsigned grid, unsigned threads, size_t bytes, Stream st,
                     const P& params) {
    return launch_grid<P>(fn, dim3(grid), threads, st, params, bytes);
}

template <class K>
static int launch(const typename K::Params& p, long long grid, Stream st) {
    if (grid <= 0) return FIELDS_OK;
    if (grid > 0x7fffffffLL) return FIELDS_ERR_UNSUPPORTED;
    return launch_on<typename K::Params>(kernel_entry<K>, (unsigned)grid, K::kThreads,
                                         K::kSmemFloats * sizeof(float), st, p);
}

static int fill_zero(float* p, size_t n, Stream st) {
    return check_cuda(cudaMemsetAsync(p, 0, n * sizeof(float), st));
}

// Phases FIRST..LAST of one tile, with the block barriers between them.
template <class K, int PH, int LAST>
__device__ __forceinline__ void run_phases(const typename K::Params& p, int tile, float* smem,
                                           typename K::State& st) {
    K::template phase<PH>(p, tile, (int)threadIdx.x, smem, st);
    if constexpr (PH < LAST) {
        if constexpr (K::barrier_after(PH)) __syncthreads();
        run_phases<K, PH + 1, LAST>(p, tile, smem, st);
    }
}

// One block per tile, taken in block-index order (time-major): every tile a block may wait
// for has a smaller index, so the hardware has already started it. (A persistent variant
// that claimed tiles from a counter was measured and was no faster: the claim sits on the
// critical path and the loop costs registers.) After the look-back, while the last sweep
// runs, the block can warm L2 with the inputs of the tile `prefetch` positions ahead, which
// is about the tile that the block taking this one's place will read.
// The order in which tiles are handed out. By default the tile is the block index: a tile's
// predecessors then have smaller block indices, and the kernels rely on the hardware starting
// blocks in index order (what every CUDA GPU so far does, though the programming model does not
// promise it; if a GPU ever did otherwise a block could wait, up to its bound, for a block that
// has not started, and the call would end with FIELDS_ERR_TIMEOUT, not hang). With `s.ticket` set
// a block instead takes its tile from a counter in the workspace header (word 1, which the fill
// leaves at 0xFFFFFFFF, so the first ticket is 0): predecessors then belong to blocks that took
// their tickets earlier and are running, whatever the dispatch order. The atomic's round trip
// sits at the head of every tile: measured +9.5 % on the forward, +3.7 % on the fp32 step and
// +10 % on the bfloat16 step at 8 x 2,048 tokens, which is why it is off in the product and
// selectable (FIELDS_TILE_TICKET=1) only in the test build, where the GPU tests run it.
// EXTRA: the block also does its share of cleaning a kept workspace, and the last block of a channel group folds
// the partial rows. A second instantiation, because the code costs registers (the bfloat16 backward lost
// its fourth block per SM to it: 55.6 -> 61.1 us at 8 x 2,048).
template <class K, bool EXTRA = false>
__global__ void __launch_bounds__(K::kThreads, K::kMinBlocks) stateful_entry(const typename K::Params p) {
    extern __shared__ __align__(16) float smem[];
    typename K::State st;
    wait_for_previous_kernel();
    int tile = (int)blockIdx.x;
#ifdef FIELDS_ALL_VARIANTS
    if (p.s.ticket) {
        // handed round through the first word of the carry area, which no phase writes before
        // the barrier that follows phase 0
        int* ticket = reinterpret_cast<int*>(smem + K::kSumFloats);
        if (threadIdx.x == 0) *ticket = (int)(atomicAdd(p.ctrl + 1, 1u) + 1u);
        __syncthreads();
        tile = *ticket;
        if ((unsigned)tile >= gridDim.x) return;  // (one ticket per block: only a stale counter gets here)
    }
#endif
    run_phases<K, 0, K::kClaimAfter>(p, tile, smem, st);
    __syncthreads();
    if (p.s.prefetch > 0) {
        const long long next = (long long)tile + p.s.prefetch;
        if (next < (long long)p.s.B * p.s.G * p.s.NT) K::prefetch(p, (int)next, (int)threadIdx.x);
    }
    run_phases<K, K::kClaimAfter + 1, K::kPhases - 1>(p, tile, smem, st);
    if constexpr (EXTRA) {
        for (unsigned i = blockIdx.x * K::kThreads + threadIdx.x; i < p.s.clean_n; i += gridDim.x * K::kThreads)
            p.s.clean[i] = make_uint4(kUnsetBits, kUnsetBits, kUnsetBits, kUnsetBits);
        K::finish(p, tile, (int)threadIdx.x, smem);
    }
}

// Kernels that need more than the default 48 KB of dynamic shared memory opt in once per device.
// `ready` is the caller's per-kernel, per-device record (kernels of equal signature share a
// function-pointer type, so the record cannot live in this template).
template <class Fn>
static int allow_shared_memory(Fn fn, size_t bytes, bool* ready) {
    if (bytes <= 48 * 1024) return FIELDS_OK;
    static std::mutex mu;
    int dev = 0;
    int rc = check_cuda(cudaGetDevice(&dev));
    if (rc) return rc;
    if (dev < 0 || dev >= 64) return FIELDS_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> lock(mu);
    if (!ready[dev]) {
        rc = check_cuda(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)bytes));
        if (rc) return rc;
        ready[dev] = true;
    }
    return FIELDS_OK;
}

// (the third argument, the number of chains, only matters to the host emulation)
template <class K>
static int launch_stateful(const typename K::Params& p, long long tiles, long long, Stream st, bool extra = false) {
    if (tiles <= 0) return FIELDS_OK;
    if (tiles > 0x7fffffffLL) return FIELDS_ERR_UNSUPPORTED;
    constexpr size_t bytes = K::kSmemFloats * sizeof(float);
    static bool ready[2][64] = {};
    const auto fn = extra ? stateful_entry<K, true> : stateful_entry<K, false>;
    const int rc = allow_shared_memory(fn, bytes, ready[extra]);
    if (rc) return rc;
    return launch_on<typename K::Params>(fn, (unsigned)tiles, K::kThreads, bytes, st, p);
}

// Fills with the "not yet written" pattern. A kernel rather than a memset, so that it takes part
// in the dependent-launch chain: a memset would make the kernel after it wait for a full drain.
struct FillParams {
    uint4* p;
    size_t n;  // 16-byte words
};
constexpr int kFillThreads = 256, kFillPerThread = 4;

__global__ void __launch_bounds__(kFillThreads) fill_entry(const FillParams q) {
    wait_for_previous_kernel();
    const size_t base = (size_t)blockIdx.x * (kFillThreads * kFillPerThread) + threadIdx.x;
#pragma unroll
    for (int j = 0; j < kFillPerThread; ++j) {
        const size_t i = base + (size_t)j * kFillThreads;
        if (i < q.n) q.p[i] = make_uint4(kUnsetBits, kUnsetBits, kUnsetBits, kUnsetBits);
    }
}

static int fill_unset(void* p, size_t bytes, Stream st) {
    if (!dependent_launch_enabled() || (reinterpret_cast<uintptr_t>(p) & 15) || (bytes & 15))
        return check_cuda(cudaMemsetAsync(p, kUnsetByte, bytes, st));
    const size_t n = bytes / 16, per_block = (size_t)kFillThreads * kFillPerThread;
    if (n == 0) return FIELDS_OK;
    return launch_on<FillParams>(fill_entry, (unsigned)((n + per_block - 1) / per_block), kFillThreads,
                                 0, st, FillParams{static_cast<uint4*>(p), n});
}

// Blocks of kernel K that the current GPU holds at once (occupancy x SM count), asked once per device.
template <class K>
static int resident_blocks() {
    static std::mutex mu;
    static int cached[64] = {};
    int per_sm = 0, dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    std::lock_guard<std::mutex> lock(mu);
    if (cached[dev] > 0) return cached[dev];
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, stateful_entry<K, false>, K::kThreads,
                                                      K::kSmemFloats * sizeof(float)) != cudaSuccess)
        return 0;
    cached[dev] = per_sm * sms;
    return cached[dev];
}

// Persistent block program over an executor: the calling thread, then a block barrier.
template <class K>
struct DeviceExec {
    typename K::State& st;
    template <class F> __device__ __forceinline__ void all(F f) { f((int)threadIdx.x, st); __syncthreads(); }
    template <class F> __device__ __forceinline__ void run(F f) { f((int)threadIdx.x, st); }
    __device__ __forceinline__ int blocks() const { return (int)gridDim.x; }
};

template <class K>
__global__ void __launch_bounds__(K::kThreads, K::kMinBlocks) span_entry(const typename K::Params p) {
    extern __shared__ __align__(16) float smem[];
    typename K::State st;
    DeviceExec<K> ex{st};
    wait_for_previous_kernel();
    if (p.epoch_word == nullptr) {
        K::run_block(p, (int)blockIdx.x, smem, ex);
        return;
    }
    // Epoch kept on the device: every block reads the last completed epoch when it starts; the
    // block that finishes last (all others have read it long before) stores the new one. The
    // ranks' counters advance together because every rank makes the same calls.
    typename K::Params q = p;
    unsigned last;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(last) : "l"(p.epoch_word) : "memory");
    q.epoch = last + 1u ? last + 1u : 1u;   // never 0
    K::run_block(q, (int)blockIdx.x, smem, ex);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(p.epoch_word + 1, 1u) == gridDim.x - 1) {
            p.epoch_word[1] = 0;
            __threadfence();
            asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p.epoch_word), "r"(q.epoch) : "memory");
        }
    }
}

// Blocks of span_entry<K> that the current device holds at once, asked once per device.
template <class K>
static int span_grid() {
    static std::mutex mu;
    static int cached[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    std::lock_guard<std::mutex> lock(mu);
    if (cached[dev] <= 0) {
        int per_sm = 0, sms = 0;
        // (the opt-in to more than 48 KB of shared memory comes first: the query depends on it)
        if (K::kSmemFloats * sizeof(float) > 48 * 1024 &&
            cudaFuncSetAttribute(span_entry<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(K::kSmemFloats * sizeof(float))) != cudaSuccess)
            return 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, span_entry<K>, K::kThreads,
                                                          K::kSmemFloats * sizeof(float)) != cudaSuccess)
            return 0;
        cached[dev] = per_sm * sms;
    }
    return cached[dev];
}

// Cooperative launch (all blocks resident at once: they wait for one another), with the
// programmatic-serialization attribute beside it where the driver accepts the pair.
template <class K>
static int launch_span(const typename K::Params& p, int grid, Stream st) {
    if (grid <= 0) return FIELDS_ERR_LAUNCH;
    constexpr size_t bytes = K::kSmemFloats * sizeof(float);
    static bool ready[64] = {};
    int rc = allow_shared_memory(span_entry<K>, bytes, ready);
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(K::kThreads);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    static bool pair_refused = false;
    cfg.numAttrs = (dependent_launch_enabled() && !pair_refused) ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, span_entry<K>, p);
    if (e != cudaSuccess && cfg.numAttrs == 2) {
        (void)cudaGetLastError();
        pair_refused = true;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, span_entry<K>, p);
    }
    return check_cuda(e);
}

template <class K>
__global__ void __launch_bounds__(K::kThreads, K::kMinBlocks) walk_entry(const typename K::Params p) {
    extern __shared__ __align__(16) float smem[];
    typename K::State st;
    wait_for_previous_kernel();
    const int n = K::phases(p);
    for (int ph = 0; ph < n; ++ph) {
        K::phase(ph, p, (int)blockIdx.x, (int)threadIdx.x, smem, st);
        __syncthreads();
    }
}

template <class K>
static int launch_walk(const typename K::Params& p, long long grid, Stream st) {
    if (grid <= 0) return FIELDS_OK;
    if (grid > 0x7fffffffLL) return FIELDS_ERR_UNSUPPORTED;
    constexpr size_t bytes = K::kSmemFloats * sizeof(float);
    static bool ready[64] = {};
    const int rc = allow_shared_memory(walk_entry<K>, bytes, ready);
    if (rc) return rc;
    return launch_on<typename K::Params>(walk_entry<K>, (unsigned)grid, K::kThreads, bytes, st, p);
}

#endif

// ---------------------------------------------------------------------------
// Plan: chunk length and workspace layout, a function of the extents only.
// ---------------------------------------------------------------------------
constexpr long long kTargetWarps = 148LL * 32;  // enough warps to fill every SM of a B200

struct Plan {
    Shape s;             // with G for the vector width in use
    size_t plane;        // B * N * C floats
    size_t sum_off, carry_off, partial_off;  // in floats
    size_t fwd_floats, bwd_floats;
};

static size_t round_up(size_t x, size_t m) { return (x + m - 1) / m * m; }

static Plan make_plan(int B, int L, int C, int vec) {
    Plan pl{};
    const int nominal_vec = (C % 4 == 0) ? 4 : 1;
    const long long groups = (C + 32 * nominal_vec - 1) / (32 * nominal_vec);
    int ts = 16;
    const int candidates[3] = {64, 32, 16};
    for (int k = 0; k < 3; ++k) {
        const long long n = (L + candidates[k] - 1) / candidates[k];
        if ((long long)B * n * groups >= kTargetWarps) { ts = candidates[k]; break; }
    }
    pl.s.B = B; pl.s.L = L; pl.s.C = C;
    pl.s.ts = ts;
    pl.s.N = (L + ts - 1) / ts;
    pl.s.G = (C + 32 * vec - 1) / (32 * vec);
    pl.plane = (size_t)B * pl.s.N * C;
    pl.sum_off = 0;
    pl.carry_off = round_up(4 * pl.plane, 64);
    pl.partial_off = pl.carry_off + round_up(2 * pl.plane, 64);
    pl.fwd_floats = pl.partial_off;
    pl.bwd_floats = pl.partial_off + round_up(3 * pl.plane, 64);
    return pl;
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

static long long tile_blocks(const Shape& s) {
    const long long tasks = (long long)s.B * s.N * s.G;
    return (tasks + kWarpsPerBlock - 1) / kWarpsPerBlock;
}

#ifdef FIELDS_ALL_VARIANTS
template <int VEC>
static int run_forward(const FwdParams& p, Stream st) {
    const Shape& s = p.s;
    int rc = launch<FwdSummary<VEC, 4>>(p, tile_blocks(s), st);
    if (rc) return rc;
    CarryScan<false>::Params cp{p.sum, p.carry, p.state_in, nullptr, s};
    rc = launch<CarryScan<false>>(cp, (long long)s.B * ((s.C + 31) / 32), st);
    if (rc) return rc;
    return launch<FwdMaterialize<VEC, 4>>(p, tile_blocks(s), st);
}

template <int VEC>
static int run_backward(const BwdParams& p, Stream st) {
    const Shape& s = p.s;
    int rc = launch<BwdSummary<VEC, 4>>(p, tile_blocks(s), st);
    if (rc) return rc;
    CarryScan<true>::Params cp{p.sum, p.carry, p.grad_state_out, p.grad_state_in, s};
    rc = launch<CarryScan<true>>(cp, (long long)s.B * ((s.C + 31) / 32), st);
    if (rc) return rc;
    rc = launch<BwdMaterialize<VEC, 2>>(p, tile_blocks(s), st);
    if (rc) return rc;
    return launch<BwdReduce>(p, 3LL * ((s.C + 31) / 32), st);
}
#endif


// ---------------------------------------------------------------------------
// Single-pass forward: plan and launch.
// ---------------------------------------------------------------------------
struct SpPlan {
    SpShape s;
    long long tiles;
    size_t ctrl_words;               // header holding the error word
    size_t agg_off, incl_off;        // byte offsets into the workspace
    size_t bytes;
};

// Test build only: FIELDS_TILE_TICKET=1 hands tiles out through a counter (see stateful_entry).
#ifdef FIELDS_ALL_VARIANTS
static int tile_ticket_from_env() {
    const char* e = std::getenv("FIELDS_TILE_TICKET");
    return e && std::atoi(e) == 1 ? 1 : 0;
}
#else
static int tile_ticket_from_env() { return 0; }
#endif

static SpPlan make_sp_plan(int B, int L, int C, int tile_steps) {
    SpPlan pl{};
    pl.s.B = B; pl.s.L = L; pl.s.C = C;
    pl.s.NT = (L + tile_steps - 1) / tile_steps;
    pl.s.G = (C + kGroup - 1) / kGroup;
    pl.s.zp = pl.s.gp = 3 * C;
    pl.s.max_polls = kMaxPolls;
    pl.s.ticket = tile_ticket_from_env();
    pl.tiles = (long long)B * pl.s.G * pl.s.NT;
    pl.ctrl_words = kCtrlHeader;
    pl.agg_off = pl.ctrl_words * sizeof(unsigned);
    pl.incl_off = pl.agg_off + (size_t)pl.tiles * 4 * kGroup * sizeof(float);
    pl.bytes = pl.incl_off + (size_t)pl.tiles * 2 * kGroup * sizeof(float);
    return pl;
}


enum Algo { kAlgoAuto = 0, kAlgoThreePhase = 1, kAlgoSinglePass = 2, kAlgoWalk = 3 };

// The product library runs one kernel family, single pass (with 32-bit accesses where 128-bit ones are not
// possible). The measured alternatives (other tile
// shapes, the two-sweep forward, the direct-load and tile-resident backward, the chain walkers,
// the three-phase kernels, L2 prefetch) are compiled only into the test build
// (FIELDS_ALL_VARIANTS), which picks them per call from the environment:
//   FIELDS_READ_ALGO = three_phase | single_pass | walk, FIELDS_FWD_VARIANT, FIELDS_BWD_VARIANT,
//   FIELDS_READ_PREFETCH.
#ifdef FIELDS_ALL_VARIANTS
static Algo algo_from_env() {
    const char* e = std::getenv("FIELDS_READ_ALGO");
    if (!e) return kAlgoAuto;
    const std::string v(e);
    if (v == "three_phase") return kAlgoThreePhase;
    if (v == "single_pass") return kAlgoSinglePass;
    if (v == "walk") return kAlgoWalk;
    return kAlgoAuto;
}
#else
static Algo algo_from_env() { return kAlgoAuto; }
#endif

// Instantiations of the single-pass kernels. The first of each list is the default; the
// others are tuning alternatives selected with FIELDS_FWD_VARIANT / FIELDS_BWD_VARIANT.
//   forward  <steps per warp, warps, blocks per SM the registers must allow>
// Three blocks of four warps per SM at 168 registers hold 108 steps of 128 channels (four blocks at 128
// registers with 24-step tiles: 96). At 1 x 65,536 x 512 189 -> 183 us against the earlier two blocks of
// eight warps and 48-step tiles, at 1 x 16,384 54.2 -> 51.8, at 2 x 3,001 x 384 20.6 -> 19.5, equal at
// 8 x 2,048. From eight rounds of blocks on, where the last one weighs little, 40-step tiles are a little
// faster in spite of a few spilled registers: 184 -> 179 us at 1 x 65,536, 173 -> 169 at 4 x 16,384.
using FwdSp0 = FwdSinglePass<9, 4, 3>;
using FwdSpDeep = FwdSinglePass<10, 4, 3>;
static long long tiles_of(int B, int L, int C, int steps) {
    return (long long)B * ((C + kGroup - 1) / kGroup) * ((L + steps - 1) / steps);
}
// Tensors without 128-bit access (F32Any), forward and backward: the same kernels with four 32-bit accesses. Eight steps
// per warp against six (a tile below what the workspace is counted for): 127 / 143 us at 1 x 30,000 x 513, 44.9 / 47.0
// at 8 x 2,048 x 333, 12.5 / 12.0 at 3 x 777 x 333; blocks of six and eight warps 13.2 to 15.7 at the last.
using FwdSpAny = FwdSinglePass<8, 4, 3, F32Any>;
using FwdSpRows = FwdSinglePass<9, 4, 3, float, false, true>;  // also writes state rows
#ifdef FIELDS_ALL_VARIANTS
using FwdSp1 = FwdSinglePass<4, 8, 2>;        // tile 32
//   two-sweep forward <steps per warp, warps, unroll, blocks per SM, ring slots>
using FwdSp2 = FwdTwoSweep<8, 4, 2, 4, 3>;    // tile 32, 16 warps per SM
#endif
//   backward <steps per warp, warps, sweep-1 unroll, sweep-2 unroll, blocks per SM, rings, ring slots>
using BwdSp0 = BwdSinglePass<8, 4, 2, 1, 3, true, 3>;  // tile 32, 3-slot cp.async rings, 12 warps per SM
using BwdSpAny = BwdSinglePass<8, 4, 2, 1, 3, true, 3, F32Any>;
#ifdef FIELDS_ALL_VARIANTS
using BwdSp1 = BwdSinglePass<8, 4, 2, 1, 4>;           // direct loads, 16 warps per SM
#endif
//   backward with recomputed states <steps per warp, warps, steps per ring slot, blocks per SM, ring slots>
using BwdSp2 = BwdRecompute<8, 4, 1, 3, 2>;   // 73 KB per block, 12 warps per SM
//   tile resident in shared memory, recomputed states <steps per warp, warps, blocks per SM>
#ifdef FIELDS_ALL_VARIANTS
using BwdSp3 = BwdTileResident<4, 4, 3>;      // tile 16, 68 KB per block, 12 warps per SM
#endif
//   bfloat16 raw / read / grad_read / grad_raw (bits as uint16_t); state and arithmetic stay fp32
// The forward: blocks of four warps, four to an SM, ten steps per warp of which six wait in shared memory (figures at FwdSinglePass).
template <bool STATS> using FwdSpBf16 = FwdSinglePass<10, 4, 4, uint16_t, STATS, false, 6>;  // STATS: per-token sums of squares too
// bfloat16 ring cells are half the size, so a 64-step tile (4 warps x 16 steps) still leaves room for
// four blocks per SM; measured 54.9 us against 59.7 us for the 32-step tile (and 71.5 us with
// 16-byte cells) on 8 x 2,048 tokens. (The bound of 128 registers keeps the fourth block: without it the second sweep's early
// batches take 138.)
using BwdSpBf16 = BwdSinglePass<16, 4, 2, 1, 4, true, 3, uint16_t>;
// Smallest time tile of any instantiation above, for the workspace bound (the run functions assert it). The
// bound also decides which extents fields_read_forward_noalloc takes.
constexpr int kSpMinTile = 32;
constexpr int kSpMinTileBwd = 16;

#ifdef FIELDS_ALL_VARIANTS
static int variant_from_env(const char* name) {
    const char* e = std::getenv(name);
    return e ? std::atoi(e) : 0;
}
#endif

// L2 prefetch of the next tile (test build: FIELDS_READ_PREFETCH = 1 for a distance of the
// number of resident blocks, a larger number for that distance). It gained 5 to 9 % on the
// batch-8 forward and lost as much on the backward and on long sequences: off in the product.
#ifdef FIELDS_ALL_VARIANTS
static int prefetch_from_env(int resident) {
    const char* e = std::getenv("FIELDS_READ_PREFETCH");
    const int v = e ? std::atoi(e) : 0;
    return v == 1 ? resident : (v > 1 ? v : 0);
}
#else
static int prefetch_from_env(int) { return 0; }
#endif

// The calling thread's next pass runs on a kept workspace (fields_read_use_kept); null: the workspace holds
// anything and is filled first.
static thread_local fields_kept* g_next_kept = nullptr;

struct ReadyWorkspace {
    unsigned* ctrl;
    float *agg, *incl, *partial;
    fields_kept* kept;  // null: not a kept workspace
    char* half[2];
};

// Makes a workspace ready for a pass of the single-pass kernels. cleaned_after: a kernel behind the pass fills
// what is used of a kept workspace (BwdReduceClean).
static int ready_workspace(void* workspace, SpPlan& pl, Stream st, ReadyWorkspace* out, bool cleaned_after = false) {
    char* ws = static_cast<char*>(workspace);
    fields_kept* k = g_next_kept;
    g_next_kept = nullptr;
    char* slots = ws + pl.agg_off;
    const size_t slot_bytes = pl.bytes - pl.agg_off;
    out->ctrl = reinterpret_cast<unsigned*>(ws);
    out->partial = reinterpret_cast<float*>(ws + pl.bytes);
    out->kept = k;
    int rc = FIELDS_OK;
    if (k) {
        // A pass publishes in one half. Where that half is unset no fill is needed; a small pass (up to 592
        // tiles, four per SM) also fills what was used of the other: there the fill launch shows, in host time
        // above all (20.1 -> 19.2 us of GPU at 2 x 3,001 x 384, 13.6 -> 12.7 at 1 x 2,048 x 512); above, the code in
        // the kernel costs as much, and the half stays as it is until the reduction of a backward pass fills
        // both, or a pass meets it and fills it first.
        if (slot_bytes > k->half_bytes) return FIELDS_ERR_WORKSPACE;
        const unsigned h = k->parity & 1;
        char** half = out->half;
        half[0] = ws + pl.agg_off;
        half[1] = half[0] + k->half_bytes;
        slots = half[h];
        out->partial = reinterpret_cast<float*>(half[1] + k->half_bytes);
        const size_t used = k->dirty[1 - h];
        if (pl.tiles <= 592 && k->dirty[h] == 0 && !cleaned_after) {
            if (used > (size_t)pl.tiles * 16384) {  // a much larger pass was before: too much for these blocks
                rc = fill_unset(half[1 - h], used, st);
            } else {
                pl.s.clean = reinterpret_cast<uint4*>(half[1 - h]);
                pl.s.clean_n = (unsigned)(used / 16);
            }
            k->dirty[1 - h] = 0;
            k->dirty[h] = slot_bytes;
            k->parity = 1 - h;
        } else {
            if (k->dirty[h]) rc = fill_unset(slots, slot_bytes, st);
            if (k->dirty[h] < slot_bytes) k->dirty[h] = slot_bytes;
            if (used == 0) k->parity = 1 - h;
        }
    } else {
        rc = fill_unset(ws, pl.bytes, st);  // error word, counters and every publication slot
    }
    out->agg = reinterpret_cast<float*>(slots);
    out->incl = reinterpret_cast<float*>(slots + (pl.incl_off - pl.agg_off));
    return rc;
}

template <class K, typename IO = float>
static int run_forward_single_pass(const IO* raw, const float* tr, const float* ti,
                                   const float* gamma, const float* state_in, IO* read,
                                   float* state_out, void* workspace, int B, int L, int C,
                                   Stream st, float* sumsq = nullptr, long long pitch = 0,
                                   float* rows = nullptr) {
    static_assert(K::kTile >= kSpMinTile, "fields_read_workspace_bytes counts the slots of tiles of kSpMinTile steps");
    SpPlan pl = make_sp_plan(B, L, C, K::kTile);
    pl.s.prefetch = prefetch_from_env(resident_blocks<K>());
    if (pitch) pl.s.zp = (int)pitch;
    ReadyWorkspace ws;
    const int rc = ready_workspace(workspace, pl, st, &ws);
    if (rc) return rc;
    SpFwdParamsT<IO> p{raw, tr, ti, gamma, state_in, read, state_out, ws.agg, ws.incl, ws.ctrl, pl.s};
    p.sumsq = sumsq;
    p.rows = rows;
    return launch_stateful<K>(p, pl.tiles, (long long)B * pl.s.G, st, pl.s.clean_n > 0);
}

template <class K, typename IO = float>
static int run_backward_single_pass(const IO* raw, const float* tr, const float* ti,
                                    const float* gamma, const float* state_in, const IO* read,
                                    const IO* grad_read, const float* grad_state_out,
                                    IO* grad_raw, float* grad_tr, float* grad_ti,
                                    float* grad_gamma, float* grad_state_in, void* workspace,
                                    int B, int L, int C, Stream st,
                                    const float* states = nullptr, long long raw_pitch = 0,
                                    long long grad_pitch = 0) {
    static_assert(K::kTile >= kSpMinTileBwd, "fields_read_workspace_bytes counts the slots of tiles of that many steps");
    SpPlan pl = make_sp_plan(B, L, C, K::kTile);
    pl.s.prefetch = prefetch_from_env(resident_blocks<K>());
    if (raw_pitch) pl.s.zp = (int)raw_pitch;
    if (grad_pitch) pl.s.gp = (int)grad_pitch;
    // Up to 16 partial rows the last block of a channel group adds them: a launch less, 2.5 us of GPU and as
    // much of host time. (At 64 rows that block took 5 us longer than the reduction kernel.)
#ifdef FIELDS_HOST_EMU
    const bool fold = false;
#else
    const bool fold = (long long)B * pl.s.NT <= 16 && pl.s.G <= kCtrlHeader - 2;
#endif
    ReadyWorkspace ws;
    int rc = ready_workspace(workspace, pl, st, &ws, !fold);
    if (rc) return rc;
    SpBwdParamsT<IO> p{raw, tr, ti, gamma, state_in, read, grad_read, grad_state_out, grad_raw,
                       grad_state_in, ws.agg, ws.incl, ws.ctrl, ws.partial, pl.s};
    p.states = states;
    p.state_rows = L / kStateRowEvery;
    if (fold) { p.grad_par[0] = grad_tr; p.grad_par[1] = grad_ti; p.grad_par[2] = grad_gamma; }
    rc = launch_stateful<K>(p, pl.tiles, (long long)B * pl.s.G, st, pl.s.clean_n > 0 || fold);
    if (rc || fold) return rc;
    BwdReduceClean::Params rp{};
    rp.partial = ws.partial;
    rp.grad_tr = grad_tr; rp.grad_ti = grad_ti; rp.grad_gamma = grad_gamma;
    rp.s = Shape{B, L, C, K::kTile, pl.s.NT, pl.s.G};
    rp.reduce_blocks = 3 * ((C + 31) / 32);
    if (fields_kept* k = ws.kept) {
        for (int h = 0; h < 2; ++h) {
            rp.clean[h] = reinterpret_cast<unsigned*>(ws.half[h]);
            rp.clean_n[h] = (unsigned)(k->dirty[h] / 16);
            k->dirty[h] = 0;
        }
        rp.clean_blocks = BwdReduceClean::blocks_for((long long)rp.clean_n[0] + rp.clean_n[1]);
    }
    return launch<BwdReduceClean>(rp, rp.reduce_blocks + rp.clean_blocks, st);
}

static size_t sp_backward_bytes(int B, int L, int C, int tile_steps) {
    const SpPlan pl = make_sp_plan(B, L, C, tile_steps);
    return pl.bytes + (size_t)3 * B * pl.s.NT * C * sizeof(float);
}

#ifdef FIELDS_ALL_VARIANTS
// ---------------------------------------------------------------------------
// Chain walkers: one block per (batch row, 32 channels) walks the whole sequence, no
// inter-block communication, bitwise reproducible. Measured slower than the single-pass
// kernels on B200 at every shape tried (few warps per SM, scalar shared-memory traffic), so
// they run only on request (FIELDS_READ_ALGO=walk), e.g. when run-to-run identical bits
// matter more than speed. No workspace except one partial row per chain (backward).
// ---------------------------------------------------------------------------
using FwdWalker = FwdWalk<16, 8, 3>;   // tile 128 steps, 3 x 48 KB ring, 8 warps
using BwdWalker = BwdWalk<4, 8, 4>;    // tile 32 steps, 4 x 36 KB ring, 8 warps

template <class K>
static WalkShape walk_shape(int B, int L, int C) {
    return WalkShape{B, L, C, (L + K::kTile - 1) / K::kTile, (C + kLane - 1) / kLane};
}

static bool walk_wanted(int, int, Algo algo) { return algo == kAlgoWalk; }

#endif  // FIELDS_ALL_VARIANTS

// ---------------------------------------------------------------------------
// Sequence-sharded forward in one launch (field_span.cuh): plan.
// ---------------------------------------------------------------------------
using SpanFwd = FwdSpanSweep<2, 8, 2>;   // chunks of 2 steps (two in flight per warp), 8 warps, 2 blocks per SM
constexpr int kSpanMaxItems = 1024;       // runs per launch over all chains (unless there are more chains)

static long long span_item_bound(int B, int C) {
    const long long chains = (long long)B * ((C + kGroup - 1) / kGroup);
    return chains > kSpanMaxItems ? chains : kSpanMaxItems;
}

// Runs: as many per chain as the grid has blocks for, each a whole number of warp slices.
template <class K>
static SpanShape make_span_shape(int B, int L, int C, int grid) {
    SpanShape s{};
    s.B = B; s.L = L; s.C = C;
    s.G = (C + kGroup - 1) / kGroup;
    s.chains = B * s.G;
    long long want = grid / s.chains;
    const long long cap = span_item_bound(B, C) / s.chains;
    if (want > cap) want = cap;
    if (want > (L + K::kRunQuantum - 1) / K::kRunQuantum) want = (L + K::kRunQuantum - 1) / K::kRunQuantum;
    if (want < 1) want = 1;
    int steps = (int)((L + want - 1) / want);
    steps = (steps + K::kRunQuantum - 1) / K::kRunQuantum * K::kRunQuantum;
    s.run_steps = steps;
    s.R = (L + steps - 1) / steps;
    s.items = s.chains * s.R;
    return s;
}

// Bound of a device-side wait in polls: the caller's, or the library's default.
static unsigned poll_bound(unsigned max_polls) {
    return max_polls == 0 || max_polls > kMaxPolls ? kMaxPolls : max_polls;
}

// Mailbox = [slots of the exchange][board of the one-launch forward]. The board (the run maps
// of the owner's own kernel, 4 KB per run) is never written by a peer.
static size_t mailbox_slot_bytes(int P, int B, int C) {
    return round_up((size_t)2 * P * B * 4 * C * sizeof(MailPair), 256);
}
// counters (one word per chain), then the run maps of up to span_item_bound runs (2 KB each)
// (a counter word and, 256 bytes apart from one another, a ready word per chain)
// ... and, 64 words behind them, the two words of the device-resident epoch
static size_t board_epoch_offset(int B, int C) {
    return ((size_t)B * ((C + kGroup - 1) / kGroup) * 65 + 64) * sizeof(unsigned);
}
static size_t board_count_bytes(int B, int C) {
    return round_up(board_epoch_offset(B, C) + 64 * sizeof(unsigned), 256);
}
// Behind the board: the reduction region of fields_read_sum_over_ranks, [2][P][n_max] pairs.
static int mailbox_sum_capacity(int C) { return 3 * C + 64; }
static size_t mailbox_sum_bytes(int P, int C) {
    return round_up((size_t)2 * P * mailbox_sum_capacity(C) * sizeof(MailPair), 256);
}
static size_t mailbox_board_bytes(int B, int C) {
    return board_count_bytes(B, C) + (size_t)span_item_bound(B, C) * kGroup * 4 * sizeof(float);
}

// ---------------------------------------------------------------------------
// Built-in scratch for fields_read_forward_noalloc: one fixed buffer per GPU that
// has loaded this library, held until the process exits.
// ---------------------------------------------------------------------------
constexpr size_t kStaticScratchBytes = FIELDS_STATIC_SCRATCH_BYTES;

#ifdef FIELDS_HOST_EMU
alignas(256) static unsigned char g_static_scratch[kStaticScratchBytes];

static int static_scratch(float** out) {
    *out = reinterpret_cast<float*>(g_static_scratch);
    return FIELDS_OK;
}
#else
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

constexpr int kMaxDevices = 64;
static std::mutex g_scratch_mutex;
static float* g_scratch_ptr[kMaxDevices] = {};

// In host code `g_static_scratch` is only a handle for the runtime, not an address a
// kernel may use: the device address is looked up once per device, with that device
// current, and cached.
static int static_scratch(float** out) {
    int dev = -1;
    int rc = check_cuda(cudaGetDevice(&dev));
    if (rc) return rc;
    if (dev < 0 || dev >= kMaxDevices) return FIELDS_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (!g_scratch_ptr[dev]) {
        void* p = nullptr;
        rc = check_cuda(cudaGetSymbolAddress(&p, g_static_scratch));
        if (rc) return rc;
        g_scratch_ptr[dev] = static_cast<float*>(p);
    }
    *out = g_scratch_ptr[dev];
    return FIELDS_OK;
}
#endif

}  // namespace fields

using namespace fields;

extern "C" {

const char* fields_status_string(int status) {
    switch (status) {
        case FIELDS_OK: return "ok";
        case FIELDS_ERR_ARGUMENT: return "invalid argument (null pointer or bad extent)";
        case FIELDS_ERR_WORKSPACE: return "workspace missing, too small or not 256-byte aligned";
        case FIELDS_ERR_LAUNCH: return "CUDA launch failed";
        case FIELDS_ERR_TIMEOUT: return "device-side wait timed out";
        case FIELDS_ERR_UNSUPPORTED: return "unsupported extent";
        case FIELDS_ERR_SCRATCH_LIMIT:
            return "extents need more scratch than the built-in static buffer holds";
        default: return "unknown status";
    }
}

int fields_read_version(void) { return 100; }

const char* fields_last_cuda_error(void) { return g_last_error; }

int fields_read_use_kept(struct fields_kept* kept) {
    if (kept && (kept->half_bytes % 256 || kept->half_bytes > ((size_t)1 << 32))) return FIELDS_ERR_ARGUMENT;
#ifdef FIELDS_HOST_EMU
    if (kept) return FIELDS_ERR_UNSUPPORTED;
#endif
    // (the test build's other kernel families use a workspace as plain scratch, and its ticket counter
    // starts from the fill)
    if (kept && ((algo_from_env() != kAlgoAuto && algo_from_env() != kAlgoSinglePass) || tile_ticket_from_env()))
        return FIELDS_ERR_UNSUPPORTED;
    g_next_kept = kept;
    return FIELDS_OK;
}

size_t fields_read_workspace_bytes(int B, int L, int C, int pass) {
    if (B <= 0 || L <= 0 || C <= 0) return 0;
    const Plan pl = make_plan(B, L, C, 1);
    const size_t floats = pass == FIELDS_PASS_BACKWARD ? pl.bwd_floats : pl.fwd_floats;
    size_t bytes = floats * sizeof(float);
    const size_t sp = pass == FIELDS_PASS_BACKWARD ? sp_backward_bytes(B, L, C, kSpMinTileBwd)
                                                   : make_sp_plan(B, L, C, kSpMinTile).bytes;
    return sp > bytes ? sp : bytes;
}

int fields_read_forward(const float* raw, const float* tr, const float* ti, const float* gamma,
                        const float* state_in, float* read, float* state_out, void* workspace,
                        size_t workspace_bytes, int B, int L, int C, void* stream) {
    if (B < 0 || L < 0 || C <= 0) return FIELDS_ERR_ARGUMENT;
    Stream st = reinterpret_cast<Stream>(stream);
    if (B == 0) return FIELDS_OK;
    if (!tr || !ti || !gamma) return FIELDS_ERR_ARGUMENT;
    if (L == 0) {
        // no steps: the state passes through unchanged
        if (state_out) {
            if (!state_in) return fill_zero(state_out, (size_t)B * 2 * C, st);
#ifdef FIELDS_HOST_EMU
            std::memcpy(state_out, state_in, (size_t)B * 2 * C * sizeof(float));
#else
            return check_cuda(cudaMemcpyAsync(state_out, state_in, (size_t)B * 2 * C * sizeof(float),
                                              cudaMemcpyDeviceToDevice, st));
#endif
        }
        return FIELDS_OK;
    }
    if (!raw || !read) return FIELDS_ERR_ARGUMENT;
    const bool vec4 = C % 4 == 0 && aligned16(raw) && aligned16(read) && aligned16(tr) &&
                      aligned16(ti) && aligned16(gamma) && aligned16(state_in) &&
                      aligned16(state_out) && aligned16(workspace);
    const Plan pl = make_plan(B, L, C, vec4 ? 4 : 1);
    if (!workspace || workspace_bytes < fields_read_workspace_bytes(B, L, C, FIELDS_PASS_FORWARD) ||
        (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return FIELDS_ERR_WORKSPACE;
    const Algo algo = algo_from_env();
#ifdef FIELDS_ALL_VARIANTS
    if (vec4 && walk_wanted(B, C, algo)) {
        WalkFwdParams wp{raw, tr, ti, gamma, state_in, read, state_out,
                         walk_shape<FwdWalker>(B, L, C)};
        return launch_walk<FwdWalker>(wp, (long long)B * wp.s.G, st);
    }
#endif
    if (vec4 && algo != kAlgoThreePhase) {
#define FIELDS_FWD_SP(K)                                                                      \
    return run_forward_single_pass<K>(raw, tr, ti, gamma, state_in, read, state_out, workspace, \
                                      B, L, C, st)
#ifdef FIELDS_ALL_VARIANTS
        switch (variant_from_env("FIELDS_FWD_VARIANT")) {
            case 1: FIELDS_FWD_SP(FwdSp1);
            case 2: FIELDS_FWD_SP(FwdSp2);
            default: break;
        }
#endif
        if (tiles_of(B, L, C, 40) >= 8 * 3 * 148) FIELDS_FWD_SP(FwdSpDeep);
        FIELDS_FWD_SP(FwdSp0);
#undef FIELDS_FWD_SP
    }
    if (algo != kAlgoThreePhase)
        return run_forward_single_pass<FwdSpAny, F32Any>(reinterpret_cast<const F32Any*>(raw), tr, ti, gamma, state_in,
                                                         reinterpret_cast<F32Any*>(read), state_out, workspace, B, L, C,
                                                         st);
#ifdef FIELDS_ALL_VARIANTS
    float* ws = static_cast<float*>(workspace);
    FwdParams p{raw, tr, ti, gamma, state_in, read, state_out,
                ws + pl.sum_off, ws + pl.carry_off, pl.s};
    return vec4 ? run_forward<4>(p, st) : run_forward<1>(p, st);
#else
    return FIELDS_ERR_UNSUPPORTED;  // (not reached)
#endif
}

int fields_read_backward(const float* raw, const float* tr, const float* ti, const float* gamma,
                         const float* state_in, const float* read, const float* grad_read,
                         const float* grad_state_out, float* grad_raw, float* grad_tr,
                         float* grad_ti, float* grad_gamma, float* grad_state_in, void* workspace,
                         size_t workspace_bytes, int B, int L, int C, void* stream) {
    if (B < 0 || L < 0 || C <= 0) return FIELDS_ERR_ARGUMENT;
    if (!grad_tr || !grad_ti || !grad_gamma) return FIELDS_ERR_ARGUMENT;
    Stream st = reinterpret_cast<Stream>(stream);
    if (B == 0 || L == 0) {
        // nothing depends on the parameters; the state gradient passes through
        int rc = fill_zero(grad_tr, C, st);
        if (!rc) rc = fill_zero(grad_ti, C, st);
        if (!rc) rc = fill_zero(grad_gamma, C, st);
        if (!rc && grad_state_in && B > 0) {
            if (!grad_state_out) {
                rc = fill_zero(grad_state_in, (size_t)B * 2 * C, st);
            } else {
#ifdef FIELDS_HOST_EMU
                std::memcpy(grad_state_in, grad_state_out, (size_t)B * 2 * C * sizeof(float));
#else
                rc = check_cuda(cudaMemcpyAsync(grad_state_in, grad_state_out,
                                                (size_t)B * 2 * C * sizeof(float),
                                                cudaMemcpyDeviceToDevice, st));
#endif
            }
        }
        return rc;
    }
    if (!raw || !tr || !ti || !gamma || !read || !grad_read || !grad_raw)
        return FIELDS_ERR_ARGUMENT;
    const bool vec4 = C % 4 == 0 && aligned16(raw) && aligned16(read) && aligned16(grad_read) &&
                      aligned16(grad_raw) && aligned16(tr) && aligned16(ti) && aligned16(gamma) &&
                      aligned16(state_in) && aligned16(workspace);
    const Plan pl = make_plan(B, L, C, vec4 ? 4 : 1);
    if (!workspace ||
        workspace_bytes < fields_read_workspace_bytes(B, L, C, FIELDS_PASS_BACKWARD) ||
        (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return FIELDS_ERR_WORKSPACE;
#ifdef FIELDS_ALL_VARIANTS
    if (vec4 && walk_wanted(B, C, algo_from_env())) {
        float* partial = static_cast<float*>(workspace);
        WalkBwdParams wp{raw, tr, ti, gamma, state_in, read, grad_read, grad_state_out, grad_raw,
                         grad_state_in, partial, walk_shape<BwdWalker>(B, L, C)};
        int rc = launch_walk<BwdWalker>(wp, (long long)B * wp.s.G, st);
        if (rc) return rc;
        BwdParams rp{};
        rp.partial = partial;
        rp.grad_tr = grad_tr; rp.grad_ti = grad_ti; rp.grad_gamma = grad_gamma;
        rp.s = Shape{B, L, C, L, 1, wp.s.G};
        return launch<BwdReduce>(rp, 3LL * ((C + 31) / 32), st);
    }
#endif
    if (vec4 && algo_from_env() != kAlgoThreePhase) {
#define FIELDS_BWD_SP(K)                                                                        \
    return run_backward_single_pass<K>(raw, tr, ti, gamma, state_in, read, grad_read,          \
                                       grad_state_out, grad_raw, grad_tr, grad_ti, grad_gamma, \
                                       grad_state_in, workspace, B, L, C, st)
#ifdef FIELDS_ALL_VARIANTS
        switch (variant_from_env("FIELDS_BWD_VARIANT")) {
            case 1: FIELDS_BWD_SP(BwdSp1);
            case 2: FIELDS_BWD_SP(BwdSp2);
            case 3: FIELDS_BWD_SP(BwdSp3);
            default: FIELDS_BWD_SP(BwdSp0);
        }
#else
        FIELDS_BWD_SP(BwdSp0);
#endif
#undef FIELDS_BWD_SP
    }
    if (algo_from_env() != kAlgoThreePhase) {
        auto any = [](const float* q) { return reinterpret_cast<const F32Any*>(q); };
        return run_backward_single_pass<BwdSpAny, F32Any>(any(raw), tr, ti, gamma, state_in, any(read), any(grad_read),
                                                          grad_state_out, reinterpret_cast<F32Any*>(grad_raw), grad_tr,
                                                          grad_ti, grad_gamma, grad_state_in, workspace, B, L, C, st);
    }
#ifdef FIELDS_ALL_VARIANTS
    float* ws = static_cast<float*>(workspace);
    BwdParams p{raw, tr, ti, gamma, state_in, read, grad_read, grad_state_out, grad_raw,
                grad_state_in, ws + pl.sum_off, ws + pl.carry_off, ws + pl.partial_off,
                grad_tr, grad_ti, grad_gamma, pl.s};
    return vec4 ? run_backward<4>(p, st) : run_backward<1>(p, st);
#else
    return FIELDS_ERR_UNSUPPORTED;  // (not reached)
#endif
}


int fields_read_forward_rows(const float* raw, const float* tr, const float* ti, const float* gamma,
                             const float* state_in, float* read, float* state_out, float* states,
                             void* workspace, size_t workspace_bytes, int B, int L, int C, void* stream) {
    if (B <= 0 || L <= 0 || C <= 0) return FIELDS_ERR_ARGUMENT;
    if (!raw || !tr || !ti || !gamma || !read || (!states && L >= kStateRowEvery)) return FIELDS_ERR_ARGUMENT;
    if (C % 4 != 0 || !aligned16(raw) || !aligned16(read) || !aligned16(tr) || !aligned16(ti) || !aligned16(gamma) ||
        !aligned16(states))
        return FIELDS_ERR_UNSUPPORTED;
    if (!workspace || workspace_bytes < fields_read_workspace_bytes(B, L, C, FIELDS_PASS_FORWARD) ||
        (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return FIELDS_ERR_WORKSPACE;
    return run_forward_single_pass<FwdSpRows>(raw, tr, ti, gamma, state_in, read, state_out, workspace, B, L, C,
                                              reinterpret_cast<Stream>(stream), nullptr, 0, states);
}

int fields_read_state_rows(int L) { return L > 0 ? L / kStateRowEvery : 0; }

int fields_read_backward_from_states(const float* raw, const float* tr, const float* ti,
                                     const float* gamma, const float* state_in,
                                     const float* states, const float* grad_read,
                                     const float* grad_state_out, float* grad_raw, float* grad_tr,
                                     float* grad_ti, float* grad_gamma, float* grad_state_in,
                                     void* workspace, size_t workspace_bytes, int B, int L, int C,
                                     void* stream) {
    if (B <= 0 || L <= 0 || C <= 0) return FIELDS_ERR_ARGUMENT;
    if (!raw || !tr || !ti || !gamma || !grad_read || !grad_raw || !grad_tr || !grad_ti ||
        !grad_gamma)
        return FIELDS_ERR_ARGUMENT;
    if (!states && L > kStateRowEvery) return FIELDS_ERR_ARGUMENT;
    if (C % 4 != 0 || !aligned16(raw) || !aligned16(grad_read) || !aligned16(grad_raw) ||
        !aligned16(tr) || !aligned16(ti) || !aligned16(gamma) || !aligned16(state_in) ||
        !aligned16(states))
        return FIELDS_ERR_UNSUPPORTED;
    if (!workspace ||
        workspace_bytes < fields_read_workspace_bytes(B, L, C, FIELDS_PASS_BACKWARD) ||
        (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return FIELDS_ERR_WORKSPACE;
    // `read` is never dereferenced when the rows are given; a sequence of up to 8 steps needs no row
    return run_backward_single_pass<BwdSp2>(raw, tr, ti, gamma, state_in, (const float*)nullptr,
                                            grad_read, grad_state_out, grad_raw, grad_tr, grad_ti,
                                            grad_gamma, grad_state_in, workspace, B, L, C,
                                            reinterpret_cast<Stream>(stream), states);
}

size_t fields_read_static_scratch_bytes(void) { return kStaticScratchBytes; }

int fields_read_forward_noalloc(const float* raw, const float* tr, const float* ti,
                                const float* gamma, const float* state_in, float* read,
                                float* state_out, int B, int L, int C, void* stream) {
    if (B < 0 || L < 0 || C <= 0) return FIELDS_ERR_ARGUMENT;
    const size_t need = fields_read_workspace_bytes(B, L, C, FIELDS_PASS_FORWARD);
    if (need > kStaticScratchBytes) return FIELDS_ERR_SCRATCH_LIMIT;
    float* scratch = nullptr;
    const int rc = static_scratch(&scratch);
    if (rc) return rc;
    // The forward kernels write every scratch word before they read it, so nothing has to
    // be cleared between calls.
    return fields_read_forward(raw, tr, ti, gamma, state_in, read, state_out, scratch,
                               kStaticScratchBytes, B, L, C, stream);
}


int fields_read_device_status(const void* workspace, void* stream) {
    if (!workspace) return FIELDS_ERR_ARGUMENT;
    int word = 0;
#ifdef FIELDS_HOST_EMU
    (void)stream;
    word = static_cast<const int*>(workspace)[0];
#else
    Stream st = reinterpret_cast<Stream>(stream);
    int rc = check_cuda(cudaMemcpyAsync(&word, static_cast<const int*>(workspace), sizeof(int),
                                        cudaMemcpyDeviceToHost, st));
    if (!rc) rc = check_cuda(cudaStreamSynchronize(st));
    if (rc) return rc;
#endif
    return word != -1 ? FIELDS_ERR_TIMEOUT : FIELDS_OK;
}


int fields_read_span_summary(const float* raw, const float* tr, const float* ti,
                             const float* gamma, float* summary, void* workspace,
                             size_t workspace_bytes, int B, int L, int C, void* stream) {
    if (B < 0 || L < 0 || C <= 0) return FIELDS_ERR_ARGUMENT;
    if (B == 0) return FIELDS_OK;
    if (!raw || !tr || !ti || !gamma || !summary) return FIELDS_ERR_ARGUMENT;
    if (L == 0) return FIELDS_ERR_ARGUMENT;  // an empty span has no summary to exchange
    Stream st = reinterpret_cast<Stream>(stream);
    const bool vec4 = C % 4 == 0 && aligned16(raw) && aligned16(tr) && aligned16(ti) &&
                      aligned16(gamma) && aligned16(workspace);
    Plan pl = make_plan(B, L, C, vec4 ? 4 : 1);
    if (!workspace || workspace_bytes < pl.fwd_floats * sizeof(float) ||
        (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return FIELDS_ERR_WORKSPACE;
    float* ws = static_cast<float*>(workspace);
    FwdParams p{raw, tr, ti, gamma, nullptr, nullptr, nullptr, ws + pl.sum_off, ws + pl.carry_off,
                pl.s};
    int rc;
    if (vec4) {
        // 16 steps per warp, four warps per block: one map per 64 steps (never more maps than
        // the three-phase plan, whose workspace bound therefore still holds)
        using Stream4 = ChunkSummaryStream<2, 3, 4>;
        p.s.ts = 16;
        p.s.N = (L + 63) / 64;
        p.s.G = (C + 127) / 128;
        pl.s = p.s;
        rc = launch<Stream4>(p, (long long)B * p.s.N * p.s.G, st);
    } else {
        rc = launch<FwdSummary<1, 4>>(p, tile_blocks(pl.s), st);
    }
    if (rc) return rc;
    SpanCompose::Params cp{p.sum, summary, pl.s, 0};
    return launch<SpanCompose>(cp, (long long)B * ((C + 31) / 32), st);
}

int fields_read_span_summary_backward(const float* raw, const float* tr, const float* ti,
                                      const float* grad_read, float* summary, void* workspace,
                                      size_t workspace_bytes, int B, int L, int C, void* stream) {
    if (B < 0 || L < 0 || C <= 0) return FIELDS_ERR_ARGUMENT;
    if (B == 0) return FIELDS_OK;
    if (!raw || !tr || !ti || !grad_read || !summary) return FIELDS_ERR_ARGUMENT;
    if (L == 0) return FIELDS_ERR_ARGUMENT;
    Stream st = reinterpret_cast<Stream>(stream);
    const bool vec4 = C % 4 == 0 && aligned16(raw) && aligned16(tr) && aligned16(ti) &&
                      aligned16(grad_read) && aligned16(workspace);
    const Plan pl = make_plan(B, L, C, vec4 ? 4 : 1);
    if (!workspace || workspace_bytes < pl.bwd_floats * sizeof(float) ||
        (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return FIELDS_ERR_WORKSPACE;
    float* ws = static_cast<float*>(workspace);
    BwdParams p{};
    p.raw = raw; p.tr = tr; p.ti = ti; p.grad_read = grad_read;
    p.sum = ws + pl.sum_off;
    p.s = pl.s;
    Shape cs = pl.s;
    int rc;
    if (vec4) {
        // as in fields_read_span_summary: 16 steps per warp, one map per 64 steps
        using Stream4 = ChunkDualSummaryStream<1, 3, 4>;  // 38 KB of shared memory per block
        p.s.ts = 16;
        p.s.N = (L + 63) / 64;
        p.s.G = (C + 127) / 128;
        cs = p.s;
        rc = launch<Stream4>(p, (long long)B * p.s.N * p.s.G, st);
    } else {
        rc = launch<BwdSummary<1, 4>>(p, tile_blocks(pl.s), st);
    }
    if (rc) return rc;
    SpanCompose::Params cp{p.sum, summary, cs, 1};
    return launch<SpanCompose>(cp, (long long)B * ((C + 31) / 32), st);
}

int fields_read_fold_summaries(const float* summaries, const float* state0, float* state,
                               int rank, int P, int B, int C, void* stream) {
    if (B < 0 || C <= 0 || P <= 0 || rank < 0 || rank >= P) return FIELDS_ERR_ARGUMENT;
    if (B == 0) return FIELDS_OK;
    if (!summaries || !state) return FIELDS_ERR_ARGUMENT;
    FoldSummaries::Params p{summaries, state0, state, rank, P, B, C, 0};
    const long long n = (long long)B * C;
    return launch<FoldSummaries>(p, (n + FoldSummaries::kThreads - 1) / FoldSummaries::kThreads,
                                 reinterpret_cast<Stream>(stream));
}

int fields_read_fold_summaries_backward(const float* summaries, const float* carry_end, float* carry,
                                        int rank, int P, int B, int C, void* stream) {
    if (B < 0 || C <= 0 || P <= 0 || rank < 0 || rank >= P) return FIELDS_ERR_ARGUMENT;
    if (B == 0) return FIELDS_OK;
    if (!summaries || !carry) return FIELDS_ERR_ARGUMENT;
    FoldSummaries::Params p{summaries, carry_end, carry, rank, P, B, C, 1};
    const long long n = (long long)B * C;
    return launch<FoldSummaries>(p, (n + FoldSummaries::kThreads - 1) / FoldSummaries::kThreads,
                                 reinterpret_cast<Stream>(stream));
}


}  // extern "C"

// ---------------------------------------------------------------------------
// Real-valued scan (field_scan.cuh): plan and launches.
// ---------------------------------------------------------------------------
// Blocks per cluster: as many as a sequence has tiles, while all of them fit the GPU at once (up to 16:
// the exchange costs a block Q stores and Q folds per super-tile, and its latency once).
static ScanShape make_scan_shape(int B, int L, int C, long long a_batch, long long a_step,
                                 int a_chan) {
    ScanShape s{};
    s.B = B; s.L = L; s.C = C;
    s.NT = (int)(((long long)L + kScanTile - 1) / kScanTile);
    s.CG = (C + 31) / 32;
    s.a_batch = a_batch; s.a_step = a_step; s.a_chan = a_chan;
#ifdef FIELDS_HOST_EMU
    s.Q = s.NT;
#else
    s.Q = 1;
    while (s.Q < kScanMaxCluster && s.Q < s.NT && (long long)B * s.CG * s.Q < 2 * 148) s.Q *= 2;
#endif
    s.K = (s.NT + s.Q - 1) / s.Q;
    return s;
}

// (what the host emulation exchanges maps through; the GPU kernels need no workspace, the size is kept)
static size_t scan_workspace_floats(int B, int L, int C) {
    return (size_t)3 * B * ((L + 15) / 16) * C;
}

template <bool BWD>
static int run_scan(ScanParams p, float* ws, Stream st) {
    const ScanShape& s = p.s;
    const long long blocks = (long long)s.B * s.CG * s.Q;
#ifdef FIELDS_HOST_EMU
    p.maps = ws;
    return launch_stateful<ScanWalk<BWD>>(p, blocks, 0, st);
#else
    (void)ws;
    if (blocks > 0x7fffffffLL) return FIELDS_ERR_UNSUPPORTED;
    static std::atomic<bool> ready[64];
    int dev = 0;
    int rc = check_cuda(cudaGetDevice(&dev));
    if (rc) return rc;
    if (dev < 0 || dev >= 64) return FIELDS_ERR_UNSUPPORTED;
    if (s.Q > 8 && !ready[dev]) {  // clusters of more than eight blocks are an opt-in (idempotent)
        rc = check_cuda(cudaFuncSetAttribute(scan_walk<BWD>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        if (rc) return rc;
        ready[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(ScanWalk<BWD>::kThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (dependent_launch_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (s.Q > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = s.Q;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return check_cuda(cudaLaunchKernelEx(&cfg, scan_walk<BWD>, p));
#endif
}

static int scan_check(const void* workspace, size_t workspace_bytes, int B, int L, int C,
                      long long a_batch, long long a_step, int a_chan) {
    if (a_chan != 0 && a_chan != 1) return FIELDS_ERR_ARGUMENT;
    if (a_batch < 0 || a_step < 0) return FIELDS_ERR_ARGUMENT;
#ifndef FIELDS_HOST_EMU
    if (!workspace && !workspace_bytes) return FIELDS_OK;  // the GPU kernels use none
#endif
    if (!workspace || workspace_bytes < scan_workspace_floats(B, L, C) * sizeof(float) ||
        (reinterpret_cast<uintptr_t>(workspace) & 15u))
        return FIELDS_ERR_WORKSPACE;
    return FIELDS_OK;
}

template <typename IO>
static int run_step(const IO* raw, const float* tr, const float* ti, const float* gamma,
                    float* state, IO* read, int B, int C, void* stream) {
    if (B < 0 || C <= 0) return FIELDS_ERR_ARGUMENT;
    if (B == 0) return FIELDS_OK;
    if (!raw || !tr || !ti || !gamma || !state || !read) return FIELDS_ERR_ARGUMENT;
    typename DecodeStep<IO>::Params p{raw, tr, ti, gamma, state, read, B, C};
    const long long n = (long long)B * C;
    return launch<DecodeStep<IO>>(p, (n + DecodeStep<IO>::kThreads - 1) / DecodeStep<IO>::kThreads,
                                  reinterpret_cast<Stream>(stream));
}

extern "C" {

int fields_read_step(const float* raw, const float* tr, const float* ti, const float* gamma,
                     float* state, float* read, int B, int C, void* stream) {
    return run_step<float>(raw, tr, ti, gamma, state, read, B, C, stream);
}

int fields_read_step_bf16(const void* raw, const float* tr, const float* ti, const float* gamma,
                          float* state, void* read, int B, int C, void* stream) {
    return run_step<uint16_t>(static_cast<const uint16_t*>(raw), tr, ti, gamma, state,
                              static_cast<uint16_t*>(read), B, C, stream);
}


size_t fields_scan_workspace_bytes(int B, int L, int C) {
    if (B <= 0 || L <= 0 || C <= 0) return 0;
    return scan_workspace_floats(B, L, C) * sizeof(float);
}

int fields_scan_forward(const float* a, long long a_batch, long long a_step, int a_chan,
                        const float* drive, const float* state_in, float* states,
                        float* state_out, void* workspace, size_t workspace_bytes, int B, int L,
                        int C, void* stream) {
    if (B < 0 || L < 0 || C <= 0) return FIELDS_ERR_ARGUMENT;
    Stream st = reinterpret_cast<Stream>(stream);
    if (B == 0) return FIELDS_OK;
    if (L == 0) {
        if (!state_out) return FIELDS_OK;
        if (!state_in) return fill_zero(state_out, (size_t)B * C, st);
#ifdef FIELDS_HOST_EMU
        std::memcpy(state_out, state_in, (size_t)B * C * sizeof(float));
        return FIELDS_OK;
#else
        return check_cuda(cudaMemcpyAsync(state_out, state_in, (size_t)B * C * sizeof(float),
                                          cudaMemcpyDeviceToDevice, st));
#endif
    }
    if (!a || !drive || !states) return FIELDS_ERR_ARGUMENT;
    int rc = scan_check(workspace, workspace_bytes, B, L, C, a_batch, a_step, a_chan);
    if (rc) return rc;
    ScanParams p{};
    p.a = a; p.x = drive; p.first = state_in; p.out = states; p.end = state_out;
    p.s = make_scan_shape(B, L, C, a_batch, a_step, a_chan);
    return run_scan<false>(p, static_cast<float*>(workspace), st);
}

int fields_scan_backward(const float* a, long long a_batch, long long a_step, int a_chan,
                         const float* states, const float* state_in, const float* grad_states,
                         const float* grad_state_out, float* grad_a, float* grad_drive,
                         float* grad_state_in, void* workspace, size_t workspace_bytes, int B,
                         int L, int C, void* stream) {
    if (B < 0 || L < 0 || C <= 0) return FIELDS_ERR_ARGUMENT;
    Stream st = reinterpret_cast<Stream>(stream);
    if (B == 0) return FIELDS_OK;
    if (L == 0) {
        if (!grad_state_in) return FIELDS_OK;
        if (!grad_state_out) return fill_zero(grad_state_in, (size_t)B * C, st);
#ifdef FIELDS_HOST_EMU
        std::memcpy(grad_state_in, grad_state_out, (size_t)B * C * sizeof(float));
        return FIELDS_OK;
#else
        return check_cuda(cudaMemcpyAsync(grad_state_in, grad_state_out,
                                          (size_t)B * C * sizeof(float), cudaMemcpyDeviceToDevice,
                                          st));
#endif
    }
    if (!a || !states || !grad_states || !grad_a || !grad_drive) return FIELDS_ERR_ARGUMENT;
    int rc = scan_check(workspace, workspace_bytes, B, L, C, a_batch, a_step, a_chan);
    if (rc) return rc;
    ScanParams p{};
    p.a = a; p.x = grad_states; p.states = states; p.first = state_in; p.last = grad_state_out;
    p.out = grad_drive; p.grad_a = grad_a; p.end = grad_state_in;
    p.s = make_scan_shape(B, L, C, a_batch, a_step, a_chan);
    return run_scan<true>(p, static_cast<float*>(workspace), st);
}

int fields_read_selftest_wait(void* workspace, size_t workspace_bytes, unsigned max_polls,
                              void* stream) {
    // layout: [ctrl 256 B | agg 4 tiles | incl 4 tiles | out 128 x 2]
    const size_t agg_bytes = 4 * kGroup * 4 * sizeof(float), incl_bytes = 4 * kGroup * 2 * sizeof(float);
    const size_t need = kCtrlHeader * sizeof(unsigned) + agg_bytes + incl_bytes + kGroup * 2 * sizeof(float);
    if (!workspace || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return FIELDS_ERR_WORKSPACE;
    if (max_polls == 0 || max_polls > kMaxPolls) return FIELDS_ERR_ARGUMENT;
    Stream st = reinterpret_cast<Stream>(stream);
    char* ws = static_cast<char*>(workspace);
    int rc = fill_unset(ws, need, st);
    if (rc) return rc;
    float* agg = reinterpret_cast<float*>(ws + kCtrlHeader * sizeof(unsigned));
    float* incl = reinterpret_cast<float*>(ws + kCtrlHeader * sizeof(unsigned) + agg_bytes);
    float* out = reinterpret_cast<float*>(ws + kCtrlHeader * sizeof(unsigned) + agg_bytes + incl_bytes);
    WaitSelfTest::Params p{agg, incl, reinterpret_cast<unsigned*>(ws), out, max_polls};
    rc = launch<WaitSelfTest>(p, 1, st);
    if (rc) return rc;
    return fields_read_device_status(workspace, stream);
}


static bool aligned8(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 7u) == 0; }

}  // extern "C"

template <bool STATS>
static int run_forward_bf16(const void* raw, long long pitch, const float* tr, const float* ti, const float* gamma,
                            const float* state_in, void* read, float* sumsq, float* state_out, void* workspace,
                            int B, int L, int C, void* stream) {
    return run_forward_single_pass<FwdSpBf16<STATS>, uint16_t>(static_cast<const uint16_t*>(raw), tr, ti, gamma, state_in,
                                                               static_cast<uint16_t*>(read), state_out, workspace, B, L, C,
                                                               reinterpret_cast<Stream>(stream), sumsq, pitch);
}

extern "C" {

int fields_read_forward_bf16(const void* raw, const float* tr, const float* ti, const float* gamma,
                             const float* state_in, void* read, float* state_out, void* workspace,
                             size_t workspace_bytes, int B, int L, int C, void* stream) {
    if (B < 0 || L < 0 || C <= 0) return FIELDS_ERR_ARGUMENT;
    if (B == 0 || L == 0) {
        // nothing to scan: the fp32 entry point handles the state pass-through
        return fields_read_forward(nullptr, tr, ti, gamma, state_in, nullptr, state_out, workspace,
                                   workspace_bytes, B, 0, C, stream);
    }
    if (!raw || !read || !tr || !ti || !gamma) return FIELDS_ERR_ARGUMENT;
    if (C % 4 || !aligned8(raw) || !aligned8(read) || !aligned16(tr) || !aligned16(ti) ||
        !aligned16(gamma))
        return FIELDS_ERR_UNSUPPORTED;  // 64-bit accesses only: C % 4 == 0, 8-byte aligned rows
    if (!workspace || workspace_bytes < fields_read_workspace_bytes(B, L, C, FIELDS_PASS_FORWARD) ||
        (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return FIELDS_ERR_WORKSPACE;
    return run_forward_bf16<false>(raw, 3LL * C, tr, ti, gamma, state_in, read, nullptr, state_out, workspace, B,
                                   L, C, stream);
}

int fields_read_forward_bf16_stats(const void* raw, const float* tr, const float* ti,
                                   const float* gamma, const float* state_in, void* read,
                                   float* sumsq, float* state_out, void* workspace,
                                   size_t workspace_bytes, int B, int L, int C, void* stream) {
    if (B <= 0 || L <= 0 || C <= 0) return FIELDS_ERR_ARGUMENT;
    if (!raw || !read || !sumsq || !tr || !ti || !gamma) return FIELDS_ERR_ARGUMENT;
    if (C % 4 || !aligned8(raw) || !aligned8(read) || !aligned16(tr) || !aligned16(ti) ||
        !aligned16(gamma))
        return FIELDS_ERR_UNSUPPORTED;
    if (!workspace || workspace_bytes < fields_read_workspace_bytes(B, L, C, FIELDS_PASS_FORWARD) ||
        (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return FIELDS_ERR_WORKSPACE;
    return run_forward_bf16<true>(raw, 3LL * C, tr, ti, gamma, state_in, read, sumsq, state_out, workspace, B, L,
                                  C, stream);
}

int fields_read_backward_bf16(const void* raw, const float* tr, const float* ti, const float* gamma,
                              const float* state_in, const void* read, const void* grad_read,
                              const float* grad_state_out, void* grad_raw, float* grad_tr,
                              float* grad_ti, float* grad_gamma, float* grad_state_in,
                              void* workspace, size_t workspace_bytes, int B, int L, int C,
                              void* stream) {
    if (B < 0 || L < 0 || C <= 0) return FIELDS_ERR_ARGUMENT;
    if (B == 0 || L == 0)
        return fields_read_backward(nullptr, tr, ti, gamma, state_in, nullptr, nullptr, grad_state_out,
                                    nullptr, grad_tr, grad_ti, grad_gamma, grad_state_in, workspace,
                                    workspace_bytes, B, 0, C, stream);
    if (!raw || !read || !grad_read || !grad_raw || !tr || !ti || !gamma || !grad_tr || !grad_ti ||
        !grad_gamma)
        return FIELDS_ERR_ARGUMENT;
    if (C % 4 || !aligned8(raw) || !aligned8(read) || !aligned8(grad_read) || !aligned8(grad_raw) ||
        !aligned16(tr) || !aligned16(ti) || !aligned16(gamma) || !aligned16(state_in))
        return FIELDS_ERR_UNSUPPORTED;
    if (!workspace ||
        workspace_bytes < fields_read_workspace_bytes(B, L, C, FIELDS_PASS_BACKWARD) ||
        (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return FIELDS_ERR_WORKSPACE;
    return run_backward_single_pass<BwdSpBf16, uint16_t>(
        static_cast<const uint16_t*>(raw), tr, ti, gamma, state_in,
        static_cast<const uint16_t*>(read), static_cast<const uint16_t*>(grad_read), grad_state_out,
        static_cast<uint16_t*>(grad_raw), grad_tr, grad_ti, grad_gamma, grad_state_in, workspace,
        B, L, C, reinterpret_cast<Stream>(stream));
}


size_t fields_read_mailbox_bytes(int P, int B, int C) {
    if (P <= 0 || B <= 0 || C <= 0) return 0;
    return mailbox_slot_bytes(P, B, C) + mailbox_board_bytes(B, C) + mailbox_sum_bytes(P, C);
}

int fields_read_sum_over_ranks(const float* values, float* out, int n, void* const* mailboxes,
                               unsigned* error_word, int rank, int P, unsigned epoch,
                               unsigned max_polls, int B, int C, void* stream) {
    if (B <= 0 || C <= 0 || P <= 0 || P > kMaxRanks || rank < 0 || rank >= P || epoch == 0 || n < 0 ||
        n > mailbox_sum_capacity(C))
        return FIELDS_ERR_ARGUMENT;
    if (n == 0) return FIELDS_OK;
    if (!values || !out || !mailboxes || !error_word) return FIELDS_ERR_ARGUMENT;
    SumMailbox::Params p{};
    p.values = values; p.out = out; p.error = error_word;
    const size_t off = mailbox_slot_bytes(P, B, C) + mailbox_board_bytes(B, C);
    for (int r = 0; r < P; ++r) {
        if (!mailboxes[r] || (reinterpret_cast<uintptr_t>(mailboxes[r]) & 7u)) return FIELDS_ERR_ARGUMENT;
        p.region[r] = reinterpret_cast<MailPair*>(static_cast<char*>(mailboxes[r]) + off);
    }
    p.rank = rank; p.P = P; p.n = n; p.n_max = mailbox_sum_capacity(C);
    p.epoch = epoch; p.max_polls = poll_bound(max_polls);
    p.stages = 3;
#ifdef FIELDS_HOST_EMU
    p.stages = g_emu_span_stages & 3;  // the CPU tests run every rank's stores before any rank's wait
#endif
    return launch<SumMailbox>(p, (n + SumMailbox::kThreads - 1) / SumMailbox::kThreads,
                              reinterpret_cast<Stream>(stream));
}

int fields_read_forward_sharded(const float* raw, const float* tr, const float* ti,
                                const float* gamma, const float* state0, float* read,
                                float* state_out, float* summary, void* const* mailboxes,
                                unsigned* error_word, int rank, int P, unsigned epoch,
                                unsigned max_polls, int B, int L, int C, void* stream) {
    if (B < 0 || L <= 0 || C <= 0 || P <= 0 || P > kMaxRanks || rank < 0 || rank >= P)
        return FIELDS_ERR_ARGUMENT;
#ifdef FIELDS_HOST_EMU
    if (epoch == 0) return FIELDS_ERR_ARGUMENT;  // the emulation runs a call as several partial launches
#endif
    if (B == 0) return FIELDS_OK;
    if (!raw || !tr || !ti || !gamma || !read || !mailboxes || !error_word) return FIELDS_ERR_ARGUMENT;
    for (int r = 0; r < P; ++r)
        if (!mailboxes[r] || (reinterpret_cast<uintptr_t>(mailboxes[r]) & 255u)) return FIELDS_ERR_ARGUMENT;
    if (C % 4 != 0 || !aligned16(raw) || !aligned16(read) || !aligned16(tr) || !aligned16(ti) ||
        !aligned16(gamma))
        return FIELDS_ERR_UNSUPPORTED;
    Stream st = reinterpret_cast<Stream>(stream);
    const int grid_max = span_grid<SpanFwd>();
    if (grid_max <= 0) return FIELDS_ERR_LAUNCH;
    SpanFwdParams p{};
    p.raw = raw; p.tr = tr; p.ti = ti; p.gamma = gamma; p.state0 = state0;
    p.read = read; p.state_out = state_out; p.summary = summary;
    p.s = make_span_shape<SpanFwd>(B, L, C, grid_max);
    char* board = static_cast<char*>(mailboxes[rank]) + mailbox_slot_bytes(P, B, C);
    p.count = reinterpret_cast<unsigned*>(board);
    p.ready = p.count + p.s.chains;
    p.runmap = reinterpret_cast<float*>(board + board_count_bytes(B, C));
    p.emu_round = -1;
    p.error = error_word;
    for (int r = 0; r < P; ++r) p.mailbox[r] = static_cast<MailPair*>(mailboxes[r]);
    p.own = static_cast<const MailPair*>(mailboxes[rank]);
    p.rank = rank; p.P = P; p.epoch = epoch;
    // epoch 0: the epoch lives on the rank's board and the kernel advances it itself
    p.epoch_word = epoch == 0 ? reinterpret_cast<unsigned*>(board + board_epoch_offset(B, C)) : nullptr;
    p.max_polls = poll_bound(max_polls);
    p.stages = 3;
#ifdef FIELDS_HOST_EMU
    p.stages = g_emu_span_stages;  // the CPU tests run the ranks' first sweeps before any rank's wait
#endif
    const int grid = p.s.items < grid_max ? p.s.items : grid_max;
    return launch_span<SpanFwd>(p, grid, st);
}

int fields_read_span_summary_put(const float* raw, const float* tr, const float* ti,
                                 const float* gamma, void* const* mailboxes, float* summary,
                                 int rank, int P, unsigned epoch, void* workspace,
                                 size_t workspace_bytes, int B, int L, int C, void* stream) {
    if (B < 0 || L <= 0 || C <= 0 || P <= 0 || P > kMaxRanks || rank < 0 || rank >= P || epoch == 0)
        return FIELDS_ERR_ARGUMENT;
    if (B == 0) return FIELDS_OK;
    if (!raw || !tr || !ti || !gamma || !mailboxes) return FIELDS_ERR_ARGUMENT;
    for (int r = 0; r < P; ++r)
        if (!mailboxes[r] || (reinterpret_cast<uintptr_t>(mailboxes[r]) & 7u)) return FIELDS_ERR_ARGUMENT;
    Stream st = reinterpret_cast<Stream>(stream);
    const bool vec4 = C % 4 == 0 && aligned16(raw) && aligned16(tr) && aligned16(ti) &&
                      aligned16(gamma) && aligned16(workspace);
    Plan pl = make_plan(B, L, C, vec4 ? 4 : 1);
    if (!workspace || workspace_bytes < pl.fwd_floats * sizeof(float) ||
        (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return FIELDS_ERR_WORKSPACE;
    float* ws = static_cast<float*>(workspace);
    FwdParams p{raw, tr, ti, gamma, nullptr, nullptr, nullptr, ws + pl.sum_off, ws + pl.carry_off,
                pl.s};
    int rc;
    if (vec4) {
        using Stream4 = ChunkSummaryStream<2, 3, 4>;
        p.s.ts = 16;
        p.s.N = (L + 63) / 64;
        p.s.G = (C + 127) / 128;
        rc = launch<Stream4>(p, (long long)B * p.s.N * p.s.G, st);
    } else {
        rc = launch<FwdSummary<1, 4>>(p, tile_blocks(pl.s), st);
    }
    if (rc) return rc;
    PutSummary::Params pp{};
    pp.sum = p.sum;
    for (int r = 0; r < P; ++r) pp.mailbox[r] = static_cast<MailPair*>(mailboxes[r]);
    pp.summary = summary;
    pp.rank = rank; pp.P = P; pp.epoch = epoch;
    pp.s = p.s;
    pp.reverse = 0;
    return launch<PutSummary>(pp, (long long)B * ((C + 31) / 32), st);
}

int fields_read_span_summary_backward_put(const float* raw, const float* tr, const float* ti,
                                          const float* grad_read, void* const* mailboxes,
                                          float* summary, int rank, int P, unsigned epoch,
                                          void* workspace, size_t workspace_bytes, int B, int L,
                                          int C, void* stream) {
    if (B < 0 || L <= 0 || C <= 0 || P <= 0 || P > kMaxRanks || rank < 0 || rank >= P || epoch == 0)
        return FIELDS_ERR_ARGUMENT;
    if (B == 0) return FIELDS_OK;
    if (!raw || !tr || !ti || !grad_read || !mailboxes) return FIELDS_ERR_ARGUMENT;
    for (int r = 0; r < P; ++r)
        if (!mailboxes[r] || (reinterpret_cast<uintptr_t>(mailboxes[r]) & 7u)) return FIELDS_ERR_ARGUMENT;
    Stream st = reinterpret_cast<Stream>(stream);
    const bool vec4 = C % 4 == 0 && aligned16(raw) && aligned16(tr) && aligned16(ti) &&
                      aligned16(grad_read) && aligned16(workspace);
    const Plan pl = make_plan(B, L, C, vec4 ? 4 : 1);
    if (!workspace || workspace_bytes < pl.bwd_floats * sizeof(float) ||
        (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return FIELDS_ERR_WORKSPACE;
    float* ws = static_cast<float*>(workspace);
    BwdParams p{};
    p.raw = raw; p.tr = tr; p.ti = ti; p.grad_read = grad_read;
    p.sum = ws + pl.sum_off;
    p.s = pl.s;
    int rc;
    if (vec4) {
        using Stream4 = ChunkDualSummaryStream<1, 3, 4>;
        p.s.ts = 16;
        p.s.N = (L + 63) / 64;
        p.s.G = (C + 127) / 128;
        rc = launch<Stream4>(p, (long long)B * p.s.N * p.s.G, st);
    } else {
        rc = launch<BwdSummary<1, 4>>(p, tile_blocks(pl.s), st);
    }
    if (rc) return rc;
    PutSummary::Params pp{};
    pp.sum = p.sum;
    for (int r = 0; r < P; ++r) pp.mailbox[r] = static_cast<MailPair*>(mailboxes[r]);
    pp.summary = summary;
    pp.rank = rank; pp.P = P; pp.epoch = epoch;
    pp.s = p.s;
    pp.reverse = 1;
    return launch<PutSummary>(pp, (long long)B * ((C + 31) / 32), st);
}

int fields_read_fold_mailbox(const void* mailbox, const float* state0, float* state,
                             unsigned* error_word, int rank, int P, unsigned epoch,
                             unsigned max_polls, int B, int C, void* stream) {
    if (B < 0 || C <= 0 || P <= 0 || P > kMaxRanks || rank < 0 || rank >= P || epoch == 0)
        return FIELDS_ERR_ARGUMENT;
    if (B == 0) return FIELDS_OK;
    if (!mailbox || !state || !error_word) return FIELDS_ERR_ARGUMENT;
    FoldMailbox::Params p{static_cast<const MailPair*>(mailbox), state0, state, error_word,
                          rank, P, B, C, epoch, poll_bound(max_polls), 0};
    const long long n = (long long)B * C;
    return launch<FoldMailbox>(p, (n + FoldMailbox::kThreads - 1) / FoldMailbox::kThreads,
                               reinterpret_cast<Stream>(stream));
}

int fields_read_fold_mailbox_backward(const void* mailbox, const float* carry_end, float* carry,
                                      unsigned* error_word, int rank, int P, unsigned epoch,
                                      unsigned max_polls, int B, int C, void* stream) {
    if (B < 0 || C <= 0 || P <= 0 || P > kMaxRanks || rank < 0 || rank >= P || epoch == 0)
        return FIELDS_ERR_ARGUMENT;
    if (B == 0) return FIELDS_OK;
    if (!mailbox || !carry || !error_word) return FIELDS_ERR_ARGUMENT;
    FoldMailbox::Params p{static_cast<const MailPair*>(mailbox), carry_end, carry, error_word,
                          rank, P, B, C, epoch, poll_bound(max_polls), 1};
    const long long n = (long long)B * C;
    return launch<FoldMailbox>(p, (n + FoldMailbox::kThreads - 1) / FoldMailbox::kThreads,
                               reinterpret_cast<Stream>(stream));
}

int fields_read_forward_bf16_tensor(const void* raw, const float* tr, const float* ti,
                                    const float* gamma, const float* state_in, void* read,
                                    float* state_out, unsigned* error_word, int B, int L, int C,
                                    void* stream) {
    if (B < 0 || L <= 0 || C <= 0) return FIELDS_ERR_ARGUMENT;
    if (B == 0) return FIELDS_OK;
    if (!raw || !read || !tr || !ti || !gamma || !error_word) return FIELDS_ERR_ARGUMENT;
    if (C % 4 || !aligned8(raw) || !aligned8(read)) return FIELDS_ERR_UNSUPPORTED;
    TensorFwdParams p{static_cast<const uint16_t*>(raw), tr, ti, gamma, state_in,
                      static_cast<uint16_t*>(read), state_out, error_word, B, L, C, kMaxPolls};
    const long long grid = (long long)B * ((C + kTcChannels - 1) / kTcChannels);
    if (grid > 0x7fffffffLL) return FIELDS_ERR_UNSUPPORTED;
#ifdef FIELDS_HOST_EMU
    (void)stream;
    std::vector<double> store(kTcSmemBytesEmu / 8 + 2);
    for (long long block = 0; block < grid; ++block)
        FwdTensorChain::run_block_emu(p, (int)block, reinterpret_cast<char*>(store.data()));
    return FIELDS_OK;
#else
    static bool ready[64] = {};
    const int rc = allow_shared_memory(tensor_chain_entry, (size_t)kTcSmemBytes, ready);
    if (rc) return rc;
    return launch_on<TensorFwdParams>(tensor_chain_entry, (unsigned)grid, kTcThreads, kTcSmemBytes,
                                      reinterpret_cast<Stream>(stream), p);
#endif
}

#ifdef FIELDS_HOST_EMU
// Host emulation only: which parts fields_read_forward_sharded runs (bit 0: first sweep,
// bit 2: prefix maps and the store of the span's map into the mailboxes, bit 1: the same plus
// the wait and the second sweep), so a test can emulate several ranks in turn.
void fields_emu_span_stages(int stages) { g_emu_span_stages = stages; }
#endif

#ifndef FIELDS_HOST_EMU
size_t fields_mixer_epilogue_bias_rows(long long N) {
    return N > 0 ? (size_t)((N + kEpiRows - 1) / kEpiRows) : 0;
}

int fields_mixer_epilogue_forward(const float* x, const void* acc, const void* gate,
                                  const float* sumsq, const float* bias, const float* gate_bias,
                                  float* y, float eps, int features, long long N, int D,
                                  void* stream) {
    if (N < 0 || D <= 0 || features <= 0) return FIELDS_ERR_ARGUMENT;
    if (N == 0) return FIELDS_OK;
    if (!x || !acc || !gate || !sumsq || !bias || !y) return FIELDS_ERR_ARGUMENT;
    if (D % 4 || !aligned16(x) || !aligned16(y) || !aligned16(bias) || !aligned16(gate_bias) ||
        !aligned8(acc) || !aligned8(gate))
        return FIELDS_ERR_UNSUPPORTED;
    const long long blocks = (N + kEpiRows - 1) / kEpiRows;
    if (blocks > 0x7fffffffLL) return FIELDS_ERR_UNSUPPORTED;
    EpilogueParams p{x, static_cast<const uint16_t*>(acc), static_cast<const uint16_t*>(gate), sumsq,
                     bias, gate_bias, y, eps, 1.0f / (float)features, N, D};
    return launch_on<EpilogueParams>(epilogue_forward, (unsigned)blocks, kEpiThreads, 0,
                                     reinterpret_cast<Stream>(stream), p);
}

int fields_mixer_epilogue_backward(const float* grad_y, const void* acc, const void* gate,
                                   const float* sumsq, const float* bias, const float* gate_bias,
                                   void* grad_acc, void* grad_gate, float* grad_sumsq,
                                   float* grad_bias_rows, float* grad_gate_bias_rows, float eps,
                                   int features, long long N, int D, void* stream) {
    if (N < 0 || D <= 0 || features <= 0) return FIELDS_ERR_ARGUMENT;
    if (N == 0) return FIELDS_OK;
    if (!grad_y || !acc || !gate || !sumsq || !bias || !grad_acc || !grad_gate || !grad_sumsq ||
        !grad_bias_rows || (gate_bias && !grad_gate_bias_rows))
        return FIELDS_ERR_ARGUMENT;
    if (D % 4 || D > kEpiMaxD || !aligned16(grad_y) || !aligned16(bias) || !aligned16(gate_bias) ||
        !aligned16(grad_bias_rows) || !aligned16(grad_gate_bias_rows) || !aligned8(acc) ||
        !aligned8(gate) || !aligned8(grad_acc) || !aligned8(grad_gate))
        return FIELDS_ERR_UNSUPPORTED;
    const long long blocks = (N + kEpiRows - 1) / kEpiRows;
    if (blocks > 0x7fffffffLL) return FIELDS_ERR_UNSUPPORTED;
    EpilogueGradParams p{grad_y, static_cast<const uint16_t*>(acc),
                         static_cast<const uint16_t*>(gate), sumsq, bias, gate_bias,
                         static_cast<uint16_t*>(grad_acc), static_cast<uint16_t*>(grad_gate),
                         grad_sumsq, grad_bias_rows, grad_gate_bias_rows, eps,
                         1.0f / (float)features, N, D};
    return launch_on<EpilogueGradParams>(epilogue_backward, (unsigned)blocks, kEpiThreads, 0,
                                         reinterpret_cast<Stream>(stream), p);
}

int fields_read_norm_grad_combine(const void* grad_read, const void* read, const float* grad_sumsq,
                                  void* total, long long N, int F, void* stream) {
    if (N < 0 || F <= 0) return FIELDS_ERR_ARGUMENT;
    if (N == 0) return FIELDS_OK;
    if (!read || !grad_sumsq || !total) return FIELDS_ERR_ARGUMENT;
    if (F % 4 || !aligned8(grad_read) || !aligned8(read) || !aligned8(total))
        return FIELDS_ERR_UNSUPPORTED;
    const long long blocks = (N + kEpiRows - 1) / kEpiRows;
    if (blocks > 0x7fffffffLL) return FIELDS_ERR_UNSUPPORTED;
    NormGradParams p{static_cast<const uint16_t*>(grad_read), static_cast<const uint16_t*>(read),
                     grad_sumsq, static_cast<uint16_t*>(total), N, F};
    return launch_on<NormGradParams>(norm_grad_combine, (unsigned)blocks, kEpiThreads, 0,
                                     reinterpret_cast<Stream>(stream), p);
}

}  // extern "C"

// The layout of one block; the number of thread blocks it takes in *blocks.
static int layout_params(const struct fields_stack_weights* w, const float* ff_norm_w, int parts, LayoutParams& p,
                         long long* blocks) {
    if (!w || w->dim <= 0 || w->hidden < 0) return FIELDS_ERR_ARGUMENT;
    const bool rest = parts & FIELDS_LAYOUT_REST, w12 = parts & (FIELDS_LAYOUT_W12 | FIELDS_LAYOUT_W12_STEP),
               step = parts & FIELDS_LAYOUT_W12_STEP;
    if (step && (!ff_norm_w || !aligned16(ff_norm_w))) return ff_norm_w ? FIELDS_ERR_UNSUPPORTED : FIELDS_ERR_ARGUMENT;
    if (!w->write_w || !w->write_b || !w->gate_w || !w->out_w || !w->read_norm_w || !w->radius_logit ||
        !w->theta || !w->in_w || !w->in_b || !w->out_w16 || !w->par ||
        (w->hidden && (!w->w3 || !w->w3_16 || (w12 && (!w->w12 || !w->w12_16)))))
        return FIELDS_ERR_ARGUMENT;
    const long long D = w->dim, H = w->hidden, C = D / 2;
    const void* all[] = {w->write_w, w->write_b, w->gate_w, w->out_w, w->read_norm_w, w->w12, w->w3,
                         w->in_w, w->in_b, w->out_w16, w->w12_16, w->w3_16};
    if (D % 8 || H % 8) return FIELDS_ERR_UNSUPPORTED;
    for (const void* q : all)
        if (!aligned16(q)) return FIELDS_ERR_UNSUPPORTED;
    uint16_t* in_w = static_cast<uint16_t*>(w->in_w);
    p.piece[0] = {w->write_w, in_w, nullptr, 3 * C * D, (int)D};
    p.piece[1] = {w->gate_w, in_w + 3 * C * D, nullptr, D * D, (int)D};
    p.piece[2] = {w->write_b, static_cast<uint16_t*>(w->in_b), nullptr, 3 * C, (int)(3 * C)};
    p.piece[3] = {w->out_w, static_cast<uint16_t*>(w->out_w16), w->read_norm_w, D * 2 * D, (int)(2 * D)};
    p.piece[4] = {w->w12, static_cast<uint16_t*>(w->w12_16), step ? ff_norm_w : nullptr, 2 * H * D, (int)D, step ? (int)H : 0};
    p.piece[5] = {w->w3, static_cast<uint16_t*>(w->w3_16), nullptr, D * H, (int)H};
    p.piece[6] = {nullptr, static_cast<uint16_t*>(w->in_b) + 3 * C, nullptr, D, (int)D};
    p.radius_logit = w->radius_logit; p.theta = w->theta; p.par = w->par; p.C = (int)C;
    p.piece[7] = {nullptr, nullptr, nullptr, 0, 4};
    for (int k = 0; k < kLayoutPieces; ++k)
        if (!(k == 4 ? w12 : rest)) p.piece[k].n = 0;
    long long at = 0;
    for (int k = 0; k < kLayoutPieces; ++k) {
        p.first[k] = at;
        at += (p.piece[k].n + kLayoutChunk - 1) / kLayoutChunk;
    }
    p.first[kLayoutPieces] = at;
    *blocks = at + (rest ? (C + kRowThreads - 1) / kRowThreads : 0);
    return *blocks > 0x7fffffffLL ? FIELDS_ERR_UNSUPPORTED : FIELDS_OK;
}

extern "C" {

int fields_stack_layout(const struct fields_stack_weights* w, int count, void* stream) {
    return fields_stack_layout_parts(w, nullptr, count, FIELDS_LAYOUT_REST | FIELDS_LAYOUT_W12, stream);
}

int fields_stack_layout_parts(const struct fields_stack_weights* w, const float* const* ff_norm_w, int count, int parts,
                              void* stream) {
    const int both = FIELDS_LAYOUT_W12 | FIELDS_LAYOUT_W12_STEP;
    if (!w || count <= 0 || parts <= 0 || (parts & ~(FIELDS_LAYOUT_REST | both)) || (parts & both) == both ||
        ((parts & FIELDS_LAYOUT_W12_STEP) && !ff_norm_w))
        return FIELDS_ERR_ARGUMENT;
    for (int i = 0; i < count; i += kLayoutBlocks) {
        LayoutBatch batch{};
        const int n = count - i < kLayoutBlocks ? count - i : kLayoutBlocks;
        long long blocks = 0;
        for (int k = 0; k < n; ++k) {
            if (w[i + k].dim != w[0].dim || w[i + k].hidden != w[0].hidden) return FIELDS_ERR_ARGUMENT;
            const int rc = layout_params(&w[i + k], ff_norm_w ? ff_norm_w[i + k] : nullptr, parts, batch.block[k], &blocks);
            if (rc) return rc;
        }
        if (blocks == 0) continue;
        const int rc = launch_grid<LayoutBatch>(layout_block, dim3((unsigned)blocks, (unsigned)n), kRowThreads,
                                                reinterpret_cast<Stream>(stream), batch);
        if (rc) return rc;
    }
    return FIELDS_OK;
}

int fields_stack_step_norm(const void* raw, long long raw_stride, const float* par, float* state,
                           void* out, float eps, long long N, int C, void* stream) {
    if (N < 0 || C <= 0) return FIELDS_ERR_ARGUMENT;
    if (N == 0) return FIELDS_OK;
    if (!raw || !par || !state || !out) return FIELDS_ERR_ARGUMENT;
    if (C % 4 || C > 2048 || raw_stride % 4 || N > 0x7fffffffLL || !aligned8(raw) || !aligned16(par) ||
        !aligned16(state) || !aligned8(out))
        return FIELDS_ERR_UNSUPPORTED;
    StepNormParams p{static_cast<const uint16_t*>(raw), par, state, static_cast<uint16_t*>(out), N,
                     raw_stride, C, eps};
    return launch_on<StepNormParams>(C <= 512 ? step_norm<1> : step_norm<4>, (unsigned)N, 128, 0,
                                     reinterpret_cast<Stream>(stream), p);
}

}  // extern "C"

// Which of the row kernels: one warp per row where that already fills the GPU (148 SMs of 32 warps) and
// a row fits a warp's registers, four warps per row otherwise (fewer rows: shorter chains per thread).
template <class P>
static int launch_rows(void (*one)(const P), void (*four)(const P), void (*wide)(const P), long long N,
                       int D, void* stream, const P& p) {
    const bool single = D <= 1024 && N >= 148 * 32;
    const long long per_block = single ? kRowThreads / 32 : kRowThreads / 128;
    const long long blocks = (N + per_block - 1) / per_block;
    if (blocks > 0x7fffffffLL) return FIELDS_ERR_UNSUPPORTED;
    return launch_on<P>(single ? one : D <= 1024 ? four : wide, (unsigned)blocks, kRowThreads, 0,
                        reinterpret_cast<Stream>(stream), p);
}

extern "C" {

int fields_stack_close_mixer(const float* x, const void* acc, const void* gate, long long gate_stride,
                             const float* groups, int G, const float* bias, const float* gate_bias,
                             const float* norm_w, float* y, void* h, float eps, int features,
                             float norm_eps, long long N, int D, void* stream) {
    if (N < 0 || D <= 0 || features <= 0 || G < 0) return FIELDS_ERR_ARGUMENT;
    if (N == 0) return FIELDS_OK;
    if (!x || !acc || !gate || !bias || !y || (h && !norm_w)) return FIELDS_ERR_ARGUMENT;
    if (D % 4 || D > 4096 || gate_stride % 4 || !aligned16(x) || !aligned16(y) || !aligned16(bias) ||
        !aligned16(gate_bias) || !aligned16(norm_w) || !aligned8(acc) || !aligned8(gate) || !aligned8(h))
        return FIELDS_ERR_UNSUPPORTED;
    CloseMixerParams p{x, static_cast<const uint16_t*>(acc), static_cast<const uint16_t*>(gate), groups,
                       bias, gate_bias, norm_w, y, static_cast<uint16_t*>(h), N, gate_stride, D, G, eps,
                       1.0f / (float)features, norm_eps};
    return launch_rows<CloseMixerParams>(close_mixer<1, 8>, close_mixer<4, 2>, close_mixer<4, 8>, N, D,
                                         stream, p);
}

int fields_stack_swiglu(const void* uv, void* out, long long N, int H, void* stream) {
    if (N < 0 || H <= 0) return FIELDS_ERR_ARGUMENT;
    if (N == 0) return FIELDS_OK;
    if (!uv || !out) return FIELDS_ERR_ARGUMENT;
    if (H % 8 || !aligned16(uv) || !aligned16(out)) return FIELDS_ERR_UNSUPPORTED;
    const long long blocks = (N * (H / 8) + kRowThreads - 1) / kRowThreads;
    if (blocks > 0x7fffffffLL) return FIELDS_ERR_UNSUPPORTED;
    SwigluParams p{static_cast<const uint16_t*>(uv), static_cast<uint16_t*>(out), N, H};
    return launch_on<SwigluParams>(swiglu, (unsigned)blocks, kRowThreads, 0,
                                   reinterpret_cast<Stream>(stream), p);
}

int fields_stack_close_ff(const float* x, const void* f, const float* norm_w, float* y, void* h,
                          float norm_eps, long long N, int D, void* stream) {
    if (N < 0 || D <= 0) return FIELDS_ERR_ARGUMENT;
    if (N == 0) return FIELDS_OK;
    if (!x || (!h && !y)) return FIELDS_ERR_ARGUMENT;
    if (D % 4 || D > 4096 || !aligned16(x) || !aligned16(y) || !aligned16(norm_w) || !aligned8(f) ||
        !aligned8(h))
        return FIELDS_ERR_UNSUPPORTED;
    if (!norm_w) {
        const long long n = N * D, per = 4LL * 4 * kRowThreads, blocks = (n + per - 1) / per;
        if (blocks > 0x7fffffffLL) return FIELDS_ERR_UNSUPPORTED;
        AddCastParams p{x, static_cast<const uint16_t*>(f), y, static_cast<uint16_t*>(h), n};
        return launch_on<AddCastParams>(add_cast, (unsigned)blocks, kRowThreads, 0, reinterpret_cast<Stream>(stream), p);
    }
    CloseFfParams p{x, static_cast<const uint16_t*>(f), norm_w, y, static_cast<uint16_t*>(h), N, D, norm_eps};
    return launch_rows<CloseFfParams>(close_ff<1, 8>, close_ff<4, 2>, close_ff<4, 8>, N, D, stream, p);
}

int fields_read_forward_bf16_rows(const void* raw, long long raw_pitch, const float* tr, const float* ti,
                                  const float* gamma, const float* state_in, void* read, float* sumsq,
                                  float* state_out, void* workspace, size_t workspace_bytes, int B, int L,
                                  int C, void* stream) {
    if (B <= 0 || L <= 0 || C <= 0 || raw_pitch < 3LL * C || raw_pitch > 0x7fffffffLL) return FIELDS_ERR_ARGUMENT;
    if (!raw || !read || !tr || !ti || !gamma) return FIELDS_ERR_ARGUMENT;
    if (C % 4 || raw_pitch % 4 || !aligned8(raw) || !aligned8(read) || !aligned16(tr) || !aligned16(ti) ||
        !aligned16(gamma))
        return FIELDS_ERR_UNSUPPORTED;
    if (!workspace || workspace_bytes < fields_read_workspace_bytes(B, L, C, FIELDS_PASS_FORWARD) ||
        (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return FIELDS_ERR_WORKSPACE;
    if (sumsq)
        return run_forward_bf16<true>(raw, raw_pitch, tr, ti, gamma, state_in, read, sumsq, state_out, workspace, B,
                                      L, C, stream);
    return run_forward_bf16<false>(raw, raw_pitch, tr, ti, gamma, state_in, read, nullptr, state_out, workspace, B, L,
                                   C, stream);
}

int fields_read_backward_bf16_rows(const void* raw, long long raw_pitch, const float* tr, const float* ti,
                                   const float* gamma, const void* read, const void* grad_read, void* grad_raw,
                                   long long grad_pitch, float* grad_tr, float* grad_ti, float* grad_gamma,
                                   void* workspace, size_t workspace_bytes, int B, int L, int C, void* stream) {
    if (B <= 0 || L <= 0 || C <= 0 || raw_pitch < 3LL * C || raw_pitch > 0x7fffffffLL || grad_pitch < 3LL * C ||
        grad_pitch > 0x7fffffffLL)
        return FIELDS_ERR_ARGUMENT;
    if (!raw || !read || !grad_read || !grad_raw || !tr || !ti || !gamma || !grad_tr || !grad_ti || !grad_gamma)
        return FIELDS_ERR_ARGUMENT;
    if (C % 4 || raw_pitch % 4 || grad_pitch % 4 || !aligned8(raw) || !aligned8(read) || !aligned8(grad_read) ||
        !aligned8(grad_raw) || !aligned16(tr) || !aligned16(ti) || !aligned16(gamma))
        return FIELDS_ERR_UNSUPPORTED;
    if (!workspace || workspace_bytes < fields_read_workspace_bytes(B, L, C, FIELDS_PASS_BACKWARD) ||
        (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return FIELDS_ERR_WORKSPACE;
    return run_backward_single_pass<BwdSpBf16, uint16_t>(
        static_cast<const uint16_t*>(raw), tr, ti, gamma, nullptr, static_cast<const uint16_t*>(read),
        static_cast<const uint16_t*>(grad_read), nullptr, static_cast<uint16_t*>(grad_raw), grad_tr, grad_ti,
        grad_gamma, nullptr, workspace, B, L, C, reinterpret_cast<Stream>(stream), nullptr, raw_pitch, grad_pitch);
}

// Rows of one block of open_grad: one round of blocks over the GPU, within what its shared memory holds.
static int grad_rows_per_block(long long N) {
    long long per = (N + kGradBlocks - 1) / kGradBlocks;
    per = (per + 3) / 4 * 4;
    return (int)(per < 4 ? 4 : per > kGradRowsMax ? kGradRowsMax : per);
}
constexpr int kColumnBlocks = 296, kWeightBlocks = 64;  // row blocks of column_sums and out_weight_grad

size_t fields_mixer_grad_rows(long long N) {
    const long long per = grad_rows_per_block(N);
    return N > 0 ? (size_t)((N + per - 1) / per) : 0;
}

size_t fields_mixer_grad_scratch_bytes(int D) {
    return D > 0 ? ((size_t)kColumnBlocks * (3 * (D / 2)) + (size_t)kWeightBlocks * 2 * D) * sizeof(float) : 0;
}

int fields_mixer_open_grad(const float* grad_y, const void* acc, const void* gate, long long gate_pitch,
                           const float* groups, int G, const float* bias, const float* gate_bias, void* grad_acc,
                           void* grad_gate, long long grad_pitch, float* grad_sumsq, float* rows, float eps,
                           int features, long long N, int D, void* stream) {
    if (N <= 0 || D <= 0 || features <= 0 || G <= 0) return FIELDS_ERR_ARGUMENT;
    if (!grad_y || !acc || !gate || !groups || !bias || !gate_bias || !grad_acc || !grad_gate || !grad_sumsq || !rows)
        return FIELDS_ERR_ARGUMENT;
    if (D % 4 || D > 4096 || gate_pitch % 4 || grad_pitch % 4 || !aligned16(grad_y) || !aligned16(bias) ||
        !aligned16(gate_bias) || !aligned16(rows) || !aligned8(acc) || !aligned8(gate) || !aligned8(grad_acc) ||
        !aligned8(grad_gate))
        return FIELDS_ERR_UNSUPPORTED;
    OpenGradParams p{grad_y, static_cast<const uint16_t*>(acc), static_cast<const uint16_t*>(gate), groups, bias,
                     gate_bias, static_cast<uint16_t*>(grad_acc), static_cast<uint16_t*>(grad_gate), grad_sumsq,
                     rows, N, gate_pitch, grad_pitch, D, G, grad_rows_per_block(N), eps, 1.0f / (float)features};
    const size_t blocks = fields_mixer_grad_rows(N);
    if (blocks > 0x7fffffffu) return FIELDS_ERR_UNSUPPORTED;
    Stream st = reinterpret_cast<Stream>(stream);
    if (D <= 4 * kRowThreads) {
        int threads = (D / 4 + 31) / 32 * 32;
        if (threads < kGradRowsMax) threads = kGradRowsMax;  // one thread per row at the end
        return launch_on<OpenGradParams>(open_grad<1, 2>, (unsigned)blocks, (unsigned)threads, 0, st, p);
    }
    if (D <= 8 * kRowThreads) return launch_on<OpenGradParams>(open_grad<2, 1>, (unsigned)blocks, kRowThreads, 0, st, p);
    return launch_on<OpenGradParams>(open_grad<4, 1>, (unsigned)blocks, kRowThreads, 0, st, p);
}

int fields_mixer_close_grad(const struct fields_mixer_grads* g, long long N, int D, void* stream) {
    if (!g || N <= 0 || D <= 0) return FIELDS_ERR_ARGUMENT;
    const bool biases = g->grad_out_b || g->grad_gate_b, transition = g->grad_radius || g->grad_theta;
    if ((biases && !g->rows) || (g->grad_write_b && !g->grad_raw) || (g->grad_norm_w && !g->grad_out) ||
        (g->grad_out && (!g->out_w || !g->norm_w)) || ((g->grad_write_b || g->grad_out) && !g->scratch) ||
        (transition && (!g->radius_logit || !g->theta || !g->grad_tr || !g->grad_ti || !g->grad_gamma)))
        return FIELDS_ERR_ARGUMENT;
    if (D % 8 || g->grad_pitch % 4 || !aligned8(g->grad_raw) || !aligned16(g->grad_out) || !aligned16(g->out_w) ||
        !aligned16(g->norm_w) || !aligned16(g->scratch))
        return FIELDS_ERR_UNSUPPORTED;
    Stream st = reinterpret_cast<Stream>(stream);
    const int C = D / 2, cols = 3 * C, wide = 2 * D, per_x = kRowThreads * 4;
    float* col_rows = g->scratch;
    float* weight_rows = col_rows + (size_t)kColumnBlocks * cols;
    FinishGradParams p{};
    int first = 0, rc;
    // (a set without an output has no columns, and so no blocks)
    auto add = [&](int k, const float* rows, float* out, int count, int width) {
        p.set[k] = PartialRows{rows, out, count, out ? width : 0, first};
        first += (p.set[k].cols + 31) / 32;
    };
    const int n = (int)fields_mixer_grad_rows(N);
    add(0, g->rows, g->grad_out_b, n, D);
    add(1, g->rows + (size_t)n * D, g->grad_gate_b, n, D);
    const long long per = (N + kColumnBlocks - 1) / kColumnBlocks;
    if (per > 0x7fffffffLL) return FIELDS_ERR_UNSUPPORTED;
    const int col_blocks = (int)((N + per - 1) / per);
    if (g->grad_write_b) {
        ColumnSumParams cp{static_cast<const uint16_t*>(g->grad_raw), col_rows, N, g->grad_pitch, cols, (int)per};
        rc = launch_grid<ColumnSumParams>(column_sums, dim3((cols + per_x - 1) / per_x, col_blocks), kRowThreads, st, cp);
        if (rc) return rc;
    }
    add(2, col_rows, g->grad_write_b, col_blocks, cols);
    const int wper = (D + kWeightBlocks - 1) / kWeightBlocks, weight_blocks = (D + wper - 1) / wper;
    if (g->grad_out) {
        OutWeightGradParams wp{g->grad_out, g->out_w, g->norm_w, weight_rows, D, wide, wper};
        rc = launch_grid<OutWeightGradParams>(out_weight_grad, dim3((wide + per_x - 1) / per_x, weight_blocks), kRowThreads,
                                              st, wp);
        if (rc) return rc;
    }
    add(3, weight_rows, g->grad_norm_w, weight_blocks, wide);
    p.transition_block = first;
    p.radius_logit = g->radius_logit; p.theta = g->theta;
    p.g_tr = g->grad_tr; p.g_ti = g->grad_ti; p.g_gm = g->grad_gamma;
    p.g_radius = g->grad_radius; p.g_theta = g->grad_theta; p.C = C;
    const int blocks = first + (transition ? (C + kRowThreads - 1) / kRowThreads : 0);
    if (blocks == 0) return FIELDS_OK;
    return launch_on<FinishGradParams>(finish_grad, (unsigned)blocks, kRowThreads, 0, st, p);
}

int fields_step_w12_rows(int hidden) { return hidden > 0 ? (hidden + 19) / 20 * 40 : 0; }

static bool step_sizes(int D, int H) { return D > 0 && D % 16 == 0 && D <= 4096 && H > 0 && H % 8 == 0; }

int fields_step_layout(const struct fields_step_weights* w, void* stream) {
    if (!w || !w->write_w || !w->write_b || !w->gate_w || !w->gate_b || !w->in_w || !w->in_b ||
        (w->w12_w && (!w->w12 || !w->ff_norm_w)) || (!w->w12_w && w->w12))
        return FIELDS_ERR_ARGUMENT;
    if (!step_sizes(w->dim, w->hidden) || !aligned16(w->write_w) || !aligned16(w->gate_w) || !aligned16(w->w12) ||
        !aligned16(w->ff_norm_w) || !aligned16(w->in_w) || !aligned16(w->w12_w))
        return FIELDS_ERR_UNSUPPORTED;
    const int D = w->dim, C = D / 2;
    StepLayoutParams p{w->write_w, w->write_b, w->gate_w, w->gate_b, w->w12, w->ff_norm_w,
                       static_cast<uint16_t*>(w->in_w), static_cast<uint16_t*>(w->w12_w), w->in_b, D, C, w->hidden};
    return launch_on<StepLayoutParams>(step_layout, (unsigned)(5 * C + (w->w12_w ? fields_step_w12_rows(w->hidden) : 0)),
                                       kRowThreads, 0, reinterpret_cast<Stream>(stream), p);
}

}  // extern "C"

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver's encoder of tensor maps, looked up once.
static EncodeTiled encode_tiled() {
    static const EncodeTiled fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &found) !=
                cudaSuccess || found != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<EncodeTiled>(f);
    }();
    return fn;
}

// A dense bfloat16 matrix [rows, cols] in boxes of 64 columns x box_rows rows with the 128-byte swizzle.
static bool operand_map(CUtensorMap* map, const void* base, long long rows, int cols, int box_rows) {
    const EncodeTiled encode = encode_tiled();
    if (!encode) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    const cuuint32_t box[2] = {kStepKBox, (cuuint32_t)box_rows}, ones[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, ones,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A matrix of fp32 or bfloat16 in boxes of 32 rows x box_cols columns, of 128 or 64 bytes, with the swizzle of that length.
static bool box_map(CUtensorMap* map, const void* base, long long rows, int cols, long long pitch, int box_cols, bool f32) {
    const EncodeTiled encode = encode_tiled();
    if (!encode) return false;
    const int size = f32 ? 4 : 2;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)pitch * size};
    const cuuint32_t box[2] = {(cuuint32_t)box_cols, 32}, ones[2] = {1, 1};
    return encode(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims,
                  strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  box_cols * size == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <class Epi, int NT, bool BY_DEPTH>
static int launch_product(const struct fields_product_args& g, ProductParams p, int pairs, Stream st) {
    using T = ProductShape<Epi, NT>;
    p.k_blocks = (g.depth + T::kBox - 1) / T::kBox;
    p.tiles_n = (p.N + NT - 1) / NT;
    p.tiles = (p.M + 2 * kProductRows - 1) / (2 * kProductRows) * p.tiles_n;
    ProductMaps maps;
    std::memset(&maps, 0, sizeof(maps));
    bool ok = operand_map(&maps.a, g.a, p.M, g.depth, kProductRows) &&
              (BY_DEPTH ? operand_map(&maps.b, g.b, g.depth, p.N, T::kBox) : operand_map(&maps.b, g.b, p.N, g.depth, NT / 2));
    if (Epi::kF32) ok = ok && box_map(&maps.x, g.x, p.M, p.N, p.N, T::kChunk, true) && box_map(&maps.y, g.y, p.M, p.N, p.N, T::kChunk, true);
    if (Epi::kIn && !p.direct_in) ok = ok && box_map(&maps.in16, p.in16, p.M, p.N, p.in_pitch, T::kHalfColumns, false);
    if (!p.direct_out) {
        if (p.has_h) ok = ok && box_map(&maps.out16, p.h, p.M, Epi::kSwiglu ? p.N / 2 : p.N, p.h_pitch, T::kHalfColumns, false);
        else if (p.has_acc) ok = ok && box_map(&maps.out16, p.acc, p.M, p.N, p.N, T::kHalfColumns, false);
    }
    if (!ok) return FIELDS_ERR_UNSUPPORTED;
    static bool ready[64] = {};
    const int rc = allow_shared_memory(pair_product<Epi, NT, BY_DEPTH>, T::kSmemBytes, ready);
    if (rc) return rc;
    p.pairs = p.tiles < pairs ? (int)p.tiles : pairs;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)p.pairs * 2);
    cfg.blockDim = dim3(32 * (kProductWarps + 2));
    cfg.dynamicSmemBytes = T::kSmemBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = dependent_launch_enabled() ? 2 : 1;
    return check_cuda(cudaLaunchKernelEx(&cfg, pair_product<Epi, NT, BY_DEPTH>, maps, p));
}

// Tiles of 256 or of 128 columns: by the rounds of tiles that a pair takes, each as long as its columns and about 64 more
// (loads and a wave's end; 2,048 rows: 2,560 columns of depth 1,024 16.9 and 15.3 us, 1,024 of depth 2,528 21.4 and 14.4; 8,192
// rows: 32.1 and 35.9, 41.7 and 47.2).
template <class Epi, bool BY_DEPTH = false>
static int run_product(const struct fields_product_args& g, const ProductParams& p, Stream st) {
    int dev = 0, sms = 0;
    int rc = check_cuda(cudaGetDevice(&dev));
    if (!rc) rc = check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (rc) return rc;
    const int pairs = sms > 1 ? sms / 2 : 1;
    auto rounds = [&](int nt) {
        const long long tiles = (p.M + 2 * kProductRows - 1) / (2 * kProductRows) * ((p.N + nt - 1) / nt);
        return (tiles + pairs - 1) / pairs * (nt + 64);
    };
    return rounds(128) < rounds(256) ? launch_product<Epi, 128, BY_DEPTH>(g, p, pairs, st)
                                     : launch_product<Epi, 256, BY_DEPTH>(g, p, pairs, st);
}

// How a launch of step_stack covers the GPU: `clusters` are resident at once.
template <bool NARROW>
static void step_phases(StepStackParams& p, int clusters) {
    using T = StepShape<NARROW>;
    p.groups = p.row_tiles < clusters ? p.row_tiles : clusters;
    const int most = clusters / p.groups, blocks = most * kStepCluster;
    const int K[kStepPhases] = {p.D, 4 * p.C, p.D, p.H};
    const int cols[kStepPhases] = {5 * p.C, p.D, fields_step_w12_rows(p.H), p.D};
    const int split[kStepPhases] = {T::In::kMaxSplit, T::Out::kMaxSplit, T::Uv::kMaxSplit, T::Ff::kMaxSplit};
    p.group_clusters = 1;
    for (int i = 0; i < kStepPhases; ++i) {
        StepPhase& h = p.phase[i];
        h.tiles_n = (cols[i] + T::nt(i) - 1) / T::nt(i);
        h.k_blocks = (K[i] + kStepKBlock - 1) / kStepKBlock;
        h.S = 1;  // K over as many blocks as there are, every one of them with a part of K
        for (int S = 2; S <= split[i] && h.tiles_n * S <= blocks; S *= 2)
            if ((S - 1) * ((h.k_blocks + S - 1) / S) < h.k_blocks) h.S = S;
        h.per = (h.k_blocks + h.S - 1) / h.S;
        const int subs = kStepCluster / h.S, want = (h.tiles_n + subs - 1) / subs;
        if (p.group_clusters < (want < most ? want : most)) p.group_clusters = want < most ? want : most;
    }
    for (StepPhase& h : p.phase) {
        const int per = p.group_clusters * (kStepCluster / h.S);
        h.iters = (h.tiles_n + per - 1) / per;
    }
}

// Clusters of step_stack that the device holds at once.
template <bool NARROW>
static int step_clusters(cudaLaunchConfig_t cfg, int* clusters) {
    static std::atomic<int> known[64];
    int dev = 0;
    const int rc = check_cuda(cudaGetDevice(&dev));
    if (rc) return rc;
    if (dev < 0 || dev >= 64) return FIELDS_ERR_UNSUPPORTED;
    *clusters = known[dev].load();
    if (*clusters > 0) return FIELDS_OK;
    cfg.gridDim = dim3(kStepCluster);
    const int rc2 = check_cuda(cudaOccupancyMaxActiveClusters(clusters, step_stack<NARROW>, &cfg));
    if (rc2) return rc2;
    if (*clusters < 1) return FIELDS_ERR_UNSUPPORTED;
    known[dev].store(*clusters);
    return FIELDS_OK;
}

// Phases [first, last) of the blocks in p: as one cooperative launch (p.sync), or one phase by itself.
template <bool NARROW>
static int launch_step(StepStackParams& p, bool cooperative, Stream st) {
    using T = StepShape<NARROW>;
    static bool ready[64] = {};
    int rc = allow_shared_memory(step_stack<NARROW>, T::kSmemBytes, ready);
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kStepThreads);
    cfg.dynamicSmemBytes = T::kSmemBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kStepCluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    rc = step_clusters<NARROW>(cfg, &clusters);
    if (rc) return rc;
    step_phases<NARROW>(p, clusters);
    if (cooperative) {
        attr[1].id = cudaLaunchAttributeCooperative;
        attr[1].val.cooperative = 1;
        cfg.numAttrs = 2;
    } else if (dependent_launch_enabled()) {
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.numAttrs = 2;
    }
    cfg.gridDim = dim3((unsigned)(p.groups * p.group_clusters * kStepCluster));
    const cudaError_t e = cudaLaunchKernelEx(&cfg, step_stack<NARROW>, p);
    if (cooperative && e == cudaErrorCooperativeLaunchTooLarge) {
        (void)cudaGetLastError();
        return FIELDS_ERR_UNSUPPORTED;
    }
    return check_cuda(e);
}

// Whether the narrow tiles leave less of the GPU without one.
static bool step_narrow(int rows, int dim) { return (rows + kStepRows - 1) / kStepRows * ((dim + 63) / 64) * 8 <= 148; }

// One product of a block: A [M, K] activations, B [n_rows, K] weights, `slices` column slices.
template <class Epi>
static int launch_phase(const void* a, const void* b, int n_rows, int K, int slices, PhaseParams p, Stream st) {
    using T = PhaseTile<Epi>;
    p.k_blocks = (K + kStepKBox - 1) / kStepKBox;
    p.tiles_n = (slices + Epi::kSlices - 1) / Epi::kSlices;
    const int tiles = p.tiles_n * ((p.M + kStepRows - 1) / kStepRows);
    // K over as many blocks as share the GPU in one round, every one of them with a part of K (clusters of four or more
    // do not find room for 144 blocks: 384 features, 384 rows took 250 us instead of 215 for eight blocks)
    p.S = 1;
    for (int S = 2; S <= Epi::kMaxSplit && tiles * S <= (S > 2 ? 132 : 148); S *= 2)
        if ((S - 1) * ((p.k_blocks + S - 1) / S) < p.k_blocks) p.S = S;
    CUtensorMap a_map, b_map;
    if (!operand_map(&a_map, a, p.M, K, kStepRows) || !operand_map(&b_map, b, n_rows, K, T::kNT))
        return FIELDS_ERR_UNSUPPORTED;
    static bool ready[64] = {};
    const int rc = allow_shared_memory(step_phase<Epi>, T::kSmemBytes, ready);
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * p.S));
    cfg.blockDim = dim3(kPhaseThreads);
    cfg.dynamicSmemBytes = T::kSmemBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (dependent_launch_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (p.S > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = (unsigned)p.S;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return check_cuda(cudaLaunchKernelEx(&cfg, step_phase<Epi>, a_map, b_map, p));
}

// A block as four launches.
static int step_block(const struct fields_step_args& g, Stream st) {
    const int D = g.dim, C = D / 2, H = g.hidden;
    auto h = [](void* q) { return static_cast<uint16_t*>(q); };
    PhaseParams p{};
    p.x = g.x; p.gate = h(g.gate); p.read = h(g.read); p.state = g.state; p.y = g.y; p.yb = h(g.yb);
    p.act = h(g.act); p.xb = h(g.xb); p.read_sq = g.read_sq; p.y_sq = g.y_sq;
    p.in_b = g.in_b; p.par = g.par; p.out_b = g.out_b;
    p.read_eps = g.read_eps; p.ff_eps = g.ff_eps; p.M = g.rows; p.D = D; p.C = C; p.H = H;
    // the first product waits where a parameter may still be on its way; it lets the second in afterwards
    p.wait_first = !g.settled;
    int rc = launch_phase<PhaseIn>(g.xb, g.in_w, 5 * C, D, C / 8, p, st);
    p.wait_first = 0;
    const bool narrow = step_narrow(g.rows, D);
    if (!rc) rc = narrow ? launch_phase<PhaseOut<4>>(g.read, g.out_w16, D, 2 * D, D / 8, p, st)
                         : launch_phase<PhaseOut<8>>(g.read, g.out_w16, D, 2 * D, D / 8, p, st);
    if (!rc) rc = narrow ? launch_phase<PhaseUv<5>>(g.yb, g.w12_w, fields_step_w12_rows(H), D, H / 8, p, st)
                         : launch_phase<PhaseUv<10>>(g.yb, g.w12_w, fields_step_w12_rows(H), D, H / 8, p, st);
    if (!rc) rc = narrow ? launch_phase<PhaseFf<4>>(g.act, g.w3_16, D, H, D / 8, p, st)
                         : launch_phase<PhaseFf<8>>(g.act, g.w3_16, D, H, D / 8, p, st);
    return rc;
}

template <bool NARROW>
static int run_step(const struct fields_step_args* g, int count, unsigned* sync, Stream st) {
    using T = StepShape<NARROW>;
    auto h = [](void* q) { return static_cast<uint16_t*>(q); };
    StepStackParams p;
    std::memset(&p, 0, sizeof(p));
    const int M = g->rows, D = g->dim, C = D / 2, H = g->hidden;
    p.gate = h(g->gate); p.read = h(g->read); p.yb = h(g->yb); p.act = h(g->act); p.xb = h(g->xb);
    p.y = g->y; p.read_sq = g->read_sq; p.y_sq = g->y_sq;
    p.M = M; p.D = D; p.C = C; p.H = H;
    p.row_tiles = (M + kStepRows - 1) / kStepRows;
    p.a_rows = M < kStepRows ? (M + 7) / 8 * 8 : kStepRows;
    const void* a[kStepPhases] = {g->xb, g->read, g->yb, g->act};
    const int K[kStepPhases] = {D, 4 * C, D, H};
    const int rows[kStepPhases] = {5 * C, D, fields_step_w12_rows(H), D};
    for (int i = 0; i < kStepPhases; ++i)
        if (!operand_map(&p.a[i], a[i], M, K[i], p.a_rows)) return FIELDS_ERR_UNSUPPORTED;
    for (int at = 0; at < count; at += kStepMaxBlocks) {
        const int n = count - at < kStepMaxBlocks ? count - at : kStepMaxBlocks;
        for (int j = 0; j < n; ++j) {
            const struct fields_step_args& q = g[at + j];
            StepWeights& w = p.block[j];
            w.x = q.x; w.in_b = q.in_b; w.par = q.par; w.out_b = q.out_b; w.state = q.state;
            w.read_eps = q.read_eps; w.ff_eps = q.ff_eps;
            const void* b[kStepPhases] = {q.in_w, q.out_w16, q.w12_w, q.w3_16};
            for (int i = 0; i < kStepPhases; ++i)
                if (!operand_map(&w.b[i], b[i], rows[i], K[i], T::box(i))) return FIELDS_ERR_UNSUPPORTED;
        }
        int rc = FIELDS_ERR_UNSUPPORTED;
        if (sync) {
            p.sync = sync;
            p.first = 0;
            p.last = n * kStepPhases;
            rc = check_cuda(cudaMemsetAsync(sync, 0, kStepSyncBytes, st));
            if (!rc) rc = launch_step<NARROW>(p, true, st);
            if (rc == FIELDS_ERR_UNSUPPORTED) {  // no such launch on this device
                rc = FIELDS_OK;
                for (int i = 0; i < n && !rc; ++i) rc = step_block(g[at + i], st);
            }
        } else {  // one launch per phase: none of them waits for another
            rc = FIELDS_OK;
            for (int i = 0; i < n * kStepPhases && !rc; ++i) {
                p.first = i;
                p.last = i + 1;
                rc = launch_step<NARROW>(p, false, st);
            }
        }
        if (rc) return rc;
    }
    return FIELDS_OK;
}

static int step_arguments(const struct fields_step_args& q) {
    const void* all[] = {q.x, q.state, q.y, q.xb, q.yb, q.read, q.gate, q.act, q.read_sq, q.y_sq, q.in_w,
                         q.out_w16, q.w12_w, q.w3_16, q.in_b, q.par, q.out_b};
    for (const void* v : all)
        if (!v) return FIELDS_ERR_ARGUMENT;
    if (!step_sizes(q.dim, q.hidden) || q.rows > 512) return FIELDS_ERR_UNSUPPORTED;
    for (const void* v : all)
        if (!aligned16(v)) return FIELDS_ERR_UNSUPPORTED;
    return FIELDS_OK;
}

extern "C" {

int fields_transpose_bf16(const struct fields_transpose* parts, int count, void* stream) {
    if (!parts || count < 1 || count > 2) return FIELDS_ERR_ARGUMENT;
    TransposeParams p{};
    long long tiles = 0;
    for (int i = 0; i < count; ++i) {
        const struct fields_transpose& q = parts[i];
        if (!q.in || !q.out || q.rows <= 0 || q.cols <= 0) return FIELDS_ERR_ARGUMENT;
        if (q.rows % 2 || q.cols % 2 || (reinterpret_cast<uintptr_t>(q.in) | reinterpret_cast<uintptr_t>(q.out)) % 4)
            return FIELDS_ERR_UNSUPPORTED;
        const long long across = (q.cols + 63) / 64, n = (q.rows + 63) / 64 * across;
        tiles += n;
        if (tiles > 0x7fffffffLL) return FIELDS_ERR_UNSUPPORTED;
        p.part[i] = {static_cast<const uint16_t*>(q.in), static_cast<uint16_t*>(q.out), q.rows, q.cols, (int)across, (int)n};
    }
    return launch_on<TransposeParams>(transpose_bf16, (unsigned)tiles, kRowThreads, 0, reinterpret_cast<Stream>(stream), p);
}

int fields_product(const struct fields_product_args* g, int kind, void* stream) {
    const bool by_depth = kind >= 0 && (kind & FIELDS_PRODUCT_BY_DEPTH);
    if (by_depth) {
        kind -= FIELDS_PRODUCT_BY_DEPTH;
        if (kind != FIELDS_PRODUCT_RESIDUAL && kind != FIELDS_PRODUCT_NORM_GRAD) return FIELDS_ERR_ARGUMENT;
    }
    if (!g || g->rows < 0 || g->cols <= 0 || g->depth <= 0) return FIELDS_ERR_ARGUMENT;
    if (g->rows == 0) return FIELDS_OK;
    if (!g->a || !g->b) return FIELDS_ERR_ARGUMENT;
    constexpr int kWidest = 1 << 26;  // 32 rows of a tensor are addressed with 32 bits
    const int h_cols = kind == FIELDS_PRODUCT_SWIGLU ? g->cols / 2 : g->cols;
    const long long gate_pitch = g->gate_pitch ? g->gate_pitch : g->cols, h_pitch = g->h_pitch ? g->h_pitch : h_cols;
    if ((kind == FIELDS_PRODUCT_GATE && gate_pitch < g->cols) || (g->h && h_pitch < h_cols))
        return FIELDS_ERR_ARGUMENT;  // rows would overlap
    if (g->cols > kWidest || gate_pitch > kWidest || h_pitch > kWidest || gate_pitch < 0 || h_pitch < 0)
        return FIELDS_ERR_UNSUPPORTED;
    if (g->cols % (by_depth ? 8 : 4) || g->depth % 8 || g->rows > 0x7fffff00LL || !aligned16(g->a) || !aligned16(g->b) || !aligned16(g->x) ||
        !aligned16(g->y) || !aligned16(g->bias) || !aligned16(g->gate_bias) || !aligned8(g->bias16) || !aligned8(g->gate) ||
        !aligned8(g->read) || !aligned8(g->h) || !aligned8(g->acc) || gate_pitch % 4 || h_pitch % 4)
        return FIELDS_ERR_UNSUPPORTED;
    ProductParams p{};
    auto h = [](const void* q) { return static_cast<const uint16_t*>(q); };
    p.M = g->rows; p.N = g->cols;
    const bool gated = kind == FIELDS_PRODUCT_GATE;
    p.bias16 = h(g->bias16); p.bias = g->bias; p.gate_bias = g->gate_bias;
    p.sums = g->sums; p.entries = g->entries;
    p.inv_features = g->features > 0 ? 1.0f / (float)g->features : 0.0f; p.eps = g->eps;
    p.row = g->row; p.sums_out = g->sums_out;
    p.in16 = h(gated ? g->gate : g->read); p.in_pitch = gated ? gate_pitch : p.N;
    p.h = static_cast<uint16_t*>(g->h); p.h_pitch = h_pitch; p.acc = static_cast<uint16_t*>(g->acc);
    p.has_h = p.h != nullptr; p.has_acc = gated && p.acc;
    p.direct_in = !aligned16(p.in16) || p.in_pitch % 8;
    p.direct_out = p.has_h ? !aligned16(p.h) || h_pitch % 8 : p.has_acc && (!aligned16(p.acc) || p.N % 8);
    Stream st = reinterpret_cast<Stream>(stream);
    switch (kind) {
        case FIELDS_PRODUCT_BIAS:
            if (!p.bias16 || !p.h) return FIELDS_ERR_ARGUMENT;
            return run_product<ProductBias>(*g, p, st);
        case FIELDS_PRODUCT_GATE:
            if (!g->x || !p.bias || !p.gate_bias || !p.in16 || !p.sums || p.entries <= 0 || g->features <= 0 || !g->y)
                return FIELDS_ERR_ARGUMENT;
            return run_product<ProductGate>(*g, p, st);
        case FIELDS_PRODUCT_SWIGLU:
            if (!p.sums || p.entries <= 0 || g->features <= 0 || !p.h || p.N % 16) return FIELDS_ERR_ARGUMENT;
            return run_product<ProductSwiglu>(*g, p, st);
        case FIELDS_PRODUCT_RESIDUAL:
            if (!g->x || !g->y) return FIELDS_ERR_ARGUMENT;
            return by_depth ? run_product<ProductResidual, true>(*g, p, st) : run_product<ProductResidual>(*g, p, st);
        case FIELDS_PRODUCT_NORM_GRAD:
            if (!p.in16 || !p.row || !p.h) return FIELDS_ERR_ARGUMENT;
            return by_depth ? run_product<ProductNormGrad, true>(*g, p, st) : run_product<ProductNormGrad>(*g, p, st);
    }
    return FIELDS_ERR_ARGUMENT;
}

int fields_step_stack(const struct fields_step_args* g, int count, void* sync, void* stream) {
    if (!g || count < 0 || g->rows < 0) return FIELDS_ERR_ARGUMENT;
    if (g->rows == 0 || count == 0) return FIELDS_OK;
    for (int i = 0; i < count; ++i) {
        const struct fields_step_args& q = g[i];
        const int rc = step_arguments(q);
        if (rc) return rc;
        // one block goes on from the other
        if (q.y != g->y || q.xb != g->xb || q.yb != g->yb || q.read != g->read || q.gate != g->gate || q.act != g->act ||
            q.read_sq != g->read_sq || q.y_sq != g->y_sq || q.rows != g->rows || q.dim != g->dim ||
            q.hidden != g->hidden || (i > 0 && q.x != g->y))
            return FIELDS_ERR_ARGUMENT;
    }
    if (sync && !aligned16(sync)) return FIELDS_ERR_UNSUPPORTED;
    return step_narrow(g->rows, g->dim) ? run_step<true>(g, count, static_cast<unsigned*>(sync), reinterpret_cast<Stream>(stream))
                  : run_step<false>(g, count, static_cast<unsigned*>(sync), reinterpret_cast<Stream>(stream));
}

int fields_step_block(const struct fields_step_args* g, void* stream) {
    if (!g || g->rows < 0) return FIELDS_ERR_ARGUMENT;
    if (g->rows == 0) return FIELDS_OK;
    const int rc = step_arguments(*g);
    return rc ? rc : step_block(*g, reinterpret_cast<Stream>(stream));
}

#endif  // FIELDS_HOST_EMU

}  // extern "C"
