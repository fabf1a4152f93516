// Exchange of small records between the blocks of a cluster through distributed shared memory: a store
// that completes a transaction barrier in the receiving block (st.async), so no block waits for more
// than the records themselves, and nothing in global memory has to be cleared or polled.
//
// Use, per exchange k of a kernel: every block expects Q records per thread on its barrier k & 1, stores
// its own record into slot [k & 1][rank] of every block of the cluster, and waits for its barrier. Two
// parities suffice: a block stores for exchange k + 2 only after it has the records of k + 1 from
// all blocks, each of which sent those after it had read the slots of k.
//
// Waits are bounded; device only.
#pragma once

#include "field_math.cuh"

#ifndef FIELDS_HOST_EMU

namespace fields {

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
template <bool PEERS>
__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned parity) {
    unsigned done;
    if constexpr (PEERS)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
    return done != 0;
}
// Waits for a phase, with a bound (a try suspends for a while by itself, so 2^20 of them are a second
// or more). `dead` is the thread's record that a wait has run out: it is set then, and later waits
// give up at once, so a kernel always terminates. Acquires at cluster scope; mbar_wait_local, for barriers
// that only this block and its own copies arrive on, at block scope.
template <bool PEERS>
__device__ __forceinline__ void mbar_wait_scope(unsigned bar, unsigned parity, bool& dead) {
    unsigned tries = 0;
    while (!mbar_try<PEERS>(bar, parity)) {
        if (dead || ++tries >= (1u << 20)) {
            dead = true;
            return;
        }
    }
}
__device__ __forceinline__ void mbar_wait(unsigned bar, unsigned parity, bool& dead) { mbar_wait_scope<true>(bar, parity, dead); }
__device__ __forceinline__ void mbar_wait_local(unsigned bar, unsigned parity, bool& dead) {
    mbar_wait_scope<false>(bar, parity, dead);
}
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned peer_addr(unsigned addr, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void send2(unsigned dst, float x, float y, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(dst),
                 "f"(x), "f"(y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

}  // namespace fields

#endif  // FIELDS_HOST_EMU
