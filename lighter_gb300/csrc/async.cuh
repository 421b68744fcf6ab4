// Shared-memory barriers and bulk asynchronous copies (sm_100 family PTX), with
// bounded waits: a wait gives up after a cycle limit, records an error bit and
// returns false, so no kernel spins forever on a copy that never lands.
#pragma once

#include <cstdint>

namespace lg {

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t) __cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(bar)), "r"(count) : "memory");
}

// Makes initialised barriers visible to the asynchronous proxy (the copy engine).
__device__ __forceinline__ void mbar_init_fence()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(bar)) : "memory");
}

// An arrival on the barrier at the same place in CTA `rank` of this cluster.
__device__ __forceinline__ void mbar_arrive_rank(uint64_t* bar, uint32_t rank)
{
    asm volatile(
        "{\n\t.reg .b32 a;\n\t"
        "mapa.shared::cluster.u32 a, %0, %1;\n\t"
        "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [a];\n\t}" ::"r"(saddr(bar)),
        "r"(rank)
        : "memory");
}

// CLUSTER: arrivals by other CTAs of the cluster are acquired too.
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    if (CLUSTER)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(saddr(bar)), "r"(parity)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(saddr(bar)), "r"(parity)
            : "memory");
    return ok != 0;
}

// Bounded wait for the phase of parity `parity`: false (and the error bit)
// after `limit` SM clock cycles.
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t* err, uint32_t bit,
                                          unsigned long long limit)
{
    if (mbar_try<CLUSTER>(bar, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try<CLUSTER>(bar, parity)) {
        if (clock64() - t0 > (long long) limit) {
            if (err) atomicOr(err, bit);
            return false;
        }
    }
    return true;
}

// Bulk copy of `bytes` from global to this CTA's shared memory, completing on
// `bar` (both addresses 16-byte aligned, bytes a multiple of 16). The line is
// marked evict-first in L2: the source is streamed once.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar, uint64_t policy)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
            saddr(dst)),
        "l"(src), "r"(bytes), "r"(saddr(bar)), "l"(policy)
        : "memory");
}

__device__ __forceinline__ uint64_t l2_evict_first_policy()
{
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}

}  // namespace lg
