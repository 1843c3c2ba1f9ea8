// mbarriers, bulk copies and asynchronous stores to a cluster's other CTAs.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"

namespace nricp_b200 {

__device__ __forceinline__ uint32_t shared_address(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(void* bar, int arrivals) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(shared_address(bar)), "r"(arrivals) : "memory");
    // the copies' and the other CTAs' view of the initialised barrier
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_invalidate(void* bar) {
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(shared_address(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive(void* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(shared_address(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect(void* bar, int bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(shared_address(bar)), "r"(bytes)
                 : "memory");
}
// Waits for the phase of this parity, at most `tries` times (kWaitTries): false
// if they ran out.
__device__ __forceinline__ bool mbar_wait(void* bar, int parity, int tries) {
    const uint32_t at = shared_address(bar);
    for (int i = 0; i < tries; ++i) {
        uint32_t done;
        asm volatile("{\n.reg .pred p;\n"
                     "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
                     "selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(done)
                     : "r"(at), "r"(parity)
                     : "memory");
        if (done) return true;
    }
    return false;
}
// Global to shared, both 16-byte aligned, a multiple of 16 bytes.
__device__ __forceinline__ void bulk_to_shared(void* dst, const void* src, int bytes, void* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     shared_address(dst)),
                 "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(shared_address(bar))
                 : "memory");
}

// The same shared-memory address in another CTA of the cluster.
__device__ __forceinline__ uint32_t peer_address(const void* p, int rank) {
    uint32_t out;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(shared_address(p)), "r"(rank));
    return out;
}
// This CTA's shared memory to a peer's, completing on the peer's mbarrier;
// 16-byte aligned, a multiple of 16 bytes.
__device__ __forceinline__ void bulk_to_peer(uint32_t dst, const void* src, int bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     dst),
                 "r"(shared_address(src)), "r"(bytes), "r"(bar)
                 : "memory");
}
// Two doubles into a peer's shared memory, completing on its mbarrier.
__device__ __forceinline__ void store_to_peer(uint32_t dst, double a, double b, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(dst),
                 "l"(__double_as_longlong(a)), "l"(__double_as_longlong(b)), "r"(bar)
                 : "memory");
}

}  // namespace nricp_b200
