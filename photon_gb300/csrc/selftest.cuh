// Self-test of the failure path of a bounded device wait (phx_selftest_wait_timeout).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace phx {

__device__ __forceinline__ unsigned smemAddr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbarInit(uint64_t* b, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smemAddr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void fenceBarrierInit() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
// try_wait suspends the thread until the phase completes or the hint (ns)
// runs out, so a waiting warp takes no issue slots from the working ones
__device__ __forceinline__ bool mbarTryWait(uint64_t* b, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smemAddr(b)), "r"(parity), "r"(20000u)
        : "memory");
    return ok != 0;
}
// Self-test of the failure path of a bounded wait: one thread waits, with a
// limit of `limitCycles`, on an mbarrier that nothing arrives on. The wait
// runs out, the kernel records bit 4 in the context's error word and
// returns; no copy is in flight and nothing else waits on it. R is the
// engine's precision (one instance per engine).
template <class R>
__global__ void k_selftest_wait(unsigned* errWord, long long limitCycles) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x != 0) return;
    mbarInit(&bar, 1);
    fenceBarrierInit();
    const long long t0 = clock64();
    bool arrived = false;
    while (!(arrived = mbarTryWait(&bar, 0))) {
        if (clock64() - t0 > limitCycles) break;
        __nanosleep(1000);
    }
    if (!arrived) atomicOr(errWord, 4u);
}

}  // namespace phx
