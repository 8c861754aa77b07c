// Self-test of the failure path of a bounded device wait (phx_selftest_wait_timeout).
#pragma once
#include "pressure_kernels.cuh"

namespace phx {

constexpr unsigned ERR_SELFTEST = 4u;   // error-word bit

// One thread waits, as the solve's threads do, for a tagged value that nothing writes. The
// wait runs out after limitCycles, sets its bit and this one in the context's error
// word and returns; nothing else waits on it. R is the engine's precision (one
// instance per engine).
template <class R>
__global__ void k_selftest_wait(unsigned* errWord, const unsigned long long* never, long long limitCycles) {
    __shared__ int gaveUp;
    if (threadIdx.x != 0) return;
    gaveUp = 0;
    const TagWait wait{&gaveUp, &errWord, &limitCycles};
    float v;
    waitFor(wait, [&] { return tagLoad(never, 0, 1u, v); });
    if (gaveUp) atomicOr(errWord, ERR_SELFTEST);
}

}  // namespace phx
