// The coarse levels of the pressure multigrid (src/sim/pressure_mg.cpp:237-300)
// and the scalars of the CG iteration (src/sim/gasphase.cpp:551-626), as the
// device functions the solve kernel (solve.cuh) is made of.
//
// Coarse levels are CSR rows: damped Jacobi (omega 0.7) and a gather of the
// children's residuals in ascending order. The coarsest level's 20 forward +
// backward Gauss-Seidel sweeps from x = 0 are a fixed linear map of b; it is
// applied as a dense operator built on the host from those sweeps (on the
// mixed path: the exact inverse).
#pragma once
#include "level0.cuh"

namespace phx {

constexpr double OMEGA = 0.7;

// a + b c, rounded once in either precision
__device__ __forceinline__ double madd(double a, double b, double c) { return fma(b, c, a); }
__device__ __forceinline__ float madd(float a, float b, float c) { return fmaf(b, c, a); }

// A damped Jacobi value (jacobi, pressure_mg.cpp:237-247) from the row's sum s and
// its old x. FP64 path: s times omega / diagonal from the host (an FP64
// division costs some twenty FP64 instructions, which the pipe issues at a
// sixteenth of a warp per clock); FP32 path: the division itself.
__device__ __forceinline__ double jacobiValue(double s, double x, double, double omd) {
    return omd > 0 ? madd((1.0 - OMEGA) * x, omd, s) : 0.0;
}
__device__ __forceinline__ float jacobiValue(float s, float x, float dg, float) {
    const float om = (float)OMEGA;
    return dg <= 0.f ? 0.f : (1.f - om) * x + om * s / dg;
}

// ---- tagged values ------------------------------------------------------------------
// Values that one CTA's thread hands to another's inside a kernel travel with a
// tag in the same 64-bit word (FP64: each half of the number in a word of its
// own), so the reader needs neither a barrier nor the writer a fence: it reads
// until the tag is the one it waits for. A word is written and read whole. A
// barrier of the solve's team takes 1.4 us (the fence alone 0.4), a tagged value
// one store and one load through L2. The coarse levels and the d.q sum of an iteration
// without their barriers: FP32 room step 0.52 -> 0.45 ms, house 1.33 -> 1.25,
// 1.3e6 cells 3.75 -> 3.63; 24 scenarios (2400 rows of level 1 a CTA, whose values no
// longer come from L1) 5.9 -> 6.0; FP64 room 0.77 -> 0.72.
template <class R>
constexpr int TAG_WORDS = sizeof(R) == 8 ? 2 : 1;

__device__ __forceinline__ void tagStore(unsigned long long* a, int i, float v, unsigned tag) {
    const unsigned long long w = ((unsigned long long)tag << 32) | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(a + i), "l"(w) : "memory");
}
__device__ __forceinline__ void tagStore(unsigned long long* a, int i, double v, unsigned tag) {
    const unsigned long long t = (unsigned long long)tag << 32, b = (unsigned long long)__double_as_longlong(v);
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(a + 2 * (size_t)i), "l"(t | (b & 0xffffffffull)),
                 "l"(t | (b >> 32))
                 : "memory");
}
// the value at i; false where it does not have the tag yet
__device__ __forceinline__ bool tagLoad(const unsigned long long* a, int i, unsigned tag, float& v) {
    unsigned long long w;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(a + i) : "memory");
    v = __uint_as_float((unsigned)w);
    return (unsigned)(w >> 32) == tag;
}
__device__ __forceinline__ bool tagLoad(const unsigned long long* a, int i, unsigned tag, double& v) {
    unsigned long long lo, hi;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(a + 2 * (size_t)i) : "memory");
    v = __hiloint2double((int)(unsigned)hi, (int)(unsigned)lo);
    return (unsigned)(lo >> 32) == tag && (unsigned)(hi >> 32) == tag;
}
// a thread's wait for tagged values: true while it should read again. After a scenario's
// limit it gives up for the whole CTA: *gaveUp (shared memory) ends every
// later wait at once, and the kernel at its next team barrier.
constexpr unsigned ERR_TEAM_WAIT = 8u;                     // error-word bit
struct TagWait {
    volatile int* gaveUp;
    unsigned* const* errWord;    // the descriptor's, in shared memory
    const long long* limit;
    __device__ __forceinline__ bool again(int& spins, long long& since) const {
        if (*gaveUp) return false;
        if (++spins < 64) return true;
        const long long now = clock64();
        if (spins == 64) since = now;
        if (now - since <= *limit) return true;
        atomicOr(*errWord, ERR_TEAM_WAIT);
        *gaveUp = 1;
        return false;
    }
};
// read(): loads everything the thread needs, true when all tags match
template <class F>
__device__ __forceinline__ void waitFor(const TagWait& w, F read) {
    int spins = 0;
    long long since = 0;
    while (!read() && w.again(spins, since)) {}
}

// coarsest level: x = M b with the dense operator of the reference's 20
// forward + backward Gauss-Seidel sweeps (pressure_mg.cpp:258-266, 279).
// One warp per row.
template <class R>
__device__ __forceinline__ R coarseDenseRow(const Level<R>& L, int row, const R* b) {
    using T = R;
    const int lane = threadIdx.x & 31;
    const R* M = L.dense + (size_t)row * L.n;
    T acc = 0;
    for (int j0 = 0; j0 < L.n; j0 += 256) {   // eight columns a lane at a time: their loads are in flight together
        T m[8], v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int j = j0 + 32 * e + lane;
            m[e] = j < L.n ? M[j] : T(0);
            v[e] = j < L.n ? b[j] : T(0);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) acc = madd(acc, m[e], v[e]);
    }
    return warpSum(acc);
}

// coarsest level solved as the reference does it: 20 forward + backward
// sweeps, serially in one thread (used when the level is too large for a dense
// operator); b and x are plain arrays of the CTA's own
template <class R>
__device__ __forceinline__ void coarseSerial(const Level<R>& L, const R* b, R* x) {
    using T = R;
    for (int I = 0; I < L.n; ++I) x[I] = 0;
    for (int it = 0; it < 20; ++it)
        for (int dir = 0; dir < 2; ++dir)
            for (int t = 0; t < L.n; ++t) {
                int I = dir == 0 ? t : L.n - 1 - t;
                T dg = L.diag[I];
                if (dg <= 0) { x[I] = 0; continue; }
                T s = b[I];
                for (int q = L.rowStart[I]; q < L.rowStart[I + 1]; ++q) s += L.val[q] * x[L.col[q]];
                x[I] = s / dg;
            }
}

// The CG scalars of a scenario while it is being solved, one copy per CTA of its team.
struct CgState {
    double rz, alpha, beta, dq;
    double rmax, r64;        // last max|r| of the recursion; of the FP64 residual where it was formed (mixed path)
    // bars on max|r|: the absolute one and half of it; the relative one and twice it (-1: none)
    double absStop, absHalf, relStop, relStop2;
    int it, done, repl;      // repl: the residual is replaced this iteration (mixed path)
    int brk;                 // mixed path: 1 after a breakdown (next update skipped), 2 restart pending
};

// a > b for numbers of which b is not a NaN and a is not negative, by their bits:
// an FP64 comparison takes some hundred cycles here, and closing an iteration is a
// chain of them on one thread
__device__ __forceinline__ bool above(double a, double b) { return __double_as_longlong(a) > __double_as_longlong(b); }

// closes a CG iteration once r.z = tot is known: the iteration count and the stop
// test (src/sim/gasphase.cpp:589-605; the optional relative test is max|r| <=
// relTol max|b|). beta is tot / rz. phase 0: the first preconditioning before the
// loop; 1: inside the loop. One thread.
template <class R>
__device__ __forceinline__ void closeCgIteration(const Scn<R>& g, CgState& c, int phase, double tot, double beta,
                                                 double rmax, double r64) {
    const int it = phase == 0 ? 0 : c.it + 1;
    const bool positive = tot > 0;
    c.it = it;
    c.rmax = rmax;
    if (!g.mixed) {
        if (phase != 0) c.beta = beta;
        c.rz = tot;
        if (!(above(rmax, c.absStop) && it < g.maxIters && positive && above(rmax, c.relStop))) c.done = 1;
        return;
    }
    // mixed: the stop test uses the FP64 residual, known where it was just
    // replaced; the FP32 recursive residual schedules the next replacement
    // (every replaceEvery iterations, or once it claims convergence)
    const bool replaced = phase == 0 || c.repl != 0;
    bool converged = false, restart = false;
    if (replaced) {
        c.r64 = r64;
        converged = !above(r64, c.absStop) || !above(r64, c.relStop) || !above(r64, 0.0);
        // restart the FP32 CG from the replaced residual (d = z) where it is no
        // longer conjugate to the search direction: closed zones (their
        // operators are singular), and any scenario whose FP32 recursion had
        // drifted below the true residual (a strong preconditioner takes the
        // recursion to FP32's rounding floor within a few iterations; the old
        // direction then carries only rounding noise)
        restart = phase != 0 && (g.nClosed > 0 || above(r64, 4.0 * rmax));
    }
    // the first iteration after a breakdown's replacement restarts the FP32 CG (d = z)
    if (phase != 0 && c.brk == 2) {
        restart = true;
        c.brk = 0;
    }
    // a breakdown (r.z <= 0) of the FP32 recursion short of the FP64 bar: the recursive
    // residual has reached FP32's rounding floor, not the solution. Replace it by the FP64
    // residual on the next iteration (whose update is skipped: alpha = 0) and restart from it.
    const bool recover = !positive && !replaced && phase != 0 && !converged && it < g.maxIters;
    if (recover) c.brk = 1;
    c.rz = recover ? 1.0 : tot;   // any positive value: the skipped update does not use it
    if (phase != 0) c.beta = restart || recover ? 0.0 : beta;
    const bool stop = converged || it >= g.maxIters || (!positive && !recover);
    const bool claims = phase != 0 && (!above(rmax, c.relStop2) || !above(rmax, c.absHalf));
    c.repl = !stop && phase != 0 && ((it % g.replaceEvery) == 0 || claims || recover);
    if (stop) c.done = 1;
}

}  // namespace phx
