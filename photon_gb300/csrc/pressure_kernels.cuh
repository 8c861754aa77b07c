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

// ---- coarse levels ------------------------------------------------------------------
// damped Jacobi sweep on a coarse level (jacobi, pressure_mg.cpp:237-247).
// mode 1: y -> x; mode 2: x plus the coarser
// level's x prolongated (:290-297), into y; mode 3 (the mixed path's one-sweep
// schedule): y plus the coarser level's x prolongated, into x.
template <class R>
__device__ __forceinline__ void jacobiRow(const Scn<R>& g, int I, int l, int mode) {
    using T = R;
    const Level<R>& L = g.lv[l];
    if (I >= L.n) return;
    const bool toX = mode == 1 || mode == 3, prolong = mode == 2 || mode == 3;
    R* out = toX ? L.x : L.y;
    const R* in = toX ? L.y : L.x;
    const R* xc = prolong ? g.lv[l + 1].x : nullptr;
    const int* agg = L.agg;
    auto X = [&](int n) -> T {
        T v = in[n];
        if (prolong) v = v + xc[agg[n]];
        return v;
    };
    const int q0 = L.rowStart[I], q1 = L.rowStart[I + 1];
    const T xI = X(I);
    T s = L.b[I];
    for (int q = q0; q < q1; q += 8) {   // eight couplings at a time: their loads are in flight together
        T w[8], x[8];
        int n[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) { n[e] = L.col[min(q + e, q1 - 1)]; w[e] = L.val[min(q + e, q1 - 1)]; }
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = X(n[e]);
#pragma unroll
        for (int e = 0; e < 8; ++e) if (q + e < q1) s = madd(s, w[e], x[e]);
    }
    out[I] = jacobiValue(s, xI, L.diag[I], L.omd[I]);
}
// residual of level l fused with its restriction to level l+1 and the first
// (from-zero) Jacobi sweep of level l+1 (pressure_mg.cpp:248-257, 285-286,
// 237-247). Eight lanes serve one unknown J of level l+1: they compute the
// residuals of J's children eight at a time (children in ascending order),
// and the group's first lane sums them in that order -- the order of the
// reference's scatter -- then sets y_J = omega b_J / diag_J unless level l+1
// is the coarsest. Every lane of the warp takes part (warp shuffles).
constexpr int RRJ_LANES = 8;
template <class R>
__device__ __forceinline__ void resRestrictJac0Warp(const Scn<R>& g, int jBase, int l) {
    using T = R;
    const Level<R>& L = g.lv[l];
    const Level<R>& C = g.lv[l + 1];
    const int J = jBase + ((threadIdx.x & 31) / RRJ_LANES);
    const int c = threadIdx.x % RRJ_LANES;
    const int groupLane0 = threadIdx.x & 31 & ~(RRJ_LANES - 1);
    int nch = 0, e0 = 0;
    if (J < C.n) {
        e0 = L.childStart[J];
        nch = L.childStart[J + 1] - e0;
    }
    const int chunks = __reduce_max_sync(0xffffffffu, (nch + RRJ_LANES - 1) / RRJ_LANES);
    T acc = 0;
    for (int ch = 0; ch < chunks; ++ch) {
        const int idx = ch * RRJ_LANES + c;
        T r = 0;
        if (idx < nch) {
            const int I = L.child[e0 + idx];
            const T dg = L.diag[I];
            if (dg > 0) {
                const R* it = g.smooth1 ? L.y : L.x;   // the level's iterate after its down-leg sweeps
                const int q0 = L.rowStart[I], q1 = L.rowStart[I + 1];
                T s = madd(L.b[I], -dg, it[I]);
                for (int q = q0; q < q1; q += 8) {
                    T w[8], x[8];
                    int n[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) { n[e] = L.col[min(q + e, q1 - 1)]; w[e] = L.val[min(q + e, q1 - 1)]; }
#pragma unroll
                    for (int e = 0; e < 8; ++e) x[e] = it[n[e]];
#pragma unroll
                    for (int e = 0; e < 8; ++e) if (q + e < q1) s = madd(s, w[e], x[e]);
                }
                r = s;
            }
        }
        for (int q = 0; q < RRJ_LANES; ++q) {
            const T rq = __shfl_sync(0xffffffffu, r, groupLane0 + q);
            if (ch * RRJ_LANES + q < nch) acc = acc + rq;
        }
    }
    if (J < C.n && c == 0) {
        C.b[J] = acc;
        if (l + 1 < g.nLevels - 1) C.y[J] = jacobiValue(acc, T(0), C.diag[J], C.omd[J]);
    }
}
// coarsest level: x = M b with the dense operator of the reference's 20
// forward + backward Gauss-Seidel sweeps (pressure_mg.cpp:258-266, 279).
// One warp per row.
template <class R>
__device__ __forceinline__ void coarseDenseRow(const Scn<R>& g, int row) {
    using T = R;
    const Level<R>& L = g.lv[g.nLevels - 1];
    const int lane = threadIdx.x & 31;
    if (row >= L.n) return;
    const R* M = L.dense + (size_t)row * L.n;
    T acc = 0;
    for (int j0 = 0; j0 < L.n; j0 += 256) {   // eight columns a lane at a time: their loads are in flight together
        T m[8], v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int j = j0 + 32 * e + lane;
            m[e] = j < L.n ? M[j] : T(0);
            v[e] = j < L.n ? L.b[j] : T(0);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) acc = madd(acc, m[e], v[e]);
    }
    acc = warpSum(acc);
    if (lane == 0) L.x[row] = acc;
}
// coarsest level solved as the reference does it: 20 forward + backward
// sweeps, serially in one thread (used when the level is too large for a dense
// operator)
template <class R>
__device__ __forceinline__ void coarseSerialTile(const Scn<R>& g) {
    using T = R;
    if (threadIdx.x != 0) return;
    const Level<R>& L = g.lv[g.nLevels - 1];
    for (int I = 0; I < L.n; ++I) L.x[I] = 0;
    for (int it = 0; it < 20; ++it)
        for (int dir = 0; dir < 2; ++dir)
            for (int t = 0; t < L.n; ++t) {
                int I = dir == 0 ? t : L.n - 1 - t;
                T dg = L.diag[I];
                if (dg <= 0) { L.x[I] = 0; continue; }
                T s = L.b[I];
                for (int q = L.rowStart[I]; q < L.rowStart[I + 1]; ++q) s += L.val[q] * L.x[L.col[q]];
                L.x[I] = s / dg;
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
