// The pressure solve as one cooperative kernel: the multigrid-preconditioned
// CG of every scenario of a context (src/sim/gasphase.cpp:551-626 with the
// V-cycle of src/sim/pressure_mg.cpp:193-300), from the first residual to the
// accepted pressure.
//
// Why one kernel. A CG iteration is 12 to 18 short passes. Launched one by one
// from a graph's while node each cost about 6 us on a single building whatever
// its size (a launch, a chain of dependent loads for its tables and
// descriptor, and a drained GPU); a team barrier costs 1.0 us between 2 CTAs
// and 1.2 to 1.5 us between 152 with stores in flight, and tables, scalars and
// coarse rows stay on the SM. Measured, ms per step, launches / this kernel (the other
// stages' changes included): 36x24x24 room 2.15 / 0.72 in FP64 and 1.13 / 0.45 mixed,
// 72x52x44 house 6.8 / 2.75 and 2.77 / 1.21, 1.3 M cells mixed 5.66 / 3.58, 24 houses of
// 2.9 M cells mixed 8.1 / 5.6.
//
// What bounds it. One building: latency. Per pass a barrier, one L2 round trip
// (286 cycles) and the pass's own instructions, 2 to 3 us together; per
// reduction a chain of FP64 additions (72 cycles each) and one division (570).
// Large batches: instruction issue in FP32, the FP64 pipe (a warp's
// instruction takes it about 19 cycles) in FP64.
//
// Teams. The CTAs of the grid are divided into teams, one per scenario (teams.cuh).
// A team runs its scenario's passes one after the other with a barrier of its own
// between them, so a scenario never waits for another one's iterations and a
// stopped scenario costs nothing. Small scenarios can take turns on a CTA.
// Every CTA of a team keeps the scenario's scalars in shared memory and
// computes alpha, beta and the stop test itself from the passes' partial sums,
// in one fixed order, so all of them take the same decisions.
//
// Sums: a scenario's partial sums and the order they are added in follow from
// its size alone (SolveTiling). Neither depends on the teams, so a scenario's
// result is the same bits alone, in any batch and with any number of CTAs.
//
// Waits: a team barrier and the reader of a tagged value give up after
// Scn::waitCycles, record it in the context's error word and end the kernel; the
// launch is cooperative, so all CTAs of a team are resident.
#pragma once
#include "mixed_kernels.cuh"

namespace phx {

// dense coarse operators up to this many unknowns (n^2 reals)
constexpr int DENSE_MAX = 4096;

// PER: CTAs of the kernel per SM
template <class R, int PER>
struct SolveCfg {
    // threads per CTA. FP64 takes 128 registers a thread. FP32 trades registers for warps in
    // flight: house step 1.25 / 1.27 / 1.31 ms at 768 / 896 / 1024 threads, 24 scenarios 6.25 / 5.98 / 5.93
    static constexpr int T = sizeof(R) == 8 ? 512 : PER == 1 ? 896 : 512;
    // shared memory for the coarse rows, bytes: what it takes is missing to L1. FP32 house
    // step 1.217 / 1.222 / 1.238 / 1.254 ms at 32 / 64 / 96 / 128 KiB, 1.3e6 cells 3.69 / 3.61 /
    // 3.58 / 3.56; FP64 house 2.796 / 2.756 / 2.755 / 2.762
    static constexpr int ROWS = PER > 1 ? 32768 : sizeof(R) == 8 ? 98304 : 65536;
    // dynamic shared memory: coarse rows, then by turns the FP32 dot products' terms and
    // the coarsest level's right-hand side
    static constexpr int TERMS = sizeof(R) == 8 ? 0 : 4 * T * 8, DENSE_B = DENSE_MAX * (int)sizeof(R);
    static constexpr int SMEM = ROWS + (TERMS > DENSE_B ? TERMS : DENSE_B);
};

// CTAs per SM. Two of 512 threads divide the GPU more finely among scenarios than one of
// 896 (teams of whole CTAs, each as slow as its most loaded scenario) and wait at barriers
// in turn, but have fewer registers a thread and twice the arrivals. FP32 steps, one / two,
// ms: 8 scenarios 2.73 / 2.71, 12 3.58 / 3.59, 16 4.43 / 4.29, 24 6.54 / 6.35, 40 9.32 / 8.69,
// 60 small ones 2.45 / 2.24; 4 scenarios 2.29 / 2.46. So two where a team would have fewer
// than ten CTAs. FP64 (two of 256 threads) is slower throughout: 24 scenarios 11.46 / 11.55.
template <class R>
inline int solvePerSm(int nscn, int sms) { return sizeof(R) == 4 && nscn * 10 > sms ? 2 : 1; }

struct SolveArgs {
    TeamTable teams;
    int cap;                 // iterations after which the loop ends whatever the flags say
    int vcycleOnly;          // 1: one V-cycle z = M r without the CG (phx_precondition)
    double* maxPart;         // 2 per CTA: max |r| of the recursion, max |r| of the FP64 residual
};

// Passes over level 0. A thread owns a pair of cells along x, one red (i + j + k
// even) and one black; every pass relaxes or applies the stencil to one colour
// and reads the other colour's neighbours.
enum {
    PASS_APPLY = 0,          // q = A z + beta q, d = z + beta d, d.q
    PASS_UPDATE,             // p += alpha d, r -= alpha q, max|r|; red z = r / diag
    PASS_RED0,               // red z = r / diag
    PASS_BLACK0,             // black z from its red neighbours: the pre-smoothing pair from x = 0
    PASS_RES,                // residual restricted to level 1, level 1's first Jacobi sweep
    PASS_BLACK,              // black sweep after the prolongation
    PASS_RED                 // red sweep, r.z
};

template <class R>
struct SolveBufs {
    R *p, *r, *z, *q, *d;    // d: the direction (FP32: the previous one, dNew the one being formed)
    R* dNew;
    R alpha, beta;
    unsigned tag;            // of the V-cycle under way
    bool haveD;              // d and q hold the previous direction and its product
};

// a pair's values at c0, c0 + 1: one vector access where rows have even length
template <class R, bool EVEN>
__device__ __forceinline__ void pairLoad(const R* a, int c0, bool on1, R& v0, R& v1) {
    if constexpr (EVEN) {
        using V = typename std::conditional<sizeof(R) == 4, float2, double2>::type;
        const V v = *reinterpret_cast<const V*>(a + c0);
        v0 = v.x;
        v1 = v.y;
    } else {
        v0 = a[c0];
        v1 = a[on1 ? c0 + 1 : c0];
    }
}
template <class R, bool EVEN>
__device__ __forceinline__ void pairStore(R* a, int c0, bool on1, R v0, R v1) {
    if constexpr (EVEN) {
        using V = typename std::conditional<sizeof(R) == 4, float2, double2>::type;
        V v;
        v.x = v0;
        v.y = v1;
        *reinterpret_cast<V*>(a + c0) = v;
    } else {
        a[c0] = v0;
        if (on1) a[c0 + 1] = v1;
    }
}

// the right-hand side of level-1 unknown `at` (none: -1) and, unless level 1 is the
// coarsest, its first damped Jacobi sweep from x = 0. Every lane writes its
// cells' aggregates; the lanes of one aggregate write the same value.
template <class R>
__device__ __forceinline__ void restrictTo(const Scn<R>& g, int at, R value, unsigned tag) {
    if (at < 0) return;
    const Level<R>& L = g.lv[1];
    tagStore(L.b, at, value, tag);
    if (g.nLevels > 2) tagStore(L.yd, at, jacobiValue(value, R(0), L.diag[at], L.omd[at]), tag);
}

// A pair's place: its first cell, whether it exists (live), has a second cell (on1), has
// its red cell second (red1), and which of its neighbours lie in the grid
template <class R>
struct PairPlace {           // the pair of thread-index q: block q / 4, row and plane of the block by q % 4
    int i0, j, k, c0, nx, ny, nz;
    bool live, on1;
    __device__ __forceinline__ PairPlace(const Scn<R>& g, int q, int nblk) : nx(g.nx), ny(g.ny), nz(g.nz) {
        const int blk = min(q >> 2, nblk - 1);
        const int bz = (int)divS((unsigned)blk, g.dvL0[1]);
        const int rem = blk - bz * (int)g.dvL0[1].d;
        const int by = (int)divS((unsigned)rem, g.dvL0[0]);
        i0 = 2 * (rem - by * (int)g.dvL0[0].d);
        j = 2 * by + (q & 1);
        k = 2 * bz + ((q >> 1) & 1);
        live = (q >> 2) < nblk && j < ny && k < nz;
        on1 = live && i0 + 1 < nx;
        c0 = live ? i0 + nx * (j + ny * k) : 0;
    }
    __device__ __forceinline__ int red1() const { return (j ^ k) & 1; }
    __device__ __forceinline__ bool xm() const { return live && i0 > 0; }
    __device__ __forceinline__ bool xp() const { return live && i0 + 2 < nx; }
    __device__ __forceinline__ bool ym() const { return live && j > 0; }
    __device__ __forceinline__ bool yp() const { return live && j < ny - 1; }
    __device__ __forceinline__ bool zm() const { return live && k > 0; }
    __device__ __forceinline__ bool zp() const { return live && k < nz - 1; }
};
// One pass over a pair. All loads are issued unconditionally at clamped places and
// used through the cell's code, so one memory latency covers them. Cells
// without a diagonal hold 0 in z, d, q and r.
//
// FP64: terms of the reference's passes that are known by construction are not
// evaluated. After the pre-smoothing pair a black cell's residual is zero and a
// red cell's is the sum of its black neighbours (its z is r / diag); after the
// last red half sweep (A z)_red = r_red; and q = A d follows d's recurrence
// (q = A z + beta q), so no neighbour's d is needed. FP32 evaluates every term:
// dropping them moved the rounding of its recursion, and with it iteration
// counts and the pressure's FP32 noise.
// dot (FP64) or t0, t1 (FP32) take the pair's terms of the pass's dot product.
template <class R, int MODE, bool EVEN, class Place>
__device__ __forceinline__ void solvePair(const Scn<R>& g, const SolveBufs<R>& B, const Place& at, double& dot, F2& t0, F2& t1,
                                          R& rmax, bool writeZ) {
    using T = R;
    const int nx = g.nx, sxy = nx * g.ny;
    const bool live = at.live;
    if (MODE != PASS_RES && !live) return;
    const int c0 = at.c0;
    const bool on1 = EVEN ? live : at.on1;
    const int ro = at.red1();            // the red cell of the pair: c0 + ro
    const bool rOn = ro ? on1 : live, bOn = ro ? live : on1;
    const int cr = rOn ? c0 + ro : c0, cb = bOn ? c0 + 1 - ro : c0;
    const unsigned char* cf = g.code0;
    auto diagOf = [&](int c, unsigned cd) -> T { return (cd & CODE_GENERAL) ? g.diag[c] : codeDiag<T>(cd); };

    if constexpr (MODE == PASS_UPDATE) {
        T p0, p1, d0, d1, q0, q1, r0, r1;
        pairLoad<T, EVEN>(B.p, c0, on1, p0, p1);
        pairLoad<T, EVEN>(sizeof(R) == 4 ? B.dNew : B.d, c0, on1, d0, d1);
        pairLoad<T, EVEN>(B.q, c0, on1, q0, q1);
        pairLoad<T, EVEN>(B.r, c0, on1, r0, r1);
        const unsigned cd = cf[cr];
        p0 = madd(p0, B.alpha, d0);
        r0 = madd(r0, -B.alpha, q0);
        p1 = madd(p1, B.alpha, d1);
        r1 = madd(r1, -B.alpha, q1);
        rmax = mx(rmax, (T)fabs(r0));
        if (on1) rmax = mx(rmax, (T)fabs(r1));
        pairStore<T, EVEN>(B.p, c0, on1, p0, p1);
        pairStore<T, EVEN>(B.r, c0, on1, r0, r1);
        if (writeZ && rOn) {
            const T dg = diagOf(cr, cd);
            B.z[cr] = dg <= T(0) ? T(0) : l0Div(ro ? r1 : r0, cd, dg);
        }
        return;
    }
    if constexpr (MODE == PASS_RED0) {
        if (rOn) {
            const unsigned cd = cf[cr];
            const T rv = B.r[cr], dg = diagOf(cr, cd);
            B.z[cr] = dg <= T(0) ? T(0) : l0Div(rv, cd, dg);
        }
        return;
    }
    if constexpr (sizeof(R) == 4 && (MODE == PASS_APPLY || MODE == PASS_RES)) {
        // FP32: both cells of the pair with all their neighbours; q is A d itself and
        // the residual keeps every term (their rounding is what the FP32 recursion
        // is built on: the forms below, exact in real numbers, would let it drift)
        auto value = [&](int c) -> T {
            const T zv = B.z[c];
            if (MODE == PASS_APPLY && B.haveD) return zv + B.beta * B.d[c];
            return zv;
        };
        auto pair = [&](int c, T& v0, T& v1) {
            pairLoad<T, EVEN>(B.z, c, on1, v0, v1);
            if (MODE == PASS_APPLY && B.haveD) {
                T e0, e1;
                pairLoad<T, EVEN>(B.d, c, on1, e0, e1);
                v0 = v0 + B.beta * e0;
                v1 = v1 + B.beta * e1;
            }
        };
        T v0, v1, ym0, ym1, yp0, yp1, zm0, zm1, zp0, zp1;
        const int c1 = on1 ? c0 + 1 : c0;
        const T xm = value(at.xm() ? c0 - 1 : c0), xp = value(at.xp() ? c0 + 2 : c0);
        pair(c0, v0, v1);
        pair(at.ym() ? c0 - nx : c0, ym0, ym1);
        pair(at.yp() ? c0 + nx : c0, yp0, yp1);
        pair(at.zm() ? c0 - sxy : c0, zm0, zm1);
        pair(at.zp() ? c0 + sxy : c0, zp0, zp1);
        const unsigned cd0 = cf[c0], cd1 = cf[c1];
        const L0Nb<T> n0{xm, v1, ym0, yp0, zm0, zp0}, n1{v0, xp, ym1, yp1, zm1, zp1};
        const T dg0 = diagOf(c0, cd0), dg1 = diagOf(c1, cd1);
        if constexpr (MODE == PASS_APPLY) {
            T w0 = T(0), w1 = T(0);
            if (dg0 > T(0)) w0 = l0Sum<-1>(g, dg0 * v0, cd0, n0, c0);
            if (on1 && dg1 > T(0)) w1 = l0Sum<-1>(g, dg1 * v1, cd1, n1, c1);
            pairStore<T, EVEN>(B.dNew, c0, on1, v0, v1);
            pairStore<T, EVEN>(B.q, c0, on1, w0, w1);
            t0 = f2prod(w0, v0);
            t1 = on1 ? f2prod(w1, v1) : F2{0.f, 0.f};
        } else {
            T r0, r1;
            pairLoad<T, EVEN>(B.r, c0, on1, r0, r1);
            const int* af = g.lv[0].agg;
            const int a0 = live ? af[c0] : -1, a1 = on1 ? af[c1] : -1;
            T s0 = T(0), s1 = T(0);
            if (a0 >= 0) s0 = l0Sum<1>(g, r0 - dg0 * v0, cd0, n0, c0);
            if (a1 >= 0) s1 = l0Sum<1>(g, r1 - dg1 * v1, cd1, n1, c1);
            // the block's cells in ascending order over its four lanes
            int whole = max(a0, a1);
            whole = max(whole, __shfl_xor_sync(0xffffffffu, whole, 1));
            whole = max(whole, __shfl_xor_sync(0xffffffffu, whole, 2));
            if (__all_sync(0xffffffffu, (a0 < 0 || a0 == whole) && (a1 < 0 || a1 == whole))) {
                // one aggregate per block (a cell without one adds 0): its last lane has the sum
                T acc = s0 + s1;
#pragma unroll
                for (int l = 1; l < 4; ++l) {
                    const T before = __shfl_sync(0xffffffffu, acc, l - 1, 4);
                    if ((threadIdx.x & 3) == l) acc = (before + s0) + s1;
                }
                if ((threadIdx.x & 3) == 3) restrictTo(g, whole, acc, B.tag);
            } else {
                T acc0 = T(0), acc1 = T(0);
#pragma unroll 1
                for (int l = 0; l < 4; ++l) {
                    const int b0 = __shfl_sync(0xffffffffu, a0, l, 4), b1 = __shfl_sync(0xffffffffu, a1, l, 4);
                    const T e0 = __shfl_sync(0xffffffffu, s0, l, 4), e1 = __shfl_sync(0xffffffffu, s1, l, 4);
                    if (b0 >= 0 && b0 == a0) acc0 = acc0 + e0;
                    if (b1 >= 0 && b1 == a0) acc0 = acc0 + e1;
                    if (b0 >= 0 && b0 == a1) acc1 = acc1 + e0;
                    if (b1 >= 0 && b1 == a1) acc1 = acc1 + e1;
                }
#pragma unroll 1
                for (int h = 0; h < 2; ++h)
                    if (h == 0 || a1 != a0) restrictTo(g, h == 0 ? a0 : a1, h == 0 ? acc0 : acc1, B.tag);
            }
        }
        return;
    }
    // the cell this pass computes (o: its place in the pair) and its neighbours of
    // the other colour
    constexpr bool kRed = MODE == PASS_RES || MODE == PASS_RED;
    const int o = kRed ? ro : 1 - ro;
    const int c = kRed ? cr : cb, cIn = kRed ? cb : cr;
    const bool cOn = kRed ? rOn : bOn, inOn = kRed ? bOn : rOn;
    const int nb[5] = {(o ? at.xp() : at.xm()) ? (o ? c + 1 : c - 1) : c, at.ym() ? c - nx : c,
                       at.yp() ? c + nx : c, at.zm() ? c - sxy : c, at.zp() ? c + sxy : c};
    const T* z = B.z;
    T v[5], vIn;
    vIn = z[cIn];
#pragma unroll
    for (int f = 0; f < 5; ++f) v[f] = z[nb[f]];
    const unsigned cd = cf[c];
    if constexpr (MODE == PASS_BLACK) {   // red neighbours: z plus the prolongated correction
        const int* af = g.lv[0].agg;
        const T* x1 = g.lv[1].x;
        int ag[5], agIn;
        agIn = af[cIn];
#pragma unroll
        for (int f = 0; f < 5; ++f) ag[f] = af[nb[f]];
        T xv[5], xIn;
        xIn = x1[max(agIn, 0)];
#pragma unroll
        for (int f = 0; f < 5; ++f) xv[f] = x1[max(ag[f], 0)];
        vIn = agIn >= 0 ? (T)(vIn + xIn) : vIn;
#pragma unroll
        for (int f = 0; f < 5; ++f) v[f] = ag[f] >= 0 ? (T)(v[f] + xv[f]) : v[f];
    }
    L0Nb<T> n;
    n.xm = o ? vIn : v[0];
    n.xp = o ? v[0] : vIn;
    n.ym = v[1];
    n.yp = v[2];
    n.zm = v[3];
    n.zp = v[4];
    auto sum = [&](auto sign, T start) -> T {
        return l0Sum<decltype(sign)::value>(g, start, cd, n, c);
    };
    using Plus = std::integral_constant<int, 1>;
    using Minus = std::integral_constant<int, -1>;
    if constexpr (MODE == PASS_APPLY) {
        T z0, z1, d0 = T(0), d1 = T(0), q0 = T(0), q1 = T(0);
        const T zc = z[c], rr = B.r[cr];
        if (B.haveD) {
            pairLoad<T, EVEN>(B.d, c0, on1, d0, d1);
            pairLoad<T, EVEN>(B.q, c0, on1, q0, q1);
        }
        const T zr = rOn ? vIn : T(0), zb = bOn ? zc : T(0);
        z0 = ro ? zb : zr;
        z1 = ro ? zr : zb;
        T wb = T(0);
        if (cOn) {
            const T dg = diagOf(c, cd);
            if (dg > T(0)) wb = sum(Minus{}, dg * zb);
        }
        const T wr = rOn ? rr : T(0);
        T w0 = ro ? wb : wr, w1 = ro ? wr : wb;
        if (B.haveD) {
            z0 = madd(z0, B.beta, d0);
            z1 = madd(z1, B.beta, d1);
            w0 = madd(w0, B.beta, q0);
            w1 = madd(w1, B.beta, q1);
        }
        pairStore<T, EVEN>(B.d, c0, on1, z0, z1);
        pairStore<T, EVEN>(B.q, c0, on1, w0, w1);
        dot = fma((double)w0, (double)z0, dot);
        if (on1) dot = fma((double)w1, (double)z1, dot);
    } else if constexpr (MODE == PASS_BLACK0 || MODE == PASS_BLACK) {
        const T rv = B.r[c];
        if (cOn) {
            const T dg = diagOf(c, cd);
            T zc = T(0);
            if (dg > T(0)) zc = l0Div(sum(Plus{}, rv), cd, dg);
            B.z[c] = zc;
        }
    } else if constexpr (MODE == PASS_RED) {
        const T rv = B.r[c], rb = B.r[cIn];
        if (cOn) {
            const T dg = diagOf(c, cd);
            T zc = T(0);
            if (dg > T(0)) zc = l0Div(sum(Plus{}, rv), cd, dg);
            B.z[c] = zc;
            if constexpr (sizeof(R) == 4) (o ? t1 : t0) = f2prod(rv, zc);
            else dot = fma(rv, zc, dot);
        }
        if (inOn) {
            if constexpr (sizeof(R) == 4) (o ? t0 : t1) = f2prod(rb, vIn);
            else dot = fma(rb, vIn, dot);
        }
    } else {   // PASS_RES: the four lanes of a block hold its red cells in ascending order
        const int* af = g.lv[0].agg;
        const int a = cOn ? af[c] : -1, ab = inOn ? af[cIn] : -1;
        T res = T(0);
        if (a >= 0) res = sum(Plus{}, T(0));
        int whole = max(a, ab);
        whole = max(whole, __shfl_xor_sync(0xffffffffu, whole, 1));
        whole = max(whole, __shfl_xor_sync(0xffffffffu, whole, 2));
        if (__all_sync(0xffffffffu, (a < 0 || a == whole) && (ab < 0 || ab == whole))) {
            // one aggregate per block: its last lane has the sum
            T acc = res;
#pragma unroll
            for (int l = 1; l < 4; ++l) {
                const T before = __shfl_sync(0xffffffffu, acc, l - 1, 4);
                if ((threadIdx.x & 3) == l) acc = before + res;
            }
            if ((threadIdx.x & 3) == 3) restrictTo(g, whole, acc, B.tag);
        } else {
            T acc = T(0), accB = T(0);
#pragma unroll 1
            for (int l = 0; l < 4; ++l) {
                const int al = __shfl_sync(0xffffffffu, a, l, 4);
                const T rl = __shfl_sync(0xffffffffu, res, l, 4);
                if (al >= 0 && al == a) acc = acc + rl;
                if (al >= 0 && al == ab) accB = accB + rl;
            }
#pragma unroll 1
            for (int h = 0; h < 2; ++h)
                if (h == 0 || ab != a) restrictTo(g, h == 0 ? a : ab, h == 0 ? acc : accB, B.tag);
        }
    }
}

// ---- team barrier ---------------------------------------------------------------
struct Team {
    unsigned target;         // arrivals at g.teamBar since the start of the solve that end the next wait
    int size, rank;          // CTAs, this CTA's place
};

// every thread of every CTA of the team calls it; false, for the whole CTA: a wait ran out
// and the kernel has to end. *gaveUp and *go are shared memory, *gaveUp 0 at first.
template <class R>
__device__ __forceinline__ bool teamSync(const Scn<R>& g, Team& t, volatile int* gaveUp, volatile int* go) {
    if (t.size == 1) return __syncthreads_and(*gaveUp == 0) != 0;
    __syncthreads();
    t.target += (unsigned)t.size;
    if (threadIdx.x == 0) {
        unsigned* const bar = g.teamBar;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        unsigned seen;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
        if ((int)(seen - t.target) < 0) {
            const long long t0 = clock64();
            do {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
                if (clock64() - t0 > g.waitCycles) {
                    atomicOr(g.errWord, ERR_TEAM_WAIT);
                    *gaveUp = 1;
                    break;
                }
            } while ((int)(seen - t.target) < 0);
        }
        *go = *gaveUp == 0;   // one answer: a fast warp's next wait may run out before a slow one has looked
    }
    __syncthreads();
    return *go != 0;
}

// ---- sums ----------------------------------------------------------------------
__device__ __forceinline__ F2 f2Load(const double* p) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    return F2{v.x, v.y};
}
__device__ __forceinline__ void f2Store(double* p, F2 v) { *reinterpret_cast<float2*>(p) = make_float2(v.hi, v.lo); }
// a double-float as two tagged words
__device__ __forceinline__ void tagStorePair(double* part, int t, F2 v, unsigned tag) {
    const unsigned long long w = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(part + 2 * (size_t)t), "l"(w | __float_as_uint(v.hi)),
                 "l"(w | __float_as_uint(v.lo))
                 : "memory");
}
__device__ __forceinline__ bool tagLoadPair(const double* part, int t, unsigned tag, F2& v) {
    unsigned long long hi, lo;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(hi), "=l"(lo) : "l"(part + 2 * (size_t)t) : "memory");
    v = F2{__uint_as_float((unsigned)hi), __uint_as_float((unsigned)lo)};
    return (unsigned)(hi >> 32) == tag && (unsigned)(lo >> 32) == tag;
}
// a float as a double by its bits (a conversion instruction takes some hundred
// cycles here); zeros and numbers below the normal range take the conversion
__device__ __forceinline__ double widen(float f) {
    const unsigned b = __float_as_uint(f), e = b & 0x7f800000u;
    if (e == 0u || e == 0x7f800000u) return (double)f;
    return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(b << 29));
}
__device__ __forceinline__ double warpSumAll(double v) {   // the same value in every lane
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// FP32: the sum of a scenario's nt tiles, four to a group whose sum is rounded to
// FP64, in every lane of warp 0. The orders are those of a 128-thread CTA per 128
// blocks and one such CTA over their sums: thread i adds groups i, i + 128, ...
// All threads form the groups' sums first (sh: a value per thread of the CTA), so that
// thread i waits for one load, not for one per group.
// TAGGED: the partials are tagged words, waited for instead of a team barrier.
template <bool TAGGED>
__device__ __forceinline__ double teamTotalF2(const double* part, int nt, double* sh, double* sh4, unsigned tag,
                                              const TagWait& tw) {
    const int tid = (int)threadIdx.x, n4 = (nt + 3) / 4;
    double acc = 0;
    for (int i0 = 0; i0 < n4; i0 += (int)blockDim.x) {
        const int i = i0 + tid;
        if (i < n4) {
            F2 w[4];
            auto read = [&] {
                bool ok = true;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    w[e] = F2{0.f, 0.f};
                    if (4 * i + e < nt) {
                        if (TAGGED) {
                            ok &= tagLoadPair(part, 4 * i + e, tag, w[e]);
                        } else {
                            const float2 v = __ldcg(reinterpret_cast<const float2*>(part + 4 * i + e));
                            w[e] = F2{v.x, v.y};
                        }
                    }
                }
                return ok;
            };
            waitFor(tw, read);
            const F2 v = f2add(f2add(w[0], w[2]), f2add(w[1], w[3]));
            sh[tid] = widen(v.hi) + widen(v.lo);
        }
        __syncthreads();
        if (tid < 128) {
            const int n = min(n4 - i0, (int)blockDim.x);
#pragma unroll 1
            for (int q = tid; q < n; q += 128) acc += sh[q];
        }
        if (i0 + (int)blockDim.x < n4) __syncthreads();
    }
    if (tid < 128) {
        acc = warpSum(acc);
        if ((tid & 31) == 0) sh4[tid >> 5] = acc;
    }
    __syncthreads();
    return (sh4[0] + sh4[2]) + (sh4[1] + sh4[3]);
}
// The sum of a scenario's nt partials, in every lane of warp 0; the whole CTA
// calls it and may read what other warps wrote to shared memory before the call.
// Up to 512 partials warp 0 adds alone, beyond that eight warps add 256 columns
// first. What counts here is the chain of FP64 instructions (an addition takes
// some hundred cycles, an FP32-to-FP64 conversion more): the loads of sixteen
// values are in flight together, and they are added as a tree.
template <bool TAGGED>
__device__ __forceinline__ double teamTotal(const double* part, int nt, double* sh256, unsigned tag, const TagWait& tw) {
    const int tid = (int)threadIdx.x;
    double acc = 0;
    const int step = nt > 512 ? 256 : 32;
    if (tid < step) {
        for (int i0 = tid; i0 < nt; i0 += 16 * step) {
            double v[16];
            waitFor(tw, [&] {
                bool ok = true;
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const int i = i0 + e * step;
                    v[e] = 0.0;
                    if (i < nt) {
                        if (TAGGED) ok &= tagLoad(reinterpret_cast<const unsigned long long*>(part), i, tag, v[e]);
                        else v[e] = __ldcg(part + i);
                    }
                }
                return ok;
            });
#pragma unroll
            for (int e = 0; e < 16; e += 4)
                if ((i0 & ~31) + e * step < nt) acc += (v[e] + v[e + 1]) + (v[e + 2] + v[e + 3]);
        }
        if (step == 256) sh256[tid] = acc;
    }
    __syncthreads();
    if (tid < 32) {
        if (step == 256) {
            double v[8];
#pragma unroll
            for (int w = 0; w < 8; ++w) v[w] = sh256[w * 32 + tid];
            acc = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
        }
        acc = warpSumAll(acc);
    }
    return acc;
}

// The maximum of non-negative values through their bit patterns, in integer
// instructions (a NaN never enters: the callers' mx drops it)
__device__ __forceinline__ float warpMaxPos(float v) {
    return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v)));
}
__device__ __forceinline__ double warpMaxPos(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const unsigned hi = (unsigned)(b >> 32), mhi = __reduce_max_sync(0xffffffffu, hi);
    const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? (unsigned)b : 0u);
    return __longlong_as_double((long long)(((unsigned long long)mhi << 32) | mlo));
}
// CTA-wide max of non-negative values into *dst (this CTA's slot)
template <class V>
__device__ __forceinline__ void ctaMaxStore(double* dst, V v, V* sh) {
    v = warpMaxPos(v);
    const int w = (int)(threadIdx.x >> 5), l = (int)(threadIdx.x & 31), nw = (int)(blockDim.x >> 5);
    if (l == 0) sh[w] = v;   // the previous call's reader is past a team barrier
    __syncthreads();
    if (w == 0) {
        const V x = warpMaxPos(l < nw ? sh[l] : V(0));
        if (l == 0) *dst = (double)x;
    }
}

constexpr int RRJ_LANES = 8;   // lanes per unknown of a restriction

// ---- coarse rows ----------------------------------------------------------------
// A coarse level's rows lie in sets of 32, transposed over a warp's lanes (Level::rows):
// a coupling of 32 rows is one access. The sets of a warp's first ROW_CHUNKS groups are
// copied to the CTA's shared memory as far as the pool goes, since they are the same in
// every V-cycle: a sweep then waits for one memory latency (its neighbours' values); other
// sets are read from the level each time. Rows without a set take the level's arrays.
// Against rows read one by one (a lane's own row start, columns and values): house step in
// FP32 1.26 -> 1.21 ms, 1.3e6 cells 3.64 -> 3.57, 24 scenarios 6.07 -> 5.99.
constexpr int ROW_CHUNKS = 2;
template <class R>
struct RowView {
    const R* diag;           // [32]: the diagonal; FP64 sweeps (toNext): omega / diagonal
    const R* val;            // [width][32]
    const int *own, *col, *next;   // [32], [width][32] each
};
template <class R>
__device__ __forceinline__ RowView<R> rowView(const unsigned* pool, const RowSet& s) {
    RowView<R> v;
    v.diag = reinterpret_cast<const R*>(pool + s.off);
    v.val = v.diag + 32;
    v.own = reinterpret_cast<const int*>(v.val + 32 * s.width);
    v.col = v.own + 32;
    v.next = v.col + 32 * s.width;
    return v;
}
// a warp's set copied to the pool where it fits, for the whole solve: its place there, in
// the level (~off, below 0 and above -1), or none (width -1)
template <class R>
__device__ __forceinline__ RowSet keepRows(const unsigned* rows, RowSet s, bool sweep, unsigned* pool, int* used, int words) {
    const int lane = (int)(threadIdx.x & 31);
    if (s.off < 0) return RowSet{-1, -1};
    constexpr int RW = (int)sizeof(R) / 4;
    const int need = 32 * ((1 + s.width) * RW + 1 + s.width * (sweep ? 2 : 1));
    int off = 0;
    if (lane == 0) off = atomicAdd(used, need);
    off = __shfl_sync(0xffffffffu, off, 0);
    if (off + need > words) return RowSet{~s.off, s.width};
    const uint4* from = reinterpret_cast<const uint4*>(rows + s.off);
    uint4* to = reinterpret_cast<uint4*>(pool + off);
    for (int i = lane; i < need / 4; i += 32) to[i] = from[i];
    return RowSet{off, s.width};
}
// The couplings of a level's row: of a set in shared memory (FAR: in the level), or the level's arrays
template <class R, bool IN_LEVEL>
struct SetRow {
    RowView<R> v;
    int n, lane;
    __device__ __forceinline__ int col(int e) const { return v.col[32 * e + lane]; }
    __device__ __forceinline__ int next(int e, int) const { return v.next[32 * e + lane]; }
    __device__ __forceinline__ R val(int e) const { return v.val[32 * e + lane]; }
    static constexpr bool FAR = IN_LEVEL && sizeof(R) == 4;
};
template <class R>
struct StoredRow {
    const Level<R>& L;
    int q0, n;
    __device__ __forceinline__ int col(int e) const { return L.col[q0 + e]; }
    __device__ __forceinline__ int next(int, int c) const { return L.agg[c]; }
    __device__ __forceinline__ R val(int e) const { return L.val[q0 + e]; }
    static constexpr bool FAR = sizeof(R) == 4;   // values loaded with the columns (FP64 has no registers for them)
};
// the sums of a sweep and of a residual: s plus the couplings times in[col], eight at a
// time with their loads in flight together. PROLONG: in plus the coarser level's xc.
template <class R, bool PROLONG, class Row, class Vec>
__device__ __forceinline__ R rowSum(R s, const Row& row, Vec in, Vec xc, unsigned tag, const TagWait& w) {
    for (int e0 = 0; e0 < row.n; e0 += 8) {
        int col[8], nxt[8];
        R x[8], c[8], v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            col[e] = row.col(min(e0 + e, row.n - 1));
            if (Row::FAR) v[e] = row.val(min(e0 + e, row.n - 1));
            if (PROLONG) nxt[e] = row.next(min(e0 + e, row.n - 1), col[e]);
        }
        waitFor(w, [&] {
            bool ok = true;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                ok &= tagLoad(in, col[e], tag, x[e]);
                if (PROLONG) ok &= tagLoad(xc, nxt[e], tag, c[e]);
            }
            return ok;
        });
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (e0 + e < row.n) s = madd(s, Row::FAR ? v[e] : row.val(e0 + e), PROLONG ? x[e] + c[e] : x[e]);
    }
    return s;
}
// damped Jacobi sweep of row I of level l (jacobi, pressure_mg.cpp:237-247).
// SWEEP_DOWN: the second sweep on the way down; SWEEP_UP: the first on the way up, from
// the iterate plus the coarser level's prolongated x (:290-297); SWEEP_LAST: the second
// on the way up; SWEEP_ONLY: the one on the way up of the mixed path's one-sweep
// schedule. The last value of level 1 goes to its plain array, which the black
// sweep of level 0 reads after a team barrier.
enum { SWEEP_DOWN = 0, SWEEP_UP, SWEEP_LAST, SWEEP_ONLY };
template <class R, int SWEEP, class Row>
__device__ __forceinline__ void jacobiRow(const Scn<R>& g, int l, int I, const Row& row, int own, R dg, R omd, unsigned tag,
                                          const TagWait& w) {
    using T = R;
    const Level<R>& L = g.lv[l];
    constexpr bool prolong = SWEEP == SWEEP_UP || SWEEP == SWEEP_ONLY;
    const Level<R>& C = g.lv[l + 1];
    const auto in = SWEEP == SWEEP_DOWN || SWEEP == SWEEP_ONLY ? L.yd : SWEEP == SWEEP_UP ? L.xd : L.yu;
    T s, x, c = T(0);
    waitFor(w, [&] {
        bool ok = tagLoad(L.b, I, tag, s);
        ok &= tagLoad(in, I, tag, x);
        if (prolong) ok &= tagLoad(C.xu, own, tag, c);
        return ok;
    });
    s = rowSum<R, prolong>(s, row, in, C.xu, tag, w);
    const T v = jacobiValue(s, prolong ? x + c : x, dg, omd);
    if (SWEEP == SWEEP_DOWN) tagStore(L.xd, I, v, tag);
    else if (SWEEP == SWEEP_UP) tagStore(L.yu, I, v, tag);
    else if (l == 1) L.x[I] = v;
    else tagStore(L.xu, I, v, tag);
}
// residual of level l fused with its restriction to level l+1 and the first
// (from-zero) Jacobi sweep of level l+1 (pressure_mg.cpp:248-257, 285-286,
// 237-247). Eight lanes serve one unknown J of level l+1: they compute the
// residuals of J's children eight at a time (children in ascending order), and
// the group's first lane sums them in that order -- the order of the reference's
// scatter. Every lane of the warp takes part (warp shuffles).
template <class R>
__device__ __forceinline__ void restrictRows(const Scn<R>& g, int l, int jBase, const unsigned* pool, const RowSet& rs,
                                             unsigned tag, const TagWait& w) {
    using T = R;
    const Level<R>& L = g.lv[l];
    const Level<R>& C = g.lv[l + 1];
    const int lane = (int)(threadIdx.x & 31), J = jBase + lane / RRJ_LANES, c = lane % RRJ_LANES;
    const int lane0 = lane & ~(RRJ_LANES - 1);
    const auto it = g.smooth1 ? L.yd : L.xd;   // the iterate after the way down
    T acc = T(0);
    auto residual = [&](int I, T dg, const auto& row) -> T {
        T bI, xI;
        waitFor(w, [&] {
            bool ok = tagLoad(L.b, I, tag, bI);
            return ok & tagLoad(it, I, tag, xI);
        });
        const T s = rowSum<R, false>(madd(bI, -dg, xI), row, it, it, tag, w);
        return dg > 0 ? s : T(0);
    };
    auto addChildren = [&](T s, bool on) {   // the group's eight in ascending order
        __syncwarp();
        const unsigned valid = __ballot_sync(0xffffffffu, on);
#pragma unroll
        for (int q = 0; q < RRJ_LANES; ++q) {
            const T rq = __shfl_sync(0xffffffffu, s, lane0 + q);
            if ((valid >> (lane0 + q)) & 1u) acc = acc + rq;
        }
    };
    auto fromSet = [&](const RowView<R>& v, auto inLevel) {
        const int I = v.own[lane];
        T s = T(0);
        if (I >= 0) s = residual(I, v.diag[lane], SetRow<R, decltype(inLevel)::value>{v, rs.width, lane});
        addChildren(s, I >= 0);
    };
    if (rs.off >= 0) {
        fromSet(rowView<R>(pool, rs), std::false_type{});
    } else if (rs.width >= 0) {
        fromSet(rowView<R>(L.rows, RowSet{~rs.off, rs.width}), std::true_type{});
    } else {
        const int e0 = J < C.n ? L.childStart[J] : 0, nch = J < C.n ? L.childStart[J + 1] - e0 : 0;
        const int chunks = __reduce_max_sync(0xffffffffu, (nch + RRJ_LANES - 1) / RRJ_LANES);
#pragma unroll 1
        for (int ch = 0; ch < chunks; ++ch) {
            const int I = ch * RRJ_LANES + c < nch ? L.child[e0 + ch * RRJ_LANES + c] : -1;
            T s = T(0);
            if (I >= 0) {
                const int q0 = L.rowStart[I];
                s = residual(I, L.diag[I], StoredRow<R>{L, q0, L.rowStart[I + 1] - q0});
            }
            addChildren(s, I >= 0);
        }
    }
    if (J < C.n && lane == lane0) {
        tagStore(C.b, J, acc, tag);
        if (l + 1 < g.nLevels - 1) tagStore(C.yd, J, jacobiValue(acc, T(0), C.diag[J], C.omd[J]), tag);
    }
}

// ---- the kernel ----------------------------------------------------------------------
template <class R, int PER>
__global__ void __launch_bounds__(SolveCfg<R, PER>::T, PER)
k_solve(const Scn<R>* __restrict__ S, SolveArgs a) {
    using T = R;
    constexpr int TH = SolveCfg<R, PER>::T;
    constexpr bool kMixed = sizeof(R) == 4;
    __shared__ __align__(16) unsigned long long graw[sizeof(Scn<R>) / 8];
    extern __shared__ __align__(16) unsigned pool[];
    __shared__ CgState cg;
    __shared__ double shSum[256], shZone[8 * (TH / TPB)], shMax[2];
    __shared__ RowSet rowsJ[MAX_LEVELS][TH / 32][ROW_CHUNKS], rowsR[MAX_LEVELS][TH / 32][ROW_CHUNKS];
    __shared__ int poolUsed;
    __shared__ double shDot[2][sizeof(R) == 8 ? TH : TH / 2];   // FP64: the tiles' dot products, by turns; scratch
    R* const shB = reinterpret_cast<R*>(pool + SolveCfg<R, PER>::ROWS / 4);   // the coarsest right-hand side
    double* const shTerms = reinterpret_cast<double*>(pool + SolveCfg<R, PER>::ROWS / 4);   // FP32: a tile's terms, by turns
    __shared__ double shMx[32];
    __shared__ int gaveUp, go;
    static_assert(sizeof(Scn<R>) % 8 == 0, "descriptors are copied as 8-byte words");
    const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = (int)blockIdx.x;
    if (tid == 0) gaveUp = 0;
    const SolveCta mine = a.teams.ctas[b];
    Team team{0, mine.size, mine.rank};
    const Scn<R>& g = *reinterpret_cast<const Scn<R>*>(graw);
    for (int s = mine.scenario; s >= 0; s = a.teams.next[s]) {
        __syncthreads();
        {   // the scenario's descriptor and scalars
            const unsigned long long* src = reinterpret_cast<const unsigned long long*>(S + s);
            for (int i = tid; i < (int)(sizeof(Scn<R>) / 8); i += TH) graw[i] = src[i];
            __syncthreads();
            if (tid == 0) {
                const double* sv = g.sv;
                cg.rz = 1;   // not yet known: a divisor whose quotient is not used
                cg.alpha = cg.beta = cg.dq = 0;
                cg.rmax = sv[SV_RMAX];
                cg.r64 = 0;
                const double inv = sv[SV_INV], bmax = sv[SV_BMAX];
                cg.absStop = g.tol * inv;
                cg.absHalf = 0.5 * cg.absStop;
                cg.relStop = !(g.relTol > 0) ? -1.0 : kMixed && !(bmax > 0) ? 1e300 : g.relTol * bmax;
                cg.relStop2 = 2.0 * cg.relStop;
                cg.it = cg.done = cg.repl = cg.brk = 0;
                poolUsed = 0;
            }
            __syncthreads();
        }
        const int N = g.N, nl = g.nLevels;
        const int nblk = solveBlocks(g);
        const SolveTiling tl = solveTiling<R>(nblk);
        const int nt = tl.nt;
        const int rank = team.rank, size = team.size;
        double* const partDq = g.part + (size_t)PS_DQ * g.partStride;
        double* const partRz = g.part + (size_t)PS_RZ * g.partStride;
        double* const maxR = a.maxPart + 2 * b;
        const bool closed = kMixed && g.nClosed > 0;
        SolveBufs<R> B;
        B.p = g.p; B.z = g.z; B.q = g.q; B.r = g.r; B.d = g.d;
        B.dNew = nullptr; B.alpha = T(0); B.beta = T(0); B.haveD = false;

#define PHX_TEAM_SYNC() do { if (!teamSync(g, team, &gaveUp, &go)) return; } while (0)
        // one pass over the team's tiles
        const int slot = warp / tl.warps, slots = TH / 32 / tl.warps, wt = warp - slot * tl.warps;
        int turn = 0;
        // Tiles are dealt out to the CTAs by turns: neighbouring tiles have like shares of
        // gas, so this evens out the CTAs' work (FP64 house step 2.93 -> 2.75 ms, 8
        // scenarios 4.38 -> 4.19; FP32 house 1.25 -> 1.23). An FP32 CTA with several
        // rounds of tiles takes neighbours instead, which share cached rows (24 scenarios
        // 6.06 ms against 6.14 dealt out); its many tiles even out by themselves.
        const bool deal = !kMixed || nt <= slots * team.size;
        const int tFirst = deal ? team.rank + slot * team.size : (int)((long long)nt * team.rank / team.size) + slot;
        const int tEnd = deal ? nt : (int)((long long)nt * (team.rank + 1) / team.size), tStep = deal ? slots * team.size : slots;
        auto pairs = [&](auto mode, auto even, double* part, T& rm, bool writeZ) {
            constexpr int MODE = decltype(mode)::value;
            constexpr bool kDot = MODE == PASS_APPLY || MODE == PASS_RED;
            for (int t = tFirst; t < tEnd; t += tStep) {
                double dot = 0;
                F2 e0{0.f, 0.f}, e1{0.f, 0.f};
                for (int q = 0; q < tl.reps; ++q) {
                    const PairPlace<R> at(g, ((t * tl.reps + q) * tl.warps + wt) * 32 + lane, nblk);
                    solvePair<R, MODE, decltype(even)::value>(g, B, at, dot, e0, e1, rm, writeZ);
                }
                if constexpr (kDot && kMixed) {
                    // the tile's terms side by side: the first warp adds each block's eight in
                    // ascending order (one block a lane), then its 32 blocks
                    double* const sh = shTerms + 2 * TH * turn + 256 * slot;
                    turn ^= 1;
                    f2Store(sh + 64 * wt + 2 * lane, e0);
                    f2Store(sh + 64 * wt + 2 * lane + 1, e1);
                    asm volatile("bar.sync %0, 128;" ::"r"(slot + 1) : "memory");
                    if (wt == 0) {
                        F2 acc = f2Load(sh + 8 * lane);
#pragma unroll
                        for (int u = 1; u < 8; ++u) acc = f2add(acc, f2Load(sh + 8 * lane + u));
                        acc = warpSum(acc);
                        if (lane == 0) {
                            if (MODE == PASS_APPLY) tagStorePair(part, t, acc, B.tag);
                            else f2Store(part + t, acc);
                        }
                    }
                } else if constexpr (kDot) {
                    if (tl.warps > 1) {   // the tile's first warp adds the warps' lanes
                        double* const sh = shDot[turn];
                        turn ^= 1;
                        sh[tid] = dot;
                        asm volatile("bar.sync %0, %1;" ::"r"(slot + 1), "r"(tl.warps * 32) : "memory");
                        if (wt == 0)
                            for (int w = 1; w < tl.warps; ++w) dot += sh[tid + 32 * w];
                    }
                    if (wt == 0) {
                        dot = warpSumAll(dot);
                        if (lane == 0) {
                            if (MODE == PASS_APPLY) tagStore(reinterpret_cast<unsigned long long*>(part), t, dot, B.tag);
                            else part[t] = dot;
                        }
                    }
                }
            }
        };
        auto pass = [&](auto mode, double* part, T& rm, bool writeZ) {
            if (g.nx & 1) pairs(mode, std::false_type{}, part, rm, writeZ);
            else pairs(mode, std::true_type{}, part, rm, writeZ);
        };
#define PHX_PASS(m, part, rm, wz) pass(std::integral_constant<int, m>{}, part, rm, wz)
        // rows of a coarse level: a warp takes 32 consecutive rows, warps round-robin over the team
        const int gw = warp * size + rank, nw = (TH / 32) * size;
        for (int l = 1; l < nl - 1; ++l)
            for (int m = 0; m < ROW_CHUNKS; ++m) {
                const Level<R>& L = g.lv[l];
                const Level<R>& C = g.lv[l + 1];
                const int chunk = gw + m * nw;
                RowSet j{-1, -1}, r{-1, -1};
                if (chunk * 32 < L.n) j = keepRows<R>(L.rows, L.setsJ[chunk], true, pool, &poolUsed, SolveCfg<R, PER>::ROWS / 4);
                if (chunk * (32 / RRJ_LANES) < C.n)
                    r = keepRows<R>(L.rows, L.setsR[chunk], false, pool, &poolUsed, SolveCfg<R, PER>::ROWS / 4);
                if (lane == 0) {
                    rowsJ[l][warp][m] = j;
                    rowsR[l][warp][m] = r;
                }
                __syncwarp();
            }
        const TagWait tw{&gaveUp, &g.errWord, &g.waitCycles};
        auto inLevel = [](RowSet s) { return s.off >= 0 ? RowSet{~s.off, s.width} : RowSet{-1, -1}; };
        auto jacobiLevel = [&](auto sweep, int l) {
            constexpr int SWEEP = decltype(sweep)::value;
            const Level<R>& L = g.lv[l];
            for (int m = 0, i = gw * 32; i < L.n; ++m, i += nw * 32) {
                const RowSet rs = m < ROW_CHUNKS ? rowsJ[l][warp][m] : inLevel(L.setsJ[i / 32]);
                const int I = i + lane;
                if (I >= L.n) continue;
                auto fromSet = [&](const RowView<R>& v, auto far) {
                    jacobiRow<R, SWEEP>(g, l, I, SetRow<R, decltype(far)::value>{v, rs.width, lane}, v.own[lane], v.diag[lane],
                                        v.diag[lane], B.tag, tw);
                };
                if (rs.off >= 0) {
                    fromSet(rowView<R>(pool, rs), std::false_type{});
                } else if (rs.width >= 0) {
                    fromSet(rowView<R>(L.rows, RowSet{~rs.off, rs.width}), std::true_type{});
                } else {
                    const int q0 = L.rowStart[I];
                    jacobiRow<R, SWEEP>(g, l, I, StoredRow<R>{L, q0, L.rowStart[I + 1] - q0}, L.agg[I], L.diag[I], L.omd[I], B.tag, tw);
                }
            }
        };
        auto restrictLevel = [&](int l) {
            constexpr int GROUP = 32 / RRJ_LANES;
            for (int m = 0, j = gw * GROUP; j < g.lv[l + 1].n; ++m, j += nw * GROUP)
                restrictRows(g, l, j, pool, m < ROW_CHUNKS ? rowsR[l][warp][m] : inLevel(g.lv[l].setsR[j / GROUP]), B.tag, tw);
        };
        auto coarsest = [&]() {
            const Level<R>& L = g.lv[nl - 1];
            auto put = [&](int I, T v) {
                if (nl == 2) L.x[I] = v;
                else tagStore(L.xu, I, v, B.tag);
            };
            if (L.dense) {
                for (int i = tid; i < L.n; i += TH) {
                    T v = T(0);
                    waitFor(tw, [&] { return tagLoad(L.b, i, B.tag, v); });
                    shB[i] = v;
                }
                __syncthreads();
                for (int row = gw; row < L.n; row += nw) {
                    const T v = coarseDenseRow(L, row, shB);
                    if (lane == 0) put(row, v);
                }
            } else if (rank == 0) {   // yd, which nothing writes at the coarsest level, takes the right-hand side
                R *const x = L.x, *const rhs = reinterpret_cast<R*>(L.yd);
                for (int i = tid; i < L.n; i += TH) {
                    T v = T(0);
                    waitFor(tw, [&] { return tagLoad(L.b, i, B.tag, v); });
                    rhs[i] = v;
                }
                __syncthreads();
                if (tid == 0) coarseSerial(L, rhs, x);
                __syncthreads();
                for (int I = tid; I < L.n; I += TH) put(I, x[I]);
            }
        };
        // the cells of the grid, elementwise
        auto cells = [&](auto f) {
            for (int c = rank * TH + tid; c < N; c += size * TH) f(c);
        };
        // Closed zones, dealt out to the team's CTAs; where that leaves a CTA several, as many side by
        // side as it has 256 threads for (1,000 sealed cells of 216: a step 0.591 / 0.511 ms).
        // f(cell, its zone's mean of v)
        auto zones = [&](const R* v, auto f) {
            const int side = g.nClosed > size ? TH / TPB : 1, slot = side > 1 ? warp / (TPB / 32) : 0;
            if (slot >= side) return;
            const int t = tid - TPB * slot, step = side > 1 ? TPB : TH;
            double* const sh = shZone + 8 * slot;
            auto sync = [&] {
                if (side == 1) __syncthreads();
                else asm volatile("bar.sync %0, %1;" ::"r"(8 + slot), "n"(TPB) : "memory");
            };
            for (int zi = rank * side + slot; zi < g.nClosed; zi += size * side) {
                const int e0 = g.closedStart[zi], e1 = g.closedStart[zi + 1];
                double acc = 0;   // summed by 256 threads (the order of a 256-thread CTA)
                if (t < TPB)
                    for (int e = e0 + t; e < e1; e += TPB) acc += (double)v[g.closedCells[e]];
                acc = warpSum(acc);
                sync();
                if (lane == 0 && t < TPB) sh[t >> 5] = acc;
                sync();
                const double sum = ((sh[0] + sh[4]) + (sh[2] + sh[6])) + ((sh[1] + sh[5]) + (sh[3] + sh[7]));
                const double mean = e1 > e0 ? sum / (double)(e1 - e0) : 0.0;
                for (int e = e0 + t; e < e1; e += step) {
                    const int c = g.closedCells[e];
                    if (g.diag[c] > 0) f(c, mean);
                }
            }
        };
        auto zoneCenter = [&](R* v) {
            zones(v, [&](int c, double mean) { v[c] = (R)((double)v[c] - mean); });
        };
        // mixed path: r = b - A p64 in FP64 from the FP32 right-hand side and coefficients, p = 0; closed
        // zones: the zone mean of r removed
        auto residual64 = [&](double& rm) {
            const int nx = g.nx, ny = g.ny, nz = g.nz, sxy = nx * ny;
            const double* x = g.p64;
            cells([&](int c) {
                // every load up front at clamped places; a coded cell's coefficients are 0 or 1
                const unsigned cd = g.code0[c];
                const double x0 = x[c], xm = x[max(c - 1, 0)], xp = x[min(c + 1, N - 1)], ym = x[max(c - nx, 0)],
                             yp = x[min(c + nx, N - 1)], zm = x[max(c - sxy, 0)], zp = x[min(c + sxy, N - 1)];
                const double bc = (double)g.b[c];
                double r = 0;
                if (!(cd & CODE_GENERAL)) {
                    const int cnt = __popc(cd & 63u) + (cd >> 7);
                    double acc = __dmul_rn((double)cnt, x0);
                    acc -= (cd & 1u) ? xm : 0.0;
                    acc -= (cd & 2u) ? xp : 0.0;
                    acc -= (cd & 4u) ? ym : 0.0;
                    acc -= (cd & 8u) ? yp : 0.0;
                    acc -= (cd & 16u) ? zm : 0.0;
                    acc -= (cd & 32u) ? zp : 0.0;
                    r = cnt > 0 ? bc - acc : 0.0;
                } else {
                    const double dg = (double)g.diag[c];
                    int i, j, k;
                    ijkOf(g, 0, c, i, j, k);
                    const int fx0 = i + (nx + 1) * (j + ny * k), fy0 = i + nx * (j + (ny + 1) * k);
                    double acc = dg * x0;
                    if (i > 0) acc -= (double)g.a0x[fx0] * xm;
                    if (i < nx - 1) acc -= (double)g.a0x[fx0 + 1] * xp;
                    if (j > 0) acc -= (double)g.a0y[fy0] * ym;
                    if (j < ny - 1) acc -= (double)g.a0y[fy0 + nx] * yp;
                    if (k > 0) acc -= (double)g.a0z[c] * zm;
                    if (k < nz - 1) acc -= (double)g.a0z[c + sxy] * zp;
                    if (dg > 0) r = bc - acc;
                }
                B.r[c] = (R)r;
                g.p[c] = 0;
                const int z = g.nClosed > 0 ? g.zone[c] : -1;
                if (!(z >= 0 && !g.zoneOpen[z])) rm = mx(rm, fabs(r));
            });
        };
        auto zoneProject = [&](double& rm) {
            zones(B.r, [&](int c, double mean) {
                const R v = (R)((double)B.r[c] - mean);
                B.r[c] = v;
                rm = fmax(rm, fabs((double)v));
            });
        };

        if (kMixed && !a.vcycleOnly) {
            double rm = 0;
            residual64(rm);
            if (closed) {
                PHX_TEAM_SYNC();
                zoneProject(rm);
            }
            ctaMaxStore(maxR + 1, rm, shMx);
            PHX_TEAM_SYNC();
        }

        const unsigned tag0 = *g.tagBase;
        T none = T(0);
        for (int phase = a.vcycleOnly ? 2 : 0, loop = 0;; phase = 1, ++loop) {
            B.tag = tag0 + 1u + (unsigned)loop;
            bool haveRed = false;   // the update has set the red cells of z
            if (phase == 1) {
                B.beta = (T)cg.beta;
                B.haveD = cg.it > 0;
                if (kMixed) {   // the neighbours' previous d is read: two buffers by turns
                    B.d = cg.it & 1 ? g.tmp[0] : g.d;
                    B.dNew = cg.it & 1 ? g.d : g.tmp[0];
                }
                PHX_PASS(PASS_APPLY, partDq, none, false);
                // tagged partial sums take no barrier: a thread updates the cells it has just formed
                // q and d for, and every read of z was done before the reader's partial sum
                __syncthreads();
                const double total = kMixed ? teamTotalF2<true>(partDq, nt, shDot[0], shSum, B.tag, tw)
                                            : teamTotal<true>(partDq, nt, shSum, B.tag, tw);
                if (tid == 0) {
                    cg.dq = total;
                    if (cg.brk == 1) {   // the iteration after a breakdown: no update, then a restart
                        cg.alpha = 0;
                        cg.brk = 2;
                    } else if (total <= 0) {
                        cg.done = 1;
                    } else {
                        cg.alpha = cg.rz / total;
                    }
                }
                __syncthreads();
                if (cg.done != 0) break;
                B.alpha = (T)cg.alpha;
                const bool repl = kMixed && cg.repl != 0;
                haveRed = !repl && !closed;
                T rm = T(0);
                PHX_PASS(PASS_UPDATE, nullptr, rm, haveRed);
                ctaMaxStore(maxR, rm, reinterpret_cast<T*>(shMx));
                PHX_TEAM_SYNC();
                if (closed) {
                    zoneCenter(B.r);
                    PHX_TEAM_SYNC();
                }
                if (repl) {
                    cells([&](int c) { if (g.diag[c] > 0) g.p64[c] += (double)g.p[c]; });
                    PHX_TEAM_SYNC();
                    double rm64 = 0;
                    residual64(rm64);
                    if (closed) {
                        PHX_TEAM_SYNC();
                        zoneProject(rm64);
                    }
                    ctaMaxStore(maxR + 1, rm64, shMx);
                    PHX_TEAM_SYNC();
                }
            }
            // the V-cycle z = M r
            if (!haveRed) {
                PHX_PASS(PASS_RED0, nullptr, none, true);
                PHX_TEAM_SYNC();
            }
            PHX_PASS(PASS_BLACK0, nullptr, none, true);
            PHX_TEAM_SYNC();
            PHX_PASS(PASS_RES, nullptr, none, true);
            using Down = std::integral_constant<int, SWEEP_DOWN>;
            using Up = std::integral_constant<int, SWEEP_UP>;
            using Last = std::integral_constant<int, SWEEP_LAST>;
            using Only = std::integral_constant<int, SWEEP_ONLY>;
            // the coarse levels: with tagged values no barrier until level 1's correction is whole
            for (int l = 1; l < nl - 1; ++l) {
                if (!g.smooth1) {
                    jacobiLevel(Down{}, l);
                }
                restrictLevel(l);
            }
            coarsest();
            for (int l = nl - 2; l >= 1; --l) {
                if (g.smooth1) {
                    jacobiLevel(Only{}, l);
                } else {
                    jacobiLevel(Up{}, l);
                    jacobiLevel(Last{}, l);
                }
            }
            PHX_TEAM_SYNC();
            PHX_PASS(PASS_BLACK, nullptr, none, true);
            PHX_TEAM_SYNC();
            PHX_PASS(PASS_RED, partRz, none, true);
            if (phase == 2) return;   // of one scenario only
            PHX_TEAM_SYNC();
            // r.z, the maxima, beta and the stop test
            if (warp >= TH / 32 - 2) {   // the maxima of the recursion and of the FP64 residual
                const int which = warp - (TH / 32 - 2);
                const double* mp = a.maxPart + 2 * (b - rank) + which;
                double m = 0;
                for (int i = lane; i < size; i += 32) m = mx(m, __ldcg(mp + 2 * i));
                m = warpMaxPos(m);
                if (lane == 0) shMax[which] = m;
            }
            const double total = kMixed ? teamTotalF2<false>(partRz, nt, shDot[0], shSum + 4, B.tag, tw)
                                        : teamTotal<false>(partRz, nt, shSum, B.tag, tw);
            if (warp == 0) {
                const double rmax = phase == 1 ? shMax[0] : cg.rmax;
                const double r64 = kMixed && (phase == 0 || cg.repl != 0) ? shMax[1] : 0.0;
                if (lane == 0) {
                    closeCgIteration(g, cg, phase, total, phase == 1 ? total / cg.rz : 0.0, rmax, r64);
                    if (loop >= a.cap) cg.done = 1;
                }
            }
            if (closed) {
                zoneCenter(B.z);
                PHX_TEAM_SYNC();
            }
            __syncthreads();
            if (cg.done != 0) break;
        }
        // mixed path: p64 += e and its FP32 copy (written before the team's last barrier)
        if (kMixed)
            cells([&](int c) {
                double v = g.p64[c];
                if (g.diag[c] > 0) v += (double)g.p[c];
                g.p64[c] = v;
                g.p[c] = (R)v;
            });
        if (rank == 0 && tid == 0) {
            double* sv = g.sv;
            sv[SV_IT] = cg.it;
            sv[SV_MEANITERS] = sv[SV_SOLVED] > 0 ? sv[SV_MEANITERS] + SOLVE_MEAN_SHARE * (cg.it - sv[SV_MEANITERS]) : cg.it;
            sv[SV_SOLVED] = 1;
            const double r = kMixed ? cg.r64 : cg.rmax;   // the residual the solve is judged by
            sv[SV_PRES] = r / sv[SV_INV];
            sv[SV_PREL] = sv[SV_BMAX] > 0 ? r / sv[SV_BMAX] : 0.0;
            if (kMixed) sv[SV_HAVEPREV] = 1;
        }
#undef PHX_PASS
#undef PHX_TEAM_SYNC
    }
}

}  // namespace phx
