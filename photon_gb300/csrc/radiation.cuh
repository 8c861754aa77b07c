// Radiation trace of Photon's room-scale radiation model
// (Solver::traceRadiation, src/sim/radiation.cpp:181-319) over the gas fields
// resident on the device.
//
// Four wavelength bands, 32 golden-spiral directions, an Amanatides-Woo march
// from every radiating surface element through the cells until the ray leaves
// the domain, meets a wall or a blocked cell, runs 8 m, or becomes opaque in
// every band. Everything is relative to ambient, as in the reference.
//
// What bounds it: FP64 arithmetic in the FP64 context (a warp's FP64 instruction
// occupies its SM for some 19 cycles whatever its active lanes), gathers and
// instruction issue in the FP32 one. So:
// * what depends on an element alone (band emission, hemisphere normalisation)
//   is computed with a lane per element, what depends on the ray (its weight and
//   first crossings) with a lane per direction (the reference's 32 directions
//   are one warp), the Planck series in FMA form without divisions;
// * rays are listed by direction: neighbouring lanes march neighbouring
//   elements' rays the same way, through like numbers of cells and past like
//   absorption; a persistent march kernel hands rays to lanes as they free up;
//   each element's absorbed power is its rays' results summed in direction
//   order, as the reference sums them;
// * per-cell absorption coefficient and source function of the four bands are
//   computed once per trace into one interleaved record per cell (32 B FP32,
//   64 B FP64); a cell's walls are bits beside its blocked and flame flags, so a
//   ray step gathers one record and one byte, both a step ahead of their use;
// * the band powers a ray ends on (an intact wall seen from either side, a
//   blocked cell's solid temperature) are tabulated before the march, so a
//   ray's end costs a table read instead of the Planck series;
// * numbers that cannot be negative are compared by their bits;
// * gas cells gain their rays' contributions by atomic adds in the trace's
//   precision.
#pragma once
#include "phx_dev.cuh"

namespace phx {

constexpr int RAD_NB = 4, RAD_DIRS = 32;
constexpr int RAD_ELEMS = 128;      // elements per CTA of k_rad_elems, a thread each
// elements traced at a time: an element's rays and results take 0.8 KB (FP32) or 1.5 KB of
// scratch, 420 or 770 MB for this many, however many elements a trace has
constexpr int RAD_PORTION = 1 << 19;
constexpr int RAD_EXP_N = 512;      // table of radDecay
// cells a ray advances before lanes without one take another: an FP64 step costs its warp
// the same with few lanes as with 32, an FP32 one little against the hand-out (72x52x44
// house in FP64 at 4 / 8 / 16 cells 2.16 / 2.23 / 2.85 ms, 1.3e6 cells in FP32 1.41 / 1.24 / 1.23)
template <class R>
constexpr int RAD_STEPS = sizeof(R) == 8 ? 4 : 8;

// the reference's PI is the literal 3.14159265 (src/sim/radiation.cpp:44)
template <class R> struct RadPi;
template <> struct RadPi<double> { static constexpr double v = 3.14159265; };
template <> struct RadPi<float> { static constexpr float v = 3.14159265f; };

template <class R>
struct RadConst {
    R dir[RAD_DIRS][3];
    R tD[RAD_DIRS][3];  // cells' crossing times: 1 / |component|, 1e30 along a face
    R f0[RAD_NB];       // band fractions of ambient
    R fFlame[RAD_NB];   // band fractions of the sub-grid flame (T_FLAME_RAD 1400 K)
    R dW;               // solid angle per direction
    R exp2T[sizeof(R) == 8 ? RAD_EXP_N : 1];   // 2^(-j / 512)
};

template <class R>
struct __align__(sizeof(R) * 8) RadCell {
    R kap[RAD_NB];   // 1/m; blocked cells: unused
    R src[RAD_NB];   // W/m2/sr; blocked cells: the band intensity a ray ending there sees
};

// what the march reads of an element
template <class R>
struct __align__(16) RadSource {
    R Is[RAD_NB];    // its own emission per band
    R eps;
    int cell;        // of its origin
    int skip;        // that cell, or -1: the cell a ray does not absorb in
};
// a ray's first crossings and its weight
template <class R>
struct __align__(16) RadRay {
    R tMx, tMy, tMz, w;
};

// order of numbers of which none is negative (FP64: an FP64 comparison would take the FP64 pipe)
__device__ __forceinline__ bool radLess(float a, float b) { return a < b; }
__device__ __forceinline__ bool radLess(double a, double b) { return __double_as_longlong(a) < __double_as_longlong(b); }

// exp(-x), x >= 1e-3. FP64: x = (512 k + j) ln2 / 512 + r, 2^-k 2^(-j/512) (1 + expm1(-r))
// by table and a polynomial of degree 4 (P.-T. P. Tang, "Table-driven implementation of
// the exponential function in IEEE floating-point arithmetic", ACM TOMS 15(2), 1989): 9
// FP64 operations against exp's 17. |r| <= ln2 / 1024: truncation r^5 / 120 < 2e-18;
// within 2e-16 of the result.
__device__ __forceinline__ double radDecay(double x, const double* exp2T) {
    if (!radLess(x, 40.0)) return x != x ? x : 0.0;   // below half an ulp of what it is subtracted from
    const double MAGIC = 0x1.8p52;
    const double m = fma(x, 0x1.71547652b82fep+9, MAGIC);
    const int n = __double2loint(m);
    const double k = m - MAGIC;
    const double r = fma(k, -0x1.abc9e3b39803fp-65, fma(k, -0x1.62e42fefa39efp-10, x));
    const double q = r * fma(r, fma(r, fma(r, 1.0 / 24, -1.0 / 6), 0.5), -1.0);   // expm1(-r)
    const double t = exp2T[n & (RAD_EXP_N - 1)];
    const double s = __hiloint2double(__double2hiint(t) - ((n >> 9) << 20), __double2loint(t));
    return fma(s, q, s);
}
__device__ __forceinline__ float radDecay(float x, const float*) { return expf(-x); }

__device__ __forceinline__ double radExp(double x) { return exp(x); }
__device__ __forceinline__ float radExp(float x) { return expf(x); }
__device__ __forceinline__ double radSqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float radSqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ double radFloor(double x) { return floor(x); }
__device__ __forceinline__ float radFloor(float x) { return floorf(x); }

// fraction of blackbody emission below lambda*T (um K): Chang & Rhee series
// (src/sim/radiation.cpp:54-63)
template <class R>
__device__ R radPlanckBelow(R lambdaT) {
    if (lambdaT <= 0) return 0;
    if (lambdaT > (R)1e8) return 1;
    const R PI = RadPi<R>::v;
    // term n: e^(-nx) (x^3 / n + 3 x^2 / n^2 + 6 x / n^3 + 6 / n^4)
    const R x = (R)14388.0 / lambdaT, e1 = radExp(-x);
    R s = 0, en = 1;
#pragma unroll
    for (int n = 1; n <= 12; ++n) {
        const double r = 1.0 / n;
        en *= e1;
        s = fma(en, fma(x, fma(x, fma(x, (R)r, (R)(3 * r * r)), (R)(6 * r * r * r)), (R)(6 * r * r * r * r)), s);
    }
    R v = (R)1.0 - (R)15.0 / (PI * PI * PI * PI) * s;
    return v < 0 ? (R)0 : v > 1 ? (R)1 : v;
}

template <class R>
__device__ __forceinline__ R radEdge(int b) {   // band edges, um (:46)
    return b == 1 ? (R)2.7 : b == 2 ? (R)8.0 : (R)14.0;
}

// band fractions (:64-71)
template <class R>
__device__ void radBandFractions(R T, R f[RAD_NB]) {
    R prev = 0;
#pragma unroll
    for (int b = 0; b < RAD_NB; ++b) {
        R up = b == RAD_NB - 1 ? (R)1 : radPlanckBelow<R>(radEdge<R>(b + 1) * T);
        f[b] = up - prev;
        prev = up;
    }
}

// band emissive power relative to ambient, W/m2 (:73-81), from the band fractions f
template <class R>
__device__ __forceinline__ R radPower(const RadConst<R>& k, const R f[RAD_NB], R T, int b) {
    const R a = T * T, a0 = (R)K_T0 * (R)K_T0;
    return (R)5.670374e-8 * (f[b] * a * a - k.f0[b] * a0 * a0);
}

// directions, band tables (:84-96, 185-192) and radDecay's; RAD_EXP_N threads
template <class R>
__global__ void k_rad_setup(RadConst<R>* k) {
    const int i = threadIdx.x;
    const R PI = RadPi<R>::v;
    if (i < RAD_DIRS) {
        const R ga = PI * ((R)3.0 - radSqrt((R)5.0));
        R z = (R)1.0 - (R)2.0 * (i + (R)0.5) / RAD_DIRS;
        R r = radSqrt(mx((R)0, 1 - z * z));
        R ang = ga * i;
        k->dir[i][0] = r * (R)cos((double)ang);
        k->dir[i][1] = r * (R)sin((double)ang);
        k->dir[i][2] = z;
        for (int a = 0; a < 3; ++a) {
            const R v = k->dir[i][a];
            k->tD[i][a] = v > (R)1e-9 ? 1 / v : v < (R)-1e-9 ? -1 / v : (R)1e30;
        }
    }
    if (sizeof(R) == 8) k->exp2T[i] = (R)exp2(-i / (double)RAD_EXP_N);
    if (i == 0) {
        radBandFractions<R>((R)K_T0, k->f0);
        radBandFractions<R>((R)1400.0, k->fFlame);
        k->dW = (R)4.0 * PI / RAD_DIRS;
    }
}

// end-of-ray band intensities of every wall, seen from below (0-3) and above (4-7), and
// the wall's bit in the flags of the cells on its two sides (after k_rad_cells)
template <class R>
__global__ void k_rad_walls(const phx_rad_wall* __restrict__ wl, int nW, int nx, int ny, int nz, int* __restrict__ wallOf,
                            unsigned* __restrict__ flags, R* __restrict__ wallI, const RadConst<R>* __restrict__ kc) {
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= nW) return;
    const phx_rad_wall x = wl[w];
    const int mx_ = nx + (x.axis == 0), my = ny + (x.axis == 1);
    const int i = x.face % mx_, j = (x.face / mx_) % my, k = x.face / (mx_ * my);
    const int at = x.axis == 0 ? i : x.axis == 1 ? j : k, n = x.axis == 0 ? nx : x.axis == 1 ? ny : nz;
    const int above = i + nx * (j + ny * k), below = above - (x.axis == 0 ? 1 : x.axis == 1 ? nx : nx * ny);
    wallOf[(x.axis == 0 ? 0 : x.axis == 1 ? (nx + 1) * ny * nz : (nx + 1) * ny * nz + nx * (ny + 1) * nz) + x.face] = w;
    if (at < n) atomicOr(flags + (above >> 2), 4u << (2 * x.axis + 8 * (above & 3)));
    if (at > 0) atomicOr(flags + (below >> 2), 8u << (2 * x.axis + 8 * (below & 3)));
    const R PI = RadPi<R>::v;
    R f[RAD_NB];
#pragma unroll
    for (int side = 0; side < 2; ++side) {
        const R T = (R)(side == 0 ? x.t_lower : x.t_upper);
        radBandFractions<R>(T, f);
#pragma unroll
        for (int q = 0; q < RAD_NB; ++q) wallI[8 * w + 4 * side + q] = radPower<R>(*kc, f, T, q) * ((R)0.9 / PI);
    }
}

// per-cell absorption and source of the four bands (:193-222); flags bit 0
// blocked, bit 1 flame cell, bits 2-7 (k_rad_walls) a wall on its x-, x+, ... z+ face
template <class R>
__global__ void k_rad_cells(const Scn<R>* __restrict__ S, int s, const double* __restrict__ solidT,
                            RadCell<R>* __restrict__ cells, uint8_t* __restrict__ flags,
                            const RadConst<R>* __restrict__ kc) {
    const Scn<R>& g = S[s];
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= g.N) return;
    const R PI = RadPi<R>::v;
    R f[RAD_NB];
    RadCell<R> o;
    if (g.blocked[c]) {
        const R T = solidT ? (R)solidT[c] : (R)K_T0;
        radBandFractions<R>(T, f);
#pragma unroll
        for (int q = 0; q < RAD_NB; ++q) { o.kap[q] = 0; o.src[q] = radPower<R>(*kc, f, T, q) * ((R)0.9 / PI); }
        cells[c] = o;
        flags[c] = 1;
        return;
    }
    const R T = tAbs(g.sc[0][c]), Ys = g.sc[3][c], Yc = g.sc[6][c], Yw = g.sc[7][c], Pb = g.Pb[c], hrr = g.hrr[c];
    const R rho = Pb / ((R)K_RS * T);
    const R fv = rho * Ys / (R)1800.0;
    const R pg = (Yw * (R)28.96 / (R)18.02 + Yc * (R)28.96 / (R)44.01) * Pb / (R)K_P0;
    radBandFractions<R>(T, f);
    const R jfTot = hrr > 0 ? (R)K_CHI_R * hrr / ((R)4.0 * PI) : (R)0;
    const R lam[RAD_NB] = {(R)1.5, (R)4.5, (R)11.0, (R)25.0};
    const R kg[RAD_NB] = {(R)0.05, (R)3.0, (R)0.1, (R)6.0};
    R k[RAD_NB], Eb[RAD_NB], jTot = 0;
#pragma unroll
    for (int q = 0; q < RAD_NB; ++q) {
        Eb[q] = radPower<R>(*kc, f, T, q);
        k[q] = (R)5.5 * fv / (lam[q] * (R)1e-6) + kg[q] * pg + (R)1e-4;
        jTot += k[q] * Eb[q] / PI;
    }
    const bool fl = jfTot > jTot;
#pragma unroll
    for (int q = 0; q < RAD_NB; ++q) {
        const R j = fl ? jfTot * kc->fFlame[q] : k[q] * Eb[q] / PI;
        o.kap[q] = k[q];
        o.src[q] = j / k[q];
    }
    cells[c] = o;
    flags[c] = fl ? 2 : 0;
}

// Rays (:225-248). A thread per element first: its own emission in each band, its origin's
// cell and the hemisphere normalisation, summed in direction order. Then a warp takes its
// 32 elements one by one, lane = direction: which directions an element emits into (weight
// w > 0, origin inside the grid), and after the CTA has taken room in each direction's
// part of the ray list (nE places each, counts[d] of them used), weights and first
// crossings. A direction that is not emitted into gets its result here: 0.
template <class R>
__global__ void __launch_bounds__(RAD_ELEMS)
k_rad_elems(const Scn<R>* __restrict__ S, int s, const double* __restrict__ els, int elWords, int nE,
            const RadConst<R>* __restrict__ kc, RadSource<R>* __restrict__ sources, RadRay<R>* __restrict__ rays,
            int* __restrict__ rayElem, R* __restrict__ rayVal, int* __restrict__ counts) {
    constexpr int WARPS = RAD_ELEMS / 32;
    __shared__ R dir[RAD_DIRS][3];
    __shared__ R shN[RAD_ELEMS][3], shP[RAD_ELEMS][3], shW[RAD_ELEMS], shA[RAD_ELEMS];
    __shared__ int kind[RAD_ELEMS];              // 0 no rays, 1 hemisphere, 2 sphere
    __shared__ int room[WARPS][RAD_DIRS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int e0 = blockIdx.x * RAD_ELEMS;
    const Scn<R>& g = S[s];
    const R PI = RadPi<R>::v;
    const R dW = kc->dW;
    for (int q = tid; q < RAD_DIRS * 3; q += RAD_ELEMS) dir[q / 3][q % 3] = kc->dir[q / 3][q % 3];
    __syncthreads();
    kind[tid] = 0;
    if (e0 + tid < nE) {
        // a phx_rad_elem, or its 11 numbers as doubles
        static_assert(sizeof(phx_rad_elem) == 80, "nine doubles and two ints");
        const double* el = els + (size_t)(e0 + tid) * elWords;
        const R eps = (R)el[7], temp = (R)el[8], area = (R)el[6];
        const bool sphere = elWords == 11 ? (int)el[9] != 0 : reinterpret_cast<const int*>(el + 9)[0] != 0;
        const bool skipOwn = elWords == 11 ? (int)el[10] != 0 : reinterpret_cast<const int*>(el + 9)[1] != 0;
        const R n0 = (R)el[3], n1 = (R)el[4], n2 = (R)el[5];
        RadSource<R> o;
        R f[RAD_NB];
        radBandFractions<R>(temp, f);
#pragma unroll
        for (int q = 0; q < RAD_NB; ++q) {   // own emission, relative to ambient
            o.Is[q] = radPower<R>(*kc, f, temp, q);
            o.Is[q] *= eps / PI;
        }
        // hemisphere weights normalised so that sum(cos dW) = pi, in direction order
        R wsum = 0;
        if (!sphere) {
#pragma unroll 4
            for (int d = 0; d < RAD_DIRS; ++d) {
                const R cs = dir[d][0] * n0 + dir[d][1] * n1 + dir[d][2] * n2;
                if (cs > 0) wsum += cs * dW;
            }
        }
        const R norm = sphere ? (R)1 : (wsum > 0 ? PI / wsum : (R)0);
        const R px = ((R)el[0] - (R)g.ox) / (R)g.dx, py = ((R)el[1] - (R)g.oy) / (R)g.dx,
                pz = ((R)el[2] - (R)g.oz) / (R)g.dx;
        const int ci = (int)radFloor(px), cj = (int)radFloor(py), ck = (int)radFloor(pz);
        const bool inside = !(ci < 0 || cj < 0 || ck < 0 || ci >= g.nx || cj >= g.ny || ck >= g.nz);
        o.eps = eps;
        o.cell = inside ? ci + g.nx * (cj + g.ny * ck) : 0;
        o.skip = skipOwn ? o.cell : -1;
        sources[e0 + tid] = o;
        kind[tid] = !inside ? 0 : sphere ? 2 : 1;
        shN[tid][0] = n0; shN[tid][1] = n1; shN[tid][2] = n2;
        shP[tid][0] = px; shP[tid][1] = py; shP[tid][2] = pz;
        shW[tid] = sphere ? dW * (R)0.25 * area : norm;
        shA[tid] = area;
    }
    __syncthreads();
    const R v0 = dir[lane][0], v1 = dir[lane][1], v2 = dir[lane][2];
    auto cosine = [&](int q) { return v0 * shN[q][0] + v1 * shN[q][1] + v2 * shN[q][2]; };
    unsigned on = 0;   // this direction's elements of the warp's 32
#pragma unroll 1
    for (int m = 0; m < 32; ++m) {
        const int q = warp * 32 + m, e = e0 + q;
        if (e >= nE) break;
        const bool emits = kind[q] == 2 || (kind[q] == 1 && cosine(q) > 0);
        on |= emits ? 1u << m : 0u;
        if (!emits) rayVal[(size_t)e * RAD_DIRS + lane] = 0;
    }
    room[warp][lane] = __popc(on);
    __syncthreads();
    if (warp == 0) {
        int n = 0;
        for (int w = 0; w < WARPS; ++w) { const int c = room[w][lane]; room[w][lane] = n; n += c; }
        const int base = n ? atomicAdd(counts + lane, n) : 0;
        for (int w = 0; w < WARPS; ++w) room[w][lane] += base;
    }
    __syncthreads();
    size_t at = (size_t)lane * nE + room[warp][lane];
#pragma unroll 1
    for (int m = 0; m < 32; ++m) {
        if (!((on >> m) & 1u)) continue;
        const int q = warp * 32 + m;
        const R px = shP[q][0], py = shP[q][1], pz = shP[q][2];
        const R fx = radFloor(px), fy = radFloor(py), fz = radFloor(pz);
        auto crossing = [](R p, R f, R v) -> R {
            return v > (R)1e-9 ? (f + 1 - p) / v : v < (R)-1e-9 ? (p - f) / -v : (R)1e30;
        };
        RadRay<R> r;
        r.tMx = crossing(px, fx, v0);
        r.tMy = crossing(py, fy, v1);
        r.tMz = crossing(pz, fz, v2);
        r.w = kind[q] == 2 ? shW[q] : cosine(q) * dW * shW[q] * shA[q];
        rays[at] = r;
        rayElem[at] = e0 + q;
        ++at;
    }
}

// A trace of a 72x52x44 house (31,000 elements) takes 2.2 ms in FP64, 7.7 with rays listed by
// element, exp and comparisons in FP64 and the series with divisions; of 1.3e6 cells (210,000
// elements) in FP32 1.24 ms, before 2.07.
// The march (:249-306), persistent: every lane takes the next ray of the list when its
// own has ended (a warp-aggregated atomic hands out rays). A ray's result eps w It lands
// in its element's slot of its direction; gas cells gain by atomic adds. counts:
// rays per direction, then the next ray to hand out.
template <class R>
__global__ void __launch_bounds__(256, sizeof(R) == 8 ? 2 : 4)
k_rad_march(const Scn<R>* __restrict__ S, int s, int nE, const RadSource<R>* __restrict__ sources,
            const RadCell<R>* __restrict__ cells, const uint8_t* __restrict__ flags, const int* __restrict__ wallOf,
            const R* __restrict__ wallI, const RadConst<R>* __restrict__ kc, const RadRay<R>* __restrict__ rays,
            const int* __restrict__ rayElem, R* __restrict__ rayVal, int* __restrict__ counts, R* __restrict__ radGas) {
    __shared__ int first[RAD_DIRS + 1];
    __shared__ R exp2T[sizeof(R) == 8 ? RAD_EXP_N : 1];
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 32) {
        const int n = counts[lane];
        int v = n;
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        first[lane] = v - n;
        if (lane == 31) first[32] = v;
    }
    if (sizeof(R) == 8)
        for (int q = threadIdx.x; q < RAD_EXP_N; q += blockDim.x) exp2T[q] = kc->exp2T[q];
    __syncthreads();
    const Scn<R>& g = S[s];
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const int NX = g.NX, NY = g.NY;
    const R dx = (R)g.dx;
    const int nRays = first[RAD_DIRS];
    const R tEnd = (R)8.0 / dx;
    int slot = -1;        // ray in flight (32 e + d); -1 none, -2 the list is exhausted
    int ci = 0, cj = 0, ck = 0, c = 0, skip = -1, ups = 0;
    R tMx = 0, tMy = 0, tMz = 0, tDx = 0, tDy = 0, tDz = 0, t = 0, w = 0, eps = 0;
    R tau[RAD_NB], Is[RAD_NB], I = 0;
    RadCell<R> cell;
    unsigned fl = 0;
    for (;;) {
        const bool need = slot == -1;
        const unsigned mNeed = __ballot_sync(0xffffffffu, need);
        if (mNeed) {
            const int leader = __ffs(mNeed) - 1;
            int base = 0;
            if (lane == leader) base = atomicAdd(counts + RAD_DIRS, __popc(mNeed));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (need) {
                const int k = base + __popc(mNeed & ((1u << lane) - 1u));
                if (k >= nRays) slot = -2;
                else {
                    int d = 0;   // the last direction whose rays start at or before k
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) d += first[d + o] <= k ? o : 0;
                    const size_t at = (size_t)d * nE + (k - first[d]);
                    const int e = rayElem[at];
                    const RadRay<R> r = rays[at];
                    const RadSource<R> src = sources[e];
                    slot = e * RAD_DIRS + d;
                    tMx = r.tMx; tMy = r.tMy; tMz = r.tMz; w = r.w;
                    eps = src.eps;
                    c = src.cell;
                    skip = src.skip;
                    fl = flags[c];
                    cell = cells[c];
#pragma unroll
                    for (int q = 0; q < RAD_NB; ++q) { Is[q] = src.Is[q]; tau[q] = 1; }
                    I = 0;
                    tDx = kc->tD[d][0]; tDy = kc->tD[d][1]; tDz = kc->tD[d][2];
                    ups = (kc->dir[d][0] > 0 ? 1 : 0) | (kc->dir[d][1] > 0 ? 2 : 0) | (kc->dir[d][2] > 0 ? 4 : 0);
                    t = 0;
                    ijkOf(g, 0, c, ci, cj, ck);
                }
            }
        }
        if (__ballot_sync(0xffffffffu, slot >= 0) == 0) break;   // every lane exhausted
        if (slot < 0) continue;
        // advance this lane's ray by up to RAD_STEPS cells
        bool ended = false;
        R Iend[RAD_NB] = {0, 0, 0, 0};
#pragma unroll 1
        for (int it = 0; it < RAD_STEPS<R>; ++it) {
            const int a = radLess(tMx, tMy) ? (radLess(tMx, tMz) ? 0 : 2) : (radLess(tMy, tMz) ? 1 : 2);
            const R tMa = a == 0 ? tMx : a == 1 ? tMy : tMz;
            const bool last = !radLess(tMa, tEnd);
            const R tn = last ? tEnd : tMa;
            const R ds = (tn - t) * dx;
            // the cell beyond the face crossed next, loaded before this one is evaluated
            const int upf = (ups >> a) & 1;
            const bool wall = (fl >> (2 + 2 * a + upf)) & 1u;
            const int at = a == 0 ? ci : a == 1 ? cj : ck;
            const bool out = upf ? at + 1 >= (a == 0 ? nx : a == 1 ? ny : nz) : at == 0;
            const int stride = a == 0 ? 1 : a == 1 ? nx : nx * ny;
            const int nb = upf ? c + stride : c - stride;
            unsigned nfl = 0;
            RadCell<R> next = cell;
            if (!last && !wall && !out) {
                nfl = flags[nb];
                next = cells[nb];
            }
            if (ds > 0 && !(fl & 1) && c != skip) {
                // per band the part u of the ray that the cell takes away, and so gives
                R taken = 0, given = 0;
#pragma unroll
                for (int q = 0; q < RAD_NB; ++q) {
                    const R x = cell.kap[q] * ds;
                    R u, left;
                    if (radLess(x, (R)1e-3)) {
                        u = tau[q] * (x * fma((R)-0.5, x, (R)1));
                        left = tau[q] - u;
                    } else {
                        left = tau[q] * radDecay(x, exp2T);
                        u = tau[q] - left;
                    }
                    tau[q] = left;
                    taken = fma(u, Is[q], taken);
                    given = fma(u, cell.src[q], given);
                }
                I += given;
                atomicAdd(radGas + c, w * ((fl & 2) ? taken : fma(-eps, given, taken)));   // a flame cell's own radiation is accounted elsewhere
            }
            t = tn;
            if (last || (radLess(tau[0], (R)1e-3) && radLess(tau[1], (R)1e-3) && radLess(tau[2], (R)1e-3) &&
                         radLess(tau[3], (R)1e-3))) {
                ended = true;
                break;
            }
            if (wall) {   // an intact wall ends the ray with its surface seen from c
                const int f = a == 0 ? (ci + upf) + (nx + 1) * (cj + ny * ck)
                            : a == 1 ? NX + ci + nx * ((cj + upf) + (ny + 1) * ck)
                                     : NX + NY + ci + nx * (cj + ny * (ck + upf));
                const int wi = wallOf[f];
#pragma unroll
                for (int q = 0; q < RAD_NB; ++q) Iend[q] = wallI[8 * wi + (upf ? 0 : 4) + q];
                ended = true;
                break;
            }
            if (out) { ended = true; break; }
            if (nfl & 1) {
#pragma unroll
                for (int q = 0; q < RAD_NB; ++q) Iend[q] = next.src[q];
                ended = true;
                break;
            }
            c = nb;
            fl = nfl;
            cell = next;
            const int step = upf ? 1 : -1;
            if (a == 0) { tMx += tDx; ci += step; }
            else if (a == 1) { tMy += tDy; cj += step; }
            else { tMz += tDz; ck += step; }
        }
        if (ended) {
            R It = I;
#pragma unroll
            for (int q = 0; q < RAD_NB; ++q) It = fma(tau[q], Iend[q], It);
            rayVal[slot] = eps * w * It;
            slot = -1;
        }
    }
}

// absorbed power of each element: its directions' results summed in direction
// order (:305, directions it does not emit into hold 0)
template <class R>
__global__ void k_rad_absorbed(const R* __restrict__ rayVal, int nE, double* __restrict__ radAbs) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nE) return;
    const R* v = rayVal + (size_t)e * RAD_DIRS;
    R acc = 0;
#pragma unroll
    for (int d = 0; d < RAD_DIRS; ++d) acc += v[d];
    radAbs[e] = (double)acc;
}

}  // namespace phx
