// The level-0 pressure operator: the 7-point structured grid of the multigrid
// V-cycle and of q = A d, with the matrix coefficients coded in one byte per
// cell. Both precisions use it (R = double: the FP64 path; R = float: the
// mixed path); solve.cuh has the passes.
//
// Coefficient codes. On the grids Photon discretizes, the level-0 matrix
// coefficients (a0x, a0y, a0z: open fractions of a cell's six faces) are 0 or
// 1 nearly everywhere, and the diagonal is their sum. A cell's code holds, in
// bits 0-5, which of its interior faces (x-, x+, y-, y+, z-, z+) couple it to
// its neighbour with a coefficient of exactly 1, and in bit 7 one open
// domain-boundary face (it adds 1 to the diagonal and has no neighbour). Its
// diagonal is then the number of those bits. A cell with any other
// coefficient, more than one open boundary face, or a diagonal that is not
// that count gets bit 6 ("general") and its coefficients are read from the
// arrays as before. The host builds and checks every code. Multiplying by a
// coefficient of 1 is exact and adding a zero term changes nothing, so a
// coded cell computes what the array form computes, in the same order. A pass
// then streams 1 byte per cell of matrix data instead of four coefficient
// arrays.
#pragma once
#include <type_traits>

#include "fdiv.cuh"
#include "step_kernels.cuh"

namespace phx {

// bits 0-5: interior faces x-, x+, y-, y+, z-, z+ with coefficient 1; bit 7:
// one open boundary face; bit 6: read the arrays
constexpr unsigned char CODE_GENERAL = 64;
constexpr unsigned char CODE_BOUNDARY = 128;

// diagonal of a coded cell
template <class T>
__device__ __forceinline__ T codeDiag(unsigned cd) { return (T)(__popc(cd & 63u) + (cd >> 7)); }

// a smoothing sweep's division by the diagonal: on the FP64 path the reference's
// quotient, for a coded cell by the integer diagonal in three FP64 operations
// (fdiv.cuh); on the FP32 path the fast reciprocal-based division (a
// preconditioner; diagonals are far from the range where it loses accuracy)
__device__ __forceinline__ double gsDiv(double a, double b) { return a / b; }
__device__ __forceinline__ float gsDiv(float a, float b) { return __fdividef(a, b); }
template <class T>
__device__ __forceinline__ T l0Div(T a, unsigned cd, T dg) {
    if constexpr (sizeof(T) == 8) {
        if (!(cd & CODE_GENERAL)) return divSmall(a, (int)(__popc(cd & 63u) + (cd >> 7)));
    }
    return gsDiv(a, dg);
}

// neighbour values of one cell in the reference's term order
template <class R>
struct L0Nb {
    R xm, xp, ym, yp, zm, zp;
};

// the general-cell form of the stencil: the interior neighbours times the arrays'
// coefficients. Out of line: few cells take it, and its code would stand in the
// instruction stream of every pass.
template <int SIGN, class R>
__device__ __noinline__ R l0SumGeneral(const Scn<R>& g, R sacc, L0Nb<R> n, int c) {
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    int i, j, k;
    ijkOf(g, 0, c, i, j, k);
    const long long fx = i + (long long)(nx + 1) * (j + (long long)ny * k);
    const long long fy = i + (long long)nx * (j + (long long)(ny + 1) * k);
    const R xm = g.a0x[fx], xp = g.a0x[fx + 1], ym = g.a0y[fy], yp = g.a0y[fy + nx], zm = g.a0z[c],
            zp = g.a0z[c + (long long)nx * ny];
    if (SIGN > 0) {
        if (i > 0) sacc += xm * n.xm;
        if (i < nx - 1) sacc += xp * n.xp;
        if (j > 0) sacc += ym * n.ym;
        if (j < ny - 1) sacc += yp * n.yp;
        if (k > 0) sacc += zm * n.zm;
        if (k < nz - 1) sacc += zp * n.zp;
    } else {
        if (i > 0) sacc -= xm * n.xm;
        if (i < nx - 1) sacc -= xp * n.xp;
        if (j > 0) sacc -= ym * n.ym;
        if (j < ny - 1) sacc -= yp * n.yp;
        if (k > 0) sacc -= zm * n.zm;
        if (k < nz - 1) sacc -= zp * n.zp;
    }
    return sacc;
}

// sacc plus (SIGN > 0) or minus the neighbour terms of cell c in the order
// x-, x+, y-, y+, z-, z+: for a coded cell every set bit adds its neighbour
// (coefficient 1)
template <int SIGN, class R>
__device__ __forceinline__ R l0Sum(const Scn<R>& g, R sacc, unsigned cd, const L0Nb<R>& n, int c) {
    if (cd & CODE_GENERAL) return l0SumGeneral<SIGN>(g, sacc, n, c);
    if (cd & 1u) sacc = SIGN > 0 ? sacc + n.xm : sacc - n.xm;
    if (cd & 2u) sacc = SIGN > 0 ? sacc + n.xp : sacc - n.xp;
    if (cd & 4u) sacc = SIGN > 0 ? sacc + n.ym : sacc - n.ym;
    if (cd & 8u) sacc = SIGN > 0 ? sacc + n.yp : sacc - n.yp;
    if (cd & 16u) sacc = SIGN > 0 ? sacc + n.zm : sacc - n.zm;
    if (cd & 32u) sacc = SIGN > 0 ? sacc + n.zp : sacc - n.zp;
    return sacc;
}

}  // namespace phx
