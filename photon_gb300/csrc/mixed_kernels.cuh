// The mixed path's initial guess, and small per-scenario kernels of both paths.
#pragma once
#include "pressure_kernels.cuh"

namespace phx {

// start of a mixed solve: the initial guess 2 p(n) - p(n-1) when the previous
// step's pressure is known (a linear extrapolation in time), and p(n) kept
// as the next step's p(n-1). The solve stops on the same residual test, so
// only the iteration count depends on the guess.
template <class R>
__global__ void k_mx_extrap(const Scn<R>* __restrict__ S, Dom dom) {
    int s_, tile_;
    locate(dom, blockIdx.x, s_, tile_);
    const Scn<R>& g = S[s_];
    const int c = tile_ * TPB + threadIdx.x;
    if (c >= g.N || !g.p64prev) return;
    const double cur = g.p64[c];
    if (g.extrap && g.sv[SV_HAVEPREV] != 0 && g.diag[c] > 0) g.p64[c] = 2.0 * cur - g.p64prev[c];
    g.p64prev[c] = cur;
}

// simulated time of every scenario into one array (one read-back per batch)
template <class R>
__global__ void k_read_times(const Scn<R>* __restrict__ S, int n, double* out) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < n) out[s] = S[s].sv[SV_TIME];
}

// before a bare V-cycle of the first scenario (k_begin does it for a step's solves); one CTA
template <class R>
__global__ void __launch_bounds__(TEAM_TPB) k_reset(const Scn<R>* __restrict__ S, TeamTable teams) {
    if (threadIdx.x == 0) {
        startSolve(S[0]);
        offerWork(S[0], 0, teams);
    }
    __syncthreads();
    divideTeams(1, teams);
}

}  // namespace phx
