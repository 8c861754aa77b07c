// Which CTAs of the pressure solve work on which scenario (solve.cuh), decided at a
// step's begin by the last CTA of the kernel that begins it: in the solve kernel itself,
// which is short of registers, the same code costs 1 to 2 % of an FP32 step (1.3 M cells
// 3.68 ms here, 3.74 there; 24 houses 5.64 / 5.84).
#pragma once
#include "phx_dev.cuh"

namespace phx {

// How a scenario's pairs are walked: a warp takes 8 consecutive 2x2x2 blocks (four
// lanes a block) at a time; `warps` warps side by side are a tile, which walks
// `reps` such groups. A tile's dot product is one partial sum. The shape follows
// from the scenario's size alone, so its sums do not depend on the team.
// FP32: a tile is always the 32 blocks of four warps, whose products are added in
// the order of one thread per block (the block's cells in ascending order, then
// a warp's shuffle tree), four tiles to a sum that reaches FP64.
struct SolveTiling {
    int warps, reps, nt;
};
template <class R>
__host__ __device__ inline SolveTiling solveTiling(int nblk) {
    const int groups = (nblk + 7) / 8;
    SolveTiling t;
    t.reps = 1;
    if (sizeof(R) == 4) {
        t.warps = 4;
    } else {
        t.warps = groups <= 512 ? 1 : groups <= 4096 ? 4 : 8;
        while (groups / (t.warps * t.reps) >= 4096) t.reps *= 2;
    }
    const int per = t.warps * t.reps;
    t.nt = (groups + per - 1) / per;
    return t;
}
// The CTAs a scenario is given at most: two tiles a CTA cost it nothing where they are a warp
// each (FP64) or a third of the GPU and more has one (FP32, 36x24x24 room of 81 tiles: 41 / 81 /
// 152 CTAs 0.476 / 0.482 / 0.494 ms a step; 52x40x32 of 260: 130 / 152 0.526 / 0.537; but 36
// tiles: 18 / 36 0.403 / 0.383). The rest of the SMs is free for other contexts' solves: four
// closets on four threads 0.10 ms a step, when every solve bound the whole GPU 0.23; four
// FP32 rooms 0.15 and 0.30.
template <class R>
__host__ __device__ inline int solveCtas(const SolveTiling& t) {
    const int half = (t.nt + 1) / 2;
    if (sizeof(R) == 4) return t.nt < 48 ? t.nt : half < 48 ? 48 : half;
    return t.warps == 1 ? half : t.nt;
}

// The grid's CTAs among the scenarios. A scenario has a team of CTAs, in proportion to its
// work (blocks times the iterations its solves take), at least one. With many scenarios
// beside a large one that would leave the large one a few CTAs, and with more scenarios
// than CTAs nothing: then scenarios of less work than a CTA's share take turns on a CTA,
// the largest first. ms per step, a CTA each at least / shared: a 165 k-cell house with 280
// closets of 1.3 k cells in FP64 89 / 4.8, a 1.3 M-cell house with 290 of them in FP32 43 / 5.2.
struct SolveCta {
    int scenario, size, rank;    // the first it works on (-1: none), the CTAs of that one's team, its place there
};
struct TeamTable {
    SolveCta* ctas;              // of the solve's grid
    int* next;                   // per scenario: the one its CTA takes after it, -1 none
    float2* work;                // per scenario: its work, the most CTAs it can use (bits)
    unsigned* arrived;           // CTAs of k_begin that have written theirs; 0 between launches
    int grid;
};

// A scenario that has not solved yet, new or restored, counts as this many iterations: a large one that
// joins a running batch would else get a CTA or two for its longest solve (serving 32 requests of
// 20 k to 1.3 M cells, mixed: 343 M cell-updates/s and 28 ms at the 99th percentile of a
// step, 292 M and 90 ms with the count of 0).
constexpr float SOLVE_FIRST_ITERS = 40.0f;
// After it a running mean of its iterations counts, each solve with this share, and two more.
// Under the reference's absolute stop counts go up and down (0, 5, 5, 4, 3, 0, ... where the warm
// start is good enough now and then), and the last one alone gives the solve after a 0 a
// CTA or two: 64 houses of 20 k to 400 k cells 10.6 ms a step with it, 9.1 with the mean
// (10.0 when every pass was a launch over all of them), 24 houses 3.80 and 3.55. At a relative
// stop counts are steady: 24 houses 5.75 ms with either, 8 in FP64 4.31. Mean step of 40
// to 60; a share of 0.5 and four more are within 1 %.
constexpr double SOLVE_MEAN_SHARE = 0.3, SOLVE_MORE_ITERS = 2.0;
template <class R>
__device__ __forceinline__ int solveBlocks(const Scn<R>& g) { return (int)g.dvL0[1].d * ((g.nz + 1) >> 1); }
template <class R>
__device__ __forceinline__ float solveWork(const Scn<R>& g) {
    return (float)solveBlocks(g) * (g.sv[SV_SOLVED] > 0 ? (float)(g.sv[SV_MEANITERS] + SOLVE_MORE_ITERS) : SOLVE_FIRST_ITERS);
}

// a scenario's share in the division, from the CTA that begins its step
template <class R>
__device__ __forceinline__ void offerWork(const Scn<R>& g, int s, const TeamTable& t) {
    t.work[s] = make_float2(solveWork(g), __int_as_float(solveCtas<R>(solveTiling<R>(solveBlocks(g)))));
}

// The division of the first n scenarios' work, by one CTA of TEAM_TPB threads: the smallest bound
// on a CTA's work that the grid can meet, a scenario taking at most a CTA per tile.
// Sharing is weighed only where a CTA for every scenario would bind a fourth of the grid, and
// taken where it halves the bound or there are too few CTAs. Shared CTAs are dealt the
// scenarios in descending order of work up and down, so that the one with a round's
// largest has the next round's smallest. With it k_begin takes 10 us for one scenario, 15 for 24,
// 24 for 100 and 45 for 600 (9, 10, 11 and 11 without, and the division in every CTA of k_solve
// 4, 8, 27 and none).
constexpr int TEAM_TPB = 256;
inline __device__ void divideTeams(int n, const TeamTable& t) {
    constexpr int WARPS = TEAM_TPB / 32;
    __shared__ __align__(16) float work[MAX_BATCH];
    __shared__ int most[MAX_BATCH], first[MAX_BATCH + 1];
    __shared__ short order[MAX_BATCH];
    __shared__ float sums[2][WARPS], largests[WARPS];
    __shared__ int needs[2][WARPS], shared;
    const int G = t.grid, tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float largest = 0, all = 0;
    for (int s = tid; s < n; s += TEAM_TPB) {
        const float2 w = __ldcg(t.work + s);
        work[s] = w.x;
        most[s] = __float_as_int(w.y);
        largest = fmaxf(largest, w.x);
        all += w.x;
    }
    if (n == 1) {   // tid 0 has read it, and so does every other thread
        const int size = min(__float_as_int(__ldcg(t.work).y), G);
        for (int b = tid; b < G; b += TEAM_TPB) t.ctas[b] = SolveCta{b < size ? 0 : -1, size, b};
        if (tid == 0) t.next[0] = -1;
        return;
    }
    largest = warpMax(largest);
    for (int o = 16; o > 0; o >>= 1) all += __shfl_xor_sync(0xffffffffu, all, o);
    if (lane == 0) {
        largests[warp] = largest;
        sums[0][warp] = all;
    }
    if (tid == 0) shared = 0;
    __syncthreads();
    all = 0;
    for (int w = 0; w < WARPS; ++w) {
        largest = fmaxf(largest, largests[w]);
        all += sums[0][w];
    }
    auto ctas = [&](int s, float bound) { return min(most[s], max(1, (int)ceilf(work[s] / bound))); };
    int turn = 0;
    // the smallest bound up to hi, which can be met: a warp tries one of WARPS bounds, the
    // interval of the first that can be met is divided again. need: this lane's part
    auto search = [&](float hi, auto need) {
        float lo = 0;
        for (int it = 0; it < 5; ++it, turn ^= 1) {
            const float step = (hi - lo) / (WARPS + 1), bound = lo + step * (warp + 1);
            const int v = need(bound);
            if (lane == 0) needs[turn][warp] = v;
            __syncthreads();
            int k = 0;
            while (k < WARPS && needs[turn][k] > G) ++k;
            if (k < WARPS) hi = lo + step * (k + 1);
            lo += step * k;
        }
        return hi;
    };
    float own = 0, share = 0;   // share above 0: scenarios of at most this work share CTAs
    if (n <= G)
        own = search(largest, [&](float bound) {
            int sum = 0;
            for (int s = lane; s < n; s += 32) sum += ctas(s, bound);
            return __reduce_add_sync(0xffffffffu, sum);
        });
    if (4 * n > G) {
        share = search(fmaxf(largest, 1.001f * all / (float)G), [&](float bound) {
            int sum = 0;
            float turns = 0;
            for (int s = lane; s < n; s += 32) {
                if (work[s] > bound) sum += ctas(s, bound);
                else turns += work[s];
            }
            for (int o = 16; o > 0; o >>= 1) turns += __shfl_xor_sync(0xffffffffu, turns, o);
            return __reduce_add_sync(0xffffffffu, sum) + (int)ceilf(turns / bound);
        });
        if (n <= G && 2.0f * share > own) share = 0;
    }
    if (warp == 0) {   // the teams' CTAs
        int base = 0;
        for (int s0 = 0; s0 < n; s0 += 32) {
            const int s = s0 + lane;
            int v = s >= n || work[s] <= share ? 0 : ctas(s, share > 0 ? share : own);
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += u;
            }
            if (s < n) first[s + 1] = base + v;
            base += __shfl_sync(0xffffffffu, v, 31);
        }
        if (lane == 0) first[0] = 0;
    }
    for (int s = tid; s < n; s += TEAM_TPB) t.next[s] = -1;
    __syncthreads();
    if (share > 0) {   // the sharing scenarios' ranks; the others' work is out of the way
        for (int s = tid; s < ((n + 3) & ~3); s += TEAM_TPB)
            if (s >= n || work[s] > share) work[s] = -1.0f;
        __syncthreads();
        for (int s = tid; s < n; s += TEAM_TPB) {
            const float w = work[s];
            if (w < 0) continue;
            int rank = 0;
            for (int q = 0; q < n; q += 4) {
                const float4 v = *reinterpret_cast<const float4*>(work + q);
                rank += (v.x > w) + (v.y > w) + (v.z > w) + (v.w > w);
                rank += (v.x == w && q < s) + (v.y == w && q + 1 < s) + (v.z == w && q + 2 < s) + (v.w == w && q + 3 < s);
            }
            order[rank] = (short)s;
            atomicAdd(&shared, 1);
        }
        __syncthreads();
    }
    const int alone = first[n], bins = min(G - alone, shared);
    for (int b = tid; b < G; b += TEAM_TPB) {
        SolveCta c{-1, 1, 0};
        if (b < alone) {
            int lo = 0, hi = n - 1;   // the last scenario whose CTAs start at or before b
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (first[mid] <= b) lo = mid; else hi = mid - 1;
            }
            c = SolveCta{lo, first[lo + 1] - first[lo], b - first[lo]};
        } else if (b - alone < bins) {
            const int j = b - alone;
            c.scenario = order[j];
            for (int round = 1, s = c.scenario;; ++round) {
                const int at = round * bins + ((round & 1) ? bins - 1 - j : j);
                if (at >= shared) break;
                t.next[s] = order[at];
                s = order[at];
            }
        }
        t.ctas[b] = c;
    }
}

}  // namespace phx
