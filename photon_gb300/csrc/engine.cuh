// The GPU engine: a batch of scenarios stepped together, their device state,
// the domain tables of the launches and the launch sequence of the gas-phase
// step (src/sim/solver.cpp:226-269). A single-scenario context is a batch of
// one. Every kernel launch covers one domain (cells, faces of one axis, one
// kind of boundary, ...) of every scenario; the pressure solve is one cooperative
// launch (solve.cuh), and the whole step is captured once as a CUDA graph.
// Instantiated per precision by engine_fp64.cu and engine_mixed.cu.
#pragma once
#include <array>
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include "engine.h"
#include "host_setup.h"
#include "mixed_kernels.cuh"
#include "radiation.cuh"
#include "volume.cuh"
#include "selftest.cuh"
#include "solve.cuh"

namespace phx {

#define PHX_CK(x)                                                                        \
    do {                                                                                 \
        cudaError_t e_ = (x);                                                            \
        if (e_ != cudaSuccess) {                                                         \
            err = std::string(#x) + ": " + cudaGetErrorString(e_);                      \
            return PHX_ERR_CUDA;                                                         \
        }                                                                                \
    } while (0)
#define PHX_TRY(x) do { int r_ = (x); if (r_) return r_; } while (0)

// D_FACES, D_BND: the tiles of the x, then the y, then the z faces (boundary sides)
enum DomId { D_ONE = 0, D_CELLS, D_FACES, D_BND, D_CZ, D_CC, D_LEAK, D_COUNT };

// Widest rows the contexts take (nx); wider grids are refused, with PHX_ERR_UNSUPPORTED.
// What once set these (rows staged in shared memory) is gone, and nothing in the kernels
// depends on them now; they stay as the limits that callers have been told and that
// the tests cover, and no wider grid has been run.
template <class R>
constexpr int maxRow() { return sizeof(R) == 8 ? 410 : 776; }

template <class T>
static T* carve(char*& base, size_t& off, size_t n) {
    off = (off + 255) & ~(size_t)255;
    T* p = base ? (T*)(base + off) : nullptr;
    off += n * sizeof(T);
    return p;
}

// One scenario: host set-up results, its device arena and its descriptor.
// mixed path: CG iterations between replacements of the FP32 recursive
// residual by the FP64 residual b - A p64
constexpr int REPLACE_EVERY = 10;

// V-cycle schedules of the mixed path, per bucket of scenario size: bucket b
// holds scenarios of [20000 * 2^b, 20000 * 2^(b+1)) cells (bucket 0 also the
// smaller ones, the last one the larger ones). A bucket's entry is the
// multigrid coarsening stop the autotuner chose (0: not tuned, the
// reference's 2000). Process-wide, so scenarios admitted later (serving,
// batch_add) are built with the tuned schedule of their size.
constexpr int VC_BUCKETS = 8;
inline int vcycleBucket(long long cells) {
    int b = 0;
    long long e = 40000;
    while (cells >= e && b < VC_BUCKETS - 1) { e *= 2; ++b; }
    return b;
}
inline std::mutex& vcycleMutex() { static std::mutex m; return m; }
inline int* vcycleTable() { static int t[VC_BUCKETS] = {0}; return t; }
// the mixed path's smoothing on the coarse levels: Jacobi sweeps per level on
// each leg of the V-cycle (2, the reference's schedule, until tuned; 1 after a
// tuning that found it faster at the solve's relative residual)
inline int& vcycleSweeps() { static int v = 2; return v; }
inline int vcycleStopFor(long long cells) {
    std::lock_guard<std::mutex> lock(vcycleMutex());
    const int v = vcycleTable()[vcycleBucket(cells)];
    return v > 0 ? v : MG_COARSE_STOP_REF;
}

template <class R>
struct Scenario {
    static constexpr bool kMixed = std::is_same<R, float>::value;
    GridGeom geo;
    double cfl = 0.5, dtMaxP = 0.02, tol = 0.002, relTol = 0;
    int maxIters = 400, radiationOn = 1;
    int coarseStop = MG_COARSE_STOP_REF;   // multigrid coarsening stop (the V-cycle schedule)
    Zones Z;
    Multigrid MG;
    std::vector<double> Pb0;
    std::vector<Src> ignitions, burners;
    char* arena = nullptr;       // fields, geometry, solve vectors, scalars
    char* mgArena = nullptr;     // the multigrid levels (replaced when the V-cycle schedule changes)
    static constexpr size_t TAIL_BYTES = 256;   // of the main arena: what a saved state leaves out (tagBase)
    size_t arenaBytes = 0;       // both arenas
    size_t mainBytes = 0, mgBytes = 0;
    Scn<R> h{};                  // host copy of the device descriptor
    std::string err;

    ~Scenario() {
        if (arena) cudaFree(arena);
        if (mgArena) cudaFree(mgArena);
    }

    int setup(const phx_grid* g) {
        if (!g || g->nx <= 0 || g->ny <= 0 || g->nz <= 0 || !(g->dx > 0)) { err = "invalid grid dimensions"; return PHX_ERR_INVALID; }
        long long N = (long long)g->nx * g->ny * g->nz;
        if (N > 20000000LL) { err = "grid size out of range (the reference caps N at 20,000,000)"; return PHX_ERR_INVALID; }
        if (!g->blocked || !g->fx || !g->fy || !g->fz || !g->ax || !g->ay || !g->az) { err = "missing geometry array"; return PHX_ERR_INVALID; }
        if (g->radiation_on && !g->adiabatic_surfaces) {
            err = "radiation with non-adiabatic surfaces (the ray-traced radiation stage) is not part of the GPU step";
            return PHX_ERR_UNSUPPORTED;
        }
        geo.nx = g->nx; geo.ny = g->ny; geo.nz = g->nz;
        geo.dx = g->dx; geo.ox = g->ox; geo.oy = g->oy; geo.oz = g->oz;
        geo.windSpeed = g->wind_speed; geo.windFromDeg = g->wind_from_deg; geo.windExp = g->wind_exponent;
        const int NN = geo.N(), NX = geo.NX(), NY = geo.NY(), NZ = geo.NZ();
        geo.blocked.assign(g->blocked, g->blocked + NN);
        geo.fx.assign(g->fx, g->fx + NX); geo.fy.assign(g->fy, g->fy + NY); geo.fz.assign(g->fz, g->fz + NZ);
        geo.ax.assign(g->ax, g->ax + NX); geo.ay.assign(g->ay, g->ay + NY); geo.az.assign(g->az, g->az + NZ);
        geo.lx.assign(NX, 0); geo.ly.assign(NY, 0); geo.lz.assign(NZ, 0);
        if (g->lx) geo.lx.assign(g->lx, g->lx + NX);
        if (g->ly) geo.ly.assign(g->ly, g->ly + NY);
        if (g->lz) geo.lz.assign(g->lz, g->lz + NZ);
        geo.anyLeak = false;
        for (auto v : geo.lx) geo.anyLeak |= v != 0;
        for (auto v : geo.ly) geo.anyLeak |= v != 0;
        for (auto v : geo.lz) geo.anyLeak |= v != 0;
        if (g->nx > maxRow<R>()) {
            err = "grid rows too long for the pressure kernels (nx = " + std::to_string(g->nx) + ")";
            return PHX_ERR_UNSUPPORTED;
        }
        cfl = g->cfl; dtMaxP = g->dt_max; tol = g->tol; relTol = g->rel_tol; maxIters = g->max_iters;
        radiationOn = g->radiation_on;
        // set-up on the host: zones, multigrid
        Pb0.assign(NN, 101325.0);
        Z = computeZones(geo, Pb0);
        if (kMixed) coarseStop = vcycleStopFor(NN);   // the tuned schedule of the scenario's size, if any
        MG = buildMultigrid(geo, DENSE_MAX, coarseStop, coarseSolveFor());
        buildRowSets();
        a0Same[0] = MG.a0x == geo.ax;
        a0Same[1] = MG.a0y == geo.ay;
        a0Same[2] = MG.a0z == geo.az;
        buildLeakFaces();
        return PHX_OK;
    }

    // leak faces in the reference's order (axis, then face index) that touch no
    // blocked cell, and per zone its faces to other zones (src/sim/gasphase.cpp:410-445)
    std::vector<int> leak;       // 4 per face: axis, f, a, b
    std::vector<int> leakZStart, leakZList;
    void buildLeakFaces() {
        leak.clear();
        const int nx = geo.nx, ny = geo.ny, nz = geo.nz;
        for (int axis = 0; axis < 3 && geo.anyLeak; ++axis) {
            const std::vector<uint8_t>& lk = axis == 0 ? geo.lx : axis == 1 ? geo.ly : geo.lz;
            const int dX = nx + (axis == 0), dY = ny + (axis == 1);
            const int ncell = axis == 0 ? nx : axis == 1 ? ny : nz;
            for (int f = 0; f < (int)lk.size(); ++f) {
                if (!lk[f]) continue;
                const int i = f % dX, j = (f / dX) % dY, k = f / (dX * dY);
                int id[3] = {i, j, k}, a[3] = {i, j, k};
                a[axis] -= 1;
                const int ca = a[axis] >= 0 ? geo.cell(a[0], a[1], a[2]) : -1;
                const int cb = id[axis] < ncell ? geo.cell(i, j, k) : -1;
                if ((ca >= 0 && geo.blocked[ca]) || (cb >= 0 && geo.blocked[cb])) continue;
                leak.insert(leak.end(), {axis, f, ca, cb});
            }
        }
        const int nZ = (int)Z.zoneP.size(), nf = (int)leak.size() / 4;
        leakZStart.assign(nZ + 1, 0);
        auto zoneOf = [&](int c) { return c >= 0 ? Z.zone[c] : -1; };
        for (int q = 0; q < nf; ++q) {
            const int za = zoneOf(leak[4 * q + 2]), zb = zoneOf(leak[4 * q + 3]);
            if (za == zb) continue;
            if (za >= 0) leakZStart[za + 1]++;
            if (zb >= 0) leakZStart[zb + 1]++;
        }
        for (int z = 0; z < nZ; ++z) leakZStart[z + 1] += leakZStart[z];
        leakZList.assign(leakZStart[nZ], 0);
        std::vector<int> fill(nZ, 0);
        for (int q = 0; q < nf; ++q) {
            const int za = zoneOf(leak[4 * q + 2]), zb = zoneOf(leak[4 * q + 3]);
            if (za == zb) continue;
            if (za >= 0) leakZList[leakZStart[za] + fill[za]++] = q;
            if (zb >= 0) leakZList[leakZStart[zb] + fill[zb]++] = q;
        }
    }

    // device bytes the scenario will take (both arenas' layouts without memory)
    size_t layout(char* base) {
        if (base) return layoutMain(base) + TAIL_BYTES + layoutLevels(mgArena);
        return layoutMain(nullptr) + TAIL_BYTES + layoutLevels(nullptr);
    }

    // 2x2x2 blocks of the pressure solve
    int blocks() const { return ((geo.nx + 1) >> 1) * ((geo.ny + 1) >> 1) * ((geo.nz + 1) >> 1); }

    size_t layoutMain(char* base) {
        const int N = geo.N(), NX = geo.NX(), NY = geo.NY(), NZ = geo.NZ();
        // one reduction partial per CTA of the cell domain and per tile of the solve
        const int partStride = std::max((N + TPB - 1) / TPB, 2 * solveTiling<R>(blocks()).nt) + 2;
        size_t off = 0;
        Scn<R>& s = h;
        s.blocked = carve<uint8_t>(base, off, N);
        s.fx = carve<R>(base, off, NX); s.fy = carve<R>(base, off, NY); s.fz = carve<R>(base, off, NZ);
        s.ax = carve<R>(base, off, NX); s.ay = carve<R>(base, off, NY); s.az = carve<R>(base, off, NZ);
        // the same arrays where no wind-inflow boundary face is closed
        s.a0x = a0Same[0] ? s.ax : carve<R>(base, off, NX);
        s.a0y = a0Same[1] ? s.ay : carve<R>(base, off, NY);
        s.a0z = a0Same[2] ? s.az : carve<R>(base, off, NZ);
        s.lx = geo.anyLeak ? carve<uint8_t>(base, off, NX) : nullptr;
        s.ly = geo.anyLeak ? carve<uint8_t>(base, off, NY) : nullptr;
        s.lz = geo.anyLeak ? carve<uint8_t>(base, off, NZ) : nullptr;
        s.diag = carve<R>(base, off, N);
        s.code0 = carve<unsigned char>(base, off, N);
        s.zone = carve<int>(base, off, N);
        const int nZ = (int)Z.zoneP.size(), nC = (int)Z.closed.size();
        s.zoneOpen = carve<uint8_t>(base, off, nZ + 1);
        s.closedZone = carve<int>(base, off, nC + 1);
        s.closedStart = carve<int>(base, off, nC + 1);
        s.closedCells = carve<int>(base, off, Z.closedCells.size() + 1);
        s.zoneP = carve<double>(base, off, nZ + 1);
        s.zoneVol = carve<double>(base, off, nZ + 1);
        s.zoneDP = carve<double>(base, off, nZ + 1);
        s.zoneShift = carve<double>(base, off, nZ + 1);
        s.zoneMean = carve<double>(base, off, nZ + 1);
        s.nLeak = (int)leak.size() / 4;
        s.leak = carve<int4>(base, off, s.nLeak + 1);
        s.leakZStart = carve<int>(base, off, leakZStart.size() + 1);
        s.leakZList = carve<int>(base, off, leakZList.size() + 1);
        s.leakQ = carve<double>(base, off, s.nLeak + 1);
        s.zonePnew = carve<double>(base, off, nZ + 1);
        s.zoneDInt = carve<double>(base, off, nZ + 1);
        s.u = carve<R>(base, off, NX); s.v = carve<R>(base, off, NY); s.w = carve<R>(base, off, NZ);
        s.u2 = carve<R>(base, off, NX); s.v2 = carve<R>(base, off, NY); s.w2 = carve<R>(base, off, NZ);
        for (int q = 0; q < NSC; ++q) { s.sc[q] = carve<R>(base, off, N); s.sc2[q] = carve<R>(base, off, N); }
        s.p = carve<R>(base, off, N); s.S = carve<R>(base, off, N); s.nu = carve<R>(base, off, N);
        s.Pb = carve<R>(base, off, N); s.Q = carve<R>(base, off, N); s.Qr = carve<R>(base, off, N);
        s.hrr = carve<R>(base, off, N); s.massSrc = carve<R>(base, off, N);
        s.lit = carve<uint8_t>(base, off, N); s.lit2 = carve<uint8_t>(base, off, N); s.pilot = carve<uint8_t>(base, off, N);
        for (int q = 0; q < 7; ++q) s.tmp[q] = carve<R>(base, off, N);
        s.rho = kMixed ? nullptr : carve<R>(base, off, N);
        s.b = carve<R>(base, off, N); s.r = carve<R>(base, off, N); s.z = carve<R>(base, off, N);
        s.d = carve<R>(base, off, N); s.q = carve<R>(base, off, N);
        s.tmp[7] = s.d; s.tmp[8] = s.q;   // a solve's first iteration writes both before it reads them
        s.p64 = kMixed ? carve<double>(base, off, N) : nullptr;
        s.p64prev = kMixed ? carve<double>(base, off, N) : nullptr;
        Level<R>& L0 = s.lv[0];
        L0.diag = s.diag;
        L0.rowStart = nullptr; L0.col = nullptr; L0.val = nullptr;
        L0.childStart = nullptr; L0.child = nullptr;
        s.sv = carve<double>(base, off, SV_COUNT);
        s.part = carve<double>(base, off, (size_t)PS_COUNT * partStride);
        s.partStride = partStride;
        s.windU = carve<double>(base, off, geo.nz);
        s.cnt = carve<unsigned>(base, off, PS_COUNT + 4);
        s.teamBar = carve<unsigned>(base, off, 64);
        off = (off + 511) & ~(size_t)255;
        // past the bytes a saved state covers: tags only ever move on
        s.tagBase = base ? reinterpret_cast<unsigned*>(base + off) : nullptr;
        return off;
    }

    // the coarsest solve: the reference's 20 Gauss-Seidel sweep pairs on the FP64
    // path; on the mixed path the exact inverse of the coarsest matrix
    // (PHX_COARSE_EXACT=0: the reference's sweeps)
    static CoarseSolve coarseSolveFor() {
        CoarseSolve cs;
        if (kMixed) {
            static const bool exact = [] {
                const char* e = std::getenv("PHX_COARSE_EXACT");
                return !(e && std::atoi(e) == 0);
            }();
            cs.exact = exact;
        }
        return cs;
    }

    // the levels' arrays in their own arena: level 0's aggregation map, and per
    // coarser level its CSR rows, diagonal, iterate and scratch, child lists and,
    // at the coarsest level, the dense operator
    // A level's rows in sets of 32, each word of a set's rows side by side, so that a warp
    // reads a coupling of its rows in one access: the rows in their order for the sweeps,
    // and for the restriction eight lanes per unknown of the next level, a lane per child.
    // A set holds diag[32] (FP64 sweeps: omega / diag), val[width][32], own[32] (sweeps:
    // the row's aggregate; restriction: the row, -1 none), col[width][32] and, for the
    // sweeps, next[width][32], the columns' aggregates. Short rows end in couplings of 0 to
    // the row itself. Sets with a row of more than ROW_WIDEST couplings or an unknown of
    // more than eight children are left out.
    struct RowSets {
        size_t words = 0, nJ = 0, nR = 0;
        bool allJ = true, allR = true;   // no set is left out
        std::unique_ptr<unsigned[]> data;   // dropped once uploaded
        std::vector<RowSet> j, r;
    };
    std::vector<RowSets> rowSets;
    bool a0Same[3] = {false, false, false};   // level 0's coefficients are the faces' own, per axis
    void buildRowSets() {
        constexpr int RW = (int)sizeof(R) / 4;
        rowSets = std::vector<RowSets>(MG.lv.size());
        for (size_t l = 1; l + 1 < MG.lv.size(); ++l) {
            const MgLevel& L = MG.lv[l];
            const int nC = MG.lv[l + 1].n;
            RowSets& out = rowSets[l];
            out.nJ = (size_t)(L.n + 31) / 32;
            out.nR = (size_t)(nC + 3) / 4;
            out.j.resize(out.nJ);
            out.r.resize(out.nR);
            // widths and places first, so that the words are written once
            auto place = [&](RowSet& s, int width, bool sweep) {
                s.width = width;
                s.off = width > ROW_WIDEST ? -1 : (int)out.words;
                if (s.off >= 0) out.words += 32 * (size_t)((1 + width) * RW + 1 + width * (sweep ? 2 : 1));
                (sweep ? out.allJ : out.allR) &= s.off >= 0;
            };
            auto length = [&](int I) { return L.rowStart[I + 1] - L.rowStart[I]; };
            for (size_t c = 0; c < out.nJ; ++c) {
                int width = 0;
                for (int I = 32 * (int)c; I < std::min(32 * (int)c + 32, L.n); ++I) width = std::max(width, length(I));
                place(out.j[c], width, true);
            }
            for (size_t c = 0; c < out.nR; ++c) {
                int width = 0;
                for (int J = 4 * (int)c; J < std::min(4 * (int)c + 4, nC); ++J) {
                    if (L.childStart[J + 1] - L.childStart[J] > 8) width = ROW_WIDEST + 1;
                    for (int q = L.childStart[J]; q < L.childStart[J + 1]; ++q) width = std::max(width, length(L.child[q]));
                }
                place(out.r[c], width, false);
            }
            out.data.reset(new unsigned[out.words + 1]);
            auto fill = [&](const RowSet& s, int q, int I, bool sweep) {   // lane q's row I, -1 none
                unsigned* const w = out.data.get() + s.off;
                R* const val = reinterpret_cast<R*>(w);
                unsigned* const own = w + 32 * (1 + s.width) * RW;
                const int q0 = I >= 0 ? L.rowStart[I] : 0, n = I >= 0 ? length(I) : 0;
                val[q] = (R)(I < 0 ? 0.0 : sweep && RW == 2 ? (L.diag[I] > 0 ? OMEGA / L.diag[I] : 0.0) : L.diag[I]);
                own[q] = (unsigned)(I < 0 ? -1 : sweep ? L.agg[I] : I);
                for (int e = 0; e < s.width; ++e) {
                    const int col = e < n ? L.col[q0 + e] : std::max(I, 0);
                    val[32 * (1 + e) + q] = (R)(e < n ? L.val[q0 + e] : 0.0);
                    own[32 * (1 + e) + q] = (unsigned)col;
                    if (sweep) own[32 * (1 + s.width + e) + q] = (unsigned)L.agg[col];
                }
            };
            for (size_t c = 0; c < out.nJ; ++c)
                for (int q = 0; q < 32 && out.j[c].off >= 0; ++q) fill(out.j[c], q, 32 * (int)c + q < L.n ? 32 * (int)c + q : -1, true);
            for (size_t c = 0; c < out.nR; ++c)
                for (int q = 0; q < 32 && out.r[c].off >= 0; ++q) {
                    const int J = 4 * (int)c + q / 8, n = J < nC ? L.childStart[J + 1] - L.childStart[J] : 0;
                    fill(out.r[c], q, q % 8 < n ? L.child[L.childStart[J] + q % 8] : -1, false);
                }
        }
    }

    size_t layoutLevels(char* base) {
        const int nl = (int)MG.lv.size();
        size_t off = 0;
        Scn<R>& s = h;
        s.nLevels = nl;
        for (int l = 0; l < nl; ++l) {
            const MgLevel& L = MG.lv[l];
            Level<R>& D = s.lv[l];
            D.n = L.n;
            // the arrays that rows without a set, and a serial solve of the coarsest level, read
            const bool last = l == nl - 1, sets = rowSets[l].allJ && rowSets[l].allR;
            const bool csr = l > 0 && (last ? L.dense.empty() : !sets);
            if (l > 0) {
                D.rowStart = csr ? carve<int>(base, off, L.rowStart.size()) : nullptr;
                D.col = csr ? carve<int>(base, off, L.col.size() + 1) : nullptr;
                D.val = csr ? carve<R>(base, off, L.val.size() + 1) : nullptr;
                D.diag = carve<R>(base, off, L.n + 1);
                D.omd = carve<R>(base, off, L.n + 1);
                D.x = carve<R>(base, off, l == 1 || l == nl - 1 ? L.n + 1 : 1);
                for (unsigned long long** v : {&D.b, &D.yd, &D.xd, &D.yu, &D.xu})
                    *v = carve<unsigned long long>(base, off, TAG_WORDS<R> * (v == &D.xu && l == 1 ? 1 : (size_t)(L.n + 1)));
            }
            D.agg = L.agg.empty() || (l > 0 && !csr) ? nullptr : carve<int>(base, off, L.agg.size());
            D.childStart = (l == 0 || !csr || L.childStart.empty()) ? nullptr : carve<int>(base, off, L.childStart.size());
            D.child = (l == 0 || !csr || L.child.empty()) ? nullptr : carve<int>(base, off, L.child.size() + 1);
            D.rows = carve<unsigned>(base, off, rowSets[l].words + 1);
            D.setsJ = carve<RowSet>(base, off, rowSets[l].nJ + 1);
            D.setsR = carve<RowSet>(base, off, rowSets[l].nR + 1);
            D.dense = L.dense.empty() ? nullptr : carve<R>(base, off, L.dense.size());
        }
        return off + 256;
    }

    int allocate() {
        mainBytes = layoutMain(nullptr);
        mgBytes = layoutLevels(nullptr);
        arenaBytes = mainBytes + TAIL_BYTES + mgBytes;
        cudaError_t e = cudaMalloc(&arena, mainBytes + TAIL_BYTES);
        if (e == cudaSuccess) e = cudaMalloc(&mgArena, mgBytes);
        if (e != cudaSuccess) {
            cudaGetLastError();
            if (arena) cudaFree(arena);
            arena = nullptr;
            mgArena = nullptr;
            err = std::string("device allocation of ") + std::to_string(arenaBytes) + " bytes failed: " + cudaGetErrorString(e);
            return PHX_ERR_OOM;
        }
        layoutMain(arena);
        layoutLevels(mgArena);
        return PHX_OK;
    }

    // Replace the multigrid hierarchy by one built with another coarsening stop
    // (the V-cycle schedule): a new levels arena, uploaded; the fields and the
    // solve's state in the main arena are untouched. The caller rebuilds the
    // batch tables (the level domains change).
    int rebuildLevels(cudaStream_t st, int stop) {
        if (stop == coarseStop && mgArena) return PHX_OK;
        Multigrid M = buildMultigrid(geo, DENSE_MAX, stop, coarseSolveFor());
        PHX_CK(cudaStreamSynchronize(st));
        std::vector<RowSets> oldSets = std::move(rowSets);
        std::swap(MG, M);
        buildRowSets();
        const size_t bytes = layoutLevels(nullptr);
        char* fresh = nullptr;
        if (cudaMalloc(&fresh, bytes) != cudaSuccess) {   // the former hierarchy stays
            cudaGetLastError();
            std::swap(MG, M);
            rowSets = std::move(oldSets);
            layoutLevels(mgArena);
            err = "device allocation of the multigrid levels failed";
            return PHX_ERR_OOM;
        }
        char* const old = mgArena;
        coarseStop = stop;
        mgArena = fresh;
        mgBytes = bytes;
        arenaBytes = mainBytes + TAIL_BYTES + mgBytes;
        layoutLevels(mgArena);
        const int r = uploadLevels(st);
        if (old) cudaFree(old);
        return r;
    }

    template <class T>
    int put(cudaStream_t st, const T* dstc, const std::vector<double>& src) {
        using U = typename std::remove_const<T>::type;
        U* dst = const_cast<U*>(dstc);
        std::vector<U> tmp(src.begin(), src.end());
        if (!tmp.empty()) PHX_CK(cudaMemcpyAsync(dst, tmp.data(), tmp.size() * sizeof(U), cudaMemcpyHostToDevice, st));
        PHX_CK(cudaStreamSynchronize(st));
        return PHX_OK;
    }
    template <class T, class V>
    int putRaw(cudaStream_t st, const T* dstc, const V* src, size_t n) {
        static_assert(sizeof(T) == sizeof(V), "element size");
        void* dst = const_cast<void*>((const void*)dstc);
        if (n) PHX_CK(cudaMemcpyAsync(dst, src, n * sizeof(T), cudaMemcpyHostToDevice, st));
        PHX_CK(cudaStreamSynchronize(st));
        return PHX_OK;
    }

    int upload(cudaStream_t st) {
        const int N = geo.N();
        Scn<R>& s = h;
        PHX_CK(cudaMemsetAsync(arena, 0, mainBytes + TAIL_BYTES, st));
        s.nx = geo.nx; s.ny = geo.ny; s.nz = geo.nz; s.N = N; s.NX = geo.NX(); s.NY = geo.NY(); s.NZ = geo.NZ();
        s.dvA[0] = makeDivU(geo.nx); s.dvB[0] = makeDivU(geo.nx * geo.ny); s.dY[0] = geo.ny;
        s.dvA[1] = makeDivU(geo.nx + 1); s.dvB[1] = makeDivU((geo.nx + 1) * geo.ny); s.dY[1] = geo.ny;
        s.dvA[2] = makeDivU(geo.nx); s.dvB[2] = makeDivU(geo.nx * (geo.ny + 1)); s.dY[2] = geo.ny + 1;
        s.dvL0[0] = makeDivS((geo.nx + 1) >> 1); s.dvL0[1] = makeDivS(((geo.nx + 1) >> 1) * ((geo.ny + 1) >> 1));
        s.dx = geo.dx; s.ox = geo.ox; s.oy = geo.oy; s.oz = geo.oz;
        {   // IEEE divisions in R: the values of the kernels' R(1) / dx
            const R dxr = (R)geo.dx;
            s.rdx = R(1) / dxr;
            s.rdx2 = R(1) / (dxr * dxr);
        }
        s.cfl = cfl; s.dtMaxP = dtMaxP; s.tol = tol; s.relTol = relTol; s.maxIters = maxIters; s.radiationOn = radiationOn;
        double th = geo.windFromDeg * 3.14159265 / 180.0;
        s.windSpeed = geo.windSpeed; s.windSin = std::sin(th); s.windCos = std::cos(th); s.windExp = geo.windExp;
        s.nZones = (int)Z.zoneP.size();
        s.nClosed = (int)Z.closed.size();
        s.mixed = kMixed ? 1 : 0;
        {   // PHX_REPLACE_EVERY=n: another interval, for measurements
            static const int every = [] {
                const char* e = std::getenv("PHX_REPLACE_EVERY");
                const int v = e ? std::atoi(e) : 0;
                return v >= 2 && v <= 100 ? v : REPLACE_EVERY;
            }();
            s.replaceEvery = every;
        }
        s.extrap = std::getenv("PHX_NO_EXTRAP") == nullptr;   // mixed path: extrapolated initial guess
        PHX_TRY(putRaw(st, s.blocked, geo.blocked.data(), N));
        PHX_TRY(put(st, s.fx, geo.fx)); PHX_TRY(put(st, s.fy, geo.fy)); PHX_TRY(put(st, s.fz, geo.fz));
        PHX_TRY(put(st, s.ax, geo.ax)); PHX_TRY(put(st, s.ay, geo.ay)); PHX_TRY(put(st, s.az, geo.az));
        if (s.a0x != s.ax) PHX_TRY(put(st, s.a0x, MG.a0x));
        if (s.a0y != s.ay) PHX_TRY(put(st, s.a0y, MG.a0y));
        if (s.a0z != s.az) PHX_TRY(put(st, s.a0z, MG.a0z));
        PHX_TRY(put(st, s.diag, MG.lv[0].diag));
        {
            const std::vector<unsigned char> cd = levelZeroCodes();
            PHX_TRY(putRaw(st, s.code0, cd.data(), cd.size()));
        }
        PHX_TRY(putRaw(st, s.zone, Z.zone.data(), N));
        PHX_TRY(putRaw(st, s.zoneOpen, Z.zoneOpen.data(), Z.zoneOpen.size()));
        PHX_TRY(putRaw(st, s.closedZone, Z.closed.data(), Z.closed.size()));
        PHX_TRY(putRaw(st, s.closedStart, Z.closedStart.data(), Z.closedStart.size()));
        PHX_TRY(putRaw(st, s.closedCells, Z.closedCells.data(), Z.closedCells.size()));
        PHX_TRY(putRaw(st, s.zoneP, Z.zoneP.data(), Z.zoneP.size()));
        PHX_TRY(putRaw(st, s.zoneVol, Z.zoneVol.data(), Z.zoneVol.size()));
        if (geo.anyLeak) {
            PHX_TRY(putRaw(st, s.lx, geo.lx.data(), geo.lx.size()));
            PHX_TRY(putRaw(st, s.ly, geo.ly.data(), geo.ly.size()));
            PHX_TRY(putRaw(st, s.lz, geo.lz.data(), geo.lz.size()));
        }
        if (!leak.empty()) PHX_TRY(putRaw(st, s.leak, reinterpret_cast<const int4*>(leak.data()), leak.size() / 4));
        PHX_TRY(putRaw(st, s.leakZStart, leakZStart.data(), leakZStart.size()));
        PHX_TRY(putRaw(st, s.leakZList, leakZList.data(), leakZList.size()));
        // initial state (src/sim/discretize.cpp:28-31)
        const double amb[NSC] = {tStoredFromKd<R>(K_T0), K_YO2_AMB, 0, 0, 0, 0, K_YCO2_AMB, K_YH2O_AMB, 0, 0};
        for (int q = 0; q < NSC; ++q) {
            PHX_TRY(put(st, s.sc[q], std::vector<double>(N, amb[q])));
            PHX_TRY(put(st, s.sc2[q], std::vector<double>(N, amb[q])));
        }
        PHX_TRY(put(st, s.Pb, Pb0));
        return uploadLevels(st);
    }

    // How long a CTA of the solve waits for its team: two seconds, and where one thread solves the
    // coarsest level while the others wait, the cycles of its 40 sweeps as well (a row's division
    // and loads some 1,500, a coupling's load and addition some 700; twice that). The
    // environment's PHX_TEAM_WAIT_CYCLES takes the place of the two seconds.
    static long long waitCycles(const MgLevel& coarsest) {
        const char* e = std::getenv("PHX_TEAM_WAIT_CYCLES");
        const long long base = e ? std::max(0LL, std::atoll(e)) : 4000000000LL;
        if (!coarsest.dense.empty() || coarsest.rowStart.empty()) return base;
        return base + 2LL * MG_COARSE_SWEEPS_REF * (3000LL * coarsest.n + 1400LL * coarsest.rowStart.back());
    }

    int uploadLevels(cudaStream_t st) {
        Scn<R>& s = h;
        s.waitCycles = waitCycles(MG.lv.back());
        PHX_CK(cudaMemsetAsync(mgArena, 0, mgBytes, st));
        for (int l = 1; l < (int)MG.lv.size(); ++l) {
            const MgLevel& L = MG.lv[l];
            Level<R>& D = s.lv[l];
            if (D.rowStart) {
                PHX_TRY(putRaw(st, D.rowStart, L.rowStart.data(), L.rowStart.size()));
                PHX_TRY(putRaw(st, D.col, L.col.data(), L.col.size()));
                PHX_TRY(put(st, D.val, L.val));
            }
            PHX_TRY(put(st, D.diag, L.diag));
            std::vector<double> omd(L.n);
            for (int I = 0; I < L.n; ++I) omd[I] = L.diag[I] > 0 ? OMEGA / L.diag[I] : 0.0;
            PHX_TRY(put(st, D.omd, omd));
        }
        for (int l = 0; l < (int)MG.lv.size(); ++l) {
            const MgLevel& L = MG.lv[l];
            Level<R>& D = s.lv[l];
            if (D.agg) PHX_TRY(putRaw(st, D.agg, L.agg.data(), L.agg.size()));
            if (D.childStart) PHX_TRY(putRaw(st, D.childStart, L.childStart.data(), L.childStart.size()));
            if (D.child) PHX_TRY(putRaw(st, D.child, L.child.data(), L.child.size()));
            if (D.dense) PHX_TRY(put(st, D.dense, L.dense));
            PHX_TRY(putRaw(st, D.rows, rowSets[l].data.get(), rowSets[l].words));
            PHX_TRY(putRaw(st, D.setsJ, rowSets[l].j.data(), rowSets[l].nJ));
            PHX_TRY(putRaw(st, D.setsR, rowSets[l].r.data(), rowSets[l].nR));
        }
        for (RowSets& r : rowSets) { r.data.reset(); r.j = {}; r.r = {}; }
        return PHX_OK;
    }

    // The level-0 coefficient code of every cell (level0.cuh): bits 0-5 for the
    // interior x-, x+, y-, y+, z-, z+ faces whose coefficient is exactly 1 (they
    // couple the cell to its neighbour), bit 7 for one open domain-boundary
    // face with coefficient 1 (it adds to the diagonal only), bit 6 when the
    // cell needs the arrays (a coefficient other than 0 or 1, two or more open
    // boundary faces, or a diagonal other than the count of its bits).
    std::vector<unsigned char> levelZeroCodes() const {
        const int nx = geo.nx, ny = geo.ny, nz = geo.nz;
        std::vector<unsigned char> cd(geo.N(), 0);
        for (int k = 0; k < nz; ++k)
            for (int j = 0; j < ny; ++j)
                for (int i = 0; i < nx; ++i) {
                    const int c = geo.cell(i, j, k);
                    const double a[6] = {MG.a0x[geo.xface(i, j, k)], MG.a0x[geo.xface(i + 1, j, k)],
                                         MG.a0y[geo.yface(i, j, k)], MG.a0y[geo.yface(i, j + 1, k)],
                                         MG.a0z[geo.zface(i, j, k)], MG.a0z[geo.zface(i, j, k + 1)]};
                    const bool inner[6] = {i > 0, i < nx - 1, j > 0, j < ny - 1, k > 0, k < nz - 1};
                    unsigned bits = 0;
                    int boundary = 0;
                    bool general = false;
                    for (int f = 0; f < 6; ++f) {
                        if (a[f] == 1.0) {
                            if (inner[f]) bits |= 1u << f;
                            else ++boundary;
                        } else if (a[f] != 0.0) {
                            general = true;   // a fraction
                        }
                    }
                    if (boundary > 1) general = true;
                    int cnt = boundary;
                    for (int f = 0; f < 6; ++f) cnt += (bits >> f) & 1u;
                    if (MG.lv[0].diag[c] != (double)cnt) general = true;
                    cd[c] = general ? CODE_GENERAL : (unsigned char)(bits | (boundary ? CODE_BOUNDARY : 0u));
                }
        return cd;
    }

    // CTAs of each domain of this scenario
    void tiles(int* t) const {
        const int N = geo.N(), nx = geo.nx, ny = geo.ny, nz = geo.nz;
        auto cdiv = [](long long a, long long b) { return (int)((a + b - 1) / b); };
        for (int d = 0; d < D_COUNT; ++d) t[d] = 0;
        t[D_ONE] = 1;
        t[D_CELLS] = cdiv(N, TPB);
        t[D_LEAK] = cdiv((long long)leak.size() / 4, TPB);
        t[D_FACES] = cdiv(geo.NX(), TPB) + cdiv(geo.NY(), TPB) + cdiv(geo.NZ(), TPB);
        t[D_BND] = cdiv(2LL * ny * nz, TPB) + cdiv(2LL * nx * nz, TPB) + cdiv((long long)nx * ny, TPB);
        t[D_CZ] = (int)Z.closed.size();
        t[D_CC] = cdiv((long long)Z.closedCells.size(), TPB);
    }
};

template <class R>
class Ctx : public CtxBase {
public:
    // the float instantiation is the mixed path: FP32 fields and stencils, FP64
    // refinement of the pressure solve, FP64 dots and global sums
    static constexpr bool kMixed = std::is_same<R, float>::value;

    std::vector<std::unique_ptr<Scenario<R>>> sc;
    cudaStream_t st = nullptr;
    // batch-wide device tables
    int cap = 0;                 // scenario capacity of the tables
    char* tab = nullptr;
    Scn<R>* dS = nullptr;        // descriptors
    int* dDomStart = nullptr;    // D_COUNT x (cap + 1)
    double* dDtMax = nullptr;    // per-scenario dtMax of the step
    unsigned* dErr = nullptr;    // error word of the device side (bounded waits that ran out); [2..3] stay 0
    unsigned* ownTab = nullptr;  // CTA -> (scenario, tile) of every domain (Dom::owner)
    size_t ownCap = 0;
    double* dTimes = nullptr;    // simulated time of each scenario (read-back staging)
    double* dMaxPart = nullptr;  // k_solve: two maxima per CTA
    TeamTable teams{};           // ... and which scenario each CTA works on
    int solveGrid = 0;           // k_solve: CTAs resident at once
    int solvePer = 1;            // ... per SM
    bool smoothOne = false;            // mixed path: one Jacobi sweep per coarse level and leg (vcycleSweeps)
    double* hPin = nullptr;      // pinned scratch for read-backs
    Dom dom[D_COUNT];
    bool anyLeak = false;
    bool tablesDirty = true;
    int launches = 0;
    cudaEvent_t ev[4] = {};

    // radiation trace work space, grown on demand (traces are seconds of
    // simulated time apart)
    struct RadWork {
        enum { EL, WL, WALLI, ABS, WALLOF, CELLS, FLAGS, SOLIDT, GAS, KC, SOURCES, RAYS, RAYELEM, RAYVAL, CNT, NBUF };
        int marchCtas = 0;
        void* buf[NBUF] = {};
        size_t cap[NBUF] = {};
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        double lastMs = 0;
        void release() {
            for (void* p : buf) if (p) cudaFree(p);
            if (e0) cudaEventDestroy(e0);
            if (e1) cudaEventDestroy(e1);
        }
    } rad;

    ~Ctx() override {
        if (st) cudaStreamSynchronize(st);
        rad.release();
        volw.release();
        destroyGraph();
        sc.clear();
        if (tab) cudaFree(tab);
        if (ownTab) cudaFree(ownTab);
        if (hPin) cudaFreeHost(hPin);
        if (flushBuf) cudaFree(flushBuf);
        for (auto e : evPool) cudaEventDestroy(e);
        for (auto& e : ev) if (e) cudaEventDestroy(e);
        if (st) cudaStreamDestroy(st);
    }

    int nscn() const { return (int)sc.size(); }

    int initStream() {
        if (st) return PHX_OK;
        PHX_CK(cudaGetDevice(&device));
        PHX_CK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
        PHX_CK(cudaMallocHost(&hPin, 8192 * sizeof(double)));
        for (auto& e : ev) PHX_CK(cudaEventCreate(&e));
        return PHX_OK;
    }

    // ---- membership ---------------------------------------------------------------
    int addScenario(const phx_grid* g, int* id) override {
        if (nscn() >= MAX_BATCH) { err = "batch is full (1024 scenarios)"; return PHX_ERR_BUDGET; }
        size_t bytes = 0;
        // validation and host set-up first: no device needed to reject bad input
        void* p = prepare(g, &bytes, err);
        if (!p) return lastPrepareStatus;
        return admit(p, id);
    }

    int lastPrepareStatus = PHX_OK;
    void* prepare(const phx_grid* g, size_t* bytes, std::string& e) override {
        auto s = std::make_unique<Scenario<R>>();
        const int r = s->setup(g);
        lastPrepareStatus = r;
        if (r != PHX_OK) { e = s->err; return nullptr; }
        if (bytes) *bytes = s->layout(nullptr);
        return s.release();
    }
    int admit(void* prepared, int* id) override {
        std::unique_ptr<Scenario<R>> s(static_cast<Scenario<R>*>(prepared));
        if (nscn() >= MAX_BATCH) { err = "batch is full (1024 scenarios)"; return PHX_ERR_BUDGET; }
        PHX_TRY(initStream());
        int r = s->allocate();
        if (r == PHX_OK) r = s->upload(st);
        if (r != PHX_OK) { err = s->err.empty() ? err : s->err; return r; }
        sc.push_back(std::move(s));
        if (id) *id = nscn() - 1;
        tablesDirty = true;
        return PHX_OK;
    }
    void discard(void* prepared) override { delete static_cast<Scenario<R>*>(prepared); }
    // Solver::traceRadiation (src/sim/radiation.cpp:181-319) for scenario s
    // (el: phx_rad_elem records, or rows of 11 doubles; elWords: their doubles)
    int radTrace(int s, const void* el, int elWords, int nE, const phx_rad_wall* wl, int nW, const double* solidT,
                 double* radAbs, double* radGas) override {
        PHX_TRY(checkScn(s));
        if (nE < 0 || nW < 0 || (nE > 0 && (!el || !radAbs)) || (nW > 0 && !wl)) {
            err = "invalid radiation trace arguments";
            return PHX_ERR_INVALID;
        }
        const Scenario<R>& S = *sc[s];
        const int nx = S.geo.nx, ny = S.geo.ny, nz = S.geo.nz;
        const size_t N = (size_t)nx * ny * nz;
        const size_t NF[3] = {(size_t)(nx + 1) * ny * nz, (size_t)nx * (ny + 1) * nz, (size_t)nx * ny * (nz + 1)};
        const size_t nF = NF[0] + NF[1] + NF[2];
        {   // at most one wall per face, every face in range (an error of the range comes first)
            std::vector<uint64_t> seen((nF + 63) / 64);
            bool two = false;
            for (int w = 0; w < nW; ++w) {
                if (wl[w].axis < 0 || wl[w].axis > 2 || wl[w].face < 0 || (size_t)wl[w].face >= NF[wl[w].axis]) {
                    err = "radiation wall " + std::to_string(w) + ": axis or face out of range";
                    return PHX_ERR_INVALID;
                }
                const size_t key = (wl[w].axis == 0 ? 0 : wl[w].axis == 1 ? NF[0] : NF[0] + NF[1]) + (size_t)wl[w].face;
                const uint64_t bit = 1ull << (key & 63);
                two |= (seen[key >> 6] & bit) != 0;
                seen[key >> 6] |= bit;
            }
            if (two) { err = "two radiation walls on one face"; return PHX_ERR_INVALID; }
        }
        PHX_TRY(ensureTables());
        PHX_TRY(initStream());
        // buffer b holds at least `bytes` (device memory is allocated here only)
        auto grow = [&](int b, size_t bytes) -> int {
            bytes = std::max<size_t>(bytes, 16);
            if (rad.buf[b] && rad.cap[b] >= bytes) return PHX_OK;
            if (rad.buf[b]) { PHX_CK(cudaStreamSynchronize(st)); cudaFree(rad.buf[b]); rad.buf[b] = nullptr; rad.cap[b] = 0; }
            if (cudaMalloc(&rad.buf[b], bytes) != cudaSuccess) {
                cudaGetLastError();
                rad.buf[b] = nullptr;
                err = "out of device memory for the radiation trace";
                return PHX_ERR_OOM;
            }
            rad.cap[b] = bytes;
            return PHX_OK;
        };
        const size_t elBytes = (size_t)nE * elWords * sizeof(double);
        PHX_TRY(grow(RadWork::EL, elBytes));
        PHX_TRY(grow(RadWork::ABS, nE * sizeof(double)));
        PHX_TRY(grow(RadWork::WL, nW * sizeof(phx_rad_wall)));
        PHX_TRY(grow(RadWork::WALLI, nW * 8 * sizeof(R)));
        PHX_TRY(grow(RadWork::WALLOF, nF * sizeof(int)));
        PHX_TRY(grow(RadWork::CELLS, N * sizeof(RadCell<R>)));
        PHX_TRY(grow(RadWork::FLAGS, (N + 3) & ~(size_t)3));
        PHX_TRY(grow(RadWork::SOLIDT, N * sizeof(double)));
        PHX_TRY(grow(RadWork::GAS, N * sizeof(R)));
        PHX_TRY(grow(RadWork::KC, sizeof(RadConst<R>)));
        const size_t nAt = std::min(nE, RAD_PORTION);   // elements at a time
        PHX_TRY(grow(RadWork::SOURCES, nAt * sizeof(RadSource<R>)));
        PHX_TRY(grow(RadWork::RAYS, nAt * RAD_DIRS * sizeof(RadRay<R>)));
        PHX_TRY(grow(RadWork::RAYVAL, nAt * RAD_DIRS * sizeof(R)));
        PHX_TRY(grow(RadWork::RAYELEM, nAt * RAD_DIRS * sizeof(int)));
        PHX_TRY(grow(RadWork::CNT, (RAD_DIRS + 1) * sizeof(int)));
        if (!rad.marchCtas) {
            int dev = 0, sms = 0, per = 0;
            PHX_CK(cudaGetDevice(&dev));
            PHX_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
            PHX_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_rad_march<R>, 256, 0));
            rad.marchCtas = std::max(1, sms * std::max(1, per));
        }
        if (!rad.e0) {
            PHX_CK(cudaEventCreate(&rad.e0));
            PHX_CK(cudaEventCreate(&rad.e1));
        }
        double* dEl = static_cast<double*>(rad.buf[RadWork::EL]);
        phx_rad_wall* dWl = static_cast<phx_rad_wall*>(rad.buf[RadWork::WL]);
        R* dWallI = static_cast<R*>(rad.buf[RadWork::WALLI]);
        double* dAbs = static_cast<double*>(rad.buf[RadWork::ABS]);
        int* dWallOf = static_cast<int*>(rad.buf[RadWork::WALLOF]);
        RadCell<R>* dCells = static_cast<RadCell<R>*>(rad.buf[RadWork::CELLS]);
        uint8_t* dFlags = static_cast<uint8_t*>(rad.buf[RadWork::FLAGS]);
        double* dSolid = static_cast<double*>(rad.buf[RadWork::SOLIDT]);
        R* dGas = static_cast<R*>(rad.buf[RadWork::GAS]);
        RadConst<R>* dKc = static_cast<RadConst<R>*>(rad.buf[RadWork::KC]);
        RadSource<R>* dSources = static_cast<RadSource<R>*>(rad.buf[RadWork::SOURCES]);
        RadRay<R>* dRays = static_cast<RadRay<R>*>(rad.buf[RadWork::RAYS]);
        R* dRayVal = static_cast<R*>(rad.buf[RadWork::RAYVAL]);
        int* dRayElem = static_cast<int*>(rad.buf[RadWork::RAYELEM]);
        int* dCnt = static_cast<int*>(rad.buf[RadWork::CNT]);
        if (nE) PHX_CK(cudaMemcpyAsync(dEl, el, elBytes, cudaMemcpyHostToDevice, st));
        if (nW) PHX_CK(cudaMemcpyAsync(dWl, wl, nW * sizeof(phx_rad_wall), cudaMemcpyHostToDevice, st));
        if (solidT) PHX_CK(cudaMemcpyAsync(dSolid, solidT, N * sizeof(double), cudaMemcpyHostToDevice, st));
        PHX_CK(cudaMemsetAsync(dGas, 0, N * sizeof(R), st));
        PHX_CK(cudaMemsetAsync(dCnt, 0, (RAD_DIRS + 1) * sizeof(int), st));
        PHX_CK(cudaEventRecord(rad.e0, st));
        k_rad_setup<R><<<1, RAD_EXP_N, 0, st>>>(dKc);
        k_rad_cells<R><<<(unsigned)((N + 255) / 256), 256, 0, st>>>(dS, s, solidT ? dSolid : nullptr, dCells, dFlags,
                                                                    dKc);
        if (nW) k_rad_walls<R><<<(nW + 127) / 128, 128, 0, st>>>(dWl, nW, nx, ny, nz, dWallOf,
                                                                 reinterpret_cast<unsigned*>(dFlags), dWallI, dKc);
        for (long long e0 = 0; e0 < nE; e0 += RAD_PORTION) {
            const int n = (int)std::min<long long>(nE - e0, RAD_PORTION);
            if (e0) PHX_CK(cudaMemsetAsync(dCnt, 0, (RAD_DIRS + 1) * sizeof(int), st));
            k_rad_elems<R><<<(n + RAD_ELEMS - 1) / RAD_ELEMS, RAD_ELEMS, 0, st>>>(dS, s, dEl + e0 * elWords, elWords, n, dKc,
                                                                                 dSources, dRays, dRayElem, dRayVal, dCnt);
            k_rad_march<R><<<rad.marchCtas, 256, 0, st>>>(dS, s, n, dSources, dCells, dFlags, dWallOf, dWallI, dKc,
                                                          dRays, dRayElem, dRayVal, dCnt, dGas);
            k_rad_absorbed<R><<<(n + 255) / 256, 256, 0, st>>>(dRayVal, n, dAbs + e0);
        }
        PHX_CK(cudaGetLastError());
        PHX_CK(cudaEventRecord(rad.e1, st));
        if (nE) PHX_CK(cudaMemcpyAsync(radAbs, dAbs, nE * sizeof(double), cudaMemcpyDeviceToHost, st));
        if (radGas) PHX_TRY(getReal(dGas, N, radGas));
        else PHX_CK(cudaStreamSynchronize(st));
        float ms = 0;
        PHX_CK(cudaEventElapsedTime(&ms, rad.e0, rad.e1));
        rad.lastMs = ms;
        return checkDeviceError();
    }
    double radLastMs() const override { return rad.lastMs; }

    // ---- V-cycle schedule autotuner ----------------------------------------------
    // For each size bucket present in the batch (largest total first), every
    // candidate coarsening stop is applied to the bucket's scenarios and the
    // whole batch is stepped from the same saved state: one untimed step (the
    // step graph is rebuilt), then `steps` steps timed with CUDA events. Every
    // candidate solves to the same relative residual, so the fastest one
    // delivers the most cell-updates per second at equal residual; it is kept
    // and recorded in the process-wide table. The batch's state is restored at
    // the end. The FP64 path keeps the reference's schedule (its parity with
    // the reference needs the reference's V-cycle).
    int tuneVcycle(int steps, double dtMax, int* out, int cap) override {
        if (steps < 1 || steps > 50 || !(dtMax > 0)) { err = "invalid tuning arguments"; return PHX_ERR_INVALID; }
        auto report = [&]() {
            std::lock_guard<std::mutex> lock(vcycleMutex());
            for (int b = 0; b < cap && b < VC_BUCKETS && out; ++b) {
                const int v = vcycleTable()[b];
                out[b] = v > 0 ? v : MG_COARSE_STOP_REF;
            }
            if (out && cap > VC_BUCKETS) out[VC_BUCKETS] = kMixed ? vcycleSweeps() : 2;
        };
        if (!kMixed || nscn() == 0) { report(); return PHX_OK; }
        PHX_TRY(ensureTables());
        PHX_CK(cudaStreamSynchronize(st));
        // the batch's state: every scenario's main arena (fields, solve vectors, scalars)
        size_t snapBytes = 0;
        for (auto& S : sc) snapBytes += S->mainBytes;
        char* snap = nullptr;
        if (cudaMalloc(&snap, snapBytes) != cudaSuccess) {
            cudaGetLastError();
            err = "device allocation of the tuner's state copy failed";
            return PHX_ERR_OOM;
        }
        auto copyState = [&](bool save) -> int {
            size_t o = 0;
            for (auto& S : sc) {
                if (save) PHX_CK(cudaMemcpyAsync(snap + o, S->arena, S->mainBytes, cudaMemcpyDeviceToDevice, st));
                else PHX_CK(cudaMemcpyAsync(S->arena, snap + o, S->mainBytes, cudaMemcpyDeviceToDevice, st));
                o += S->mainBytes;
            }
            return PHX_OK;
        };
        // host descriptors: the swap state of the double buffers is part of the state
        std::vector<Scn<R>> hostSaved;
        for (auto& S : sc) hostSaved.push_back(S->h);
        auto restoreHost = [&]() {
            for (int i = 0; i < nscn(); ++i) {
                Scn<R>& h = sc[i]->h;
                const Scn<R>& o = hostSaved[i];
                h.u = o.u; h.v = o.v; h.w = o.w; h.u2 = o.u2; h.v2 = o.v2; h.w2 = o.w2;
                h.lit = o.lit; h.lit2 = o.lit2;
                for (int q = 0; q < NSC; ++q) { h.sc[q] = o.sc[q]; h.sc2[q] = o.sc2[q]; }
            }
        };
        int r = copyState(true);
        std::vector<long long> bucketCells(VC_BUCKETS, 0);
        for (auto& S : sc) bucketCells[vcycleBucket(S->geo.N())] += S->geo.N();
        std::vector<int> order;
        for (int b = 0; b < VC_BUCKETS; ++b) if (bucketCells[b] > 0) order.push_back(b);
        std::sort(order.begin(), order.end(), [&](int a, int b) { return bucketCells[a] > bucketCells[b]; });
        const int cands[] = {MG_COARSE_STOP_REF, 1000, 500};
        auto trial = [&](double* ms) -> int {
            PHX_TRY(copyState(false));
            restoreHost();
            tablesDirty = true;
            PHX_TRY(step(1, dtMax, nullptr, nullptr));
            double t = 0;
            int nl = 0;
            PHX_TRY(timeSteps(steps, dtMax, 0, &t, &nl));
            *ms = t;
            return PHX_OK;
        };
        // the coarse levels' smoothing first, one schedule for the batch (two Jacobi
        // sweeps per level and leg, the reference's, or one; PHX_COARSE_SWEEPS=1|2
        // fixes it), then the coarsening stop per size bucket
        auto setSweeps = [&](int v) {
            std::lock_guard<std::mutex> lock(vcycleMutex());
            vcycleSweeps() = v;
        };
        if (r == PHX_OK) {
            const char* fixed = std::getenv("PHX_COARSE_SWEEPS");
            if (fixed && (std::atoi(fixed) == 1 || std::atoi(fixed) == 2)) {
                setSweeps(std::atoi(fixed));
            } else {
                double ms2 = 0, ms1 = 0;
                setSweeps(2);
                r = trial(&ms2);
                if (r == PHX_OK) {
                    setSweeps(1);
                    r = trial(&ms1);
                }
                setSweeps(r == PHX_OK && ms1 < ms2 ? 1 : 2);
            }
        }
        for (int b : order) {
            if (r != PHX_OK) break;
            int best = MG_COARSE_STOP_REF;
            double bestMs = 1e300;
            for (int c : cands) {
                for (auto& S : sc)
                    if (vcycleBucket(S->geo.N()) == b && (r = S->rebuildLevels(st, c)) != PHX_OK) { err = S->err; break; }
                if (r != PHX_OK) break;
                double ms = 0;
                if ((r = trial(&ms)) != PHX_OK) break;
                if (ms < bestMs) { bestMs = ms; best = c; }
            }
            if (r != PHX_OK) break;
            for (auto& S : sc)
                if (vcycleBucket(S->geo.N()) == b && (r = S->rebuildLevels(st, best)) != PHX_OK) { err = S->err; break; }
            std::lock_guard<std::mutex> lock(vcycleMutex());
            vcycleTable()[b] = best;
        }
        const int back = copyState(false);   // also after a failure: the trials have stepped the fields
        if (r == PHX_OK) r = back;
        restoreHost();
        tablesDirty = true;
        cudaStreamSynchronize(st);
        cudaFree(snap);
        if (r != PHX_OK) return r;
        report();
        return checkDeviceError();
    }

    // one bounded wait that nothing satisfies: the failure path of a solve's wait that
    // runs out (error word, host report, context still usable)
    int selftestWait(double limitMs) override {
        if (!(limitMs > 0) || limitMs > 1000) { err = "self-test limit must be in (0, 1000] ms"; return PHX_ERR_INVALID; }
        PHX_TRY(ensureTables());
        PHX_TRY(initStream());
        int dev = 0, khz = 0;
        PHX_CK(cudaGetDevice(&dev));
        PHX_CK(cudaDeviceGetAttribute(&khz, cudaDevAttrClockRate, dev));
        const long long cycles = (long long)(limitMs * (double)std::max(khz, 1000000));
        k_selftest_wait<R><<<1, 32, 0, st>>>(dErr, reinterpret_cast<const unsigned long long*>(dErr + 2), cycles);
        PHX_CK(cudaGetLastError());
        PHX_CK(cudaStreamSynchronize(st));
        return checkDeviceError();
    }

    // the viewer's volume ray march for scenario s (src/render/renderer.cpp:119-283)
    struct VolWork {
        float4* vol = nullptr;
        size_t capVol = 0;
        uint8_t* bricks = nullptr;
        size_t capBricks = 0;
        float* depth = nullptr;
        float* rgb = nullptr;
        size_t capPix = 0;
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        double lastMs = 0;
        void release() {
            if (vol) cudaFree(vol);
            if (bricks) cudaFree(bricks);
            if (depth) cudaFree(depth);
            if (rgb) cudaFree(rgb);
            if (e0) cudaEventDestroy(e0);
            if (e1) cudaEventDestroy(e1);
        }
    } volw;

    int volRender(int s, const phx_vol_params* p, const float* depth, float* rgb) override {
        PHX_TRY(checkScn(s));
        if (!p || !rgb || p->width <= 0 || p->height <= 0 || (size_t)p->width * p->height > (size_t)1 << 26 ||
            p->n_lights < 0 || p->n_lights > 8 || !(p->step > 0)) {
            err = "invalid volume render parameters";
            return PHX_ERR_INVALID;
        }
        const Scenario<R>& S = *sc[s];
        const size_t N = (size_t)S.geo.nx * S.geo.ny * S.geo.nz, npx = (size_t)p->width * p->height;
        PHX_TRY(ensureTables());
        PHX_TRY(initStream());
        auto alloc = [&](auto*& ptr, size_t& cap, size_t n, size_t esz) -> int {
            if (ptr && cap >= n) return PHX_OK;
            if (ptr) { PHX_CK(cudaStreamSynchronize(st)); cudaFree(ptr); ptr = nullptr; cap = 0; }
            void* q = nullptr;
            if (cudaMalloc(&q, n * esz) != cudaSuccess) {
                cudaGetLastError();
                err = "out of device memory for the volume render";
                return PHX_ERR_OOM;
            }
            ptr = static_cast<std::remove_reference_t<decltype(ptr)>>(q);
            cap = n;
            return PHX_OK;
        };
        PHX_TRY(alloc(volw.vol, volw.capVol, N, sizeof(float4)));
        VolGrid G;
        G.bx = (S.geo.nx + VOL_BRICK - 1) / VOL_BRICK;
        G.by = (S.geo.ny + VOL_BRICK - 1) / VOL_BRICK;
        const size_t nBricks = (size_t)G.bx * G.by * ((S.geo.nz + VOL_BRICK - 1) / VOL_BRICK);
        PHX_TRY(alloc(volw.bricks, volw.capBricks, nBricks, 1));
        if (volw.capPix < npx || !volw.rgb) {
            size_t c1 = volw.capPix, c2 = volw.capPix;
            PHX_TRY(alloc(volw.rgb, c1, npx, 3 * sizeof(float)));
            PHX_TRY(alloc(volw.depth, c2, npx, sizeof(float)));
            volw.capPix = npx;
        }
        if (!volw.e0) { PHX_CK(cudaEventCreate(&volw.e0)); PHX_CK(cudaEventCreate(&volw.e1)); }
        if (depth) PHX_CK(cudaMemcpyAsync(volw.depth, depth, npx * sizeof(float), cudaMemcpyHostToDevice, st));
        G.vol = volw.vol;
        G.bricks = volw.bricks;
        G.nx = S.geo.nx; G.ny = S.geo.ny; G.nz = S.geo.nz;
        const float dxf = (float)S.geo.dx;
        G.bmin = v3((float)S.geo.ox, (float)S.geo.oy, (float)S.geo.oz);
        G.bmax = v3((float)S.geo.ox + G.nx * dxf, (float)S.geo.oy + G.ny * dxf, (float)S.geo.oz + G.nz * dxf);
        PHX_CK(cudaEventRecord(volw.e0, st));
        PHX_CK(cudaMemsetAsync(volw.bricks, 0, nBricks, st));
        k_vol_pack<R><<<(unsigned)((N + 255) / 256), 256, 0, st>>>(dS, s, volw.vol, volw.bricks, G.bx, G.by, p->smoke_scale);
        dim3 grid((p->width + 15) / 16, (p->height + 7) / 8);
        k_vol_render<R><<<grid, 128, 0, st>>>(G, *p, depth ? volw.depth : nullptr, volw.rgb);
        PHX_CK(cudaGetLastError());
        PHX_CK(cudaEventRecord(volw.e1, st));
        PHX_CK(cudaMemcpyAsync(rgb, volw.rgb, npx * 3 * sizeof(float), cudaMemcpyDeviceToHost, st));
        PHX_CK(cudaStreamSynchronize(st));
        float ms = 0;
        PHX_CK(cudaEventElapsedTime(&ms, volw.e0, volw.e1));
        volw.lastMs = ms;
        return checkDeviceError();
    }
    double volLastMs() const override { return volw.lastMs; }

    int readTimes(double* out) override {
        const int n = nscn();
        if (n == 0) return PHX_OK;
        PHX_TRY(ensureTables());
        k_read_times<R><<<(n + 127) / 128, 128, 0, st>>>(dS, n, dTimes);
        ++launches;
        PHX_CK(cudaMemcpyAsync(out, dTimes, n * sizeof(double), cudaMemcpyDeviceToHost, st));
        PHX_CK(cudaStreamSynchronize(st));
        return checkDeviceError();
    }

    int removeScenario(int s) override {
        if (s < 0 || s >= nscn()) { err = "no such scenario"; return PHX_ERR_INVALID; }
        PHX_CK(cudaStreamSynchronize(st));
        sc.erase(sc.begin() + s);
        tablesDirty = true;
        return PHX_OK;
    }

    int scenarioCount() const override { return nscn(); }
    size_t scenarioBytes(int s) const override { return s >= 0 && s < nscn() ? sc[s]->arenaBytes : 0; }

    // batch tables: descriptors, domain prefixes, CG buffers; invalidates the graph
    int rebuildTables() {
        destroyGraph();
        const int n = nscn();
        if (n > cap || !tab) {
            if (tab) { PHX_CK(cudaStreamSynchronize(st)); cudaFree(tab); tab = nullptr; }
            cap = std::max(n, std::max(1, cap * 2));
            char* base = nullptr;
            for (int pass = 0; pass < 2; ++pass) {
                size_t off = 0;
                dS = carve<Scn<R>>(base, off, cap);
                dDomStart = carve<int>(base, off, (size_t)D_COUNT * (cap + 1));
                dDtMax = carve<double>(base, off, cap);
                dErr = carve<unsigned>(base, off, 4);
                dTimes = carve<double>(base, off, cap);
                dMaxPart = carve<double>(base, off, 2 * MAX_SOLVE_CTAS);
                teams.ctas = carve<SolveCta>(base, off, MAX_SOLVE_CTAS);
                teams.next = carve<int>(base, off, cap);
                teams.work = carve<float2>(base, off, cap);
                teams.arrived = carve<unsigned>(base, off, 4);
                if (pass == 0) {
                    cudaError_t e = cudaMalloc(&tab, off + 256);
                    if (e != cudaSuccess) { tab = nullptr; err = "device allocation of the batch tables failed"; return PHX_ERR_OOM; }
                    PHX_CK(cudaMemsetAsync(tab, 0, off + 256, st));
                    base = tab;
                }
            }
        }
        std::vector<int> starts((size_t)D_COUNT * (n + 1), 0);
        std::vector<int> tilesAll((size_t)D_COUNT * cap, 0);
        anyLeak = false;
        {
            std::lock_guard<std::mutex> lock(vcycleMutex());
            smoothOne = kMixed && vcycleSweeps() == 1;
        }
        int t[D_COUNT];
        for (int s = 0; s < n; ++s) {
            Scenario<R>& S = *sc[s];
            S.tiles(t);
            for (int d = 0; d < D_COUNT; ++d) {
                starts[(size_t)d * (n + 1) + s + 1] = starts[(size_t)d * (n + 1) + s] + t[d];
                tilesAll[(size_t)d * cap + s] = t[d];
            }
            anyLeak |= !S.leak.empty();
            S.h.dtMaxArg = dDtMax + s;
            S.h.errWord = dErr;
            S.h.smooth1 = smoothOne ? 1 : 0;
        }
        // per domain, the scenario and tile of every CTA (packed 11 + 20 bits)
        size_t ownTotal = 0;
        bool packable = true;
        for (int d = 0; d < D_COUNT; ++d) {
            ownTotal += (size_t)starts[(size_t)d * (n + 1) + n];
            for (int s = 0; s < n; ++s) packable &= tilesAll[(size_t)d * cap + s] < (1 << 20);
        }
        std::vector<unsigned> own;
        if (packable && n <= 2048) {
            own.reserve(ownTotal);
            for (int d = 0; d < D_COUNT; ++d)
                for (int s = 0; s < n; ++s)
                    for (int t = 0; t < tilesAll[(size_t)d * cap + s]; ++t) own.push_back(((unsigned)s << 20) | (unsigned)t);
            if (own.size() > ownCap) {
                if (ownTab) { PHX_CK(cudaStreamSynchronize(st)); cudaFree(ownTab); ownTab = nullptr; ownCap = 0; }
                if (cudaMalloc(&ownTab, own.size() * sizeof(unsigned)) != cudaSuccess) {
                    ownTab = nullptr;
                    err = "device allocation of the CTA owner tables failed";
                    return PHX_ERR_OOM;
                }
                ownCap = own.size();
            }
            if (!own.empty())
                PHX_CK(cudaMemcpyAsync(ownTab, own.data(), own.size() * sizeof(unsigned), cudaMemcpyHostToDevice, st));
        }
        size_t ownOff = 0;
        for (int d = 0; d < D_COUNT; ++d) {
            dom[d].start = dDomStart + (size_t)d * (n + 1);
            dom[d].nscn = n;
            dom[d].total = starts[(size_t)d * (n + 1) + n];
            dom[d].owner = own.empty() ? nullptr : ownTab + ownOff;
            ownOff += (size_t)dom[d].total;
        }
        PHX_CK(cudaMemcpyAsync(dDomStart, starts.data(), starts.size() * sizeof(int), cudaMemcpyHostToDevice, st));
        tablesDirty = false;
        for (int s = 0; s < n; ++s) PHX_TRY(pushDescriptor(s, false));
        if (n > 0) k_wind<R><<<dom[D_ONE].total, 128, 0, st>>>(dS, dom[D_ONE]);
        PHX_CK(cudaStreamSynchronize(st));
        return n > 0 ? setupSolve() : PHX_OK;
    }

    // the solve kernel's grid: every CTA resident, since its teams wait on one
    // another. PHX_PERSIST_CTAS caps it (tests: several scenarios per CTA)
    static constexpr int MAX_SOLVE_CTAS = 1024;
    int setupSolve() {
        int dev = 0, sms = 0, occ[2] = {0, 0};
        PHX_CK(cudaGetDevice(&dev));
        PHX_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        auto fit = [&](auto per) -> cudaError_t {
            constexpr int PER = decltype(per)::value;
            using Cfg = SolveCfg<R, PER>;
            const cudaError_t e = cudaFuncSetAttribute(k_solve<R, PER>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM);
            return e != cudaSuccess ? e : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ[PER - 1], k_solve<R, PER>, Cfg::T, Cfg::SMEM);
        };
        PHX_CK(fit(std::integral_constant<int, 1>{}));
        if constexpr (kMixed) PHX_CK(fit(std::integral_constant<int, 2>{}));
        if (occ[0] < 1) { err = "the solve kernel does not fit an SM"; return PHX_ERR_CUDA; }
        solvePer = occ[1] >= 2 ? solvePerSm<R>(nscn(), sms) : 1;
        solveGrid = std::min(sms * (solvePer == 2 ? 2 : occ[0]), MAX_SOLVE_CTAS);
        // no more than all scenarios can use, so that contexts share the GPU, but half the SMs:
        // a smaller grid's CTAs are placed otherwise, and its steps take 2 to 3 % longer (medians of
        // 12 contexts below 76 CTAs / from there: closet FP64 0.410 / 0.402 ms, room FP32
        // 0.535 / 0.520). CTAs without work leave at once.
        long long usable = 0;
        for (auto& S : sc) usable += solveCtas<R>(solveTiling<R>(S->blocks()));
        solveGrid = (int)std::min<long long>(solveGrid, std::max<long long>(usable, sms / 2));
        if (const char* c = std::getenv("PHX_PERSIST_CTAS")) solveGrid = std::max(1, std::min(solveGrid, std::atoi(c)));
        teams.grid = solveGrid;
        return PHX_OK;
    }

    int ensureTables() { return tablesDirty ? rebuildTables() : PHX_OK; }

    int pushDescriptor(int s, bool sync = true) {
        Scenario<R>& S = *sc[s];
        S.h.nsrc = (int)(S.ignitions.size() + S.burners.size());
        int q = 0;
        for (auto& x : S.ignitions) S.h.src[q++] = x;
        for (auto& x : S.burners) S.h.src[q++] = x;
        if (tablesDirty) return PHX_OK;   // uploaded with the tables
        PHX_CK(cudaMemcpyAsync(dS + s, &S.h, sizeof(Scn<R>), cudaMemcpyHostToDevice, st));
        if (sync) PHX_CK(cudaStreamSynchronize(st));
        return PHX_OK;
    }

    int checkScn(int s) {
        if (s < 0 || s >= nscn()) { err = "no such scenario"; return PHX_ERR_INVALID; }
        return PHX_OK;
    }

    // ---- sources ------------------------------------------------------------------
    int addBurner(int s, double x0, double y0, double x1, double y1, double z, double peakW, double rampS,
                  double start, double duration, int* index) override {
        if (index) *index = -1;
        PHX_TRY(checkScn(s));
        Scenario<R>& S = *sc[s];
        std::vector<int> cells = burnerCells(S.geo, x0, y0, x1, y1, z);
        if (cells.empty()) { err = "burner covers no gas cell"; return PHX_ERR_INVALID; }
        if ((int)(S.ignitions.size() + S.burners.size()) >= MAX_SRC) { err = "too many burners and ignitions (16)"; return PHX_ERR_INVALID; }
        Src b{};
        b.kind = 1;
        b.i0 = b.j0 = 1 << 30; b.i1 = b.j1 = -1; b.k = -1;
        for (int c : cells) {
            int i = c % S.geo.nx, j = (c / S.geo.nx) % S.geo.ny, k = c / (S.geo.nx * S.geo.ny);
            b.i0 = std::min(b.i0, i); b.i1 = std::max(b.i1, i); b.j0 = std::min(b.j0, j); b.j1 = std::max(b.j1, j);
            if (b.k >= 0 && b.k != k) { err = "burner cells span several layers"; return PHX_ERR_UNSUPPORTED; }
            b.k = k;
        }
        // the device selects the unblocked cells of the box: check that this is the same set
        size_t inBox = 0;
        for (int j = b.j0; j <= b.j1; ++j)
            for (int i = b.i0; i <= b.i1; ++i) inBox += !S.geo.blocked[S.geo.cell(i, j, b.k)];
        if (inBox != cells.size()) { err = "burner cells do not form a box of gas cells"; return PHX_ERR_UNSUPPORTED; }
        b.ncells = (int)cells.size();
        b.peakW = peakW; b.rampS = rampS; b.start = start; b.duration = duration;
        S.burners.push_back(b);
        if (index) *index = (int)S.burners.size() - 1;
        return pushDescriptor(s);
    }

    int addIgnition(int s, int cell, double power, double duration) override {
        PHX_TRY(checkScn(s));
        Scenario<R>& S = *sc[s];
        if (cell < 0 || cell >= S.geo.N()) return PHX_OK;   // the reference ignores it
        if ((int)(S.ignitions.size() + S.burners.size()) >= MAX_SRC) { err = "too many burners and ignitions (16)"; return PHX_ERR_INVALID; }
        PHX_CK(cudaMemcpyAsync(hPin, S.h.sv + SV_TIME, sizeof(double), cudaMemcpyDeviceToHost, st));
        PHX_CK(cudaStreamSynchronize(st));
        Src x{};
        x.kind = 0;
        x.i0 = x.i1 = cell % S.geo.nx; x.j0 = x.j1 = (cell / S.geo.nx) % S.geo.ny; x.k = cell / (S.geo.nx * S.geo.ny);
        x.ncells = 1;
        x.power = power; x.start = hPin[0]; x.duration = duration;
        S.ignitions.push_back(x);
        return pushDescriptor(s);
    }

    // ---- launch helpers -------------------------------------------------------------
    bool prof = false;
    std::vector<cudaEvent_t> evPool;
    std::vector<std::pair<const char*, int>> evUse;   // (kernel name, first event index)
    int evNext = 0;
    struct KStat { std::string name; int launches = 0; double ms = 0; };
    std::vector<KStat> kstats;
    void* flushBuf = nullptr;
    size_t flushBytes = 0;

    template <class K, class... A>
    void launch(const char* name, int d, int threads, K kern, A... args) {
        if (dom[d].total <= 0) return;
        if (prof) {
            if (evNext + 2 > (int)evPool.size()) {
                for (int i = 0; i < 64; ++i) { cudaEvent_t e; cudaEventCreate(&e); evPool.push_back(e); }
            }
            cudaEventRecord(evPool[evNext], st);
            kern<<<dom[d].total, threads, 0, st>>>(args...);
            cudaEventRecord(evPool[evNext + 1], st);
            evUse.push_back({name, evNext});
            evNext += 2;
        } else {
            kern<<<dom[d].total, threads, 0, st>>>(args...);
        }
        ++launches;
    }

    // the same with every CTA's tile split over `split` smaller CTAs
    template <class K, class... A>
    void launchSplit(const char* name, int d, int split, int threads, K kern, A... args) {
        const int total = dom[d].total;
        dom[d].total = total * split;
        launch(name, d, threads, kern, args...);
        dom[d].total = total;
    }

    // the device error word: a bounded wait inside a kernel that ran out
    int checkDeviceError() {
        if (!dErr) return PHX_OK;
        unsigned w = 0;
        PHX_CK(cudaMemcpyAsync(&w, dErr, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
        PHX_CK(cudaStreamSynchronize(st));
        if (w) {
            // report once and clear, so that the context stays usable
            PHX_CK(cudaMemsetAsync(dErr, 0, sizeof(unsigned), st));
            PHX_CK(cudaStreamSynchronize(st));
            err = (w & ERR_SELFTEST) ? "a bounded device wait ran out (self-test, device error word " + std::to_string(w) + ")"
                                     : "a CTA of the pressure solve waited too long for its team; the step's results are not "
                                       "valid (device error word " + std::to_string(w) + ")";
            return PHX_ERR_TIMEOUT;
        }
        return PHX_OK;
    }

    int collectProfile() {
        PHX_CK(cudaStreamSynchronize(st));
        for (auto& u : evUse) {
            float ms = 0;
            cudaEventElapsedTime(&ms, evPool[u.second], evPool[u.second + 1]);
            KStat* k = nullptr;
            for (auto& x : kstats) if (x.name == u.first) k = &x;
            if (!k) { kstats.push_back(KStat{u.first, 0, 0}); k = &kstats.back(); }
            k->launches++;
            k->ms += ms;
        }
        evUse.clear();
        evNext = 0;
        return PHX_OK;
    }

    void swapHost(int what) {
        for (auto& S : sc) {
            Scn<R>& h = S->h;
            if (what & 1) std::swap(h.lit, h.lit2);
            if (what & 2) { std::swap(h.u, h.u2); std::swap(h.v, h.v2); std::swap(h.w, h.w2); }
            if (what & 4) for (int q = 0; q < NSC; ++q) std::swap(h.sc[q], h.sc2[q]);
        }
    }
    void swapBoth(int what) {
        launch("k_swap", D_ONE, 32, k_swap<R>, dS, dom[D_ONE], what);
        swapHost(what);
    }

    int setDtMax(double dtMax, const double* per) {
        std::vector<double> v(nscn(), dtMax);
        if (per) for (int s = 0; s < nscn(); ++s) v[s] = per[s];
        // pageable source: staged at the call, safe to reuse at once
        if (!v.empty()) PHX_CK(cudaMemcpyAsync(dDtMax, v.data(), v.size() * sizeof(double), cudaMemcpyHostToDevice, st));
        return PHX_OK;
    }

    // ---- stages ---------------------------------------------------------------------
    void stBegin(bool computeDt, double dt) {
        launch("k_begin", D_ONE, TEAM_TPB, k_begin<R>, (const Scn<R>*)dS, dom[D_ONE], computeDt ? 1 : 0, dt, teams);
    }
    // Stages. In the full step the double buffers are exchanged by kernels that do not
    // read them (turbulence: the burning flags; energy: the velocities, ahead of
    // momentum; the end of the step: the scalars); a stage on its own (alone) does it
    // by k_swap, so that its result is in place when it returns.
    void stCombustion(bool alone) {
        launch("k_combust", D_CELLS, TPB, k_combust<R>, (const Scn<R>*)dS, dom[D_CELLS]);
        if (alone) swapBoth(1);
    }
    void stTurbulence(bool alone) {
        const Scn<R>* S = dS;
        launch("k_turb_x", D_CELLS, TPB, k_turb_x<R>, S, dom[D_CELLS], alone ? nullptr : dS);
        if (!alone) swapHost(1);
        launch("k_turb_y", D_CELLS, TPB, k_turb_y<R>, S, dom[D_CELLS]);
        launch("k_turb_nu", D_CELLS, TPB, k_turb_nu<R>, S, dom[D_CELLS]);
    }
    void stHeat() {
        launch("k_heat", D_CELLS, TPB, k_heat<R>, (const Scn<R>*)dS, dom[D_CELLS]);
    }
    // FP64, a stage on its own: the density the full step's earlier kernels leave behind
    void stDensity() {
        if (!kMixed) launch("k_rho", D_CELLS, TPB, k_rho<R>, (const Scn<R>*)dS, dom[D_CELLS]);
    }
    void stEnergy(bool alone) {
        launch("k_energy", D_CELLS, TPB, k_energy<R>, (const Scn<R>*)dS, dom[D_CELLS], alone ? nullptr : dS);
        if (!alone) swapHost(2);
    }
    void stMomentum(bool alone) {
        if (alone) swapBoth(2);
        launch("k_momentum", D_FACES, TPB, k_momentum<R>, (const Scn<R>*)dS, dom[D_FACES]);
        launch("k_mom_bnd", D_BND, TPB, k_mom_bnd<R>, (const Scn<R>*)dS, dom[D_BND]);
    }
    void stLeakage() {
        launch("k_zone_integral", D_CZ, TPB, k_zone_integral<R>, (const Scn<R>*)dS, dom[D_CZ]);
        if (anyLeak) {
            launch("k_leak_faces", D_LEAK, TPB, k_leak_faces<R>, (const Scn<R>*)dS, dom[D_LEAK]);
            launch("k_leak_finish", D_CZ, TPB, k_leak_finish<R>, (const Scn<R>*)dS, dom[D_CZ]);
        }
    }
    // the whole pressure solve in one cooperative launch (solve.cuh)
    int launchSolve(int vcycleOnly) {
        SolveArgs a;
        a.teams = teams;
        a.cap = maxItersAll() + 2;
        a.vcycleOnly = vcycleOnly;
        a.maxPart = dMaxPart;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)solveGrid);
        constexpr int PER2 = kMixed ? 2 : 1;
        const bool two = solvePer == 2;
        cfg.blockDim = dim3(two ? SolveCfg<R, PER2>::T : SolveCfg<R, 1>::T);
        cfg.dynamicSmemBytes = two ? SolveCfg<R, PER2>::SMEM : SolveCfg<R, 1>::SMEM;
        cfg.stream = st;
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeCooperative;
        at.val.cooperative = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        const Scn<R>* S = dS;
        int e0 = -1;
        if (prof) {
            if (evNext + 2 > (int)evPool.size()) {
                for (int i = 0; i < 64; ++i) { cudaEvent_t e; cudaEventCreate(&e); evPool.push_back(e); }
            }
            e0 = evNext;
            evNext += 2;
            cudaEventRecord(evPool[e0], st);
        }
        PHX_CK(two ? cudaLaunchKernelEx(&cfg, k_solve<R, PER2>, S, a) : cudaLaunchKernelEx(&cfg, k_solve<R, 1>, S, a));
        if (prof) {
            cudaEventRecord(evPool[e0 + 1], st);
            evUse.push_back({"k_solve", e0});
        }
        ++launches;
        return PHX_OK;
    }
    // right-hand side (and the mixed path's initial guess), then the solve
    int solveStage() {
        const Scn<R>* S = dS;
        if (kMixed) launch("k_mx_extrap", D_CELLS, TPB, k_mx_extrap<R>, S, dom[D_CELLS]);
        launch("k_rhs", D_CELLS, TPB, k_rhs<R>, S, dom[D_CELLS]);
        return launchSolve(0);
    }
    // zone mean removal and velocity correction (:629-676)
    void projectEpilogue() {
        const Scn<R>* S = dS;
        launch("k_zone_mean", D_CZ, TPB, k_zone_mean<R>, S, dom[D_CZ]);
        launch("k_zone_mean_sub", D_CC, TPB, k_zone_mean_sub<R>, S, dom[D_CC]);
        launch("k_velcorr", D_FACES, TPB, k_velcorr<R>, S, dom[D_FACES]);
    }
    int maxItersAll() const {
        int m = 0;
        for (auto& S : sc) m = std::max(m, S->maxIters);
        return m;
    }

    int stProject() {
        PHX_TRY(solveStage());
        projectEpilogue();
        return PHX_OK;
    }
    void stAdvect(bool alone) {
        launchSplit("k_advect", D_CELLS, TPB / ADV_TPB<R>, ADV_TPB<R>, k_advect<R>, (const Scn<R>*)dS, dom[D_CELLS]);
        if (alone) swapBoth(4);
    }
    void stEnd(bool alone) {
        const Scn<R>* S = dS;
        launch("k_zone_pressure", D_ONE, 32, k_zone_pressure<R>, S, dom[D_ONE], alone ? nullptr : dS);
        if (!alone) swapHost(4);
        launch("k_zone_pb", D_CC, TPB, k_zone_pb<R>, S, dom[D_CC]);
        launch("k_stats", D_CELLS, TPB, k_stats<R>, S, dom[D_CELLS]);
    }

    int checkLaunch() {
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) { err = std::string("kernel launch: ") + cudaGetErrorString(e); return PHX_ERR_CUDA; }
        return PHX_OK;
    }

    // ---- captured step graph -----------------------------------------------------------
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t gexec = nullptr;
    int graphKernels = 0;        // kernel nodes of the step graph
    // the step runs as one CUDA graph; PHX_NO_GRAPH=1 launches the same kernels
    // one by one
    bool useGraph = std::getenv("PHX_NO_GRAPH") == nullptr;

    void destroyGraph() {
        if (gexec) cudaGraphExecDestroy(gexec);
        if (graph) cudaGraphDestroy(graph);
        gexec = nullptr;
        graph = nullptr;
    }

    int buildGraph() {
        destroyGraph();
        std::vector<Scn<R>> saved;
        for (auto& S : sc) saved.push_back(S->h);
        PHX_CK(cudaGraphCreate(&graph, 0));
        PHX_CK(cudaStreamBeginCaptureToGraph(st, graph, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
        launches = 0;
        stBegin(true, 0.0);
        stCombustion(false);
        stTurbulence(false);
        stHeat();
        stEnergy(false);
        stMomentum(false);
        stLeakage();
        PHX_TRY(stProject());
        stAdvect(false);
        stEnd(false);
        cudaGraph_t done = nullptr;
        PHX_CK(cudaStreamEndCapture(st, &done));
        graphKernels = launches;
        for (int s = 0; s < nscn(); ++s) sc[s]->h = saved[s];
        PHX_CK(cudaGraphInstantiate(&gexec, graph, 0));
        return checkLaunch();
    }

    int graphStep(double dtMax, const double* per) {
        if (!gexec) PHX_TRY(buildGraph());
        PHX_TRY(setDtMax(dtMax, per));
        PHX_CK(cudaGraphLaunch(gexec, st));
        swapHost(1 | 2 | 4);
        return PHX_OK;
    }

    int oneStep(double dtMax, const double* per = nullptr) {
        PHX_TRY(ensureTables());
        if (nscn() == 0) return PHX_OK;
        if (useGraph && !prof) return graphStep(dtMax, per);
        PHX_TRY(setDtMax(dtMax, per));
        stBegin(true, 0.0);
        stCombustion(false);
        stTurbulence(false);
        stHeat();
        stEnergy(false);
        stMomentum(false);
        stLeakage();
        PHX_TRY(stProject());
        stAdvect(false);
        stEnd(false);
        return checkLaunch();
    }

    int step(int n, double dtMax, const double* per, double* dtOut) override {
        for (int i = 0; i < n; ++i) {
            launches = 0;
            PHX_TRY(oneStep(dtMax, per));
            if (dtOut) {
                const int m = nscn();
                for (int s = 0; s < m; ++s)
                    PHX_CK(cudaMemcpyAsync(hPin + 16 + s % 4000, sc[s]->h.sv + SV_DT, sizeof(double), cudaMemcpyDeviceToHost, st));
                PHX_CK(cudaStreamSynchronize(st));
                if (per) for (int s = 0; s < m; ++s) dtOut[(size_t)i * m + s] = hPin[16 + s % 4000];
                else dtOut[i] = hPin[16];
                PHX_TRY(checkDeviceError());
            }
        }
        return PHX_OK;
    }

    int stage(int which, double arg) override {
        PHX_TRY(ensureTables());
        switch (which) {
        case PHX_STAGE_BEGIN: PHX_TRY(setDtMax(arg, nullptr)); stBegin(true, 0.0); break;
        case PHX_STAGE_COMBUSTION: stBegin(false, arg); stCombustion(true); break;
        case PHX_STAGE_TURBULENCE: stTurbulence(true); break;
        case PHX_STAGE_HEAT: stBegin(false, arg); stDensity(); stHeat(); break;
        case PHX_STAGE_ENERGY: stBegin(false, arg); stEnergy(true); break;
        case PHX_STAGE_MOMENTUM: stBegin(false, arg); stDensity(); stMomentum(true); break;
        case PHX_STAGE_LEAKAGE: stBegin(false, arg); stLeakage(); break;
        case PHX_STAGE_PROJECT: stBegin(false, arg); PHX_TRY(stProject()); break;
        case PHX_STAGE_ADVECT: stBegin(false, arg); stDensity(); stAdvect(true); break;
        case PHX_STAGE_END: stBegin(false, arg); stEnd(true); break;
        default: err = "unknown stage"; return PHX_ERR_INVALID;
        }
        PHX_TRY(checkLaunch());
        PHX_CK(cudaStreamSynchronize(st));
        return PHX_OK;
    }

    // z = M^-1 r with one V-cycle of the multigrid (single-scenario contexts)
    int precondition(const double* r, double* z) override {
        PHX_TRY(ensureTables());
        if (nscn() != 1) { err = "precondition needs a single-scenario context"; return PHX_ERR_STATE; }
        Scenario<R>& S = *sc[0];
        const int N = S.geo.N();
        PHX_TRY(S.put(st, S.h.r, std::vector<double>(r, r + N)));
        k_reset<R><<<1, TEAM_TPB, 0, st>>>(dS, teams);
        PHX_TRY(launchSolve(1));
        PHX_TRY(checkLaunch());
        return getReal(S.h.z, N, z);
    }

    // ---- fields -----------------------------------------------------------------------
    int getReal(const R* src, size_t n, double* out) {
        if (std::is_same<R, double>::value) {
            PHX_CK(cudaMemcpyAsync(out, src, n * sizeof(double), cudaMemcpyDeviceToHost, st));
            PHX_CK(cudaStreamSynchronize(st));
            return PHX_OK;
        }
        PHX_CK(cudaMemcpyAsync(upperHalf(out, n), src, n * sizeof(R), cudaMemcpyDeviceToHost, st));
        PHX_CK(cudaStreamSynchronize(st));
        widenUpperHalf(out, n);
        return PHX_OK;
    }
    // A caller's n doubles take the device's n reals in their upper half first and are
    // widened from the front: number i is read before anything that covers it is written
    // (8 i + 8 <= 4 n + 4 i + 4 for every i < n), block by block through a copy on the
    // stack. No second array whose pages are touched for the first time on every call
    // (a trace's C call over 1.3e6 cells, with the walls' bitmap instead of a sort: 3.1 -> 2.2 ms).
    static void* upperHalf(double* out, size_t n) { return reinterpret_cast<char*>(out) + n * (sizeof(double) - sizeof(R)); }
    static void widenUpperHalf(double* out, size_t n) {
        constexpr size_t B = 1024;
        R part[B];
        for (size_t i = 0; i < n; i += B) {
            const size_t m = std::min(B, n - i);
            std::memcpy(part, static_cast<char*>(upperHalf(out, n)) + i * sizeof(R), m * sizeof(R));
            for (size_t q = 0; q < m; ++q) out[i + q] = (double)part[q];
        }
    }

    bool fieldPtr(int s, int f, void** p, size_t* n, int* type) const {
        if (s < 0 || s >= nscn()) return false;
        const Scenario<R>& S = *sc[s];
        const Scn<R>& h = S.h;
        const size_t N = S.geo.N(), NX = S.geo.NX(), NY = S.geo.NY(), NZ = S.geo.NZ();
        *type = 0;
        switch (f) {
        case PHX_FIELD_U: *p = h.u; *n = NX; return true;
        case PHX_FIELD_V: *p = h.v; *n = NY; return true;
        case PHX_FIELD_W: *p = h.w; *n = NZ; return true;
        case PHX_FIELD_P: *p = h.p; *n = N; return true;
        case PHX_FIELD_S: *p = h.S; *n = N; return true;
        case PHX_FIELD_NU: *p = h.nu; *n = N; return true;
        case PHX_FIELD_PB: *p = h.Pb; *n = N; return true;
        case PHX_FIELD_Q: *p = h.Q; *n = N; return true;
        case PHX_FIELD_QR: *p = h.Qr; *n = N; return true;
        case PHX_FIELD_HRR: *p = h.hrr; *n = N; return true;
        case PHX_FIELD_MASSSRC: *p = h.massSrc; *n = N; return true;
        case PHX_FIELD_RHS: *p = h.b; *n = N; return true;
        case PHX_FIELD_CGR: *p = h.r; *n = N; return true;
        case PHX_FIELD_CGZ: *p = h.z; *n = N; return true;
        case PHX_FIELD_LIT: *p = h.lit; *n = N; *type = 1; return true;
        case PHX_FIELD_ZONE: *p = (void*)h.zone; *n = N; *type = 2; return true;
        case PHX_FIELD_ZONEP: *p = (void*)h.zoneP; *n = S.Z.zoneP.size(); *type = 3; return true;
        default:
            if (f >= PHX_FIELD_T && f <= PHX_FIELD_YAI) { *p = h.sc[f - PHX_FIELD_T]; *n = N; return true; }
            return false;
        }
    }

    size_t fieldCount(int s, int f) const override {
        void* p;
        size_t n;
        int t;
        return fieldPtr(s, f, &p, &n, &t) ? n : 0;
    }

    int getField(int s, int f, void* host, size_t bytes) override {
        void* p;
        size_t n;
        int t;
        if (!fieldPtr(s, f, &p, &n, &t)) { err = "unknown field or scenario"; return PHX_ERR_INVALID; }
        size_t want = n * (t == 0 || t == 3 ? sizeof(double) : t == 1 ? 1 : 4);
        if (bytes != want) { err = "field size mismatch: expected " + std::to_string(want) + " bytes"; return PHX_ERR_INVALID; }
        if (kMixed && f == PHX_FIELD_P) {   // the FP64 pressure of the refinement loop
            PHX_CK(cudaMemcpyAsync(host, sc[s]->h.p64, bytes, cudaMemcpyDeviceToHost, st));
            PHX_CK(cudaStreamSynchronize(st));
            return PHX_OK;
        }
        if (t == 0) {
            PHX_TRY(getReal((const R*)p, n, (double*)host));
            if (tempIsOffset<R>() && f == PHX_FIELD_T)   // the stored offset back to kelvin, in FP64
                for (size_t i = 0; i < n; ++i) ((double*)host)[i] = tKFromStoredd<R>(((double*)host)[i]);
            return PHX_OK;
        }
        PHX_CK(cudaMemcpyAsync(host, p, bytes, cudaMemcpyDeviceToHost, st));
        PHX_CK(cudaStreamSynchronize(st));
        return PHX_OK;
    }

    int setField(int s, int f, const void* host, size_t bytes) override {
        void* p;
        size_t n;
        int t;
        if (!fieldPtr(s, f, &p, &n, &t) || f == PHX_FIELD_ZONE) { err = "unknown or read-only field"; return PHX_ERR_INVALID; }
        size_t want = n * (t == 0 || t == 3 ? sizeof(double) : t == 1 ? 1 : 4);
        if (bytes != want) { err = "field size mismatch: expected " + std::to_string(want) + " bytes"; return PHX_ERR_INVALID; }
        Scenario<R>& S = *sc[s];
        if (t == 0) {
            const double* d = (const double*)host;
            if (kMixed && f == PHX_FIELD_P) {
                PHX_TRY(S.putRaw(st, S.h.p64, d, n));
                const double zero = 0;   // the previous step's pressure no longer applies
                PHX_CK(cudaMemcpyAsync(S.h.sv + SV_HAVEPREV, &zero, sizeof(double), cudaMemcpyHostToDevice, st));
                PHX_CK(cudaStreamSynchronize(st));
            }
            std::vector<double> v(d, d + n);
            if (tempIsOffset<R>() && f == PHX_FIELD_T)   // kelvin to the stored offset, in FP64
                for (auto& x : v) x = tStoredFromKd<R>(x);
            return S.put(st, (R*)p, v);
        }
        PHX_CK(cudaMemcpyAsync(p, host, bytes, cudaMemcpyHostToDevice, st));
        PHX_CK(cudaStreamSynchronize(st));
        return PHX_OK;
    }

    int getStats(int s, phx_stats* o) override {
        PHX_TRY(checkScn(s));
        PHX_CK(cudaMemcpyAsync(hPin + 4096, sc[s]->h.sv, SV_COUNT * sizeof(double), cudaMemcpyDeviceToHost, st));
        PHX_CK(cudaStreamSynchronize(st));
        const double* sv = hPin + 4096;
        o->time = sv[SV_TIME]; o->dt = sv[SV_DT];
        o->max_vel = sv[SV_MAXVEL]; o->max_nu = sv[SV_MAXNU]; o->max_div = sv[SV_MAXDIV];
        o->pressure_iters = (int)sv[SV_IT];
        o->pressure_residual = sv[SV_PRES]; o->pressure_rel_residual = sv[SV_PREL];
        o->hrr = sv[SV_HRR]; o->max_gas_t = sv[SV_MAXGAST]; o->burning_cells = (int)sv[SV_BURNING];
        o->fuel_in = sv[SV_FUELIN]; o->fuel_burned = sv[SV_FUELBURNED]; o->fuel_in_domain = sv[SV_FUELINDOMAIN];
        o->zones = (int)sc[s]->Z.zoneP.size(); o->leak_faces = (int)sc[s]->leak.size() / 4;
        return PHX_OK;
    }

    int setScalars(int s, double time, double maxVel, double maxNu, double maxDiv) override {
        PHX_TRY(checkScn(s));
        double v[4] = {time, maxVel, maxNu, maxDiv};
        double* sv = sc[s]->h.sv;
        PHX_CK(cudaMemcpyAsync(sv + SV_TIME, &v[0], sizeof(double), cudaMemcpyHostToDevice, st));
        PHX_CK(cudaMemcpyAsync(sv + SV_MAXVEL, &v[1], sizeof(double), cudaMemcpyHostToDevice, st));
        PHX_CK(cudaMemcpyAsync(sv + SV_MAXNU, &v[2], sizeof(double), cudaMemcpyHostToDevice, st));
        PHX_CK(cudaMemcpyAsync(sv + SV_MAXDIV, &v[3], sizeof(double), cudaMemcpyHostToDevice, st));
        PHX_CK(cudaStreamSynchronize(st));
        return PHX_OK;
    }

    // the scalar slots a checkpoint restores (src/sim/state.cpp:144-145,186)
    int setStats(int s, const phx_stats* in) override {
        PHX_TRY(checkScn(s));
        const int slot[10] = {SV_TIME, SV_MAXVEL, SV_MAXNU, SV_MAXDIV, SV_HRR, SV_MAXGAST, SV_BURNING,
                              SV_FUELIN, SV_FUELBURNED, SV_FUELINDOMAIN};
        const double v[10] = {in->time, in->max_vel, in->max_nu, in->max_div, in->hrr, in->max_gas_t,
                              (double)in->burning_cells, in->fuel_in, in->fuel_burned, in->fuel_in_domain};
        double* sv = sc[s]->h.sv;
        for (int q = 0; q < 10; ++q)
            PHX_CK(cudaMemcpyAsync(sv + slot[q], &v[q], sizeof(double), cudaMemcpyHostToDevice, st));
        PHX_CK(cudaStreamSynchronize(st));
        return PHX_OK;
    }

    size_t deviceBytes() const override {
        size_t b = 0;
        for (auto& S : sc) b += S->arenaBytes;
        return b;
    }
    int sync() override {
        if (st) PHX_CK(cudaStreamSynchronize(st));
        return checkDeviceError();
    }
    int deviceView(int s, const void** descriptor, int* cells, void** stream) override {
        PHX_TRY(checkScn(s));
        if (tablesDirty || !dS) {
            // building the tables would allocate: the caller steps (or syncs) the context first
            err = "the context's device tables are not built yet: step the context once after adding scenarios";
            return PHX_ERR_STATE;
        }
        *descriptor = dS + s;
        *cells = sc[s]->geo.N();
        *stream = (void*)st;
        return PHX_OK;
    }
    int mgInfo(int s, int* levels, int* rows, int cap) override {
        PHX_TRY(checkScn(s));
        const Multigrid& M = sc[s]->MG;
        if (levels) *levels = (int)M.lv.size();
        for (int l = 0; rows && l < cap && l < (int)M.lv.size(); ++l) rows[l] = M.lv[l].n;
        return PHX_OK;
    }
    int mgNnz(int s, int* nnz, int cap) override {
        PHX_TRY(checkScn(s));
        const Multigrid& M = sc[s]->MG;
        for (int l = 0; nnz && l < cap && l < (int)M.lv.size(); ++l)
            nnz[l] = M.lv[l].rowStart.empty() ? 0 : M.lv[l].rowStart.back();
        return PHX_OK;
    }
    int lastLaunches() const override {
        if (useGraph && gexec) return graphKernels;
        return launches;
    }

    // n steps timed with CUDA events on the context's stream; with flushL2 a
    // buffer larger than L2 is written (untimed) before each step
    int timeSteps(int n, double dtMax, int flushL2, double* totalMs, int* launchesOut) override {
        PHX_TRY(ensureTables());
        if (flushL2 && !flushBuf) {
            flushBytes = (size_t)512 << 20;
            PHX_CK(cudaMalloc(&flushBuf, flushBytes));
        }
        PHX_CK(cudaStreamSynchronize(st));
        double total = 0;
        int nl = 0;
        for (int i = 0; i < n; ++i) {
            if (flushL2) PHX_CK(cudaMemsetAsync(flushBuf, i & 0xff, flushBytes, st));
            PHX_CK(cudaEventRecord(ev[0], st));
            launches = 0;
            PHX_TRY(oneStep(dtMax));
            PHX_CK(cudaEventRecord(ev[1], st));
            PHX_CK(cudaEventSynchronize(ev[1]));
            float ms = 0;
            PHX_CK(cudaEventElapsedTime(&ms, ev[0], ev[1]));
            total += ms;
            nl += useGraph ? graphKernels : launches;
        }
        if (totalMs) *totalMs = total;
        if (launchesOut) *launchesOut = nl;
        return checkDeviceError();
    }

    // one step with an event pair around every launch; per-kernel totals
    int profileStep(double dtMax, int flushL2, phx_kernel_time* out, int cap_, int* count) override {
        PHX_TRY(ensureTables());
        if (flushL2) {
            if (!flushBuf) { flushBytes = (size_t)512 << 20; PHX_CK(cudaMalloc(&flushBuf, flushBytes)); }
            PHX_CK(cudaMemsetAsync(flushBuf, 0x5a, flushBytes, st));
        }
        kstats.clear();
        prof = true;
        launches = 0;
        int r = oneStep(dtMax);
        prof = false;
        PHX_TRY(r);
        PHX_TRY(collectProfile());
        int n = 0;
        for (auto& k : kstats) {
            if (n < cap_ && out) {
                std::memset(&out[n], 0, sizeof(phx_kernel_time));
                std::strncpy(out[n].name, k.name.c_str(), sizeof(out[n].name) - 1);
                out[n].launches = k.launches;
                out[n].ms = k.ms;
            }
            ++n;
        }
        if (count) *count = n;
        return PHX_OK;
    }
};

#undef PHX_TRY
}  // namespace phx
