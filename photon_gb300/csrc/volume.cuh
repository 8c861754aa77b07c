// Smoke and flame volume ray march of Photon's viewer (the VOL_FS fragment
// shader, src/render/renderer.cpp:119-283, over the volume uploadVolume packs,
// src/app/viewer.cpp:941-949) as a CUDA kernel writing an RGB image into a
// device buffer: no window, no GL. One thread per pixel; the volume is one
// float4 per cell (soot density, aerosol density, T, heat release), sampled
// trilinearly with clamp-to-edge addressing as the shader's GL_LINEAR 3D
// texture is. The scene behind the volume is a constant background colour
// with an optional depth buffer (the opaque pass's colour and depth
// textures). All arithmetic is FP32, as in the shader.
#pragma once
#include "phx_dev.cuh"

namespace phx {

struct V3 { float x, y, z; };
__host__ __device__ __forceinline__ V3 v3(float a, float b, float c) { return {a, b, c}; }
__host__ __device__ __forceinline__ V3 operator+(V3 a, V3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__host__ __device__ __forceinline__ V3 operator-(V3 a, V3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__host__ __device__ __forceinline__ V3 operator*(V3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
__host__ __device__ __forceinline__ V3 operator*(V3 a, V3 b) { return {a.x * b.x, a.y * b.y, a.z * b.z}; }

// floor for |x| < 2^22: x + 1.5 * 2^23 rounded down has no fraction bits left, and its low
// bits are the integer. Two additions at full rate; the rounding and conversion
// instructions of floorf and (int) run at an eighth of it and bounded the march.
constexpr float V_ROUND = 12582912.0f;
constexpr float V_SMALL = 4194304.0f;
__device__ __forceinline__ float vFloorSmall(float x) { return __fadd_rd(x, V_ROUND) - V_ROUND; }

// GLSL built-ins (GLSL 3.30 definitions)
__device__ __forceinline__ float vFract(float x) { return x - floorf(x); }
__device__ __forceinline__ float vClamp(float x, float a, float b) { return fminf(fmaxf(x, a), b); }
__device__ __forceinline__ float vMix(float a, float b, float t) { return a * (1.0f - t) + b * t; }
__device__ __forceinline__ V3 vMix(V3 a, V3 b, float t) { return a * (1.0f - t) + b * t; }
__device__ __forceinline__ float vSmooth(float e0, float e1, float x) {
    float t = vClamp((x - e0) / (e1 - e0), 0.0f, 1.0f);
    return t * t * (3.0f - 2.0f * t);
}
__device__ __forceinline__ float vDot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

__device__ __forceinline__ V3 vHeatmap(float t) {
    t = vClamp(t, 0.0f, 1.0f);
    const V3 c0 = v3(0.10f, 0.15f, 0.55f), c1 = v3(0.10f, 0.65f, 0.85f), c2 = v3(0.95f, 0.90f, 0.20f),
             c3 = v3(0.95f, 0.35f, 0.05f), c4 = v3(0.85f, 0.05f, 0.05f);
    if (t < 0.25f) return vMix(c0, c1, t / 0.25f);
    if (t < 0.5f) return vMix(c1, c2, (t - 0.25f) / 0.25f);
    if (t < 0.75f) return vMix(c2, c3, (t - 0.5f) / 0.25f);
    return vMix(c3, c4, (t - 0.75f) / 0.25f);
}
__device__ __forceinline__ V3 vGlow(float T) {
    float t = vClamp((T - 700.0f) / 1000.0f, 0.0f, 1.0f);
    return v3(1.0f, 0.22f + 0.6f * t, 0.04f + 0.45f * t * t) * t * t;
}
// the fraction of a large product: where its sum is contracted (FP32 context) decides
// every pixel's dither, so the operations are written out
template <bool FUSED>
__device__ __forceinline__ float vHash2(float px, float py) {
    const float b = __fmul_rn(py, 78.233f), a = FUSED ? fmaf(px, 12.9898f, b) : __fadd_rn(__fmul_rn(px, 12.9898f), b);
    return vFract(__fmul_rn(sinf(a), 43758.5453f));
}
// the shader's hash3 of a lattice point takes each coordinate through the same function
// first, so a cube's eight points need it six times, not 24. SMALL: every coordinate is
// below V_SMALL (a point's hash argument always is: 17^3 * 51)
template <bool SMALL>
__device__ __forceinline__ float vFloor(float x) { return SMALL ? vFloorSmall(x) : floorf(x); }
template <bool SMALL>
__device__ __forceinline__ float vHashAxis(float c) {
    const float x = c * 0.3183099f + 0.1f;
    return (x - vFloor<SMALL>(x)) * 17.0f;
}
template <bool SMALL>
__device__ __forceinline__ float vNoise(V3 x) {
    const V3 i = v3(vFloor<SMALL>(x.x), vFloor<SMALL>(x.y), vFloor<SMALL>(x.z));
    V3 f = v3(x.x - i.x, x.y - i.y, x.z - i.z);
    f = v3(f.x * f.x * (3.0f - 2.0f * f.x), f.y * f.y * (3.0f - 2.0f * f.y), f.z * f.z * (3.0f - 2.0f * f.z));
    const float x0 = vHashAxis<SMALL>(i.x), x1 = vHashAxis<SMALL>(i.x + 1.0f), y0 = vHashAxis<SMALL>(i.y),
                y1 = vHashAxis<SMALL>(i.y + 1.0f), z0 = vHashAxis<SMALL>(i.z), z1 = vHashAxis<SMALL>(i.z + 1.0f);
    auto point = [](float a, float b, float c) {
        const float h = a * b * c * (a + b + c);
        return h - vFloorSmall(h);
    };
    auto line = [&](float y, float z) { return vMix(point(x0, y, z), point(x1, y, z), f.x); };
    return vMix(vMix(line(y0, z0), line(y1, z0), f.y), vMix(line(y0, z1), line(y1, z1), f.y), f.z);
}
template <bool SMALL>
__device__ __forceinline__ float vFlameNoiseAt(V3 p, float time) {
    const V3 q = p * v3(5.0f, 5.0f, 2.6f) - v3(0.0f, 0.0f, time * 3.2f);
    return 0.55f * vNoise<SMALL>(q) + 0.30f * vNoise<SMALL>(q * 2.1f + v3(0.0f, 0.0f, -time * 2.0f)) + 0.15f * vNoise<SMALL>(q * 4.3f);
}
template <bool SMALL>
__device__ __forceinline__ float vSmokeNoiseAt(V3 p, float time) {
    V3 q = p * 1.6f - v3(0.0f, 0.0f, time * 0.35f);
    q = q + (v3(vNoise<SMALL>(q + v3(5.2f, 1.3f, 0.0f)), vNoise<SMALL>(q + v3(1.7f, 9.2f, 3.1f)), vNoise<SMALL>(q + v3(8.3f, 2.8f, 4.7f))) * 0.6f -
             v3(0.3f, 0.3f, 0.3f));
    float n = 0.5f * vNoise<SMALL>(q) + 0.3f * vNoise<SMALL>(q * 2.03f + v3(1.7f, 1.7f, 1.7f)) + 0.2f * vNoise<SMALL>(q * 4.1f + v3(3.3f, 3.3f, 3.3f));
    return vSmooth(0.2f, 0.8f, n);
}
// far from the origin or late: floorf
inline __device__ __noinline__ float vFlameNoiseFar(V3 p, float time) { return vFlameNoiseAt<false>(p, time); }
inline __device__ __noinline__ float vSmokeNoiseFar(V3 p, float time) { return vSmokeNoiseAt<false>(p, time); }
// every coordinate above stays within V_SMALL: at most 21.5 |p| + 14 |time| + 20. The test is on
// p and not on q, whose products are contracted into the noise's own additions
__device__ __forceinline__ bool vNear(V3 p, float time) {
    return fmaxf(fmaxf(fabsf(p.x), fabsf(p.y)), fmaxf(fabsf(p.z), fabsf(time))) < V_SMALL / 64.0f;
}
__device__ __forceinline__ float vFlameNoise(V3 p, float time) {
    return vNear(p, time) ? vFlameNoiseAt<true>(p, time) : vFlameNoiseFar(p, time);
}
__device__ __forceinline__ float vSmokeNoise(V3 p, float time) {
    return vNear(p, time) ? vSmokeNoiseAt<true>(p, time) : vSmokeNoiseFar(p, time);
}
__device__ __forceinline__ V3 vFlameColor(float k) {
    return vMix(vMix(v3(0.9f, 0.18f, 0.02f), v3(1.0f, 0.5f, 0.08f), vSmooth(0.0f, 0.4f, k)), v3(1.0f, 0.9f, 0.55f),
                vSmooth(0.45f, 1.0f, k));
}

// cells per side of a brick: bricks whose samples cannot add anything to a pixel are marked
// when the volume is packed, and the march steps over them
constexpr int VOL_BRICK = 4;
struct VolGrid {
    const float4* vol;
    const uint8_t* bricks;   // 1: something there
    int bx, by;              // bricks per row, rows per plane
    int nx, ny, nz;
    V3 bmin, bmax;
};
// x / d for a d whose reciprocal y is rounded to nearest: two of Markstein's correction
// steps ("Computation of elementary functions on the IBM RISC System/6000 processor", IBM
// J. Res. Dev. 34(1), 1990), the IEEE quotient in five operations without a branch (numbers
// in the normal range; below it the last bit may differ)
__device__ __forceinline__ float vDivBy(float x, float d, float y) {
    float q = x * y;
    q = fmaf(fmaf(-q, d, x), y, q);
    return fmaf(fmaf(-q, d, x), y, q);
}
// the box's extents and their reciprocals, once per thread
struct VolBox {
    V3 ext, rcp;
    __device__ __forceinline__ explicit VolBox(const VolGrid& G)
        : ext(G.bmax - G.bmin), rcp(v3(1.0f / ext.x, 1.0f / ext.y, 1.0f / ext.z)) {}
};
__device__ __forceinline__ float2 vLerp(float2 a, float2 b, float t) {
    return make_float2(a.x * (1.0f - t) + b.x * t, a.y * (1.0f - t) + b.y * t);
}
__device__ __forceinline__ float4 vLerp(float4 a, float4 b, float t) {
    return make_float4(a.x * (1.0f - t) + b.x * t, a.y * (1.0f - t) + b.y * t, a.z * (1.0f - t) + b.z * t,
                       a.w * (1.0f - t) + b.w * t);
}
// where a sample lies: its lower corner (may be outside the grid) and the position between
// the corners. A sample lies in the box or a few shadow steps beyond it, so well within
// V_SMALL cells.
struct VolAt {
    int i, j, k;
    float ax, ay, az;
    __device__ __forceinline__ VolAt(const VolGrid& G, const VolBox& B, V3 p) {
        const V3 u = v3(vDivBy(p.x - G.bmin.x, B.ext.x, B.rcp.x), vDivBy(p.y - G.bmin.y, B.ext.y, B.rcp.y),
                        vDivBy(p.z - G.bmin.z, B.ext.z, B.rcp.z));
        const float x = u.x * G.nx - 0.5f, y = u.y * G.ny - 0.5f, z = u.z * G.nz - 0.5f;
        const float fx = __fadd_rd(x, V_ROUND), fy = __fadd_rd(y, V_ROUND), fz = __fadd_rd(z, V_ROUND);
        ax = x - (fx - V_ROUND);
        ay = y - (fy - V_ROUND);
        az = z - (fz - V_ROUND);
        i = __float_as_int(fx) - __float_as_int(V_ROUND);
        j = __float_as_int(fy) - __float_as_int(V_ROUND);
        k = __float_as_int(fz) - __float_as_int(V_ROUND);
    }
};
__device__ __forceinline__ int vEdge(int v, int n) { return min(max(v, 0), n - 1); }
// texture(uVol, (p - boxMin) / (boxMax - boxMin)) with GL_LINEAR, CLAMP_TO_EDGE; V = float2:
// its first two channels
template <class V>
__device__ __forceinline__ V vSample(const VolGrid& G, const VolAt& at) {
    const int i0 = vEdge(at.i, G.nx), i1 = vEdge(at.i + 1, G.nx), j0 = vEdge(at.j, G.ny), j1 = vEdge(at.j + 1, G.ny),
              k0 = G.ny * vEdge(at.k, G.nz), k1 = G.ny * vEdge(at.k + 1, G.nz);
    auto line = [&](int row) {   // a grid has fewer than 2^31 cells
        return vLerp(__ldg(reinterpret_cast<const V*>(G.vol + (G.nx * row + i0))),
                     __ldg(reinterpret_cast<const V*>(G.vol + (G.nx * row + i1))), at.ax);
    };
    const V c00 = line(j0 + k0), c10 = line(j1 + k0), c01 = line(j0 + k1), c11 = line(j1 + k1);
    return vLerp(vLerp(c00, c10, at.ay), vLerp(c01, c11, at.ay), at.az);
}

// uploadVolume (src/app/viewer.cpp:941-949): soot and aerosol density, T, heat release.
// A cell that can change a pixel marks the bricks of every sample it is a corner of (lower
// corner i or i - 1 in each direction). It cannot where its smoke is thinner than the
// shader's 0.02 threshold, it is colder than the 700 K at which smoke begins to glow and its
// heat release drives less than the 0.01 of a flame: an interpolated value lies between its
// corners', and each bound leaves more than that interpolation's rounding. A NaN marks.
template <class R>
__global__ void k_vol_pack(const Scn<R>* __restrict__ S, int s, float4* __restrict__ vol, uint8_t* __restrict__ bricks,
                           int bx, int by, float smokeScale) {
    const Scn<R>& g = S[s];
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= g.N) return;
    float4 v = make_float4(0, 0, 0, 0);
    if (!g.blocked[c]) {
        const float T = (float)tAbs(g.sc[0][c]);
        const float rho = (float)g.Pb[c] / (287.0f * T);
        v = make_float4((float)g.sc[3][c] * rho, (float)g.sc[4][c] * rho, T, (float)g.hrr[c]);
    }
    vol[c] = v;
    const float sigma = (8700.0f * fmaxf(v.x, 0.0f) + 3000.0f * fmaxf(v.y, 0.0f)) * smokeScale;
    if (sigma <= 0.0199f && v.z <= 699.0f && v.w <= 11000.0f && v.x == v.x && v.y == v.y) return;
    int i, j, k;
    ijkOf(g, 0, c, i, j, k);
    const int i0 = max(i - 1, 0) / VOL_BRICK, j0 = max(j - 1, 0) / VOL_BRICK, k0 = max(k - 1, 0) / VOL_BRICK;
    for (int bk = k0; bk <= k / VOL_BRICK; ++bk)
        for (int bj = j0; bj <= j / VOL_BRICK; ++bj)
            for (int bi = i0; bi <= i / VOL_BRICK; ++bi) bricks[bi + bx * (bj + by * bk)] = 1;
}

// the fragment shader's main(), one thread per pixel; rgb rows from the bottom
// (GL window order). R is the engine's precision; the render is FP32 in both.
// Bound by instruction issue (0.74 of the active cycles, 29.5 of 32 lanes; 98 % of the
// loads hit L1). A 1280x720 frame of a 72x52x44 house with smoke in a fifth of its cells,
// pack and march, ms: 1.76; a cube's hashes shared, the phase function taken out of the
// loop, terms that are 0 not evaluated, divisions by the box in five operations, two
// channels for the shadow samples 1.17; floors in additions 1.08; empty bricks stepped
// over 0.93.
template <class R>
__global__ void __launch_bounds__(128) k_vol_render(VolGrid G, phx_vol_params P, const float* __restrict__ depth,
                                                    float* __restrict__ rgb) {
    // 16x8 pixels a CTA, 8x4 a warp: its rays stay together longer than 16x2's
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int px = blockIdx.x * 16 + (warp & 1) * 8 + (lane & 7), py = blockIdx.y * 8 + (warp >> 1) * 4 + (lane >> 3);
    if (px >= P.width || py >= P.height) return;
    const float uvx = (px + 0.5f) / P.width, uvy = (py + 0.5f) / P.height;
    const float* M = P.inv_vp;
    auto worldAt = [&](float d) {
        const float a = uvx * 2.0f - 1.0f, b = uvy * 2.0f - 1.0f, c = d * 2.0f - 1.0f;
        const float X = M[0] * a + M[4] * b + M[8] * c + M[12], Y = M[1] * a + M[5] * b + M[9] * c + M[13];
        const float Z = M[2] * a + M[6] * b + M[10] * c + M[14], W = M[3] * a + M[7] * b + M[11] * c + M[15];
        return v3(X / W, Y / W, Z / W);
    };
    const V3 base = v3(P.background[0], P.background[1], P.background[2]);
    const float d = depth ? depth[(size_t)py * P.width + px] : 1.0f;
    const V3 ro = v3(P.eye[0], P.eye[1], P.eye[2]);
    V3 rd = worldAt(1.0f) - ro;
    rd = rd * (1.0f / sqrtf(vDot(rd, rd)));
    const float tScene = d < 1.0f ? sqrtf(vDot(worldAt(d) - ro, worldAt(d) - ro)) : 1e9f;
    const V3 bmax = v3(G.bmax.x, G.bmax.y, fminf(G.bmax.z, P.clip_z));
    const V3 inv = v3(1.0f / rd.x, 1.0f / rd.y, 1.0f / rd.z);
    const V3 ta = (G.bmin - ro) * inv, tb = (bmax - ro) * inv;
    const V3 tmn = v3(fminf(ta.x, tb.x), fminf(ta.y, tb.y), fminf(ta.z, tb.z));
    const V3 tmx = v3(fmaxf(ta.x, tb.x), fmaxf(ta.y, tb.y), fmaxf(ta.z, tb.z));
    const float t0 = fmaxf(fmaxf(fmaxf(tmn.x, tmn.y), tmn.z), 0.0f);
    const float t1 = fminf(fminf(tmx.x, tmx.y), tmx.z);
    const float tEnd = fminf(t1, tScene);
    V3 col = v3(0, 0, 0);
    float tr = 1.0f;
    const float tS = (P.slice_z - ro.z) / rd.z;
    const bool sliceHit = P.slice == 1 && tS > t0 && tS < tEnd && P.slice_z < bmax.z;
    const V3 sun = v3(P.sun_dir[0], P.sun_dir[1], P.sun_dir[2]);
    const VolBox box(G);
    // the phase function of this ray (Henyey-Greenstein): the same at every step
    const float gg = 0.35f, ct = vDot(rd, sun);
    const float hg = (1.0f - gg * gg) / powf(1.0f + gg * gg - 2.0f * gg * ct, 1.5f) * 0.25f;
    auto slice = [&]() {
        float4 sv = vSample<float4>(G, VolAt(G, box, ro + rd * tS));
        if (sv.z > 150.0f) {
            float tn = (sv.z - P.t_min) / (P.t_max - P.t_min);
            float sa = vMix(0.12f, 0.88f, vSmooth(0.0f, 0.2f, tn));
            col = col + vHeatmap(tn) * (tr * sa);
            tr *= 1.0f - sa;
        }
    };
    bool sliceDone = !sliceHit;
    if (t0 < tEnd) {
        const float ds = P.step;
        const float jit = vHash2<sizeof(R) == 4>(px + 0.5f, py + 0.5f);
        const int n = (int)fminf(600.0f, (tEnd - t0) / ds + 1.0f);
        // steps per cell along each axis, and the cells by which a step's computed place may
        // be off (coordinates far from the origin): steps over a brick stop that far before its side
        const V3 cells = v3(G.nx / box.ext.x, G.ny / box.ext.y, G.nz / box.ext.z);
        const V3 per = v3(1.0f / fabsf(rd.x * ds * cells.x), 1.0f / fabsf(rd.y * ds * cells.y), 1.0f / fabsf(rd.z * ds * cells.z));
        auto big = [](V3 a) { return fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fabsf(a.z)); };
        const float off = 0.01f + 1e-6f * (big(ro) + big(G.bmin) + big(G.bmax) + tEnd) * big(cells);
        // steps that stay in a brick along one axis, from lower corner c (clamped: q) and position a
        auto inside = [&](int c, int q, float a, float dir, float per1, int n1) {
            const int b = q & ~(VOL_BRICK - 1);
            const float ahead = dir > 0.0f ? (float)(b + VOL_BRICK - c) - a : (float)(c - b) + a;
            const bool open = dir > 0.0f ? b + VOL_BRICK >= n1 : b == 0;   // the edge cells continue outside
            return open ? 1e6f : (ahead - off) * per1;
        };
        int i = 0;
        for (;;) {
            // to the next step that can add something
            float t = 0.0f;
            V3 p = ro;
            bool found = false;
            VolAt at(G, box, ro);
            while (i < n) {
                t = t0 + ((float)i + jit) * ds;
                if (t > tEnd) { i = n; break; }
                if (!sliceDone && t >= tS) { slice(); sliceDone = true; }
                if (P.smoke == 0 && P.fire == 0) { ++i; continue; }
                p = ro + rd * t;
                at = VolAt(G, box, p);
                const int qi = vEdge(at.i, G.nx), qj = vEdge(at.j, G.ny), qk = vEdge(at.k, G.nz);
                found = G.bricks[qi / VOL_BRICK + G.bx * (qj / VOL_BRICK + G.by * (qk / VOL_BRICK))] != 0;
                if (found) break;
                if (tr < 0.004f) { i = n; break; }
                float m = fminf(fminf(inside(at.i, qi, at.ax, rd.x, per.x, G.nx), inside(at.j, qj, at.ay, rd.y, per.y, G.ny)),
                                inside(at.k, qk, at.az, rd.z, per.z, G.nz));
                if (!sliceDone) m = fminf(m, (tS - t) / ds - 1.0f);   // the slice's own step is visited
                i += 1 + (int)fminf(fmaxf(m, 0.0f), 1e6f);
            }
            if (!found) break;
            ++i;
            const float4 v = vSample<float4>(G, at);
            const float soot = fmaxf(v.x, 0.0f), aero = fmaxf(v.y, 0.0f);
            const float sigma0 = (8700.0f * soot + 3000.0f * aero) * P.smoke_scale;
            float sigma = sigma0;
            float a = 0.0f;
            V3 scat = v3(0, 0, 0);
            if (P.smoke == 1 && sigma0 > 0.02f) {
                const float lightFrac = aero / (soot * 3.0f + aero + 1e-12f);
                const float bill = vSmokeNoise(p, P.time);
                sigma = sigma0 * vMix(0.25f, 1.75f, bill);
                a = 1.0f - expf(-sigma * ds);
                float od = 0.0f;
                for (int sh = 1; sh <= 4; ++sh) {
                    const float2 sv2 = vSample<float2>(G, VolAt(G, box, p + sun * (0.35f * (float)sh)));
                    od += (8700.0f * fmaxf(sv2.x, 0.0f) + 3000.0f * fmaxf(sv2.y, 0.0f)) * P.smoke_scale * 0.35f;
                }
                const float sunT = expf(-od);
                const V3 albedo = vMix(v3(0.10f, 0.095f, 0.09f), v3(0.86f, 0.84f, 0.78f), lightFrac);
                const float amb = 0.45f + 0.25f * vClamp((p.z - G.bmin.z) * 0.15f, 0.0f, 1.0f);
                scat = albedo * (amb * vMix(0.55f, 1.0f, sunT) + 1.6f * hg * sunT);
                scat = scat * vMix(0.85f, 1.1f, bill);
                if (P.fire == 1) {   // fire light is scattered where there is smoke (a > 0) only
                    const float alb = vMix(0.45f, 0.95f, lightFrac);
                    float fl = 0.0f;
                    for (int li = 0; li < P.n_lights; ++li) {
                        const V3 dl = v3(P.lights[li][0], P.lights[li][1], P.lights[li][2]) - p;
                        fl += P.lights[li][3] / (0.6f + vDot(dl, dl));
                    }
                    scat = scat + v3(1.0f, 0.45f, 0.15f) * fl * alb * 0.9f;
                }
            }
            V3 emit = v3(0, 0, 0);
            if (P.fire == 1) {   // terms that are 0 are not evaluated: no heat release, below 1000 K, no smoke or below 700 K
                const float hot = v.z > 1000.0f ? vSmooth(1000.0f, 1600.0f, v.z) : 0.0f;
                const float drive = (v.w > 0.0f ? vClamp(v.w / 1.0e6f * 0.9f, 0.0f, 3.0f) : 0.0f) + hot * 0.9f;
                if (drive > 0.01f) {
                    const float nn = vFlameNoise(p, P.time);
                    const float shape = vSmooth(0.62f - 0.25f * vClamp(drive, 0.0f, 1.5f), 0.85f, nn + 0.15f * fminf(drive, 1.5f));
                    const float k = vClamp(0.25f * drive + 0.6f * nn * shape, 0.0f, 1.0f);
                    emit = vFlameColor(k) * shape * drive * 6.0f;
                }
                if (v.z > 700.0f && sigma > 0.0f) emit = emit + vGlow(v.z) * vClamp(sigma * 0.6f, 0.0f, 1.0f) * 4.0f;
            }
            col = col + (scat * a + emit * ds) * tr;
            tr *= 1.0f - a;
            if (tr < 0.004f) break;
        }
        if (!sliceDone) slice();
    }
    float* o = rgb + 3 * ((size_t)py * P.width + px);
    o[0] = base.x * tr + (1.0f - expf(-col.x * 1.1f));
    o[1] = base.y * tr + (1.0f - expf(-col.y * 1.1f));
    o[2] = base.z * tr + (1.0f - expf(-col.z * 1.1f));
}

}  // namespace phx
