// nb_tile.cuh -- the mixed-precision pair term over unordered pairs: 64 x 64
// body tiles whose j side rotates through the lanes of a warp.
//
// A sum over ordered pairs evaluates a pair's displacement, r^2 and r^-3 twice,
// once for each body.  Here a warp holds a tile of 64 i-bodies (two per lane)
// and meets a tile of 64 j-bodies, two at a time as an f32x2 pair: at step s
// lane l meets j-bodies (l + s) mod 32 and 32 + (l + s) mod 32, adds the pair
// terms to its own bodies' sums in registers and to the j-bodies' running sums,
// which move one lane down per step by shuffles.  Per unordered pair the far
// term costs 17 FP32 lane operations and the near one 26, where ordered pairs
// cost 2 x 12 and 2 x 21; two MUFU operations become one.  The FP32 pipe bounds the
// loop (34 packed operations, 68 cycles, per step against 50 issue slots).
//
// Rounding is as in the sums over ordered pairs: 16 terms per f32x2 lane in
// plain FP32, then a Kahan-compensated add -- after every 16 steps on the i side
// (one term per lane and step) and every 8 on the j side (two).  The Kahan pairs
// live in shared memory (the registers they would take cost more), the j side's
// indexed by the j-body the lane holds then.
#pragma once

#include "nb_pair.cuh"

namespace nb {

constexpr int kTile = 64;  // bodies per tile

// A staged j-tile: index l holds bodies l and 32 + l side by side.
struct TileJ {
    float4 a[32];  // (x_l, x_32+l, y_l, y_32+l)
    float4 b[32];  // (z_l, z_32+l, m_l, m_32+l)
    float4 c[32];  // low parts of x and y
    float2 d[32];  // low parts of z
};

// Sums of a tile, one f32x2 per component and index (bodies l and 32 + l): Kahan
// sum and the negated compensation (so that only additions are needed).
struct TileSums {
    float2 s[3][32], c[3][32];
};

// The warp's i-tile: body 32 k + lane in k = 0, 1, coordinates negated and
// duplicated.
struct TileI {
    float2 nx[2], ny[2], nz[2];     // high parts
    float2 ex[2], ey[2], ez[2];     // low parts
    float2 nm[2];                   // negated mass
};

__device__ __forceinline__ void tile_sums_zero(TileSums &t, int lane)
{
#pragma unroll
    for (int c = 0; c < 3; ++c) t.s[c][lane] = t.c[c][lane] = dup2(0.f);
}

__device__ __forceinline__ void tile_i_set(TileI &t, int k, float x, float y, float z, float xl,
                                           float yl, float zl, float m)
{
    t.nx[k] = dup2(-x); t.ny[k] = dup2(-y); t.nz[k] = dup2(-z);
    t.ex[k] = dup2(-xl); t.ey[k] = dup2(-yl); t.ez[k] = dup2(-zl);
    t.nm[k] = dup2(-m);
}

// Lane `lane` stages body 32 k + lane of a j-tile (between two __syncwarp).
__device__ __forceinline__ void tile_j_put(TileJ &t, int lane, int k, float x, float y, float z,
                                           float xl, float yl, float zl, float m)
{
    float *a = reinterpret_cast<float *>(&t.a[lane]) + k;
    float *b = reinterpret_cast<float *>(&t.b[lane]) + k;
    float *c = reinterpret_cast<float *>(&t.c[lane]) + k;
    a[0] = x;
    a[2] = y;
    b[0] = z;
    b[2] = m;
    c[0] = xl;
    c[2] = yl;
    reinterpret_cast<float *>(&t.d[lane])[k] = zl;
}

// (sum, negated compensation) += t, four packed additions.
__device__ __forceinline__ void kahan_add2(float2 &s, float2 &nc, float2 t)
{
    const float2 y = add2(t, nc);
    const float2 u = add2(s, y);
    const float2 lost = fma2(u, dup2(-1.f), s);  // s - u, exact: one rounding as s + (-u)
    nc = add2(y, lost);
    s = u;
}

// One step: the lane's two i-bodies against the staged j-pair idx.  NEAR takes the
// double-single displacement and the folded Newton step (pair_term2), else the
// plain FP32 term (pair_term2_far<false>).  BOTH = false adds to the i side
// only.  The scale m r^-3 is built as (m y) y^2 for each side, not from a shared
// y^3, so that lengths of 1e13 and more (y^3 below FP32's range) still work.
template <bool NEAR, bool ZERO_SOFT, bool BOTH>
__device__ __forceinline__ void tile_step(const TileJ &t, int idx, const TileI &ti, float2 e2,
                                          float2 (&fi)[2][3], float2 (&fj)[3])
{
    const float4 A = t.a[idx], B = t.b[idx];
    float4 C = make_float4(0.f, 0.f, 0.f, 0.f);
    float2 D = make_float2(0.f, 0.f);
    if (NEAR) {
        C = t.c[idx];
        D = t.d[idx];
    }
    const float2 jx = make_float2(A.x, A.y), jy = make_float2(A.z, A.w),
                 jz = make_float2(B.x, B.y), jm = make_float2(B.z, B.w);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        float2 dx = add2(jx, ti.nx[k]), dy = add2(jy, ti.ny[k]), dz = add2(jz, ti.nz[k]);
        if (NEAR) {
            dx = add2(dx, add2(make_float2(C.x, C.y), ti.ex[k]));
            dy = add2(dy, add2(make_float2(C.z, C.w), ti.ey[k]));
            dz = add2(dz, add2(D, ti.ez[k]));
        }
        const float2 r2 = fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, e2)));
        float2 inv = make_float2(rsqrt_mufu(r2.x), rsqrt_mufu(r2.y));
        if (NEAR && ZERO_SOFT) {
            inv.x = r2.x > 0.f ? inv.x : 0.f;
            inv.y = r2.y > 0.f ? inv.y : 0.f;
        }
        float2 w = mul2(inv, inv);
        if (NEAR) w = mul2(w, fma2(dup2(-1.5f), mul2(r2, w), dup2(2.5f)));
        const float2 si = mul2(mul2(jm, inv), w);
        fi[k][0] = fma2(dx, si, fi[k][0]);
        fi[k][1] = fma2(dy, si, fi[k][1]);
        fi[k][2] = fma2(dz, si, fi[k][2]);
        if (BOTH) {
            const float2 sj = mul2(mul2(ti.nm[k], inv), w);
            fj[0] = fma2(dx, sj, fj[0]);
            fj[1] = fma2(dy, sj, fj[1]);
            fj[2] = fma2(dz, sj, fj[2]);
        }
    }
}

__device__ __forceinline__ void tile_fold_i(TileSums &is, int lane, float2 (&fi)[2][3])
{
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        kahan_add2(is.s[c][lane], is.c[c][lane],
                   make_float2(fi[0][c].x + fi[0][c].y, fi[1][c].x + fi[1][c].y));
        fi[0][c] = fi[1][c] = dup2(0.f);
    }
}

// Steps [8 g0, 8 g1) of the i-tile against a staged j-tile (g1 = 4: the whole
// pair of tiles).  is, js: the sums of either side, this warp's alone.
template <bool NEAR, bool ZERO_SOFT>
__device__ __forceinline__ void tile_pair(const TileJ &t, int lane, int g0, int g1, const TileI &ti,
                                          float2 e2, TileSums &is, TileSums &js)
{
    const int next = (lane + 1) & 31;
    float2 fi[2][3];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int c = 0; c < 3; ++c) fi[k][c] = dup2(0.f);
#pragma unroll 1
    for (int g = g0; g < g1; ++g) {
        float2 fj[3] = {dup2(0.f), dup2(0.f), dup2(0.f)};
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            tile_step<NEAR, ZERO_SOFT, true>(t, (lane + 8 * g + u) & 31, ti, e2, fi, fj);
            if (u < 7)
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    fj[c] = make_float2(__shfl_sync(0xffffffffu, fj[c].x, next),
                                        __shfl_sync(0xffffffffu, fj[c].y, next));
        }
        const int idx = (lane + 8 * g + 7) & 31;
#pragma unroll
        for (int c = 0; c < 3; ++c) kahan_add2(js.s[c][idx], js.c[c][idx], fj[c]);
        if ((g & 1) || g + 1 == g1) tile_fold_i(is, lane, fi);
        __syncwarp();  // the next group's fold takes other lanes' entries
    }
}

// A tile with itself (staged in t): every ordered pair, the i side only.
template <bool ZERO_SOFT>
__device__ __forceinline__ void tile_self(const TileJ &t, int lane, int g0, int g1, const TileI &ti,
                                          float2 e2, TileSums &is)
{
    float2 fi[2][3], none[3];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int c = 0; c < 3; ++c) fi[k][c] = dup2(0.f);
#pragma unroll 1
    for (int g = g0; g < g1; ++g) {
#pragma unroll 4
        for (int u = 0; u < 8; ++u)
            tile_step<true, ZERO_SOFT, false>(t, (lane + 8 * g + u) & 31, ti, e2, fi, none);
        if ((g & 1) || g + 1 == g1) tile_fold_i(is, lane, fi);
    }
}

} // namespace nb
