// nb_tile.cuh -- the mixed-precision pair term over unordered pairs: tiles of
// 64 j-bodies that rotate through the lanes of a warp.
//
// A sum over ordered pairs evaluates a pair's displacement, r^2 and r^-3 twice,
// once for each body.  Here a warp holds IPT i-bodies per lane (tiles of 64) and
// meets a tile of 64 j-bodies, two at a time as an f32x2 pair: at step s lane l
// meets j-bodies (l + s) mod 32 and 32 + (l + s) mod 32, adds the pair terms to its
// own bodies' sums in registers and to the j-bodies' running sums, which move one
// lane down per step by shuffles.  Per unordered pair the far term costs 17 FP32
// lane operations and the near one 26, where ordered pairs cost 2 x 12 and
// 2 x 21; two MUFU operations become one.
//
// What bounds the loop is dispatch, not the FP32 pipe alone.  Measured on GB300
// in cycles per warp instruction and SM quarter: a packed operation 2, but 3 when
// its three operands are all different registers; a MUFU, a shuffle and a
// shared-memory load 2 each; an integer operation about 0.6.  Four far pairs per
// lane took 110 cycles with two i-bodies per lane, 96 with four (half the
// shuffles and loads per pair, and tiles staged twice over so that no index
// wraps), 84 when the masses leave the loop (below).
//
// Equal masses.  Where all bodies of the i-tiles have one mass and all of the
// j-tile one (as in most N-body set-ups), the loop sums r^-3 d alone and each
// fold multiplies by the mass: 14 operations per far pair instead of 17, 23 per
// near one instead of 26.
//
// Rounding is as in the sums over ordered pairs: 16 terms per f32x2 lane in
// plain FP32, then a Kahan-compensated add -- after every 16 steps on the i side
// (one term per lane and step) and every 32 / (2 IPT) on the j side (IPT terms).
// The Kahan pairs live in shared memory (the registers they would take cost
// more), the j side's indexed by the j-body the lane holds then.
#pragma once

#include "nb_pair.cuh"

namespace nb {

constexpr int kTile = 64;  // bodies per tile

// A staged j-tile: index l (and 32 + l, a copy) holds bodies l and 32 + l side
// by side.
struct TileJ {
    float4 a[64];  // (x_l, x_32+l, y_l, y_32+l)
    float4 b[64];  // (z_l, z_32+l, m_l, m_32+l)
};
struct TileJLow {
    float4 c[64];  // low parts of x and y
    float2 d[64];  // low parts of z
};

// Sums of a tile, one f32x2 per component and index (bodies l and 32 + l): Kahan
// sum and the negated compensation (so that only additions are needed).
struct TileSums {
    float2 s[3][32], c[3][32];
};

// The warp's i-bodies, coordinates negated and duplicated: body 32 k + lane.
template <int IPT>
struct TileI {
    float2 nx[IPT], ny[IPT], nz[IPT];
    float2 nm[IPT];  // negated mass
};
template <int IPT>
struct TileILow {
    float2 ex[IPT], ey[IPT], ez[IPT];
};

__device__ __forceinline__ void tile_sums_zero(TileSums &t, int lane)
{
#pragma unroll
    for (int c = 0; c < 3; ++c) t.s[c][lane] = t.c[c][lane] = dup2(0.f);
}

template <int IPT>
__device__ __forceinline__ void tile_i_set(TileI<IPT> &t, int k, const float (&S)[3], float m)
{
    t.nx[k] = dup2(-S[0]); t.ny[k] = dup2(-S[1]); t.nz[k] = dup2(-S[2]);
    t.nm[k] = dup2(-m);
}
template <int IPT>
__device__ __forceinline__ void tile_i_set_low(TileILow<IPT> &t, int k, const float (&E)[3])
{
    t.ex[k] = dup2(-E[0]); t.ey[k] = dup2(-E[1]); t.ez[k] = dup2(-E[2]);
}

// Lane `lane` stages body 32 k + lane of a j-tile (between two __syncwarp).
__device__ __forceinline__ void tile_j_put(TileJ &t, int lane, int k, const float (&S)[3], float m)
{
#pragma unroll
    for (int r = 0; r < 64; r += 32) {
        float *a = reinterpret_cast<float *>(&t.a[lane + r]) + k;
        float *b = reinterpret_cast<float *>(&t.b[lane + r]) + k;
        a[0] = S[0];
        a[2] = S[1];
        b[0] = S[2];
        b[2] = m;
    }
}
__device__ __forceinline__ void tile_j_put_low(TileJLow &t, int lane, int k, const float (&E)[3])
{
#pragma unroll
    for (int r = 0; r < 64; r += 32) {
        float *c = reinterpret_cast<float *>(&t.c[lane + r]) + k;
        c[0] = E[0];
        c[2] = E[1];
        reinterpret_cast<float *>(&t.d[lane + r])[k] = E[2];
    }
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

// How a pair is evaluated: the plain FP32 term (pair_term2_far<false>), that with
// the folded Newton step (pair_term2_far<true>), or the double-single
// displacement and the Newton step (pair_term2).
enum TileTerm { kVeryFarTerm, kFarTerm, kNearTerm };

// One step: the lane's i-bodies against the staged j-pair idx.  BOTH = false adds to the i side
// only.  EQUAL: fi and fj receive r^-3 d without the masses, and y^3 must be in
// FP32's range (equal_range); otherwise the scale is built as (m y) y^2 for each
// side, so that lengths of 1e13 and more (y^3 below FP32's range) still work.
template <int TERM, bool EQUAL, bool ZERO_SOFT, bool BOTH, int IPT>
__device__ __forceinline__ void tile_step(const TileJ &t, const TileJLow *low, int idx,
                                          const TileI<IPT> &ti, const TileILow<IPT> *lo, float2 e2,
                                          float2 (&fi)[IPT][3], float2 (&fj)[3])
{
    constexpr bool NEAR = TERM == kNearTerm;
    const float4 A = t.a[idx], B = t.b[idx];
    float4 C = make_float4(0.f, 0.f, 0.f, 0.f);
    float2 D = make_float2(0.f, 0.f);
    if (NEAR) {
        C = low->c[idx];
        D = low->d[idx];
    }
    const float2 jx = make_float2(A.x, A.y), jy = make_float2(A.z, A.w),
                 jz = make_float2(B.x, B.y), jm = make_float2(B.z, B.w);
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        float2 dx = add2(jx, ti.nx[k]), dy = add2(jy, ti.ny[k]), dz = add2(jz, ti.nz[k]);
        if (NEAR) {
            dx = add2(dx, add2(make_float2(C.x, C.y), lo->ex[k]));
            dy = add2(dy, add2(make_float2(C.z, C.w), lo->ey[k]));
            dz = add2(dz, add2(D, lo->ez[k]));
        }
        const float2 r2 = fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, e2)));
        float2 inv = make_float2(rsqrt_mufu(r2.x), rsqrt_mufu(r2.y));
        if (NEAR && ZERO_SOFT) {
            inv.x = r2.x > 0.f ? inv.x : 0.f;
            inv.y = r2.y > 0.f ? inv.y : 0.f;
        }
        float2 w = mul2(inv, inv);
        if (TERM != kVeryFarTerm) {
            // the residual by one FMA (pair_scale rounds the product r2 w, of size
            // one, first): the same operations, a third of the scale's error
            const float2 d = fma2(r2, w, dup2(-1.f));
            w = fma2(w, mul2(d, dup2(-1.5f)), w);
        }
        const float2 si = EQUAL ? mul2(inv, w) : mul2(mul2(jm, inv), w);
        fi[k][0] = fma2(dx, si, fi[k][0]);
        fi[k][1] = fma2(dy, si, fi[k][1]);
        fi[k][2] = fma2(dz, si, fi[k][2]);
        if (BOTH) {
            const float2 sj = EQUAL ? si : mul2(mul2(ti.nm[k], inv), w);
            fj[0] = fma2(dx, sj, fj[0]);
            fj[1] = fma2(dy, sj, fj[1]);
            fj[2] = fma2(dz, sj, fj[2]);
        }
    }
}

template <bool EQUAL, int IPT>
__device__ __forceinline__ void tile_fold_i(TileSums *is, int lane, float2 (&fi)[IPT][3], float mj)
{
#pragma unroll
    for (int h = 0; h < IPT / 2; ++h)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float2 t = make_float2(fi[2 * h][c].x + fi[2 * h][c].y,
                                         fi[2 * h + 1][c].x + fi[2 * h + 1][c].y);
            kahan_add2(is[h].s[c][lane], is[h].c[c][lane], EQUAL ? mul2(t, dup2(mj)) : t);
            fi[2 * h][c] = fi[2 * h + 1][c] = dup2(0.f);
        }
}

// The i-bodies against a staged j-tile, both sides.  is[h]: the sums of the
// lane's bodies 2 h and 2 h + 1; js: those of the j-tile; this warp's alone
// meanwhile.  EQUAL: mi, mj = the masses of the i- and the j-bodies.
template <int TERM, bool EQUAL, bool ZERO_SOFT, int IPT>
__device__ __forceinline__ void tile_pair(const TileJ &t, const TileJLow *low, int lane,
                                          const TileI<IPT> &ti, const TileILow<IPT> *lo, float2 e2,
                                          float mi, float mj, TileSums *is, TileSums &js)
{
    constexpr int kRun = 16 / IPT;  // steps per j-side fold
    const int next = (lane + 1) & 31;
    float2 fi[IPT][3];
#pragma unroll
    for (int k = 0; k < IPT; ++k)
#pragma unroll
        for (int c = 0; c < 3; ++c) fi[k][c] = dup2(0.f);
#pragma unroll 1
    for (int g = 0; g < 32; g += kRun) {
        float2 fj[3] = {dup2(0.f), dup2(0.f), dup2(0.f)};
#pragma unroll
        for (int u = 0; u < kRun; ++u) {
            tile_step<TERM, EQUAL, ZERO_SOFT, true, IPT>(t, low, lane + g + u, ti, lo, e2, fi, fj);
            if (u < kRun - 1)
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    fj[c] = make_float2(__shfl_sync(0xffffffffu, fj[c].x, next),
                                        __shfl_sync(0xffffffffu, fj[c].y, next));
        }
        const int idx = (lane + g + kRun - 1) & 31;
#pragma unroll
        for (int c = 0; c < 3; ++c)
            kahan_add2(js.s[c][idx], js.c[c][idx], EQUAL ? mul2(fj[c], dup2(-mi)) : fj[c]);
        if (((g + kRun) & 15) == 0) tile_fold_i<EQUAL, IPT>(is, lane, fi, mj);
        __syncwarp();  // the next run's fold takes other lanes' entries
    }
}

// A tile with itself (staged in t): every ordered pair, the i side only.
template <bool ZERO_SOFT>
__device__ __forceinline__ void tile_self(const TileJ &t, const TileJLow *low, int lane,
                                          const TileI<2> &ti, const TileILow<2> *lo, float2 e2,
                                          TileSums &is)
{
    float2 fi[2][3], none[3];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int c = 0; c < 3; ++c) fi[k][c] = dup2(0.f);
#pragma unroll 1
    for (int g = 0; g < 32; g += 8) {
#pragma unroll 4
        for (int u = 0; u < 8; ++u)
            tile_step<kNearTerm, false, ZERO_SOFT, false, 2>(t, low, lane + g + u, ti, lo, e2, fi, none);
        if (g & 8) tile_fold_i<false, 2>(&is, lane, fi, 0.f);
    }
}

// Whether r^-3 of pairs at least sqrt(gap2 + eps2) and at most sqrt(span2 + eps2)
// apart is well inside FP32's normal range (r in [1e-11, 1e11]).
__host__ __device__ __forceinline__ bool equal_range(float gap2, float span2, float eps2)
{
    return gap2 + eps2 >= 1e-22f && span2 + eps2 <= 1e22f;
}

// A body relative to c as a normalised double-single (RELATIVE), or as it is.
template <bool RELATIVE>
__device__ __forceinline__ void tile_relative(const float4 h, const float4 l, const float (&c)[3],
                                               float (&S)[3], float (&E)[3], float &m)
{
    if (RELATIVE) {
        rel_ds(h.x, l.x, c[0], S[0], E[0]);
        rel_ds(h.y, l.y, c[1], S[1], E[1]);
        rel_ds(h.z, l.z, c[2], S[2], E[2]);
    } else {
        S[0] = h.x; S[1] = h.y; S[2] = h.z;
        E[0] = l.x; E[1] = l.y; E[2] = l.z;
    }
    m = h.w;
}
// The same for any pair of bodies that are tile_in_span, by the softening alone: decided
// on the host, once per launch.
inline bool equal_soft(double eps2) { return equal_range(0.f, 7.5e21f, (float)eps2); }
// Coordinates whose differences stay within equal_range's farthest pair.
__device__ __forceinline__ bool tile_in_span(const float (&S)[3])
{
    return fmaxf(fabsf(S[0]), fmaxf(fabsf(S[1]), fabsf(S[2]))) <= 2.5e10f;
}

// Loads IPT chunks of i-bodies from body i0 of n, relative to c.  Returns
// whether they all have one mass, mass, and coordinates within equal_range's
// span; lanes past n hold massless bodies far from every j-body.
template <bool RELATIVE, int IPT>
__device__ __forceinline__ bool tile_load_i(const float4 *__restrict__ hi,
                                             const float4 *__restrict__ lo, int n, int i0,
                                             const float (&c)[3], TileI<IPT> &ti,
                                             TileILow<IPT> &tl, float &mass)
{
    bool equal = true;
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int i = i0 + 32 * k + (int)threadIdx.x;
        float S[3] = {-1.0e18f, -1.0e18f, -1.0e18f}, E[3] = {0.f, 0.f, 0.f}, m = 0.f;
        if (i < n) tile_relative<RELATIVE>(hi[i], lo[i], c, S, E, m);
        if (k == 0) mass = __shfl_sync(0xffffffffu, m, 0);
        equal = equal && (i >= n || (m == mass && tile_in_span(S)));
        tile_i_set(ti, k, S, m);
        tile_i_set_low(tl, k, E);
    }
    return __all_sync(0xffffffffu, equal);
}

// Stages the j-tile from body j0 of n relative to c; returns as
// tile_load_i.
template <bool RELATIVE>
__device__ __forceinline__ bool tile_stage_j(const float4 *__restrict__ hi,
                                              const float4 *__restrict__ lo, int n, int j0,
                                              const float (&c)[3], TileJ &stage,
                                              TileJLow &low, float &mass)
{
    const int lane = threadIdx.x;
    bool equal = true;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int j = j0 + 32 * k + lane;
        // lanes past n stage a massless body far away: exactly 0
        float S[3] = {1.0e18f, 1.0e18f, 1.0e18f}, E[3] = {0.f, 0.f, 0.f}, m = 0.f;
        if (j < n) tile_relative<RELATIVE>(hi[j], lo[j], c, S, E, m);
        if (k == 0) mass = __shfl_sync(0xffffffffu, m, 0);
        equal = equal && (j >= n || (m == mass && tile_in_span(S)));
        tile_j_put(stage, lane, k, S, m);
        tile_j_put_low(low, lane, k, E);
    }
    equal = __all_sync(0xffffffffu, equal);
    __syncwarp();
    return equal;
}

} // namespace nb
