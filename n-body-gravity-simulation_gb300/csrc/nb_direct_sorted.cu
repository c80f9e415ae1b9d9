// nb_direct_sorted.cu -- the mixed-precision all-pairs sum over Hilbert-sorted
// bodies, in packed FP32x2 arithmetic: far 64-body tiles once for both bodies of
// a pair, near ones as ordered pairs by 32-body j-chunk, the closest pairs in
// double-single.
//
// Near/far.  The double-single displacement of the mixed pair term costs 6 of
// its 21 FP32 operations and is needed only when a pair is close compared with
// the distance of its bodies from the coordinate origin.  Here the origin
// moves to each warp: bodies are sorted along a Hilbert curve (the Barnes-Hut
// radix sort on Hilbert keys), so the 64 consecutive bodies of a tile are
// spatially compact.  The Hilbert curve never jumps between distant cells (the
// Morton curve does at every cell boundary), so its tile and chunk boxes are
// smaller: on a 65,536-body Plummer sphere 5 % of the chunk pairs are near
// instead of 11 %.
//
// direct_far_kernel takes the tile pairs that hold no close pair and lie at least
// kFarFactor D apart (D: the smaller box's diameter; 97 % of them at
// N = 65,536) over unordered pairs (nb_tile.cuh), relative to a tile's centre in
// plain FP32; at kVeryFar of the larger diameter the folded Newton step is left
// out too.  direct_near_kernel sums the others by row: a warp takes its tile's
// centre c as the origin and stages each j-chunk as a normalised double-single
// (S, E) of x - c, or S alone where the chunk's box is far or very far from its
// own.  Decisions are uniform over a warp, and a warp stages its own tiles in
// its own shared memory: no CTA-wide barrier.
//
// Measured at N = 65,536 (a velocity-Verlet step) and N = 400,003 (an
// evaluation): 1.51 and 47.7 ms, where the row kernel over every j-chunk, each
// pair evaluated twice, took 1.98 and 67 ms.
//
// Packed arithmetic.  sm_100-class SMs execute FP32 add, multiply and FMA on
// register pairs (f32x2) at the FP32 pipe's lane rate but half the issue
// slots: each thread evaluates two j at once (a j-pair, staged side by side in
// shared memory) against i-bodies held as duplicated pairs.  Every lane of an
// f32x2 operation rounds like its scalar counterpart.
//
// Error of a far term: S carries one FP32 rounding of x - c.  With
// |xi - c| <= D/2, |xj - c| <= r + D/2 and the subtraction's own rounding, the
// displacement error is at most 2^-24 (2r + D) <= 2^-24 r (2 + 1/kFarFactor)
// = 10 * 2^-24 r for kFarFactor = 1/8 -- about 6e-7 relative at worst, the
// order of the FP32 arithmetic of the term.  A very far term (gap >= D/4:
// displacement error <= 6 * 2^-24 r) also carries
// the MUFU rsqrt error three times, at most 3.7e-7 and on average -1.6e-8
// relative (measured over every FP32 input in [1, 4), i.e. every mantissa at
// both exponent parities); these terms are many and distant,
// so their errors average out: on a 65,536-body Plummer sphere the far /
// very-far factors (1/8, 1/4), (1/4, 1/4), (1/4, 1/2), (1/2, 1/2) and (1/2, 1)
// give the same errors (largest relative 5e-7 where S_i / |a_i| <= 10, RMS
// 2.5e-8), and (1/8, 1/4) the shortest kernel.  The bounds hold for both bodies of
// a far pair: they are in units of r.  Near terms keep the double-single
// displacement (absolute error ~2^-48 |x|) and the Newton step; every FP32
// accumulator takes 16 terms before its Kahan-compensated add, and the
// segments combine as a double-single.
#include "nb_internal.h"
#include "nb_check.cuh"
#include "nb_tile.cuh"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

namespace nb {
namespace {

constexpr int kChunk = 32;             // j-chunk = one body per lane
constexpr int kIpt = kTile / kChunk;   // 32-body i-chunks per warp
constexpr int kFarTiles = 4;           // tiles per block of the far kernel
// Its one-warp CTAs per SM: 12 / 14 / 16 measured 1.53 / 1.47 / 1.47 ms a step.
constexpr int kFarCtas = 16;
// Its partial planes per pass.  Each pass ends with a thinly filled last wave: with 256
// MiB an evaluation takes 3.3 % longer at N = 65,536 and 8.4 % at 400,003.
constexpr size_t kFarPlaneBytes = (size_t)1 << 30;
constexpr int kExactWarps = 8;         // warps of exact_pairs_kernel per tile
constexpr int kExactRound = 64;        // left-out pairs evaluated per round and warp
constexpr int kResortEvals = 8;        // force evaluations per re-sort

// The mass of a tile whose bodies do not all have one (compares false).
#define kNoMass __int_as_float(0x7fffffff)

// A 64-body tile: its box, squared diameter, the mass of its bodies (kNoMass:
// not all equal) and the squared left-out radius of its pairs.  Every product
// and sum here and in the functions below is an explicit round-to-nearest
// intrinsic: the kernels must take the same decisions bit for bit.
struct TileGeom {
    float mn[3], mx[3];
    float diam2, mass, thr2x;
};
__device__ __forceinline__ float box_diam2(const float (&mn)[3], const float (&mx)[3])
{
    const float sx = __fsub_rn(mx[0], mn[0]), sy = __fsub_rn(mx[1], mn[1]),
                sz = __fsub_rn(mx[2], mn[2]);
    return __fmaf_rn(sz, sz, __fmaf_rn(sy, sy, __fmul_rn(sx, sx)));
}

// Pairs closer than R leave the FP32 sum and are evaluated in double-single by
// exact_pairs_kernel (only chunks nearer than R can hold one):
// R = min(kExact D, kExactSpacing s, the global cap), s the mean body spacing of
// the tile's box, (V / 64)^(1/3) with every side padded by D / 16 so that a flat
// box keeps its in-plane spacing.
// The cap is kExactSpacing times the mean body spacing of the root cube,
// (side^3 / n)^(1/3).  A tile of sparse bodies spread over a large box would
// otherwise get a radius that takes in whole dense regions, whose terms are a
// tiny part of its bodies' sums.  per_n = kExactSpacing2 n^(-2/3), computed on
// the host.
__device__ __forceinline__ float left_out_radius2(const float (&mn)[3], const float (&mx)[3],
                                                  const double *__restrict__ root, float per_n)
{
    const float diam2 = box_diam2(mn, mx);
    const float pad = __fmul_rn(0.0625f, sqrtf(diam2));
    float vol = 1.0f;
#pragma unroll
    for (int a = 0; a < 3; ++a) vol = __fmul_rn(vol, __fadd_rn(__fsub_rn(mx[a], mn[a]), pad));
    const float s2 = exp2f(__fmul_rn(0.6666667f, log2f(__fmul_rn(vol, 1.0f / kTile))));
    const float side = __double2float_rn(root[3]);
    const float cap2 = __fmul_rn(__fmul_rn(side, side), per_n);
    return fminf(fminf(__fmul_rn(kExact2, diam2), __fmul_rn(kExactSpacing2, s2)), cap2);
}

float exact_cap_per_n(int n)
{
    return (float)((double)kExactSpacing2 / std::cbrt((double)n * (double)n));
}

// Positions in sorted order relative to the root centre, split into
// double-single hi/lo parts (mass in hi.w); the bounding box of the hi positions
// of every 32-body chunk (box[2c] = min, box[2c+1] = max; lanes past n take the
// chunk's first body); and every 64-body tile's record (tile[2t] = min and mass,
// tile[2t+1] = max and left-out radius).  A warp is a tile.
__global__ void __launch_bounds__(128)
split_sorted_kernel(const uint32_t *__restrict__ order, const double *__restrict__ x,
                    const double *__restrict__ y, const double *__restrict__ z,
                    const double *__restrict__ m, int n, const double *__restrict__ root,
                    float cap_per_n, float4 *__restrict__ hi, float4 *__restrict__ lo,
                    float4 *__restrict__ box, float4 *__restrict__ tile)
{
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (t * kTile >= n) return;
    float tmn[3] = {3.0e38f, 3.0e38f, 3.0e38f}, tmx[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
    float m0 = 0.f;
    bool equal = true;
#pragma unroll
    for (int c = 0; c < kIpt; ++c) {
        const int i = t * kTile + kChunk * c + lane;
        if (i - lane >= n) break;  // the whole chunk is past n
        float p[3] = {0.f, 0.f, 0.f}, hm = 0.f;
        const uint32_t o = i < n ? order[i] : 0u;
        if (i < n && NB_IN_RANGE(o, n)) {
            const double X = x[o] - root[0], Y = y[o] - root[1], Z = z[o] - root[2];
            p[0] = __double2float_rn(X);
            p[1] = __double2float_rn(Y);
            p[2] = __double2float_rn(Z);
            hm = __double2float_rn(m[o]);
            hi[i] = make_float4(p[0], p[1], p[2], hm);
            lo[i] = make_float4(__double2float_rn(X - (double)p[0]),
                                __double2float_rn(Y - (double)p[1]),
                                __double2float_rn(Z - (double)p[2]),
                                __double2float_rn(m[o] - (double)hm));
        }
        float mn[3], mx[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float first = __shfl_sync(0xffffffffu, p[k], 0);
            mn[k] = mx[k] = i < n ? p[k] : first;
        }
        if (c == 0) m0 = __shfl_sync(0xffffffffu, hm, 0);
        equal = equal && __all_sync(0xffffffffu, i >= n || hm == m0);
#pragma unroll
        for (int s = 16; s > 0; s >>= 1)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                mn[k] = fminf(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], s));
                mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], s));
            }
        if (lane == 0) {
            box[2 * (kIpt * t + c)] = make_float4(mn[0], mn[1], mn[2], 0.f);
            box[2 * (kIpt * t + c) + 1] = make_float4(mx[0], mx[1], mx[2], 0.f);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            tmn[k] = fminf(tmn[k], mn[k]);
            tmx[k] = fmaxf(tmx[k], mx[k]);
        }
    }
    if (lane == 0) {
        tile[2 * t] = make_float4(tmn[0], tmn[1], tmn[2], equal ? m0 : kNoMass);
        tile[2 * t + 1] = make_float4(tmx[0], tmx[1], tmx[2],
                                      left_out_radius2(tmn, tmx, root, cap_per_n));
    }
}

__device__ __forceinline__ TileGeom tile_geometry(const float4 *__restrict__ tile, int t)
{
    const float4 a = tile[2 * t], b = tile[2 * t + 1];
    TileGeom g;
    g.mn[0] = a.x; g.mn[1] = a.y; g.mn[2] = a.z;
    g.mx[0] = b.x; g.mx[1] = b.y; g.mx[2] = b.z;
    g.mass = a.w;
    g.thr2x = b.w;
    g.diam2 = box_diam2(g.mn, g.mx);
    return g;
}

// Squared gap between two boxes, the same bits whichever is called first.
__device__ __forceinline__ float box_gap2(const float (&amn)[3], const float (&amx)[3],
                                          const float (&bmn)[3], const float (&bmx)[3])
{
    float g[3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
        g[a] = fmaxf(0.f, fmaxf(__fsub_rn(bmn[a], amx[a]), __fsub_rn(amn[a], bmx[a])));
    return __fmaf_rn(g[2], g[2], __fmaf_rn(g[1], g[1], __fmul_rn(g[0], g[0])));
}

// Whether two tiles are direct_far_kernel's: an eighth of the smaller diameter
// apart (a plain FP32 displacement relative to that tile's centre is enough) and
// without left-out pairs on either side.  All other tile pairs are
// direct_near_kernel's and exact_pairs_kernel's; a chunk of such a tile lies no
// nearer than the tile, in these operations too, so neither kernel leaves out a
// pair of the far tiles.
__device__ __forceinline__ bool tiles_apart(const TileGeom &a, const TileGeom &b, float gap2)
{
    return gap2 > 0.f && gap2 >= __fmul_rn(kFarFactor2, fminf(a.diam2, b.diam2)) &&
           gap2 >= fmaxf(a.thr2x, b.thr2x);
}
// Whether they are very far apart seen from both (a quarter of the larger
// diameter): no Newton step.  Implies tiles_apart.
__device__ __forceinline__ bool tiles_very_far(const TileGeom &a, const TileGeom &b, float gap2)
{
    return tiles_apart(a, b, gap2) && gap2 >= __fmul_rn(kVeryFar2, fmaxf(a.diam2, b.diam2));
}

// A warp's tile, its centre (the origin of every staged coordinate), and the
// squared thresholds of its near/far decisions.
struct WarpGeom {
    TileGeom tile;
    float c[3];
    float thr2, thr2v;
};

__device__ __forceinline__ WarpGeom warp_geometry(const float4 *__restrict__ tiles, int t,
                                                  float far2)
{
    WarpGeom g;
    g.tile = tile_geometry(tiles, t);
#pragma unroll
    for (int a = 0; a < 3; ++a) g.c[a] = __fmul_rn(0.5f, __fadd_rn(g.tile.mn[a], g.tile.mx[a]));
    g.thr2 = __fmul_rn(far2, g.tile.diam2);        // far: double-single not needed
    g.thr2v = __fmul_rn(kVeryFar2, g.tile.diam2);  // very far: Newton step not needed
    return g;
}

// Squared gap between the warp's box and a j-chunk's box.
__device__ __forceinline__ float chunk_gap2(const WarpGeom &g, float4 jmn, float4 jmx)
{
    const float mn[3] = {jmn.x, jmn.y, jmn.z}, mx[3] = {jmx.x, jmx.y, jmx.z};
    return box_gap2(g.tile.mn, g.tile.mx, mn, mx);
}

// Stages the i-bodies (IPT chunks from i0) relative to c.
template <int IPT>
__device__ __forceinline__ void far_load_i(const float4 *__restrict__ hi,
                                           const float4 *__restrict__ lo, int n, int i0,
                                           const float (&c)[3], TileI<IPT> &ti)
{
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        // lanes past n: massless and far from every j-body (r^-3 is exactly 0)
        float S[3] = {-1.0e18f, -1.0e18f, -1.0e18f}, m = 0.f;
        const int i = i0 + 32 * k + (int)threadIdx.x;
        if (i < n) {
            const float4 h = hi[i], l = lo[i];
            S[0] = rel_s(h.x, l.x, c[0]);
            S[1] = rel_s(h.y, l.y, c[1]);
            S[2] = rel_s(h.z, l.z, c[2]);
            m = h.w;
        }
        tile_i_set(ti, k, S, m);
    }
}

// Stages the j-tile from body j0 relative to c and adds its pairs with ti.
// equal: the equal-mass loop, mi = the i-bodies' mass.
template <int TERM, int IPT>
__device__ __forceinline__ void far_tile_pair(const float4 *__restrict__ hi,
                                              const float4 *__restrict__ lo, int n, int j0,
                                              const float (&c)[3], const TileI<IPT> &ti, bool equal,
                                              float mi, float2 e2, TileJ &stage, TileSums *isum,
                                              TileSums &jsum)
{
    const int lane = threadIdx.x;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int j = j0 + 32 * k + lane;
        float S[3] = {1.0e18f, 1.0e18f, 1.0e18f}, mj = 0.f;
        if (j < n) {
            const float4 h = hi[j], l = lo[j];
            S[0] = rel_s(h.x, l.x, c[0]);
            S[1] = rel_s(h.y, l.y, c[1]);
            S[2] = rel_s(h.z, l.z, c[2]);
            mj = h.w;
        }
        tile_j_put(stage, lane, k, S, mj);
    }
    __syncwarp();
    if (equal)
        tile_pair<TERM, true, false, IPT>(stage, nullptr, lane, ti, nullptr, e2, mi, stage.b[0].z,
                                          isum, jsum);
    else
        tile_pair<TERM, false, false, IPT>(stage, nullptr, lane, ti, nullptr, e2, 0.f, 0.f, isum,
                                           jsum);
}

// The pairs of far tiles, once for both bodies (nb_tile.cuh).  One warp = one
// pair of 256-body blocks (a, a + p), the second block's sums in shared memory.
// It takes two of the first block's tiles at a time (four i-bodies per lane)
// against a tile of the second that both are very far from; they share an
// origin, the centre of their common box, which has to be D / 4 or more from the
// j-tile (D its diameter), the bound of a plain FP32 displacement without the Newton
// step (D / 8: 0.7 % faster, and twice the error there).  Other far
// tile pairs are met one by one, relative to the smaller tile's centre and with
// the Newton step.
// part: plane p - p0 holds the first side's sums of diagonal p, plane np + p - p0
// the second's, as Kahan pairs (sum, negated compensation).
__global__ void __launch_bounds__(32, kFarCtas)
direct_far_kernel(const float4 *__restrict__ hi, const float4 *__restrict__ lo,
                  const float4 *__restrict__ tile, int n, int tiles, float eps2, int blocks,
                  int p0, int np, float2 *__restrict__ part)
{
    static_assert(kFarTiles == 4, "the lanes' tile-pair tests");
    __shared__ TileJ stage;
    __shared__ TileSums jsum[kFarTiles], isum[2];
    const int lane = threadIdx.x;
    const int a = blockIdx.x % blocks, dp = blockIdx.x / blocks, p = p0 + dp;
    if (!pair_first(p, a, blocks)) return;
    const int ti0 = a * kFarTiles, tj0 = (a + p) % blocks * kFarTiles;
    const int ta = min(kFarTiles, tiles - ti0), tb = min(kFarTiles, tiles - tj0);
    // lane 4 u + v decides the tile pair (u, v), lane 16 + 4 h + v tiles 2 h and
    // 2 h + 1 together against v
    bool far = false, equal = false;
    {
        const bool two = lane >= 16;
        const int u = two ? (lane & 4) / 2 : lane / 4, v = lane & 3;
        if (lane < 24 && u + two < ta && v < tb && (p > 0 || v > u + two)) {
            TileGeom gi = tile_geometry(tile, ti0 + u);
            const TileGeom gj = tile_geometry(tile, tj0 + v);
            float gap2 = box_gap2(gi.mn, gi.mx, gj.mn, gj.mx);
            if (two) {
                const TileGeom g1 = tile_geometry(tile, ti0 + u + 1);
                far = tiles_very_far(gi, gj, gap2) &&
                      tiles_very_far(g1, gj, box_gap2(g1.mn, g1.mx, gj.mn, gj.mx));
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    gi.mn[d] = fminf(gi.mn[d], g1.mn[d]);
                    gi.mx[d] = fmaxf(gi.mx[d], g1.mx[d]);
                }
                gap2 = box_gap2(gi.mn, gi.mx, gj.mn, gj.mx);
                far = far && gap2 >= kVeryFar2 * box_diam2(gi.mn, gi.mx);
                gi.mass = gi.mass == g1.mass ? gi.mass : kNoMass;
            } else {
                far = tiles_apart(gi, gj, gap2);
            }
            float span2 = 0.f;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const float s = fmaxf(gi.mx[d], gj.mx[d]) - fminf(gi.mn[d], gj.mn[d]);
                span2 = fmaf(s, s, span2);
            }
            equal = far && gi.mass == gi.mass && gj.mass == gj.mass &&
                    equal_range(gap2, span2, eps2);
        }
    }
    const unsigned fars = __ballot_sync(0xffffffffu, far);
    const unsigned equals = __ballot_sync(0xffffffffu, equal);
    const float2 e2 = dup2(eps2);
    for (int v = 0; v < kFarTiles; ++v) tile_sums_zero(jsum[v], lane);
    const size_t plane = (size_t)n;
    float2 *pa = part + 3 * plane * dp, *pb = part + 3 * plane * (np + dp);
    for (int h = 0; 2 * h < ta; ++h) {
        tile_sums_zero(isum[0], lane);
        tile_sums_zero(isum[1], lane);
        const unsigned both = fars >> (16 + 4 * h) & 15u;
        if (both) {
            const TileGeom g = tile_geometry(tile, ti0 + 2 * h),
                           g1 = tile_geometry(tile, ti0 + 2 * h + 1);
            float c[3];
#pragma unroll
            for (int d = 0; d < 3; ++d)
                c[d] = 0.5f * (fminf(g.mn[d], g1.mn[d]) + fmaxf(g.mx[d], g1.mx[d]));
            TileI<4> ti;
            far_load_i(hi, lo, n, (ti0 + 2 * h) * kTile, c, ti);
            for (int v = 0; v < tb; ++v)
                if (both >> v & 1u)
                    far_tile_pair<kVeryFarTerm>(hi, lo, n, (tj0 + v) * kTile, c, ti,
                                                equals >> (16 + 4 * h + v) & 1u, g.mass, e2, stage,
                                                isum, jsum[v]);
        }
#pragma unroll 1
        for (int w = 0; w < 2; ++w) {
            const int u = 2 * h + w;
            const unsigned one = (fars >> (4 * u) & 15u) & ~both;
#pragma unroll 1
            for (int v = 0; v < tb; ++v) {
                if (!(one >> v & 1u)) continue;
                const TileGeom g = tile_geometry(tile, ti0 + u), gj = tile_geometry(tile, tj0 + v);
                const bool mine = g.diam2 <= gj.diam2;
                float c[3];
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    c[d] = mine ? 0.5f * (g.mn[d] + g.mx[d]) : 0.5f * (gj.mn[d] + gj.mx[d]);
                TileI<2> ti;
                far_load_i(hi, lo, n, (ti0 + u) * kTile, c, ti);
                far_tile_pair<kFarTerm>(hi, lo, n, (tj0 + v) * kTile, c, ti,
                                        equals >> (4 * u + v) & 1u, g.mass, e2, stage, isum + w,
                                        jsum[v]);
            }
        }
        __syncwarp();
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            const int u = 2 * h + w, i = (ti0 + u) * kTile + lane;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                float2 t = isum[w].s[d][lane], e = isum[w].c[d][lane];
                if (p == 0) {  // within a block: with what the tile took as a j-tile
                    const float2 js = jsum[u].s[d][lane], jc = jsum[u].c[d][lane];
                    float2 r;
                    two_sum(t.x, js.x, t.x, r.x);
                    two_sum(t.y, js.y, t.y, r.y);
                    e = make_float2(r.x + (e.x + jc.x), r.y + (e.y + jc.y));
                }
                if (i < n) pa[d * plane + i] = make_float2(t.x, e.x);
                if (i + 32 < n) pa[d * plane + i + 32] = make_float2(t.y, e.y);
            }
        }
    }
    if (p == 0) return;
    for (int v = 0; v < tb; ++v) {
        const int j = (tj0 + v) * kTile + lane;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const float2 js = jsum[v].s[d][lane], jc = jsum[v].c[d][lane];
            if (j < n) pb[d * plane + j] = make_float2(js.x, jc.x);
            if (j + 32 < n) pb[d * plane + j + 32] = make_float2(js.y, jc.y);
        }
    }
}

// All other pairs, as ordered pairs.  One warp = one tile of i-bodies (lane l of
// chunk k holds body 64 tile + 32 k + l) and the j-tiles t = y (mod segments)
// that are not far from it, chunk by chunk.  Writes per-segment Kahan sums
// and compensations (sorted order).
template <bool ZERO_SOFT>
__global__ void __launch_bounds__(32)
direct_near_kernel(const float4 *__restrict__ hi, const float4 *__restrict__ lo,
                   const float4 *__restrict__ box, const float4 *__restrict__ tile, int n,
                   int nchunks, float eps2, float *__restrict__ psum, float *__restrict__ pcomp,
                   float far2)
{
    constexpr int IPT = kIpt;
    __shared__ PairTile sg;
    const int lane = threadIdx.x;
    const int tile0 = blockIdx.x * IPT, seg = blockIdx.y, segments = gridDim.y;
    const int tiles = (nchunks + 1) / 2;

    const WarpGeom gm = warp_geometry(tile, blockIdx.x, far2);
    const float cx = gm.c[0], cy = gm.c[1], cz = gm.c[2];
    const float thr2 = gm.thr2, thr2v = gm.thr2v, thr2x = gm.tile.thr2x;
    const float thrx = __fadd_rn(thr2x, eps2);

    // i-bodies relative to c, negated and duplicated into pairs
    float2 nsx[IPT], nsy[IPT], nsz[IPT], nex[IPT], ney[IPT], nez[IPT];
    float sx[IPT], sy[IPT], sz[IPT], qx[IPT], qy[IPT], qz[IPT];
    float2 ax[IPT], ay[IPT], az[IPT];
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int i = (tile0 + k) * kChunk + lane;
        float4 h = make_float4(0.f, 0.f, 0.f, 0.f), l = h;
        if (i < n) {
            h = hi[i];
            l = lo[i];
        }
        float S, E;
        rel_ds(h.x, l.x, cx, S, E);
        nsx[k] = dup2(-S);
        nex[k] = dup2(-E);
        rel_ds(h.y, l.y, cy, S, E);
        nsy[k] = dup2(-S);
        ney[k] = dup2(-E);
        rel_ds(h.z, l.z, cz, S, E);
        nsz[k] = dup2(-S);
        nez[k] = dup2(-E);
        sx[k] = sy[k] = sz[k] = 0.f;
        qx[k] = qy[k] = qz[k] = 0.f;
        ax[k] = ay[k] = az[k] = dup2(0.f);
    }
    const float2 e2 = dup2(eps2);

    // the next chunk of a tile that is not far, in increasing order (-1: none):
    // the lanes test 32 of the segment's tiles at a time
    unsigned todo = 0;
    int scan = seg - 32 * segments, cur = -1;
    auto next_chunk = [&]() {
        if (cur >= 0 && !(cur & 1) && cur + 1 < nchunks) return ++cur;
        while (!todo) {
            scan += 32 * segments;
            if (scan >= tiles) return cur = -1;
            const int t = scan + lane * segments;
            bool near = false;
            if (t < tiles) {
                const TileGeom gj = tile_geometry(tile, t);
                near = !tiles_apart(gm.tile, gj, box_gap2(gm.tile.mn, gm.tile.mx, gj.mn, gj.mx));
            }
            todo = __ballot_sync(0xffffffffu, near);
        }
        const int b = __ffs(todo) - 1;
        todo &= todo - 1u;
        return cur = 2 * (scan + b * segments);
    };

    int jc = next_chunk();
    // the lane's body of the next chunk, loaded one chunk ahead
    float4 h = make_float4(0.f, 0.f, 0.f, 0.f), l = h;
    bool valid = jc >= 0 && jc * kChunk + lane < n;
    if (valid) {
        h = hi[jc * kChunk + lane];
        l = lo[jc * kChunk + lane];
    }
    while (jc >= 0) {
        const float gap2 = chunk_gap2(gm, box[2 * jc], box[2 * jc + 1]);
        const bool far = gap2 > 0.f && gap2 >= thr2;
        const bool vfar = far && gap2 >= thr2v;
        const bool touch = !far && gap2 < thr2x;

        // lanes past n stage a massless body far away: its terms are exactly 0
        float Sx = 1.0e18f, Sy = 1.0e18f, Sz = 1.0e18f, Ex = 0.f, Ey = 0.f, Ez = 0.f, mj = 0.f;
        if (valid) {
            if (far) {  // S alone: x - c rounded once
                Sx = rel_s(h.x, l.x, cx);
                Sy = rel_s(h.y, l.y, cy);
                Sz = rel_s(h.z, l.z, cz);
            } else {
                rel_ds(h.x, l.x, cx, Sx, Ex);
                rel_ds(h.y, l.y, cy, Sy, Ey);
                rel_ds(h.z, l.z, cz, Sz, Ez);
            }
            mj = h.w;
        }
        __syncwarp();
        if (far)
            pair_tile_put_hi(sg, lane, Sx, Sy, Sz, mj);
        else
            pair_tile_put(sg, lane, Sx, Sy, Sz, mj, Ex, Ey, Ez);
        __syncwarp();
        jc = next_chunk();
        valid = jc >= 0 && jc * kChunk + lane < n;
        if (valid) {
            h = hi[jc * kChunk + lane];
            l = lo[jc * kChunk + lane];
        }

        if (vfar) {
#pragma unroll 4
            for (int p = 0; p < kChunk / 2; ++p) {
                const JPair j = pair_tile_get(sg, p);
#pragma unroll
                for (int k = 0; k < IPT; ++k)
                    pair_term2_far<false>(j, nsx[k], nsy[k], nsz[k], e2, ax[k], ay[k], az[k]);
            }
        } else if (far) {
#pragma unroll 4
            for (int p = 0; p < kChunk / 2; ++p) {
                const JPair j = pair_tile_get(sg, p);
#pragma unroll
                for (int k = 0; k < IPT; ++k)
                    pair_term2_far<true>(j, nsx[k], nsy[k], nsz[k], e2, ax[k], ay[k], az[k]);
            }
        } else if (touch) {
            // pairs closer than R are left to exact_pairs_kernel
            bool hit = false;
#pragma unroll 4
            for (int p = 0; p < kChunk / 2; ++p) {
                const JPair j = pair_tile_get(sg, p);
#pragma unroll
                for (int k = 0; k < IPT; ++k)
                    pair_term2_excl<ZERO_SOFT>(j, nsx[k], nsy[k], nsz[k], nex[k], ney[k], nez[k],
                                               e2, thrx, ax[k], ay[k], az[k], hit);
            }
        } else {
#pragma unroll 4
            for (int p = 0; p < kChunk / 2; ++p) {
                const JPair j = pair_tile_get(sg, p);
#pragma unroll
                for (int k = 0; k < IPT; ++k)
                    pair_term2<ZERO_SOFT>(j, nsx[k], nsy[k], nsz[k], nex[k], ney[k], nez[k], e2,
                                          ax[k], ay[k], az[k]);
            }
        }
        // every accumulator lane holds 16 terms of the chunk: fold them into the
        // Kahan sums (folding after every second chunk measured no faster, and
        // raised the largest relative error at N = 65,536 from 6e-7 to 9e-7)
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            kahan_add(sx[k], qx[k], ax[k].x + ax[k].y);
            kahan_add(sy[k], qy[k], ay[k].x + ay[k].y);
            kahan_add(sz[k], qz[k], az[k].x + az[k].y);
            ax[k] = ay[k] = az[k] = dup2(0.f);
        }
    }

    const size_t plane = (size_t)n;
    const size_t base = (size_t)seg * 3 * plane;
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int i = (tile0 + k) * kChunk + lane;
        if (i < n) {
            psum[base + i] = sx[k];
            psum[base + plane + i] = sy[k];
            psum[base + 2 * plane + i] = sz[k];
            pcomp[base + i] = qx[k];
            pcomp[base + plane + i] = qy[k];
            pcomp[base + 2 * plane + i] = qz[k];
        }
    }
}

// The pairs direct_near_kernel leaves out, in double-single.  It needs
// nothing from that kernel -- it takes the same decisions from the same data
// -- so it runs beside it on a second stream.  S CTAs per tile (the same i-chunks
// and geometry) and kExactWarps warps in each: warp w
// of share y of S takes the chunks jc = kExactWarps y + w (mod kExactWarps S)
// that the near kernel tests for left-out pairs (not far, nearer than R), in increasing order, skipping those
// that no lane's i-body comes within R of.  For each it stages the chunk
// exactly as the near kernel does, recomputes the same r^2 bits, and marks the
// left-out pairs of each lane (bit 2p + u of mk[k]: tile body 2p + u against
// the lane's i-body k).  The marked pairs are evaluated one per lane,
// whole-warp, in rounds of kExactRound, and every lane adds its own bodies'
// terms into their double-single sums in increasing j; the warps' sums are
// then added in warp order.  The result does not depend on timing.
// ex[(3 y + c) n + i] = the FP64 value of body i's sum (sorted order), 0 if none.
// At most 64 registers (four CTAs per SM): beside direct_far_kernel, whose
// one-warp CTAs fill the register file, a leaner CTA displaces fewer of them.
__global__ void __launch_bounds__(kExactWarps * 32, 4)
exact_pairs_kernel(const float4 *__restrict__ hi, const float4 *__restrict__ lo,
                   const float4 *__restrict__ box, const float4 *__restrict__ tile, int n,
                   int nchunks, float eps2, float far2, double eps2d, double *__restrict__ ex)
{
    constexpr int IPT = kIpt;
    __shared__ PairTile stage[kExactWarps];
    __shared__ float ibody[IPT * 32][6];                      // (S, E) of x, y, z
    __shared__ uint16_t evt[kExactWarps][kExactRound];        // (k 32 + lane) << 5 | bit
    __shared__ float term[kExactWarps][kExactRound][6];       // (hi, lo) of x, y, z
    __shared__ float red[kExactWarps][IPT * 32][6];           // the warps' sums
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int wg = blockIdx.x;
    const int stride = kExactWarps * gridDim.y;  // candidate chunks: every stride-th
    const int tile0 = wg * IPT;
    if (tile0 >= nchunks) return;  // the whole CTA
    PairTile &sg = stage[w];
    const WarpGeom gm = warp_geometry(tile, wg, far2);
    const float thrx = __fadd_rn(gm.tile.thr2x, eps2);
    const float2 e2 = dup2(eps2);
    const DS e2ds{__double2float_rn(eps2d),
                  __double2float_rn(eps2d - (double)__double2float_rn(eps2d))};

    float2 nsx[IPT], nsy[IPT], nsz[IPT], nex[IPT], ney[IPT], nez[IPT];
    DS acc[IPT][3];
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int i = (tile0 + k) * kChunk + lane;
        float4 h = make_float4(0.f, 0.f, 0.f, 0.f), l = h;
        if (i < n) {
            h = hi[i];
            l = lo[i];
        }
        float S[3], E[3];
        rel_ds(h.x, l.x, gm.c[0], S[0], E[0]);
        rel_ds(h.y, l.y, gm.c[1], S[1], E[1]);
        rel_ds(h.z, l.z, gm.c[2], S[2], E[2]);
        nsx[k] = dup2(-S[0]); nex[k] = dup2(-E[0]);
        nsy[k] = dup2(-S[1]); ney[k] = dup2(-E[1]);
        nsz[k] = dup2(-S[2]); nez[k] = dup2(-E[2]);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (w == 0) {
                ibody[k * 32 + lane][2 * a] = S[a];
                ibody[k * 32 + lane][2 * a + 1] = E[a];
            }
            acc[k][a] = DS{0.f, 0.f};
        }
    }
    __syncthreads();

    // the lane's i-bodies' box, for the per-lane test of a chunk
    float lmn[3] = {3.0e38f, 3.0e38f, 3.0e38f}, lmx[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
    bool ival[IPT];
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        ival[k] = (tile0 + k) * kChunk + lane < n;
        if (ival[k]) {
            const float q[3] = {-nsx[k].x, -nsy[k].x, -nsz[k].x};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                lmn[a] = fminf(lmn[a], q[a]);
                lmx[a] = fmaxf(lmx[a], q[a]);
            }
        }
    }
    // The tests below only skip work, so they must never skip a chunk (or an
    // i-chunk of it) that holds a left-out pair: R grows by a slack far above
    // the FP32 roundings that separate the boxes (hi coordinates) from the
    // staged ones and the box distance from the pair's r^2 (softening included).
    const float Rw = sqrtf(gm.tile.thr2x);
    const float cmag = fmaxf(fabsf(gm.c[0]), fmaxf(fabsf(gm.c[1]), fabsf(gm.c[2])));
    const float e2slack = 1e-6f * (gm.tile.thr2x + eps2);

    int scan = kExactWarps * blockIdx.y + w;
    while (true) {
        // the next chunk of this warp's that the near kernel tests, with
        // a lane whose bodies come within R of its box
        int jc = -1;
        while (scan < nchunks) {
            const int c = scan + stride * lane;
            bool t = false;
            float4 jmn = make_float4(0.f, 0.f, 0.f, 0.f), jmx = jmn;
            if (c < nchunks) {
                jmn = box[2 * c];
                jmx = box[2 * c + 1];
                const float gap2 = chunk_gap2(gm, jmn, jmx);
                t = !(gap2 > 0.f && gap2 >= gm.thr2) && gap2 < gm.tile.thr2x;
            }
            uint32_t cand = __ballot_sync(0xffffffffu, t);
            while (cand) {
                const int src = __ffs(cand) - 1;
                cand &= cand - 1u;
                // this lane's bodies against the candidate's box (relative to c)
                const float bx0 = __shfl_sync(0xffffffffu, jmn.x, src) - gm.c[0];
                const float by0 = __shfl_sync(0xffffffffu, jmn.y, src) - gm.c[1];
                const float bz0 = __shfl_sync(0xffffffffu, jmn.z, src) - gm.c[2];
                const float bx1 = __shfl_sync(0xffffffffu, jmx.x, src) - gm.c[0];
                const float by1 = __shfl_sync(0xffffffffu, jmx.y, src) - gm.c[1];
                const float bz1 = __shfl_sync(0xffffffffu, jmx.z, src) - gm.c[2];
                const float gx = fmaxf(0.f, fmaxf(bx0 - lmx[0], lmn[0] - bx1));
                const float gy = fmaxf(0.f, fmaxf(by0 - lmx[1], lmn[1] - by1));
                const float gz = fmaxf(0.f, fmaxf(bz0 - lmx[2], lmn[2] - bz1));
                const float mag = cmag + fmaxf(fmaxf(fabsf(bx0), fabsf(bx1)),
                                               fmaxf(fmaxf(fabsf(by0), fabsf(by1)),
                                                     fmaxf(fabsf(bz0), fabsf(bz1))));
                const float Re = Rw + 1e-6f * mag;
                if (__any_sync(0xffffffffu, gx * gx + gy * gy + gz * gz <= Re * Re + e2slack)) {
                    jc = scan + stride * src;
                    break;
                }
            }
            if (jc >= 0) {
                scan = jc + stride;
                break;
            }
            scan += 32 * stride;
        }
        if (jc < 0) break;

        // the i-chunks with a body within R of the chunk's box (a lane's own
        // body against the box, the same slack)
        bool need[IPT];
        {
            const float4 jmn = box[2 * jc], jmx = box[2 * jc + 1];
            const float bx0 = jmn.x - gm.c[0], by0 = jmn.y - gm.c[1], bz0 = jmn.z - gm.c[2];
            const float bx1 = jmx.x - gm.c[0], by1 = jmx.y - gm.c[1], bz1 = jmx.z - gm.c[2];
            const float mag = cmag + fmaxf(fmaxf(fabsf(bx0), fabsf(bx1)),
                                           fmaxf(fmaxf(fabsf(by0), fabsf(by1)),
                                                 fmaxf(fabsf(bz0), fabsf(bz1))));
            const float Re = Rw + 1e-6f * mag;
#pragma unroll
            for (int k = 0; k < IPT; ++k) {
                const float px = -nsx[k].x, py = -nsy[k].x, pz = -nsz[k].x;
                const float gx = fmaxf(0.f, fmaxf(bx0 - px, px - bx1));
                const float gy = fmaxf(0.f, fmaxf(by0 - py, py - by1));
                const float gz = fmaxf(0.f, fmaxf(bz0 - pz, pz - bz1));
                need[k] = __any_sync(0xffffffffu,
                                     ival[k] && gx * gx + gy * gy + gz * gz <= Re * Re + e2slack);
            }
        }

        // stage the chunk as the near kernel does
        const int b = jc * kChunk + lane;
        float Sx = 1.0e18f, Sy = 1.0e18f, Sz = 1.0e18f, Ex = 0.f, Ey = 0.f, Ez = 0.f, mj = 0.f,
              ml = 0.f;
        if (b < n) {
            const float4 h = hi[b], l = lo[b];
            rel_ds(h.x, l.x, gm.c[0], Sx, Ex);
            rel_ds(h.y, l.y, gm.c[1], Sy, Ey);
            rel_ds(h.z, l.z, gm.c[2], Sz, Ez);
            mj = h.w;
            ml = l.w;
        }
        __syncwarp();
        pair_tile_put(sg, lane, Sx, Sy, Sz, mj, Ex, Ey, Ez);
        pair_tile_put_mlo(sg, lane, ml);
        __syncwarp();

        // the left-out pairs: the near kernel's r^2 test, same operands
        uint32_t mk[IPT];
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            mk[k] = 0u;
            if (!need[k]) continue;
            const int i = (tile0 + k) * kChunk + lane;
#pragma unroll 2
            for (int p = 0; p < kChunk / 2; ++p) {
                const JPair j = pair_tile_get(sg, p);
                const int j0 = jc * kChunk + 2 * p;
                const PairGeom g = pair_geom(j, nsx[k], nsy[k], nsz[k], nex[k], ney[k], nez[k], e2);
                const uint32_t b0 = (g.r2.x < thrx && i < n && j0 != i) ? 1u : 0u;
                const uint32_t b1 = (g.r2.y < thrx && i < n && j0 + 1 != i) ? 2u : 0u;
                mk[k] |= (b0 | b1) << (2 * p);
            }
        }
        // pairs numbered by (k, lane, bit)
        int off[IPT], total = 0;
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            const int c = __popc(mk[k]);
            int inc = c;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, inc, d);
                if (lane >= d) inc += v;
            }
            off[k] = total + inc - c;
            total += __shfl_sync(0xffffffffu, inc, 31);
        }
        for (int r = 0; r < total; r += kExactRound) {
            const int r1 = min(total, r + kExactRound);
#pragma unroll
            for (int k = 0; k < IPT; ++k) {
                uint32_t m = mk[k];
                for (int e = off[k]; m != 0u; ++e) {
                    const int bit = __ffs(m) - 1;
                    m &= m - 1u;
                    if (e >= r && e < r1) evt[w][e - r] = (uint16_t)(((k * 32 + lane) << 5) | bit);
                }
            }
            __syncwarp();
            for (int e = lane; e < r1 - r; e += 32) {
                const int code = evt[w][e];
                const int il = code >> 5, bit = code & 31;
                const int p = bit >> 1;
                const bool u = bit & 1;
                const float4 A = sg.s[p], B = sg.t[p], C = sg.e[p];
                const float2 F = sg.f[p], M = sg.g[p];
                const float *q = ibody[il];
                DS t[3];
                pair_term_ds(DS{u ? A.y : A.x, u ? C.y : C.x}, DS{u ? A.w : A.z, u ? C.w : C.z},
                             DS{u ? B.y : B.x, u ? F.y : F.x}, DS{u ? B.w : B.z, u ? M.y : M.x},
                             DS{q[0], q[1]}, DS{q[2], q[3]}, DS{q[4], q[5]}, e2ds, t);
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    term[w][e][2 * a] = t[a].hi;
                    term[w][e][2 * a + 1] = t[a].lo;
                }
            }
            __syncwarp();
#pragma unroll
            for (int k = 0; k < IPT; ++k) {
                uint32_t m = mk[k];
                for (int e = off[k]; m != 0u; ++e) {
                    m &= m - 1u;
                    if (e >= r && e < r1)
#pragma unroll
                        for (int a = 0; a < 3; ++a)
                            acc[k][a] = ds_add(acc[k][a],
                                               DS{term[w][e - r][2 * a], term[w][e - r][2 * a + 1]});
                }
            }
            __syncwarp();
        }
    }

    // the warps' sums in warp order
#pragma unroll
    for (int k = 0; k < IPT; ++k)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            red[w][k * 32 + lane][2 * a] = acc[k][a].hi;
            red[w][k * 32 + lane][2 * a + 1] = acc[k][a].lo;
        }
    __syncthreads();
    if (w != 0) return;
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int i = (tile0 + k) * kChunk + lane;
        DS sum[3] = {DS{0.f, 0.f}, DS{0.f, 0.f}, DS{0.f, 0.f}};
        for (int v = 0; v < kExactWarps; ++v)
#pragma unroll
            for (int a = 0; a < 3; ++a)
                sum[a] = ds_add(sum[a], DS{red[v][k * 32 + lane][2 * a],
                                           red[v][k * 32 + lane][2 * a + 1]});
        if (i < n)
#pragma unroll
            for (int a = 0; a < 3; ++a)
                ex[(size_t)(3 * blockIdx.y + a) * n + i] = (double)sum[a].hi + (double)sum[a].lo;
    }
}

// Body i's sum over the planes of np diagonals from p0, as a double-single: 32
// bodies per block, 8 groups of planes in strides (each group's sum in order,
// its loads ahead of it), then the groups in order.  acc: the sums of the earlier
// passes (first: none yet), written back unless this is the last pass, which
// adds the near segments (sum - comp; in strides too) and the left-out pairs:
// a[order[i]] = G * (far + near + ex_i), scaled in FP64.  Bound by memory: one
// thread per body had too few loads in flight (66 us at n = 65,536 and half of the present 410 MB).
constexpr int kCombineGroups = 8;
__global__ void __launch_bounds__(32 * kCombineGroups)
combine_sorted_kernel(const float2 *__restrict__ part, int blocks, int p0, int np, bool first,
                      bool last, float *__restrict__ acc, const float *__restrict__ psum,
                      const float *__restrict__ pcomp, int n, int segments, double G,
                      const uint32_t *__restrict__ order, const double *__restrict__ ex,
                      int shares, double *__restrict__ ax, double *__restrict__ ay,
                      double *__restrict__ az)
{
    __shared__ float2 sh[kCombineGroups][3][32];
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + lane;
    const size_t plane = (size_t)n;
    const int blk = i / (kFarTiles * kTile);
    float hi[3] = {0.f, 0.f, 0.f}, lo[3] = {0.f, 0.f, 0.f};
    if (i < n) {
        for (int k0 = g; k0 < 2 * np; k0 += 8 * kCombineGroups) {
            float2 t[8][3];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int k = k0 + u * kCombineGroups;
                const bool use = k < np ? pair_first(p0 + k, blk, blocks)
                                        : k < 2 * np && pair_second(p0 + k - np, blk, blocks);
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    t[u][c] = use ? part[((size_t)k * 3 + c) * plane + i] : dup2(0.f);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u)
#pragma unroll
                for (int c = 0; c < 3; ++c) ds_add_kahan(hi[c], lo[c], t[u][c].x, -t[u][c].y);
        }
        for (int s = g; last && s < segments; s += kCombineGroups)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const size_t at = ((size_t)s * 3 + c) * plane + i;
                ds_add_kahan(hi[c], lo[c], psum[at], pcomp[at]);
            }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) sh[g][c][lane] = make_float2(hi[c], lo[c]);
    __syncthreads();
    if (g >= 3 || i >= n) return;  // warp c finishes component c
    const int c = g;
    float2 s = first ? make_float2(0.f, 0.f)
                     : make_float2(acc[c * plane + i], acc[(3 + c) * plane + i]);
#pragma unroll
    for (int k = 0; k < kCombineGroups; ++k)
        ds_add_kahan(s.x, s.y, sh[k][c][lane].x, -sh[k][c][lane].y);
    if (!last) {
        acc[c * plane + i] = s.x;
        acc[(3 + c) * plane + i] = s.y;
        return;
    }
    const uint32_t o = order[i];
    if (!NB_IN_RANGE(o, n)) return;
    double left_out = ex[c * plane + i];
    for (int k = 1; k < shares; ++k) left_out += ex[(3 * (size_t)k + c) * plane + i];
    double *out = c == 0 ? ax : (c == 1 ? ay : az);
    out[o] = G * (((double)s.x + (double)s.y) + left_out);
}

} // namespace

void SortedBuffers::release()
{
    hi.release();
    lo.release();
    partials.release();
    boxes.release();
    tiles.release();
    exact.release();
    far.release();
    acc.release();
    if (fork) cudaEventDestroy(fork);
    fork = nullptr;
    for (int k = 0; k < 2; ++k) {
        if (side[k]) cudaStreamDestroy(side[k]);
        if (join[k]) cudaEventDestroy(join[k]);
        side[k] = nullptr;
        join[k] = nullptr;
    }
    if (sorter) bh_destroy(sorter);
    sorter = nullptr;
    order = nullptr;
    centre = nullptr;
    order_n = -1;
}

bool direct_sorted_enabled(int n, int flags)
{
    if (flags & NB_FLAG_MIXED_UNSORTED) return false;
    if (flags & NB_FLAG_MIXED_SORTED) return n > 0;
    static const bool on = [] {
        const char *e = std::getenv("NB_DIRECT_SORTED");
        return !(e && std::strcmp(e, "0") == 0);
    }();
    return on && n >= kSortedMinBodies;
}

// The near kernel's j-split: about 10,000 warps (16 per SM and four waves),
// at most 32 segments (4,000 warps: 1.93 ms a step instead of 1.48 at N = 65,536,
// the longest rows alone at the end; 20,000: the same).  A function of n alone.
static int near_segments(int tiles) { return std::min(32, std::max(2, 10000 / tiles)); }

// CTAs per tile of the exact kernel: about 1,000 CTAs, so that a tile with many
// left-out pairs is shared out where the tiles are few (at N = 16,384 one CTA
// per tile took 175 us, longer than all the other pairs).
static int exact_shares(int tiles) { return std::min(8, std::max(1, 1024 / tiles)); }

// The left-out pairs (into b.exact, 3 n doubles per share) and the near kernel's
// ordered pairs (into b.partials), each on a side stream: both wait for the
// staging on st (fork) and st waits for them before the combine (join).  The side
// streams have the highest priority, so their CTAs start at once and the longest
// chains run while the far kernel fills the GPU.
static nb_status launch_side(const float4 *hi, const float4 *lo, int n, int segments, double eps2,
                             SortedBuffers &b, cudaStream_t st)
{
    const int nchunks = (n + kChunk - 1) / kChunk, tiles = (nchunks + 1) / 2;
    const int shares = exact_shares(tiles);
    NB_TRY(b.exact.reserve(sizeof(double) * 3 * (size_t)n * shares));
    NB_TRY(b.partials.reserve(sizeof(float) * 6 * (size_t)n * segments));
    int least = 0, greatest = 0;
    if (!b.fork) {
        NB_CUDA_TRY(cudaEventCreateWithFlags(&b.fork, cudaEventDisableTiming));
    }
    for (int k = 0; k < 2; ++k)
        if (!b.side[k]) {
            NB_CUDA_TRY(cudaDeviceGetStreamPriorityRange(&least, &greatest));
            NB_CUDA_TRY(cudaEventCreateWithFlags(&b.join[k], cudaEventDisableTiming));
            NB_CUDA_TRY(cudaStreamCreateWithPriority(&b.side[k], cudaStreamNonBlocking, greatest));
        }
    NB_CUDA_TRY(cudaEventRecord(b.fork, st));
    for (int k = 0; k < 2; ++k) NB_CUDA_TRY(cudaStreamWaitEvent(b.side[k], b.fork, 0));
    const float4 *box = b.boxes.as<float4>(), *tile = b.tiles.as<float4>();
    exact_pairs_kernel<<<dim3(tiles, shares), kExactWarps * 32, 0, b.side[0]>>>(
        hi, lo, box, tile, n, nchunks, eps2 > 0.0 ? (float)eps2 : 0.0f, kFarFactor2,
        eps2 > 0.0 ? eps2 : 0.0, b.exact.as<double>());
    NB_LAUNCH_CHECK();
    float *psum = b.partials.as<float>(), *pcomp = psum + 3 * (size_t)n * segments;
    const dim3 grid(tiles, segments);
    if (eps2 > 0.0)
        direct_near_kernel<false><<<grid, 32, 0, b.side[1]>>>(
            hi, lo, box, tile, n, nchunks, (float)eps2, psum, pcomp, kFarFactor2);
    else
        direct_near_kernel<true><<<grid, 32, 0, b.side[1]>>>(hi, lo, box, tile, n, nchunks, 0.0f,
                                                             psum, pcomp, kFarFactor2);
    NB_LAUNCH_CHECK();
    for (int k = 0; k < 2; ++k) NB_CUDA_TRY(cudaEventRecord(b.join[k], b.side[k]));
    return NB_OK;
}

nb_status direct_mixed_sorted(const double *x, const double *y, const double *z, const double *m,
                              int n, double G, double eps2, double *ax, double *ay, double *az,
                              SortedBuffers &b, cudaStream_t st, const KernelTimer *timer)
{
    if (n <= 0) return NB_OK;
    NvtxRange range("direct_sorted");
    if (!b.sorter) b.sorter = bh_create();
    if (b.order_n != n || b.evals_since_sort >= kResortEvals) {
        // 2^30 cells: far smaller than a 32-body chunk
        NB_TRY(bh_hilbert_order(b.sorter, x, y, z, n, st, &b.order, &b.centre));
        b.order_n = n;
        b.evals_since_sort = 0;
    }
    ++b.evals_since_sort;
    const uint32_t *order = b.order;
    const double *centre = b.centre;
    const int nchunks = (n + kChunk - 1) / kChunk;
    NB_TRY(b.hi.reserve(sizeof(float4) * (size_t)n));
    NB_TRY(b.lo.reserve(sizeof(float4) * (size_t)n));
    NB_TRY(b.boxes.reserve(sizeof(float4) * 2 * (size_t)nchunks));
    float4 *hi = b.hi.as<float4>(), *lo = b.lo.as<float4>();
    const int tiles = (nchunks + 1) / 2;
    NB_TRY(b.tiles.reserve(sizeof(float4) * 2 * (size_t)tiles));
    split_sorted_kernel<<<(tiles + 3) / 4, 128, 0, st>>>(order, x, y, z, m, n, centre,
                                                         exact_cap_per_n(n), hi, lo,
                                                         b.boxes.as<float4>(),
                                                         b.tiles.as<float4>());
    NB_LAUNCH_CHECK();
    const int segments = near_segments(tiles);
    const int blocks = (tiles + kFarTiles - 1) / kFarTiles, diagonals = blocks / 2 + 1;
    // the diagonals in passes whose planes stay within kFarPlaneBytes
    const size_t per_diagonal = sizeof(float2) * 6 * (size_t)n;
    const int pass = (int)std::min<size_t>(diagonals,
                                           std::max<size_t>(1, kFarPlaneBytes / per_diagonal));
    NB_TRY(b.far.reserve(per_diagonal * pass));
    NB_TRY(b.acc.reserve(sizeof(float) * 6 * (size_t)n));
    if (timer && timer->start) NB_CUDA_TRY(cudaEventRecord(timer->start, st));
    NB_TRY(launch_side(hi, lo, n, segments, eps2, b, st));
    float *psum = b.partials.as<float>(), *pcomp = psum + 3 * (size_t)n * segments;
    for (int p0 = 0; p0 < diagonals; p0 += pass) {
        const int np = std::min(pass, diagonals - p0);
        direct_far_kernel<<<(unsigned)blocks * (unsigned)np, 32, 0, st>>>(
            hi, lo, b.tiles.as<float4>(), n, tiles, eps2 > 0.0 ? (float)eps2 : 0.0f, blocks, p0, np,
            b.far.as<float2>());
        NB_LAUNCH_CHECK();
        const bool last = p0 + np == diagonals;
        if (last) {
            for (int k = 0; k < 2; ++k) NB_CUDA_TRY(cudaStreamWaitEvent(st, b.join[k], 0));
            if (timer && timer->stop) NB_CUDA_TRY(cudaEventRecord(timer->stop, st));
        }
        combine_sorted_kernel<<<(n + 31) / 32, 32 * kCombineGroups, 0, st>>>(
            b.far.as<float2>(), blocks, p0, np, p0 == 0, last, b.acc.as<float>(), psum, pcomp, n,
            segments, G, order, b.exact.as<double>(), exact_shares(tiles), ax, ay, az);
        NB_LAUNCH_CHECK();
    }
    return NB_OK;
}

} // namespace nb
