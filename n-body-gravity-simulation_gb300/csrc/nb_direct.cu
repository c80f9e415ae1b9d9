// nb_direct.cu -- all-pairs gravity on sm_103a.
//
// Replaces computeAccelerationNaiveKernel (CUDA/src/force_calculator_naive.cu:4-59,
// one FP64 thread per body, 256-body tiles, ceil(N/256) CTAs).  Two kernels:
//
//  * direct_mixed_kernel -- the mixed term over ordered pairs: the no-allocation entry
//    point from 4096 bodies.  Each body is held as a float4
//    "hi" (x, y, z, m) plus a float4 "lo" (x - hi, ...): a double-single copy of
//    its FP64 position.  The pair displacement is formed as
//    (xj_hi - xi_hi) + (xj_lo - xi_lo), which is exact to FP32 rounding for close
//    pairs, so close encounters keep a relative force error near 1e-7 however far
//    the pair is from the origin.  The rest of the pair term is plain FP32 on the
//    FMA pipe with one MUFU rsqrt (rsqrt.approx.ftz.f32) whose ~1.3e-7 error is
//    removed by a Newton step folded into r^-3 (3 extra FP32 ops: 21 FP32-pipe
//    operations + 1 MUFU per pair against the 12 of the bare pair term).  The
//    FP32 work runs as packed f32x2 operations on j-pairs (two j per
//    instruction, nb_pair.cuh), which halves its issue slots.  Every thread
//    owns IPT i-bodies, so one broadcast shared-memory read of a j-pair feeds
//    IPT pair terms.  Every 32 j the FP32 partial sum is added into a Kahan-compensated
//    (sum, compensation) pair; the CTA's partial over its j-segment is written
//    as FP32 (sum, comp) and the segments are combined as a double-single,
//    scaled by G in FP64.
//    The tensor cores stay idle: a softened 1/r^3 sum is not a contraction.
//
//  * direct_mixed_small_kernel -- the same term below 4096 bodies, in one launch.
//
//  * direct_mixed_pairs_kernel -- the same term over unordered pairs from 4096
//    bodies (below 16,384, where the Hilbert-sorted path takes over).
//
//  * direct_fp64_pairs_kernel -- the 1e-12 path: an FP64 sum over unordered
//    pairs of 32-body tiles (direct_fp64_row_kernel, a warp per body, for small n).
//
// Grid of the mixed kernel: x = i-blocks of BLOCK*IPT bodies, y = j-segments.  The j-split keeps
// all 152 SMs busy at small N (the reference runs 4 CTAs at N = 1024) and the
// segment count is chosen to fill whole waves.
#include "nb_internal.h"
#include "nb_fp64pair.cuh"
#include "nb_after.cuh"
#include "nb_tile.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>
#include <string>

namespace nb {
namespace {

template <int BLOCK, int IPT, bool ZERO_SOFT>
__global__ void __launch_bounds__(BLOCK)
direct_mixed_kernel(const float4 *__restrict__ hi, const float4 *__restrict__ lo, int n,
                    float eps2, int seg_len, float *__restrict__ psum,
                    float *__restrict__ pcomp)
{
    __shared__ PairTile tiles[BLOCK / 32];

    const int tid = threadIdx.x;
    const int ibase = blockIdx.x * (BLOCK * IPT);

    // i-bodies negated and duplicated into f32x2 pairs
    float2 nxh[IPT], nyh[IPT], nzh[IPT], nxl[IPT], nyl[IPT], nzl[IPT];
    float sx[IPT], sy[IPT], sz[IPT], cx[IPT], cy[IPT], cz[IPT];
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int i = ibase + k * BLOCK + tid;
        float4 h = make_float4(0.f, 0.f, 0.f, 0.f), l = h;
        if (i < n) {
            h = hi[i];
            l = lo[i];
        }
        nxh[k] = dup2(-h.x); nyh[k] = dup2(-h.y); nzh[k] = dup2(-h.z);
        nxl[k] = dup2(-l.x); nyl[k] = dup2(-l.y); nzl[k] = dup2(-l.z);
        sx[k] = sy[k] = sz[k] = 0.f;
        cx[k] = cy[k] = cz[k] = 0.f;
    }
    const float2 e2 = dup2(eps2);

    const int j0 = blockIdx.y * seg_len;
    const int j1 = min(n, j0 + seg_len);
    for (int t0 = j0; t0 < j1; t0 += BLOCK) {
        const int j = t0 + tid;
        float4 h = far_body(), l = make_float4(0.f, 0.f, 0.f, 0.f);
        if (j < j1) {
            h = hi[j];
            l = lo[j];
        }
        __syncthreads();
        pair_tile_put(tiles[tid >> 5], tid & 31, h.x, h.y, h.z, h.w, l.x, l.y, l.z);
        __syncthreads();

        // FP32 partial sums over each 32-body tile (16 terms per f32x2 lane),
        // Kahan-added into (s, c): the rounding of a running FP32 sum grows
        // with its length, and short runs keep it below the per-term error of
        // the pair arithmetic.
#pragma unroll 1
        for (int t = 0; t < BLOCK / 32; ++t) {
            float2 ax[IPT], ay[IPT], az[IPT];
#pragma unroll
            for (int k = 0; k < IPT; ++k) ax[k] = ay[k] = az[k] = dup2(0.f);
#pragma unroll 2
            for (int p = 0; p < 16; ++p) {
                const JPair jp = pair_tile_get(tiles[t], p);
#pragma unroll
                for (int k = 0; k < IPT; ++k)
                    pair_term2<ZERO_SOFT>(jp, nxh[k], nyh[k], nzh[k], nxl[k], nyl[k], nzl[k], e2,
                                          ax[k], ay[k], az[k]);
            }
#pragma unroll
            for (int k = 0; k < IPT; ++k) {
                kahan_add(sx[k], cx[k], ax[k].x + ax[k].y);
                kahan_add(sy[k], cy[k], ay[k].x + ay[k].y);
                kahan_add(sz[k], cz[k], az[k].x + az[k].y);
            }
        }
    }

    const size_t plane = (size_t)n;
    const size_t base = (size_t)blockIdx.y * 3 * plane;
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int i = ibase + k * BLOCK + tid;
        if (i < n) {
            psum[base + i] = sx[k];
            psum[base + plane + i] = sy[k];
            psum[base + 2 * plane + i] = sz[k];
            pcomp[base + i] = cx[k];
            pcomp[base + plane + i] = cy[k];
            pcomp[base + 2 * plane + i] = cz[k];
        }
    }
}

// a_i = G * sum_s (sum_s - comp_s) as a double-single scaled in FP64: 32 bodies per
// block, 8 groups of segments in strides (their loads ahead of the ordered sums),
// then the groups in order.  Bound by the latency of those loads and sums: 22.1 us
// at n = 1000 and 32 segments with one load waiting for the last sum in 256-body
// CTAs, 6.9 with one warp per 32 bodies and 16 segments' loads at once, 6.2 now.
constexpr int kCombineGroups = 8;
__global__ void __launch_bounds__(32 * kCombineGroups)
combine_mixed_kernel(const float *__restrict__ psum,
                                     const float *__restrict__ pcomp, int n, int segments,
                                     double G, double *__restrict__ ax,
                                     double *__restrict__ ay, double *__restrict__ az)
{
    __shared__ float2 sh[kCombineGroups][3][32];
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + lane;
    const size_t plane = (size_t)n;
    float hi[3] = {0.f, 0.f, 0.f}, lo[3] = {0.f, 0.f, 0.f};
    if (i < n)
        for (int s0 = g; s0 < segments; s0 += 4 * kCombineGroups) {
            float t[4][3], q[4][3];
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const int s = s0 + u * kCombineGroups;
                    const size_t at = ((size_t)s * 3 + c) * plane + i;
                    t[u][c] = s < segments ? psum[at] : 0.f;
                    q[u][c] = s < segments ? pcomp[at] : 0.f;
                }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int c = 0; c < 3; ++c) ds_add_kahan(hi[c], lo[c], t[u][c], q[u][c]);
        }
#pragma unroll
    for (int c = 0; c < 3; ++c) sh[g][c][lane] = make_float2(hi[c], lo[c]);
    __syncthreads();
    if (g >= 3 || i >= n) return;  // warp c finishes component c
    const int c = g;
    float2 s = dup2(0.f);
#pragma unroll
    for (int k = 0; k < kCombineGroups; ++k)
        ds_add_kahan(s.x, s.y, sh[k][c][lane].x, -sh[k][c][lane].y);
    double *out = c == 0 ? ax : (c == 1 ? ay : az);
    out[i] = G * ((double)s.x + (double)s.y);
}

// ---------------------------------------------------------------- mixed, small systems
// Below kMixedPairsMin bodies a cluster of 8 CTAs sums 32 i-bodies: each of its 32 warps
// takes a share of the j-tiles (as direct_mixed_kernel does), a CTA combines its warps'
// Kahan pairs, and the first the eight CTAs': no partial sums in memory, and no second
// launch.
// Bound by latency: launch, two trips to memory, the tiles' 16 steps each, the ordered
// sums.  A velocity-Verlet step at n = 100 / 1000 / 2000 / 4000 takes 10.4 / 12.4 / 16.5 /
// 26.8 us in a row of steps, with the sums in a second kernel 14.5 / 16.5 / 21.3 / 30.8;
// 8 warps per CTA 10.4 / 14.5 / 16.5 / 25.2, two i-bodies per lane no less.
// A cluster writes its bodies' next split positions (after) while others still read the
// present ones: those are two arrays.
constexpr int kSmallCtas = 8, kSmallWarps = 4;

template <bool ZERO_SOFT>
__global__ void __cluster_dims__(kSmallCtas, 1, 1) __launch_bounds__(32 * kSmallWarps)
direct_mixed_small_kernel(const float4 *__restrict__ hi, const float4 *__restrict__ lo, int n,
                          float eps2, int warp_tiles, double G, double *__restrict__ ax,
                          double *__restrict__ ay, double *__restrict__ az,
                          const AfterForce after)
{
    __shared__ PairTile tiles[kSmallWarps];
    __shared__ float2 part[kSmallWarps][3][32];  // a warp's Kahan pairs (sum, comp)
    __shared__ float2 sum[3][32];                // the CTA's, as double-singles
    auto cluster = cooperative_groups::this_cluster();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int rank = blockIdx.x % kSmallCtas;
    const int i = blockIdx.x / kSmallCtas * 32 + lane;

    // the i-body negated and duplicated into f32x2 pairs
    float4 h = make_float4(0.f, 0.f, 0.f, 0.f), l = h;
    if (i < n) {
        h = hi[i];
        l = lo[i];
    }
    const float2 nxh = dup2(-h.x), nyh = dup2(-h.y), nzh = dup2(-h.z);
    const float2 nxl = dup2(-l.x), nyl = dup2(-l.y), nzl = dup2(-l.z);
    const float2 e2 = dup2(eps2);
    float s[3] = {0.f, 0.f, 0.f}, q[3] = {0.f, 0.f, 0.f};
    const int j0 = (rank * kSmallWarps + w) * warp_tiles * 32;
    const int j1 = min(n, j0 + warp_tiles * 32);
    for (int t0 = j0; t0 < j1; t0 += 32) {
        const int j = t0 + lane;
        h = far_body();
        l = make_float4(0.f, 0.f, 0.f, 0.f);
        if (j < j1) {
            h = hi[j];
            l = lo[j];
        }
        __syncwarp();
        pair_tile_put(tiles[w], lane, h.x, h.y, h.z, h.w, l.x, l.y, l.z);
        __syncwarp();
        float2 t[3] = {dup2(0.f), dup2(0.f), dup2(0.f)};
#pragma unroll 2
        for (int p = 0; p < 16; ++p)
            pair_term2<ZERO_SOFT>(pair_tile_get(tiles[w], p), nxh, nyh, nzh, nxl, nyl, nzl, e2,
                                  t[0], t[1], t[2]);
#pragma unroll
        for (int c = 0; c < 3; ++c) kahan_add(s[c], q[c], t[c].x + t[c].y);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) part[w][c][lane] = make_float2(s[c], q[c]);
    __syncthreads();
    if (w < 3) {
        float2 v = dup2(0.f);
#pragma unroll
        for (int u = 0; u < kSmallWarps; ++u)
            ds_add_kahan(v.x, v.y, part[u][w][lane].x, part[u][w][lane].y);
        sum[w][lane] = v;
    }
    cluster.sync();
    if (rank == 0 && w < 3 && i < n) {  // warp c finishes component c
        float2 t[kSmallCtas], v = dup2(0.f);
#pragma unroll
        for (int u = 0; u < kSmallCtas; ++u) t[u] = *cluster.map_shared_rank(&sum[w][lane], u);
#pragma unroll
        for (int u = 0; u < kSmallCtas; ++u) ds_add_kahan(v.x, v.y, t[u].x, -t[u].y);
        double *out = w == 0 ? ax : (w == 1 ? ay : az);
        const double a = G * ((double)v.x + (double)v.y);
        out[i] = a;
        after_force(after, w, i, a);
    }
    cluster.sync();  // no CTA leaves while its sums are read
}

// ---------------------------------------------------------------- mixed, unordered pairs
// From kMixedPairsMin bodies every unordered pair is evaluated once (nb_tile.cuh)
// over pairs of 256-body blocks: diagonal p pairs block a with a + p.  A one-warp
// CTA takes an eighth of a block pair's 4 x 4 tiles: two i-tiles (four bodies per
// lane) against one j-tile, whose sums it keeps in shared memory.  A body has
// kPairV planes of Kahan pairs per diagonal from its block as the first, kPairH
// as the second; the combine adds them in order.
// Bound by dispatch (nb_tile.cuh), below 8,000 bodies by how evenly the CTAs fill
// the SMs.  An evaluation at n = 5,003 / 8,000 / 16,383 takes 29 / 46 / 140 us;
// one CTA per block pair (fewer planes) 51 / 54 / 150, the ordered-pairs kernel
// 40 / 73 / 200.
constexpr int kPairTiles = 4;
constexpr int kPairBlock = kPairTiles * kTile;
constexpr int kPairH = kPairTiles / 2, kPairV = kPairTiles;

template <bool ZERO_SOFT>
__global__ void __launch_bounds__(32, 16)
direct_mixed_pairs_kernel(const float4 *__restrict__ hi, const float4 *__restrict__ lo, int n,
                          float eps2, bool soft, int blocks, int p0, int np,
                          float2 *__restrict__ part)
{
    __shared__ TileJ stage;
    __shared__ TileJLow low;
    __shared__ TileSums jsum, isum[2];
    const int lane = threadIdx.x;
    const int share = blockIdx.x % (kPairH * kPairV), item = blockIdx.x / (kPairH * kPairV);
    const int a = item % blocks, dp = item / blocks, p = p0 + dp;
    if (!pair_first(p, a, blocks)) return;
    const int h = share / kPairV, v = share % kPairV, u = 2 * h;
    const int tiles = (n + kTile - 1) / kTile;
    const int ti0 = a * kPairTiles, tj0 = (a + p) % blocks * kPairTiles;
    const int ta = min(kPairTiles, tiles - ti0), tb = min(kPairTiles, tiles - tj0);
    const bool two = u + 1 < ta;
    const float2 e2 = dup2(eps2);
    const float c[3] = {0.f, 0.f, 0.f};
    tile_sums_zero(jsum, lane);
    tile_sums_zero(isum[0], lane);
    tile_sums_zero(isum[1], lane);
    // within a block: the j-tiles after the pair's own two, and with the last of
    // those (own) the pair's tiles against themselves and each other
    const int own = p == 0 ? u + two : -1;
    float mi, mj;
    if (two && v > own && v < tb) {
        TileI<4> ti;
        TileILow<4> tl;
        const bool ei = tile_load_i<false>(hi, lo, n, (ti0 + u) * kTile, c, ti, tl, mi);
        if (tile_stage_j<false>(hi, lo, n, (tj0 + v) * kTile, c, stage, low, mj) && ei && soft)
            tile_pair<kNearTerm, true, ZERO_SOFT, 4>(stage, &low, lane, ti, &tl, e2, mi, mj, isum,
                                                     jsum);
        else
            tile_pair<kNearTerm, false, ZERO_SOFT, 4>(stage, &low, lane, ti, &tl, e2, 0.f, 0.f,
                                                      isum, jsum);
    } else if (u < ta && v < tb && (p == 0 ? v == own : !two)) {
        // one i-tile at a time: the pair's own (within), or the last of an odd number
        for (int w = 0; w < 1 + two; ++w) {
            TileI<2> ti;
            TileILow<2> tl;
            const bool ei = tile_load_i<false>(hi, lo, n, (ti0 + u + w) * kTile, c, ti, tl, mi);
            for (int t = p == 0 ? u + w : v; t <= v; ++t) {
                const bool equal =
                    tile_stage_j<false>(hi, lo, n, (tj0 + t) * kTile, c, stage, low, mj) && ei &&
                    soft;
                if (p == 0 && t == u + w)
                    tile_self<ZERO_SOFT>(stage, &low, lane, ti, &tl, e2, isum[w]);
                else if (equal)
                    tile_pair<kNearTerm, true, ZERO_SOFT, 2>(stage, &low, lane, ti, &tl, e2, mi,
                                                             mj, isum + w, jsum);
                else
                    tile_pair<kNearTerm, false, ZERO_SOFT, 2>(stage, &low, lane, ti, &tl, e2, 0.f,
                                                              0.f, isum + w, jsum);
            }
        }
    }
    __syncwarp();
    // a share without pairs writes zeros: the combine reads every plane
    const size_t plane = 3 * (size_t)n;
    float2 *pa = part + (size_t)(dp * kPairV + v) * plane;
    float2 *pb = part + (size_t)(np * kPairV + dp * kPairH + h) * plane;
    for (int w = 0; w < 3; ++w) {
        if (w < 2 ? u + w >= ta : v >= tb) continue;
        float2 *out = w < 2 ? pa : pb;
        const int i = (w < 2 ? ti0 + u + w : tj0 + v) * kTile + lane;
        const TileSums &sum = w < 2 ? isum[w] : jsum;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const float2 t = sum.s[d][lane], e = sum.c[d][lane];
            if (i < n) out[(size_t)d * n + i] = make_float2(t.x, e.x);
            if (i + 32 < n) out[(size_t)d * n + i + 32] = make_float2(t.y, e.y);
        }
    }
}

// a_i = G * the sum of body i's planes as a double-single: 32 bodies per block, 8
// groups of planes in strides (their loads ahead of the ordered sums), then the
// groups in order.  acc: the sums of earlier passes over the diagonals (first:
// none yet), written back unless this is the last.
constexpr int kPairGroups = 8;
__global__ void __launch_bounds__(32 * kPairGroups)
combine_mixed_pairs_kernel(const float2 *__restrict__ part, int n, int blocks, int p0, int np,
                           bool first, bool last, float *__restrict__ acc, double G,
                           double *__restrict__ ax, double *__restrict__ ay,
                           double *__restrict__ az, const AfterForce after)
{
    constexpr int H = kPairH, V = kPairV;
    __shared__ float2 sh[kPairGroups][3][32];
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + lane;
    float hi[3] = {0.f, 0.f, 0.f}, lo[3] = {0.f, 0.f, 0.f};
    if (i < n) {
        const int blk = i / kPairBlock, planes = np * (V + H);
        for (int k0 = g; k0 < planes; k0 += 4 * kPairGroups) {
            float2 t[4][3];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int k = k0 + u * kPairGroups, q = k - np * V;
                const bool use =
                    q < 0 ? pair_first(p0 + k / V, blk, blocks)
                          : k < planes && (p0 + q / H == 0 || pair_second(p0 + q / H, blk, blocks));
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    t[u][c] = use ? part[((size_t)k * 3 + c) * n + i] : dup2(0.f);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int c = 0; c < 3; ++c) ds_add_kahan(hi[c], lo[c], t[u][c].x, -t[u][c].y);
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) sh[g][c][lane] = make_float2(hi[c], lo[c]);
    __syncthreads();
    if (g >= 3 || i >= n) return;  // warp c finishes component c
    const int c = g;
    float2 s = first ? dup2(0.f) : make_float2(acc[(size_t)c * n + i], acc[(size_t)(3 + c) * n + i]);
#pragma unroll
    for (int k = 0; k < kPairGroups; ++k)
        ds_add_kahan(s.x, s.y, sh[k][c][lane].x, -sh[k][c][lane].y);
    if (!last) {
        acc[(size_t)c * n + i] = s.x;
        acc[(size_t)(3 + c) * n + i] = s.y;
        return;
    }
    double *out = c == 0 ? ax : (c == 1 ? ay : az);
    const double a = G * ((double)s.x + (double)s.y);
    out[i] = a;
    after_force(after, c, i, a);
}

// ---------------------------------------------------------------- FP64
// Small systems: one warp sums a body's whole row, lanes striding over j, and
// reduces it with shuffles, so no partial sums and no second launch.  Bound by
// the latency of a few dependent FP64 operations (8.1 us at n = 100; one-warp
// CTAs of 32 bodies walking all j took 77 us there).  Up to 512 bodies: beyond,
// its 16 FP64 operations per ordered pair cost more than the pairs kernel's 10
// and a combine.
template <bool ZERO_SOFT>
__global__ void __launch_bounds__(32)
direct_fp64_row_kernel(const double *__restrict__ x, const double *__restrict__ y,
                       const double *__restrict__ z, const double *__restrict__ m, int n,
                       double eps2, double G, double *__restrict__ ax, double *__restrict__ ay,
                       double *__restrict__ az, const AfterForce after)
{
    const int i = blockIdx.x;
    const double xi = x[i], yi = y[i], zi = z[i];
    double a[3] = {0.0, 0.0, 0.0};
#pragma unroll 2
    for (int j = threadIdx.x; j < n; j += 32) {
        const double dx = x[j] - xi, dy = y[j] - yi, dz = z[j] - zi;
        const double s = m[j] * inv_cube<ZERO_SOFT>(fma(dz, dz, fma(dy, dy, fma(dx, dx, eps2))));
        a[0] = fma(dx, s, a[0]);
        a[1] = fma(dy, s, a[1]);
        a[2] = fma(dz, s, a[2]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < 3; ++c) a[c] += __shfl_xor_sync(0xffffffffu, a[c], o);
    if (threadIdx.x < 3) {  // lane c finishes component c
        const int c = threadIdx.x;
        double *out = c == 0 ? ax : (c == 1 ? ay : az);
        const double t = G * (c == 0 ? a[0] : (c == 1 ? a[1] : a[2]));
        out[i] = t;
        after_force(after, c, i, t);
    }
}

// One step of a tile pair: the lane's i-body and the j-body it holds now.  The
// pair's r^-3 serves both bodies: 20 FP64 operations for two interactions,
// where a sum over ordered pairs spends 16 on each.
struct Fp64Body {
    double x, y, z, m;
};
template <bool ZERO_SOFT, bool BOTH>
__device__ __forceinline__ void fp64_pair(const Fp64Body &bi, const Fp64Body &bj, double eps2,
                                          bool valid, double (&ai)[3], double (&aj)[3])
{
    const double dx = bj.x - bi.x, dy = bj.y - bi.y, dz = bj.z - bi.z;
    double q = inv_cube<ZERO_SOFT>(fma(dz, dz, fma(dy, dy, fma(dx, dx, eps2))));
    q = valid ? q : 0.0;
    const double si = bj.m * q;
    ai[0] = fma(dx, si, ai[0]);
    ai[1] = fma(dy, si, ai[1]);
    ai[2] = fma(dz, si, ai[2]);
    if (BOTH) {
        const double sj = -(bi.m * q);
        aj[0] = fma(dx, sj, aj[0]);
        aj[1] = fma(dy, sj, aj[1]);
        aj[2] = fma(dz, sj, aj[2]);
    }
}

__device__ __forceinline__ Fp64Body fp64_load(const double *__restrict__ x,
                                              const double *__restrict__ y,
                                              const double *__restrict__ z,
                                              const double *__restrict__ m, int n, int i)
{
    if (i >= n) return Fp64Body{0.0, 0.0, 0.0, 0.0};
    return Fp64Body{x[i], y[i], z[i], m[i]};
}

__device__ __forceinline__ Fp64Body fp64_rotate(const Fp64Body &b, int src)
{
    return Fp64Body{__shfl_sync(0xffffffffu, b.x, src), __shfl_sync(0xffffffffu, b.y, src),
                    __shfl_sync(0xffffffffu, b.z, src), __shfl_sync(0xffffffffu, b.m, src)};
}

// One CTA = one block pair of diagonal p (blocks of 32 T bodies).  A warp holds
// body l of an i-tile in lane l; the bodies of a j-tile and their sums rotate
// through the lanes by shuffles, so at step s lane l meets body (l + s) mod 32
// and adds to both sums: no partial of the j side leaves the registers before
// its tile is done.  The i-tile's sums stay in registers over the second block,
// the second block's in shared memory over the first; each is written once, to
// the plane of its (diagonal, side).  Small systems (T == 1) split the 32
// rotations of their one tile pair over the WARPS warps of the CTA.
// Bound by the FP64 pipe: 86 % busy at n = 10,000, 1.98 ms for 5.0e7 pairs (the
// sum over ordered pairs: 3.63 ms); 28 us at n = 1024 (57).
template <bool ZERO_SOFT, int WARPS>
__global__ void __launch_bounds__(32 * WARPS)
direct_fp64_pairs_kernel(const double *__restrict__ x, const double *__restrict__ y,
                         const double *__restrict__ z, const double *__restrict__ m, int n,
                         double eps2, int blocks, int T, int p0, int np,
                         double *__restrict__ part)
{
    extern __shared__ double sums[];  // [WARPS][3][32 T] of the j side, [WARPS][3][32] of the i side
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, next = (lane + 1) & 31;
    const int a = blockIdx.x % blocks, dp = blockIdx.x / blocks, p = p0 + dp;
    if (!pair_first(p, a, blocks)) return;
    const int b = (a + p) % blocks;
    const int width = 32 * T;
    const int a0 = a * width, b0 = b * width;
    const int ta = min(T, (n - a0 + 31) / 32), tb = min(T, (n - b0 + 31) / 32);
    double *jsum = sums + (size_t)w * 3 * width;
    double *isum = sums + (size_t)WARPS * 3 * width;  // used when WARPS > 1
    for (int k = lane; k < 3 * width; k += 32) jsum[k] = 0.0;
    __syncwarp();
    const size_t plane = 3 * (size_t)n;
    double *pa = part + (size_t)dp * plane;
    double *pb = part + (size_t)(np + dp) * plane;
    for (int u = 0; u < ta; ++u) {
        const int i = a0 + 32 * u + lane;
        const Fp64Body bi = fp64_load(x, y, z, m, n, i);
        double ai[3] = {0.0, 0.0, 0.0};
        for (int v = p == 0 ? u : 0; v < tb; ++v) {
            const bool self = p == 0 && u == v;
            // the steps of this warp; a tile with itself needs 1 .. 16, the
            // last of which meets every pair from both sides
            const int steps = self ? 16 : 32, s0 = steps * w / WARPS + self,
                      s1 = steps * (w + 1) / WARPS + self;
            const int j0 = b0 + 32 * v;
            Fp64Body bj = fp64_load(x, y, z, m, n, j0 + ((lane + s0) & 31));
            double aj[3] = {0.0, 0.0, 0.0};
            for (int s = s0; s < s1; ++s) {
                const bool valid = i < n && j0 + ((lane + s) & 31) < n;
                if (self && s == 16)
                    fp64_pair<ZERO_SOFT, false>(bi, bj, eps2, valid, ai, aj);
                else
                    fp64_pair<ZERO_SOFT, true>(bi, bj, eps2, valid, ai, aj);
                bj = fp64_rotate(bj, next);
#pragma unroll
                for (int c = 0; c < 3; ++c) aj[c] = __shfl_sync(0xffffffffu, aj[c], next);
            }
            // the sums lane l holds now belong to body (l + s1) mod 32
            const int at = 32 * v + ((lane + s1) & 31);
#pragma unroll
            for (int c = 0; c < 3; ++c) jsum[c * width + at] += aj[c];
            __syncwarp();
        }
        if (WARPS == 1) {
            if (i < n)
#pragma unroll
                for (int c = 0; c < 3; ++c)  // within a block: what the tile took as a j-tile too
                    pa[(size_t)c * n + i] =
                        p == 0 ? ai[c] + jsum[c * width + 32 * u + lane] : ai[c];
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) isum[(w * 3 + c) * 32 + lane] = ai[c];
        }
    }
    if (WARPS == 1) {
        if (p == 0) return;
        for (int v = 0; v < tb; ++v) {
            const int j = b0 + 32 * v + lane;
            if (j < n)
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    pb[(size_t)c * n + j] = jsum[c * width + 32 * v + lane];
        }
        return;
    }
    // T == 1: warp c (mod WARPS) adds the warps' sums of component c in order
    __syncthreads();
    for (int c = w; c < 3; c += WARPS) {
        double si = 0.0, sj = 0.0;
#pragma unroll
        for (int k = 0; k < WARPS; ++k) {
            si += isum[(k * 3 + c) * 32 + lane];
            sj += sums[(k * 3 + c) * 32 + lane];
        }
        if (a0 + lane < n) pa[(size_t)c * n + a0 + lane] = p == 0 ? si + sj : si;
        if (p > 0 && b0 + lane < n) pb[(size_t)c * n + b0 + lane] = sj;
    }
}

// a_i = G * the sum of body i's planes in a fixed order: 8 bodies per block, 32
// groups of planes in strides, each group's sum in order, then a fixed tree.
// Large systems take their diagonals in several passes (add: a already holds
// the earlier passes' sums, not yet scaled; last: scale by G).
__global__ void __launch_bounds__(256)
combine_fp64_kernel(const double *__restrict__ part, int n, int blocks, int width, int p0, int np,
                    bool add, bool last, double G, double *__restrict__ ax,
                    double *__restrict__ ay, double *__restrict__ az, const AfterForce after)
{
    __shared__ double sh[8][3][8];
    const int body = threadIdx.x & 7, g = threadIdx.x >> 3;
    const int i = blockIdx.x * 8 + body;
    double s[3] = {0.0, 0.0, 0.0};
    if (i < n) {
        const int blk = i / width;
#pragma unroll 4
        for (int k = g; k < 2 * np; k += 32) {
            const int p = p0 + (k < np ? k : k - np);
            const bool use = k < np ? pair_first(p, blk, blocks) : pair_second(p, blk, blocks);
            const double *src = part + (size_t)k * 3 * n + i;
#pragma unroll
            for (int c = 0; c < 3; ++c) s[c] += use ? src[(size_t)c * n] : 0.0;
        }
    }
#pragma unroll
    for (int o = 8; o < 32; o <<= 1)
#pragma unroll
        for (int c = 0; c < 3; ++c) s[c] += __shfl_xor_sync(0xffffffffu, s[c], o);
    if ((threadIdx.x & 31) < 8)
#pragma unroll
        for (int c = 0; c < 3; ++c) sh[threadIdx.x >> 5][c][body] = s[c];
    __syncthreads();
    if (threadIdx.x >= 24 || i >= n) return;  // threads 8 c + body finish component c
    const int c = threadIdx.x >> 3;
    double *out = c == 0 ? ax : (c == 1 ? ay : az);
    double t = ((sh[0][c][body] + sh[1][c][body]) + (sh[2][c][body] + sh[3][c][body])) +
               ((sh[4][c][body] + sh[5][c][body]) + (sh[6][c][body] + sh[7][c][body]));
    if (add) t = out[i] + t;
    if (last) t = G * t;
    out[i] = t;
    if (last) after_force(after, c, i, t);
}

__global__ void split_kernel(const double *__restrict__ x, const double *__restrict__ y,
                             const double *__restrict__ z, const double *__restrict__ m, int n,
                             float4 *__restrict__ hi, float4 *__restrict__ lo)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double X = x[i], Y = y[i], Z = z[i];
    const float hx = __double2float_rn(X), hy = __double2float_rn(Y), hz = __double2float_rn(Z);
    hi[i] = make_float4(hx, hy, hz, __double2float_rn(m[i]));
    lo[i] = make_float4(__double2float_rn(X - (double)hx), __double2float_rn(Y - (double)hy),
                        __double2float_rn(Z - (double)hz), 0.0f);
}

// Picks the j-split so that i-blocks x segments fills whole waves of
// `slots` resident CTAs; longer segments are preferred on ties.
int pick_segments(int iblocks, int tiles, int slots)
{
    int best = 1;
    double best_eff = -1.0;
    const int smax = std::max(1, std::min(tiles, 64));
    for (int s = 1; s <= smax; ++s) {
        const int seg_tiles = (tiles + s - 1) / s;
        const int s_eff = (tiles + seg_tiles - 1) / seg_tiles;
        const long ctas = (long)iblocks * s_eff;
        const long waves = (ctas + slots - 1) / slots;
        // useful work / (waves * slots * longest segment): tail and
        // quantisation losses; a small penalty per extra segment.
        const double eff = (double)tiles * iblocks / ((double)waves * slots * seg_tiles) -
                           0.002 * s_eff;
        if (eff > best_eff + 1e-9) {
            best_eff = eff;
            best = s_eff;
        }
    }
    return best;
}

constexpr int kMixBlock = 256;
constexpr int kMixIpt = 4;
constexpr size_t kPairPlaneBytes = (size_t)512 << 20;  // partial planes per pass
constexpr int kF64RowMax = 512;  // largest N of the one-warp-per-body FP64 kernel
constexpr size_t kF64PlaneBytes = (size_t)512 << 20;  // FP64 partial planes per pass

int mix_slots()
{
    static const int slots = [] {
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &per_sm, (const void *)direct_mixed_kernel<kMixBlock, kMixIpt, false>, kMixBlock, 0);
        return std::max(1, per_sm) * device_props().num_sms;
    }();
    return slots;
}

// Launches the small systems' kernel.
nb_status launch_small(const float4 *hi, const float4 *lo, int n, double G, double eps2,
                       double *ax, double *ay, double *az, cudaStream_t st,
                       const AfterForce &after)
{
    const int tiles = (n + 31) / 32, warps = kSmallCtas * kSmallWarps;
    auto *kernel = eps2 > 0.0 ? direct_mixed_small_kernel<false> : direct_mixed_small_kernel<true>;
    kernel<<<tiles * kSmallCtas, 32 * kSmallWarps, 0, st>>>(
        hi, lo, n, eps2 > 0.0 ? (float)eps2 : 0.0f, (tiles + warps - 1) / warps, G, ax, ay, az,
        after);
    NB_LAUNCH_CHECK();
    return NB_OK;
}

} // namespace

nb_status split_positions(const double *x, const double *y, const double *z, const double *m,
                          int n, float4 *hi, float4 *lo, cudaStream_t st)
{
    if (n <= 0) return NB_OK;
    split_kernel<<<(n + 255) / 256, 256, 0, st>>>(x, y, z, m, n, hi, lo);
    NB_LAUNCH_CHECK();
    return NB_OK;
}

static nb_status direct_mixed_pairs(const float4 *hi, const float4 *lo, int n, double G,
                                    double eps2, double *ax, double *ay, double *az,
                                    DevBuf &partials, cudaStream_t st, const KernelTimer *timer,
                                    const AfterForce &after)
{
    const int blocks = (n + kPairBlock - 1) / kPairBlock, diagonals = blocks / 2 + 1;
    // planes of 3 n Kahan pairs, the diagonals in passes whose planes stay
    // within kPairPlaneBytes; behind them the sums between passes
    const size_t per_diagonal = sizeof(float2) * 3 * (size_t)n * (kPairH + kPairV);
    const int pass = (int)std::min<size_t>(diagonals,
                                           std::max<size_t>(1, kPairPlaneBytes / per_diagonal));
    NB_TRY(partials.reserve(per_diagonal * pass + sizeof(float) * 6 * (size_t)n));
    float2 *part = partials.as<float2>();
    float *acc = reinterpret_cast<float *>(part + per_diagonal / sizeof(float2) * pass);
    if (timer && timer->start) NB_CUDA_TRY(cudaEventRecord(timer->start, st));
    for (int p0 = 0; p0 < diagonals; p0 += pass) {
        const int np = std::min(pass, diagonals - p0);
        const unsigned grid = (unsigned)blocks * (unsigned)np * (kPairH * kPairV);
        if (eps2 > 0.0)
            direct_mixed_pairs_kernel<false><<<grid, 32, 0, st>>>(
                hi, lo, n, (float)eps2, equal_soft(eps2), blocks, p0, np, part);
        else
            direct_mixed_pairs_kernel<true><<<grid, 32, 0, st>>>(hi, lo, n, 0.0f, false, blocks,
                                                                 p0, np, part);
        NB_LAUNCH_CHECK();
        const bool last = p0 + np == diagonals;
        if (last && timer && timer->stop) NB_CUDA_TRY(cudaEventRecord(timer->stop, st));
        combine_mixed_pairs_kernel<<<(n + 31) / 32, 32 * kPairGroups, 0, st>>>(
            part, n, blocks, p0, np, p0 == 0, last, acc, G, ax, ay, az, after);
        NB_LAUNCH_CHECK();
    }
    return NB_OK;
}

nb_status direct_mixed(const float4 *hi, const float4 *lo, int n, double G, double eps2,
                       double *ax, double *ay, double *az, DevBuf &partials, cudaStream_t st,
                       const KernelTimer *timer, const AfterForce &after)
{
    if (n <= 0) return NB_OK;
    if (n >= kMixedPairsMin)
        return direct_mixed_pairs(hi, lo, n, G, eps2, ax, ay, az, partials, st, timer, after);
    if (timer && timer->start) NB_CUDA_TRY(cudaEventRecord(timer->start, st));
    NB_TRY(launch_small(hi, lo, n, G, eps2, ax, ay, az, st, after));
    if (timer && timer->stop) NB_CUDA_TRY(cudaEventRecord(timer->stop, st));
    return NB_OK;
}

// Tiles of 32 bodies per block of the FP64 block-pair sum: as many as leave 12
// warps per SM (fewer partial planes), which fill the FP64 pipes evenly.  A
// function of n and the SM count alone, so the bits of a result are too.
static int fp64_tiles(int n)
{
    auto block_pairs = [&](int T) {
        const long M = (n + 32 * T - 1) / (32 * T);
        return M * (M + 1) / 2;
    };
    int T = 1;
    while (T < 8 && block_pairs(2 * T) >= 12 * device_props().num_sms) T *= 2;
    return T;
}

template <bool ZERO_SOFT>
static void launch_fp64_pairs(const double *x, const double *y, const double *z, const double *m,
                              int n, double eps2, int blocks, int T, int p0, int np, double *part,
                              cudaStream_t st)
{
    const unsigned grid = (unsigned)blocks * (unsigned)np;
    // one tile pair per CTA: four warps share it, so that 1024 bodies still
    // give each SM 14 warps
    if (T == 1)
        direct_fp64_pairs_kernel<ZERO_SOFT, 4><<<grid, 128, sizeof(double) * 96 * 8, st>>>(
            x, y, z, m, n, eps2, blocks, T, p0, np, part);
    else
        direct_fp64_pairs_kernel<ZERO_SOFT, 1><<<grid, 32, sizeof(double) * 96 * (size_t)T, st>>>(
            x, y, z, m, n, eps2, blocks, T, p0, np, part);
}

nb_status direct_fp64(const double *x, const double *y, const double *z, const double *m, int n,
                      double G, double eps2, double *ax, double *ay, double *az,
                      DevBuf &partials, cudaStream_t st, const KernelTimer *timer,
                      const AfterForce &after)
{
    if (n <= 0) return NB_OK;
    if (n <= kF64RowMax) {
        if (timer && timer->start) NB_CUDA_TRY(cudaEventRecord(timer->start, st));
        if (eps2 > 0.0)
            direct_fp64_row_kernel<false><<<n, 32, 0, st>>>(x, y, z, m, n, eps2, G, ax, ay, az,
                                                             after);
        else
            direct_fp64_row_kernel<true><<<n, 32, 0, st>>>(x, y, z, m, n, 0.0, G, ax, ay, az,
                                                            after);
        NB_LAUNCH_CHECK();
        if (timer && timer->stop) NB_CUDA_TRY(cudaEventRecord(timer->stop, st));
        return NB_OK;
    }
    const int T = fp64_tiles(n);
    const int blocks = (n + 32 * T - 1) / (32 * T);
    const int diagonals = blocks / 2 + 1;
    // planes of 3 n doubles, two per diagonal; bounded by taking the diagonals
    // in passes
    const size_t per_diagonal = sizeof(double) * 6 * (size_t)n;
    const int pass = (int)std::min<size_t>(
        diagonals, std::max<size_t>(1, kF64PlaneBytes / per_diagonal));
    NB_TRY(partials.reserve(per_diagonal * pass));
    double *part = partials.as<double>();
    if (timer && timer->start) NB_CUDA_TRY(cudaEventRecord(timer->start, st));
    for (int p0 = 0; p0 < diagonals; p0 += pass) {
        const int np = std::min(pass, diagonals - p0);
        if (eps2 > 0.0)
            launch_fp64_pairs<false>(x, y, z, m, n, eps2, blocks, T, p0, np, part, st);
        else
            launch_fp64_pairs<true>(x, y, z, m, n, 0.0, blocks, T, p0, np, part, st);
        NB_LAUNCH_CHECK();
        const bool last = p0 + np == diagonals;
        if (last && timer && timer->stop) NB_CUDA_TRY(cudaEventRecord(timer->stop, st));
        combine_fp64_kernel<<<(n + 7) / 8, 256, 0, st>>>(part, n, blocks, 32 * T, p0, np, p0 > 0,
                                                         last, G, ax, ay, az, after);
        NB_LAUNCH_CHECK();
    }
    return NB_OK;
}

} // namespace nb

// ---------------------------------------------------------------------------
// All-pairs forces for callers that cannot allocate device memory.
//
// Some callers of this library may not call cudaMalloc/cudaFree on their hot
// path: a host application whose device memory is entirely owned by its own
// pool allocator, a plugin that is given a fixed device-memory budget at
// start-up, or a real-time loop that cannot afford the implicit device-wide
// synchronisation an allocation or free can cause.  For them,
// nb_direct_mixed_forces_noalloc keeps its scratch in the file-scope device array
// below instead of memory it allocates: the float4 hi/lo mirror of the bodies and, from
// kMixedPairsMin bodies, the per-segment Kahan partial sums of the ordered pairs.  Below,
// it launches the kernel of the NB_DIRECT_MIXED method, which needs the mirror alone.
//
// The array is kNoAllocScratchBytes (16 MiB) on every device that loads this
// library, held until the process exits, and limits n to kNoAllocMaxBodies.
// Its name is only a host-side stand-in in host code: the device address is
// fetched once per device with cudaGetSymbolAddress, by the first call made
// while that device is current (make that first call before any stream
// capture).  Every call shares the one array and leaves its contents behind;
// no part of it has to start at zero, because each call writes every element
// it later reads.  Calls whose kernels overlap on the GPU (different streams,
// or another thread) race on the array and must be serialised by the caller.
// ---------------------------------------------------------------------------
static constexpr size_t kNoAllocScratchBytes = size_t(16) << 20;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

namespace nb {
namespace {

constexpr size_t kNoAllocMaxBodies = 262144;  // hi/lo (32 B) + one segment (24 B) per body
constexpr int kNoAllocMaxDevices = 64;

std::mutex g_noalloc_mutex;
void *g_noalloc_address[kNoAllocMaxDevices] = {};

size_t round_up_256(size_t b) { return (b + 255) / 256 * 256; }

} // namespace
} // namespace nb

extern "C" nb_status nb_direct_mixed_forces_noalloc(size_t n, const double *x, const double *y,
                                                   const double *z, const double *m, double G,
                                                   double softening, double *ax, double *ay,
                                                   double *az, void *stream)
{
    using namespace nb;
    if (n > kNoAllocMaxBodies)
        return fail(NB_ERR_CAPACITY,
                    "nb_direct_mixed_forces_noalloc: n = " + std::to_string(n) +
                        " exceeds its fixed scratch limit of " +
                        std::to_string(kNoAllocMaxBodies) + " bodies");
    if (n == 0) return NB_OK;
    if (!x || !y || !z || !m || !ax || !ay || !az)
        return fail(NB_ERR_INVALID_ARGUMENT, "nb_direct_mixed_forces_noalloc: NULL array");
    if (!(softening >= 0.0))
        return fail(NB_ERR_INVALID_ARGUMENT, "nb_direct_mixed_forces_noalloc: softening < 0");
    int dev = 0;
    NB_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNoAllocMaxDevices)
        return fail(NB_ERR_UNSUPPORTED, "nb_direct_mixed_forces_noalloc: device ordinal >= 64");
    void *base = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_noalloc_mutex);
        if (!g_noalloc_address[dev]) {
            void *p = nullptr;
            cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
            if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(scratch)");
            g_noalloc_address[dev] = p;
        }
        base = g_noalloc_address[dev];
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int ni = (int)n;
    const size_t mirror = round_up_256(sizeof(float4) * n);
    float4 *hi = static_cast<float4 *>(base);
    float4 *lo = reinterpret_cast<float4 *>(static_cast<unsigned char *>(base) + mirror);
    float *psum = reinterpret_cast<float *>(static_cast<unsigned char *>(base) + 2 * mirror);

    split_kernel<<<(ni + 255) / 256, 256, 0, st>>>(x, y, z, m, ni, hi, lo);
    NB_LAUNCH_CHECK();
    const double eps2 = softening * softening;
    if (ni < kMixedPairsMin)
        return launch_small(hi, lo, ni, G, eps2, ax, ay, az, st, AfterForce{});

    // i-blocks by j-segments in whole waves, the segments few enough for their partial
    // sums to fit the remaining scratch
    const int iblocks = (ni + kMixBlock * kMixIpt - 1) / (kMixBlock * kMixIpt);
    const int tiles = (ni + kMixBlock - 1) / kMixBlock;
    const size_t per_segment = sizeof(float) * 6 * n;
    const int max_segments = (int)std::max<size_t>(1, (kNoAllocScratchBytes - 2 * mirror) /
                                                          per_segment);
    int segments = std::min(pick_segments(iblocks, tiles, mix_slots()), max_segments);
    const int seg_tiles = (tiles + segments - 1) / segments;
    segments = (tiles + seg_tiles - 1) / seg_tiles;
    float *pcomp = psum + 3 * n * (size_t)segments;
    const dim3 grid(iblocks, segments);
    if (eps2 > 0.0)
        direct_mixed_kernel<kMixBlock, kMixIpt, false><<<grid, kMixBlock, 0, st>>>(
            hi, lo, ni, (float)eps2, seg_tiles * kMixBlock, psum, pcomp);
    else
        direct_mixed_kernel<kMixBlock, kMixIpt, true><<<grid, kMixBlock, 0, st>>>(
            hi, lo, ni, 0.0f, seg_tiles * kMixBlock, psum, pcomp);
    NB_LAUNCH_CHECK();
    combine_mixed_kernel<<<(ni + 31) / 32, 32 * kCombineGroups, 0, st>>>(
        psum, pcomp, ni, segments, G, ax, ay, az);
    NB_LAUNCH_CHECK();
    return NB_OK;
}
