// nb_batch.cu -- many independent systems of uneven N in one launch.
//
// No reference counterpart: the reference simulates one system per process.
// A batch holds the bodies of every system in one pool of FP64 planes
// (x y z vx vy vz ax ay az m, 80 B/body) plus the float4 hi/lo mirror of the
// mixed pair term (32 B/body).  A system is a descriptor (SysDesc): its bodies
// are pool slots [first, first + n), in blocks of kBatchBlockBodies.
//
// Forces.  A work item is a pair of blocks of one system (or 32 rows of a small
// one); the items are ordered by cost, largest first, one one-warp CTA each.  The
// warp evaluates every unordered pair of the two blocks once (nb_tile.cuh),
// keeping the second block's sums in shared memory, and writes one partial sum
// (a Kahan pair) per body of either block to that body's plane of the (diagonal,
// side); a
// second launch adds each body's planes in order as a double-single.  Systems whose
// planes exceed a buffer of fixed size take turns in it, one of them diagonals by
// diagonals if need be.  A system's partial sums depend on that system alone: it gives
// the same bits alone and in any mix.
#include "nb_internal.h"
#include "nb_check.cuh"
#include "nb_curve.cuh"
#include "nb_tile.cuh"

#include <algorithm>
#include <cmath>

namespace nb {
namespace {

constexpr int kBatchTiles = kBatchBlockBodies / kTile;  // tiles per block
// One-warp CTAs per SM: 10 / 12 (166 registers) / 14 / 16 (128) measured 7.27 /
// 7.27 / 7.16 / 7.17 ms for two RK4 steps of the 1024-system ensemble.
constexpr int kBatchCtas = 16;

// Bounding box of a 64-body tile of sorted bodies (the union of its two chunk
// boxes, box[4 t .. 4 t + 3] = min, max, min, max; an empty chunk has an inverted
// box), or of two tiles; diam2: its squared diameter.
struct TileBox {
    float4 mn, mx;
    __device__ float diam2() const
    {
        const float dx = mx.x - mn.x, dy = mx.y - mn.y, dz = mx.z - mn.z;
        return dx * dx + dy * dy + dz * dz;
    }
};
__device__ __forceinline__ TileBox box_union(const TileBox &a, const TileBox &b)
{
    return TileBox{make_float4(fminf(a.mn.x, b.mn.x), fminf(a.mn.y, b.mn.y),
                               fminf(a.mn.z, b.mn.z), 0.f),
                   make_float4(fmaxf(a.mx.x, b.mx.x), fmaxf(a.mx.y, b.mx.y),
                               fmaxf(a.mx.z, b.mx.z), 0.f)};
}
__device__ __forceinline__ TileBox tile_box(const float4 *__restrict__ box, int t)
{
    const float4 a = box[4 * (size_t)t], b = box[4 * (size_t)t + 1], c = box[4 * (size_t)t + 2],
                 d = box[4 * (size_t)t + 3];
    TileBox r;
    r.mn = make_float4(fminf(a.x, c.x), fminf(a.y, c.y), fminf(a.z, c.z), 0.f);
    r.mx = make_float4(fmaxf(b.x, d.x), fmaxf(b.y, d.y), fmaxf(b.z, d.z), 0.f);
    return r;
}

// The row of 32 i-bodies [i0, i0 + 32) of a small system against all its
// j-bodies in 32-body chunks (ordered pairs): one warp, no partial sums.
// SORTED: the chunk's box centre is the origin of the staged coordinates, and by
// the gap to the i-chunk's box (diameter D) a j-chunk takes the double-single
// term, the plain FP32 one (D/8) or that without the Newton step (D/4).
template <bool SORTED, bool ZERO_SOFT>
__device__ __forceinline__ void batch_row(const float4 *__restrict__ hi,
                                          const float4 *__restrict__ lo,
                                          const float4 *__restrict__ box, const SysDesc &sd,
                                          int i0, float eps2, double G,
                                          const uint32_t *__restrict__ order,
                                          double *__restrict__ ax, double *__restrict__ ay,
                                          double *__restrict__ az, PairTile &sg, int total)
{
    const int lane = threadIdx.x & 31, i = i0 + lane;
    const int nch = (sd.n + 31) / 32;
    const float4 *cb = box + 4 * (size_t)sd.tile0;  // two chunk boxes per tile
    float4 bmn = make_float4(0.f, 0.f, 0.f, 0.f), bmx = bmn;
    if (SORTED) {
        bmn = cb[2 * (i0 / 32)];
        bmx = cb[2 * (i0 / 32) + 1];
    }
    const float diam2 = (bmx.x - bmn.x) * (bmx.x - bmn.x) + (bmx.y - bmn.y) * (bmx.y - bmn.y) +
                        (bmx.z - bmn.z) * (bmx.z - bmn.z);
    const float thr2 = kFarFactor2 * diam2, thr2v = kVeryFar2 * diam2;
    const float cx = 0.5f * (bmn.x + bmx.x), cy = 0.5f * (bmn.y + bmx.y),
                cz = 0.5f * (bmn.z + bmx.z);
    float4 h = make_float4(0.f, 0.f, 0.f, 0.f), l = h;
    if (i < sd.n) {
        h = hi[sd.first + i];
        l = lo[sd.first + i];
    }
    float S[3] = {h.x, h.y, h.z}, E[3] = {l.x, l.y, l.z};
    if (SORTED) {
        rel_ds(h.x, l.x, cx, S[0], E[0]);
        rel_ds(h.y, l.y, cy, S[1], E[1]);
        rel_ds(h.z, l.z, cz, S[2], E[2]);
    }
    const float2 nsx = dup2(-S[0]), nsy = dup2(-S[1]), nsz = dup2(-S[2]);
    const float2 nex = dup2(-E[0]), ney = dup2(-E[1]), nez = dup2(-E[2]), e2 = dup2(eps2);
    float sx = 0.f, sy = 0.f, sz = 0.f, qx = 0.f, qy = 0.f, qz = 0.f;
    for (int jc = 0; jc < nch; ++jc) {
        bool far = false, vfar = false;
        if (SORTED) {
            const float4 jmn = cb[2 * jc], jmx = cb[2 * jc + 1];
            const float gx = fmaxf(0.f, fmaxf(jmn.x - bmx.x, bmn.x - jmx.x));
            const float gy = fmaxf(0.f, fmaxf(jmn.y - bmx.y, bmn.y - jmx.y));
            const float gz = fmaxf(0.f, fmaxf(jmn.z - bmx.z, bmn.z - jmx.z));
            const float gap2 = gx * gx + gy * gy + gz * gz;
            far = gap2 > 0.f && gap2 >= thr2;
            vfar = far && gap2 >= thr2v;
        }
        // lanes past the system stage a massless body far away: exactly 0
        float T[3] = {1.0e18f, 1.0e18f, 1.0e18f}, U[3] = {0.f, 0.f, 0.f}, mj = 0.f;
        const int j = 32 * jc + lane;
        if (j < sd.n) {
            h = hi[sd.first + j];
            l = lo[sd.first + j];
            if (SORTED && far) {
                T[0] = rel_s(h.x, l.x, cx);
                T[1] = rel_s(h.y, l.y, cy);
                T[2] = rel_s(h.z, l.z, cz);
            } else if (SORTED) {
                rel_ds(h.x, l.x, cx, T[0], U[0]);
                rel_ds(h.y, l.y, cy, T[1], U[1]);
                rel_ds(h.z, l.z, cz, T[2], U[2]);
            } else {
                T[0] = h.x; T[1] = h.y; T[2] = h.z;
                U[0] = l.x; U[1] = l.y; U[2] = l.z;
            }
            mj = h.w;
        }
        __syncwarp();
        pair_tile_put(sg, lane, T[0], T[1], T[2], mj, U[0], U[1], U[2]);
        __syncwarp();
        float2 fx = dup2(0.f), fy = dup2(0.f), fz = dup2(0.f);
        if (vfar) {
#pragma unroll 4
            for (int p = 0; p < 16; ++p)
                pair_term2_far<false>(pair_tile_get(sg, p), nsx, nsy, nsz, e2, fx, fy, fz);
        } else if (far) {
#pragma unroll 4
            for (int p = 0; p < 16; ++p)
                pair_term2_far<true>(pair_tile_get(sg, p), nsx, nsy, nsz, e2, fx, fy, fz);
        } else {
#pragma unroll 4
            for (int p = 0; p < 16; ++p)
                pair_term2<ZERO_SOFT>(pair_tile_get(sg, p), nsx, nsy, nsz, nex, ney, nez, e2, fx,
                                      fy, fz);
        }
        kahan_add(sx, qx, fx.x + fx.y);
        kahan_add(sy, qy, fy.x + fy.y);
        kahan_add(sz, qz, fz.x + fz.y);
    }
    if (i >= sd.n) return;
    const int o = SORTED ? (int)order[sd.first + i] : sd.first + i;
    if (!NB_IN_RANGE(o, total)) return;
    ax[o] = G * ((double)sx - (double)qx);
    ay[o] = G * ((double)sy - (double)qy);
    az[o] = G * ((double)sz - (double)qz);
}

// SORTED: the bodies are in Hilbert order with one box per tile; coordinates are
// staged relative to the centre of the i-tiles' box, and a j-tile an eighth of
// that box's diameter or more away takes the plain FP32 displacement (the bound of
// nb_direct_sorted.cu, for both sides), others the double-single one.
// Otherwise every pair takes the double-single term.  Two i-tiles at a time (four
// bodies per lane), but a tile against itself and its neighbour in the pair one
// by one.  Bound by dispatch (nb_tile.cuh): two RK4 steps of the 1024-system
// ensemble (8.4e8 unordered pairs an evaluation) take 7.17 ms, with one i-tile at
// a time and the masses in the loop 7.78, with a row of 32 or 64 bodies per warp
// over ordered pairs 9.92.
template <bool SORTED, bool ZERO_SOFT, bool PARTS>
__global__ void __launch_bounds__(32, kBatchCtas)
batch_pairs_kernel(const float4 *__restrict__ hi, const float4 *__restrict__ lo,
                   const float4 *__restrict__ boxes, const SysDesc *__restrict__ sys,
                   const PairItem *__restrict__ items, float eps2, bool soft,
                   float2 *__restrict__ part, double G, const uint32_t *__restrict__ order, double *__restrict__ ax,
                   double *__restrict__ ay, double *__restrict__ az, int total, int num_tiles)
{
    __shared__ union {
        struct {
            TileJ hi;
            TileJLow lo;
        } tile;
        PairTile chunk;
    } stages;
    __shared__ TileSums sums[kBatchTiles];  // of the second block's tiles
    __shared__ TileSums isum[2];            // of the two i-tiles
    const int lane = threadIdx.x;
    const PairItem it = items[blockIdx.x];
    const SysDesc sd = sys[it.sys];
    if (!NB_IN_RANGE(sd.first, total) || !NB_IN_RANGE(sd.first + sd.n - 1, total) ||
        !NB_IN_RANGE(sd.tile0 + (sd.n - 1) / kTile, num_tiles))
        return;
    if (it.p < 0) {  // a small system: 32 rows, straight to the result
        batch_row<SORTED, ZERO_SOFT>(hi, lo, boxes, sd, 32 * it.a, eps2, G, order, ax, ay, az,
                                     stages.chunk, total);
        return;
    }
    TileJ &stage = stages.tile.hi;
    TileJLow &low = stages.tile.lo;
    const bool within = it.p == 0;  // the block with itself
    const int blk_b = (it.a + it.p) % sd.blocks;
    const int tiles = (sd.n + kTile - 1) / kTile;
    const int ti0 = it.a * kBatchTiles, tj0 = blk_b * kBatchTiles;
    const int ta = min(kBatchTiles, tiles - ti0), tb = min(kBatchTiles, tiles - tj0);
    const float4 *bhi = hi + sd.first, *blo = lo + sd.first;
    const float2 e2 = dup2(eps2);
    const size_t plane = (size_t)sd.n;
    float2 *pa = part + sd.part0 + 3 * plane * (PARTS ? it.p - sd.p0 : it.p);
    float2 *pb = part + sd.part0 +
                 3 * plane * (PARTS ? sd.np - (sd.p0 == 0) + it.p - sd.p0 : sd.blocks / 2 + it.p);
    for (int v = 0; v < kBatchTiles; ++v) tile_sums_zero(sums[v], lane);

    for (int u0 = 0; u0 < ta; u0 += 2) {
        tile_sums_zero(isum[0], lane);
        tile_sums_zero(isum[1], lane);
        const bool two = u0 + 1 < ta;
        TileBox bi{};
        float c[3] = {0.f, 0.f, 0.f};
        if (SORTED) {
            bi = tile_box(boxes, sd.tile0 + ti0 + u0);
            if (two) bi = box_union(bi, tile_box(boxes, sd.tile0 + ti0 + u0 + 1));
            c[0] = 0.5f * (bi.mn.x + bi.mx.x);
            c[1] = 0.5f * (bi.mn.y + bi.mx.y);
            c[2] = 0.5f * (bi.mn.z + bi.mx.z);
        }
        if (two && (!within || u0 + 2 < tb)) {
            TileI<4> ti;
            TileILow<4> tl;
            float mi, mj;
            const bool ei = tile_load_i<SORTED>(bhi, blo, sd.n, (ti0 + u0) * kTile, c, ti, tl, mi);
            for (int v = within ? u0 + 2 : 0; v < tb; ++v) {
                bool far = false;
                if (SORTED) {
                    const TileBox bj = tile_box(boxes, sd.tile0 + tj0 + v);
                    const float gx = fmaxf(0.f, fmaxf(bj.mn.x - bi.mx.x, bi.mn.x - bj.mx.x));
                    const float gy = fmaxf(0.f, fmaxf(bj.mn.y - bi.mx.y, bi.mn.y - bj.mx.y));
                    const float gz = fmaxf(0.f, fmaxf(bj.mn.z - bi.mx.z, bi.mn.z - bj.mx.z));
                    const float gap2 = gx * gx + gy * gy + gz * gz;
                    far = gap2 > 0.f && gap2 >= kFarFactor2 * bi.diam2();
                }
                const bool equal = tile_stage_j<SORTED>(bhi, blo, sd.n, (tj0 + v) * kTile, c,
                                                        stage, low, mj) && ei && soft;
                if (far && equal)
                    tile_pair<kFarTerm, true, ZERO_SOFT, 4>(stage, &low, lane, ti, &tl, e2, mi, mj,
                                                            isum, sums[v]);
                else if (far)
                    tile_pair<kFarTerm, false, ZERO_SOFT, 4>(stage, &low, lane, ti, &tl, e2, 0.f,
                                                             0.f, isum, sums[v]);
                else if (equal)
                    tile_pair<kNearTerm, true, ZERO_SOFT, 4>(stage, &low, lane, ti, &tl, e2, mi,
                                                             mj, isum, sums[v]);
                else
                    tile_pair<kNearTerm, false, ZERO_SOFT, 4>(stage, &low, lane, ti, &tl, e2, 0.f,
                                                              0.f, isum, sums[v]);
            }
        }
        // one tile at a time: within the block the pair's own tiles, else the
        // last tile of an odd number
        for (int u = u0; u < u0 + 1 + two; ++u) {
            if (two && !within) break;
            TileI<2> ti;
            TileILow<2> tl;
            float mi, mj;
            const bool ei = tile_load_i<SORTED>(bhi, blo, sd.n, (ti0 + u) * kTile, c, ti, tl, mi);
            const int v1 = two ? u0 + 2 : tb;
            for (int v = within ? u : 0; v < v1; ++v) {
                const bool equal = tile_stage_j<SORTED>(bhi, blo, sd.n, (tj0 + v) * kTile, c,
                                                        stage, low, mj) && ei && soft;
                if (within && u == v)
                    tile_self<ZERO_SOFT>(stage, &low, lane, ti, &tl, e2, isum[u - u0]);
                else if (equal)
                    tile_pair<kNearTerm, true, ZERO_SOFT, 2>(stage, &low, lane, ti, &tl, e2, mi,
                                                             mj, isum + (u - u0), sums[v]);
                else
                    tile_pair<kNearTerm, false, ZERO_SOFT, 2>(stage, &low, lane, ti, &tl, e2, 0.f,
                                                              0.f, isum + (u - u0), sums[v]);
            }
        }
        __syncwarp();
        // the i-tiles' partial sums; within a block with what they took as j-tiles
        for (int w = 0; w < 1 + two; ++w) {
            const int i = (ti0 + u0 + w) * kTile + lane;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                float2 t = isum[w].s[d][lane], e = isum[w].c[d][lane];
                if (within) {
                    const float2 js = sums[u0 + w].s[d][lane], jc = sums[u0 + w].c[d][lane];
                    float2 r;
                    two_sum(t.x, js.x, t.x, r.x);
                    two_sum(t.y, js.y, t.y, r.y);
                    e = make_float2(r.x + (e.x + jc.x), r.y + (e.y + jc.y));
                }
                if (i < sd.n) pa[d * plane + i] = make_float2(t.x, e.x);
                if (i + 32 < sd.n) pa[d * plane + i + 32] = make_float2(t.y, e.y);
            }
        }
    }
    if (within) return;
    for (int v = 0; v < tb; ++v) {
        const int j = (tj0 + v) * kTile + lane;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const float2 js = sums[v].s[d][lane], jc = sums[v].c[d][lane];
            if (j < sd.n) pb[d * plane + j] = make_float2(js.x, jc.x);
            if (j + 32 < sd.n) pb[d * plane + j + 32] = make_float2(js.y, jc.y);
        }
    }
}

// a = G * the sum of a body's planes in order (diagonal 0, 1, ... of the first
// side, then 1, 2, ... of the second; those of earlier passes, acc, before them), as a
// double-single: one block per block of bodies; order (sorted batches): the pool slot of
// a sorted body.
template <bool PARTS>
__global__ void __launch_bounds__(kBatchBlockBodies)
batch_combine_kernel(const float2 *__restrict__ part, float2 *__restrict__ acc,
                     const SysDesc *__restrict__ sys,
                     const PairItem *__restrict__ items, const uint32_t *__restrict__ order,
                     double G, double *__restrict__ ax, double *__restrict__ ay,
                     double *__restrict__ az, int total)
{
    const PairItem it = items[blockIdx.x];  // (system, block, 0)
    const SysDesc sd = sys[it.sys];
    const int i = it.a * kBatchBlockBodies + threadIdx.x;
    if (i >= sd.n || !NB_IN_RANGE(sd.first + i, total)) return;
    const size_t plane = (size_t)sd.n;
    const float2 *src = part + sd.part0 + i;
    // the planes of the first side, then of the second, which diagonal 0 has not
    const int p0 = PARTS ? sd.p0 : 0, from = p0 == 0;
    const int np = PARTS ? sd.np : sd.blocks / 2 + 1, planes = 2 * np - from;
    float s[3] = {0.f, 0.f, 0.f}, r[3] = {0.f, 0.f, 0.f};
    if (PARTS && p0 > 0)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float2 a = acc[sd.acc0 + c * plane + i];
            s[c] = a.x;
            r[c] = a.y;
        }
    for (int k0 = 0; k0 < planes; k0 += 4) {
        float2 t[4][3];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int k = k0 + u;
            const bool first = k < np;
            const int p = p0 + (first ? k : k - np + from);
            const bool use = k < planes && (first ? pair_first(p, it.a, sd.blocks)
                                                  : pair_second(p, it.a, sd.blocks));
#pragma unroll
            for (int c = 0; c < 3; ++c)
                t[u][c] = use ? src[(3 * (size_t)k + c) * plane] : dup2(0.f);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int c = 0; c < 3; ++c) ds_add_kahan(s[c], r[c], t[u][c].x, -t[u][c].y);
    }
    if (PARTS && p0 + np <= sd.blocks / 2) {  // a later pass has more
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[sd.acc0 + c * plane + i] = make_float2(s[c], r[c]);
        return;
    }
    const int o = order ? (int)order[sd.first + i] : sd.first + i;
    if (!NB_IN_RANGE(o, total)) return;
    ax[o] = G * ((double)s[0] + (double)r[0]);
    ay[o] = G * ((double)s[1] + (double)r[1]);
    az[o] = G * ((double)s[2] + (double)r[2]);
}

// ---------------------------------------------------------------- sorted
// The Hilbert-sorted variant (ensemble): every system's bodies are sorted
// along a Hilbert curve through the cube around that system alone, so a 64-body
// tile of sorted bodies is spatially compact.  Every quantity a system's result
// depends on -- its order, its centre, its tile boxes, each tile pair's
// classification -- is computed from that system alone, so a system still
// gives the same bits alone and in any mix.

// body_sys[i] = s for the bodies of system s; tile table entries (first body,
// count, system) of its 64-body tiles.
__global__ void batch_layout_kernel(const SysDesc *__restrict__ sys, int *__restrict__ body_sys,
                                    int4 *__restrict__ tiles)
{
    const SysDesc sd = sys[blockIdx.x];
    for (int i = threadIdx.x; i < sd.n; i += blockDim.x) body_sys[sd.first + i] = blockIdx.x;
    const int nt = (sd.n + kTile - 1) / kTile;
    for (int c = threadIdx.x; c < nt; c += blockDim.x)
        tiles[sd.tile0 + c] = make_int4(sd.first + kTile * c, min(kTile, sd.n - kTile * c),
                                        blockIdx.x, 0);
}

// geom[s] = (centre x, y, z, side) of the cube around system s: one block per
// system, min/max on order-preserving integer keys.
__global__ void __launch_bounds__(256)
batch_geom_kernel(const SysDesc *__restrict__ sys, const double *__restrict__ x,
                  const double *__restrict__ y, const double *__restrict__ z,
                  double4 *__restrict__ geom)
{
    constexpr long long kMax = 0x7fffffffffffffffll, kMin = -kMax - 1;
    __shared__ long long sh[6][8];
    const SysDesc sd = sys[blockIdx.x];
    const double *ax[3] = {x, y, z};
    long long v[6] = {kMax, kMax, kMax, kMin, kMin, kMin};
    for (int i = threadIdx.x; i < sd.n; i += 256)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double q = ax[c][sd.first + i];
            v[c] = min(v[c], order_key(q, kMax));
            v[c + 3] = max(v[c + 3], order_key(q, kMin));
        }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            v[c] = min(v[c], __shfl_xor_sync(0xffffffffu, v[c], o));
            v[c + 3] = max(v[c + 3], __shfl_xor_sync(0xffffffffu, v[c + 3], o));
        }
    if (lane == 0)
#pragma unroll
        for (int c = 0; c < 6; ++c) sh[c][warp] = v[c];
    __syncthreads();
    if (threadIdx.x != 0) return;
    double lo[3], hi[3], side = 0.0;
    for (int c = 0; c < 3; ++c) {
        long long a = sh[c][0], b = sh[c + 3][0];
        for (int w = 1; w < 8; ++w) {
            a = min(a, sh[c][w]);
            b = max(b, sh[c + 3][w]);
        }
        // only NaN coordinates: a unit cube at the origin
        lo[c] = a == kMax ? 0.0 : key_value(a);
        hi[c] = b == kMin ? 0.0 : key_value(b);
        side = fmax(side, hi[c] - lo[c]);
    }
    side = fmax(side, 1e-30) * (1.0 + 1e-6);
    geom[blockIdx.x] = make_double4(0.5 * (lo[0] + hi[0]), 0.5 * (lo[1] + hi[1]),
                                    0.5 * (lo[2] + hi[2]), side);
}

// keys[i] = (system, Hilbert index in its cube) in the top sys_bits + 30 bits,
// vals[i] = i: a stable sort keeps every system in its own index range.
__global__ void __launch_bounds__(256)
batch_key_kernel(const double *__restrict__ x, const double *__restrict__ y,
                 const double *__restrict__ z, const int *__restrict__ body_sys,
                 const double4 *__restrict__ geom, int n, int key_shift,
                 uint64_t *__restrict__ keys, uint32_t *__restrict__ vals)
{
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const int s = body_sys[i];
    const double4 g = geom[s];
    const double scale = 1024.0 / g.w;
    const double p[3] = {x[i], y[i], z[i]}, c[3] = {g.x, g.y, g.z};
    uint32_t q[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double f = floor((p[k] - (c[k] - 0.5 * g.w)) * scale);
        q[k] = (uint32_t)fmin(fmax(f, 0.0), 1023.0);
    }
    const uint64_t key = ((uint64_t)s << 30) | hilbert_index30(q[0], q[1], q[2]);
    keys[i] = key << key_shift;
    vals[i] = (uint32_t)i;
}

// Sorted positions relative to their system's centre, split into hi/lo
// (double-single) parts, mass in hi.w, and the bounding box of every 32-body
// chunk: one warp per chunk, two chunks per tile (an empty one gets an inverted
// box).
__global__ void __launch_bounds__(256)
batch_split_sorted_kernel(const uint32_t *__restrict__ order, const double *__restrict__ x,
                          const double *__restrict__ y, const double *__restrict__ z,
                          const double *__restrict__ m, const int4 *__restrict__ tiles,
                          int num_tiles, const double4 *__restrict__ geom, int total,
                          float4 *__restrict__ hi, float4 *__restrict__ lo,
                          float4 *__restrict__ box)
{
    const int ch = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (ch >= 2 * num_tiles) return;
    const int4 tl = tiles[ch >> 1];  // first body, count, system
    const double4 g = geom[tl.z];
    float mn[3] = {3.0e38f, 3.0e38f, 3.0e38f}, mx[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
    const int l = 32 * (ch & 1) + lane, i = tl.x + l;
    const uint32_t o = l < tl.y ? order[i] : 0u;
    if (l < tl.y && NB_IN_RANGE(o, total)) {
        const double X = x[o] - g.x, Y = y[o] - g.y, Z = z[o] - g.z;
        const float hx = __double2float_rn(X), hy = __double2float_rn(Y),
                    hz = __double2float_rn(Z);
        hi[i] = make_float4(hx, hy, hz, __double2float_rn(m[o]));
        lo[i] = make_float4(__double2float_rn(X - (double)hx), __double2float_rn(Y - (double)hy),
                            __double2float_rn(Z - (double)hz), 0.0f);
        mn[0] = mx[0] = hx;
        mn[1] = mx[1] = hy;
        mn[2] = mx[2] = hz;
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            mn[c] = fminf(mn[c], __shfl_xor_sync(0xffffffffu, mn[c], s));
            mx[c] = fmaxf(mx[c], __shfl_xor_sync(0xffffffffu, mx[c], s));
        }
    if (lane == 0) {
        box[2 * (size_t)ch] = make_float4(mn[0], mn[1], mn[2], 0.f);
        box[2 * (size_t)ch + 1] = make_float4(mx[0], mx[1], mx[2], 0.f);
    }
}

} // namespace

void build_batch(BatchWork &w, int pairs_min, size_t plane_bytes)
{
    const long long limit = (long long)(plane_bytes / sizeof(float2));
    const int systems = (int)w.sys.size();
    w.num_tiles = 0;
    std::vector<std::vector<int>> passes(1);  // the descriptors of each
    std::vector<int> parts;                   // systems that do not fit one
    long long used = 0, most = 0;
    for (int k = 0; k < systems; ++k) {
        SysDesc &s = w.sys[k];
        s.tile0 = w.num_tiles;
        w.num_tiles += (s.n + kTile - 1) / kTile;
        const bool pairs = s.n >= pairs_min && s.n <= kBatchPairsMax && 9ll * s.n <= limit;
        s.blocks = pairs ? (s.n + kBatchBlockBodies - 1) / kBatchBlockBodies : 0;
        s.np = s.blocks / 2 + 1;
        if (!pairs) {
            passes[0].push_back(k);
            continue;
        }
        const long long need = 3ll * s.n * (2 * s.np - 1);
        if (need > limit) {
            parts.push_back(k);
            continue;
        }
        if (used + need > limit) {
            passes.emplace_back();
            used = 0;
        }
        s.part0 = used;
        used += need;
        most = std::max(most, used);
        passes.back().push_back(k);
    }
    if (passes[0].empty()) passes.erase(passes.begin());
    for (int k : parts) {
        // the sums between passes, then two planes a diagonal
        const long long plane = 3ll * w.sys[k].n;
        const int diagonals = w.sys[k].np;
        const int np = (int)std::min<long long>(
            diagonals, std::max<long long>(1, (limit - plane) / (2 * plane)));
        for (int p0 = 0; p0 < diagonals; p0 += np) {
            SysDesc d = w.sys[k];
            d.p0 = p0;
            d.np = std::min(np, diagonals - p0);
            d.part0 = plane;  // behind the sums, at 0
            passes.push_back({(int)w.sys.size()});
            w.sys.push_back(d);
        }
        most = std::max(most, plane * (1 + 2 * np));
    }
    w.part_bytes = sizeof(float2) * (size_t)most;
    // items by cost in units of a 64 x 64 tile pair (a stable counting sort: all full
    // items of all systems cost the same; a row item is two tiles against half its
    // system's, both directions apart)
    constexpr int kMost = 64;
    for (const std::vector<int> &pass : passes) {
        std::vector<PairItem> by_cost[kMost + 1];
        BatchPass at;
        at.block0 = (int)w.blocks.size();
        at.item0 = (int)w.items.size();
        for (int s : pass) {
            const SysDesc &sd = w.sys[s];
            const int M = sd.blocks, tiles = (sd.n + kTile - 1) / kTile;
            for (int r = 0; M == 0 && r * 32 < sd.n; ++r)
                by_cost[std::min(kMost, (tiles + 1) / 2)].push_back(PairItem{s, r, -1});
            if (M == 0) continue;
            for (int a = 0; a < M; ++a) w.blocks.push_back(PairItem{s, a, 0});
            auto width = [&](int b) { return std::min(kBatchTiles, tiles - b * kBatchTiles); };
            for (int p = sd.p0; p < sd.p0 + sd.np; ++p)
                for (int a = 0; a < M; ++a) {
                    if (!pair_first(p, a, M)) continue;
                    const int ta = width(a), tb = width((a + p) % M);
                    by_cost[p == 0 ? ta * (ta + 1) / 2 : ta * tb].push_back(PairItem{s, a, p});
                }
        }
        for (int c = kMost; c >= 0; --c)
            w.items.insert(w.items.end(), by_cost[c].begin(), by_cost[c].end());
        at.parts = pass[0] >= systems;
        at.blocks = (int)w.blocks.size() - at.block0;
        at.items = (int)w.items.size() - at.item0;
        w.passes.push_back(at);
    }
}

void BatchQueue::release()
{
    d_sys.release();
    d_blocks.release();
    d_items.release();
}

nb_status reserve_batch(BatchQueue &q, const BatchWork &w)
{
    q.passes.clear();
    if (w.sys.empty()) return NB_OK;
    NB_TRY(q.d_sys.reserve(sizeof(SysDesc) * w.sys.size()));
    NB_TRY(q.d_items.reserve(sizeof(PairItem) * w.items.size()));
    if (w.blocks.empty()) return NB_OK;
    return q.d_blocks.reserve(sizeof(PairItem) * w.blocks.size());
}

nb_status upload_batch(BatchQueue &q, const BatchWork &w, cudaStream_t st)
{
    NB_TRY(reserve_batch(q, w));
    q.num_tiles = w.num_tiles;
    q.num_items = (long long)w.items.size();
    auto put = [&](DevBuf &to, const void *from, size_t bytes) -> nb_status {
        if (bytes > 0)
            NB_CUDA_TRY(cudaMemcpyAsync(to.ptr, from, bytes, cudaMemcpyHostToDevice, st));
        return NB_OK;
    };
    NB_TRY(put(q.d_sys, w.sys.data(), sizeof(SysDesc) * w.sys.size()));
    NB_TRY(put(q.d_blocks, w.blocks.data(), sizeof(PairItem) * w.blocks.size()));
    NB_TRY(put(q.d_items, w.items.data(), sizeof(PairItem) * w.items.size()));
    NB_CUDA_TRY(cudaStreamSynchronize(st));  // the host vectors may go
    q.passes = w.passes;
    return NB_OK;
}

template <bool PARTS>
static auto batch_kernel(bool sorted, double eps2)
{
    if (sorted)
        return eps2 > 0.0 ? batch_pairs_kernel<true, false, PARTS>
                          : batch_pairs_kernel<true, true, PARTS>;
    return eps2 > 0.0 ? batch_pairs_kernel<false, false, PARTS>
                      : batch_pairs_kernel<false, true, PARTS>;
}

static nb_status launch_batch(const float4 *hi, const float4 *lo, const float4 *boxes,
                              const BatchQueue &q, double G, double eps2, const uint32_t *order,
                              double *ax, double *ay, double *az, int total, int num_tiles,
                              cudaStream_t st, const KernelTimer *timer)
{
    const SysDesc *sys = q.d_sys.as<SysDesc>();
    if (timer && timer->start) NB_CUDA_TRY(cudaEventRecord(timer->start, st));
    for (const BatchPass &p : q.passes) {
        auto *kernel = p.parts ? batch_kernel<true>(boxes, eps2) : batch_kernel<false>(boxes, eps2);
        kernel<<<p.items, 32, 0, st>>>(hi, lo, boxes, sys, q.d_items.as<PairItem>() + p.item0,
                                       eps2 > 0.0 ? (float)eps2 : 0.0f, equal_soft(eps2), q.part, G,
                                       order, ax, ay, az, total, num_tiles);
        NB_LAUNCH_CHECK();
        if (timer && timer->stop && &p == &q.passes.back())
            NB_CUDA_TRY(cudaEventRecord(timer->stop, st));
        if (p.blocks == 0) continue;  // rows only: no partial sums
        auto *combine = p.parts ? batch_combine_kernel<true> : batch_combine_kernel<false>;
        combine<<<p.blocks, kBatchBlockBodies, 0, st>>>(
            q.part, q.part, sys, q.d_blocks.as<PairItem>() + p.block0, order, G, ax, ay, az, total);
        NB_LAUNCH_CHECK();
    }
    return NB_OK;
}

nb_status batch_forces(const float4 *hi, const float4 *lo, const BatchQueue &q, double G,
                       double eps2, double *ax, double *ay, double *az, int total,
                       cudaStream_t st, const KernelTimer *timer)
{
    return launch_batch(hi, lo, nullptr, q, G, eps2, nullptr, ax, ay, az, total, q.num_tiles, st,
                        timer);
}

void BatchSorted::release()
{
    if (sorter) bh_destroy(sorter);
    sorter = nullptr;
    order = nullptr;
    DevBuf *bufs[] = {&body_sys, &tiles, &geom, &boxes};
    for (DevBuf *b : bufs) b->release();
}

nb_status batch_sorted_setup(BatchSorted &b, const SysDesc *d_sys, int num_sys, int num_tiles,
                             int total, cudaStream_t st)
{
    b.num_sys = num_sys;
    b.num_tiles = num_tiles;
    b.total = total;
    int sys_bits = 1;
    while ((1 << sys_bits) < num_sys) ++sys_bits;
    const int key_bits = sys_bits + 30;
    b.key_shift = 64 - key_bits;
    b.first_shift = b.key_shift / 8 * 8;
    NB_TRY(b.body_sys.reserve(sizeof(int) * (size_t)std::max(total, 1)));
    NB_TRY(b.tiles.reserve(sizeof(int4) * (size_t)std::max(num_tiles, 1)));
    NB_TRY(b.geom.reserve(sizeof(double4) * (size_t)std::max(num_sys, 1)));
    NB_TRY(b.boxes.reserve(sizeof(float4) * 4 * (size_t)std::max(num_tiles, 1)));
    if (!b.sorter) b.sorter = bh_create();
    batch_layout_kernel<<<num_sys, 128, 0, st>>>(d_sys, b.body_sys.as<int>(), b.tiles.as<int4>());
    NB_LAUNCH_CHECK();
    return NB_OK;
}

nb_status batch_sorted_sort(BatchSorted &b, const SysDesc *d_sys, const double *x,
                            const double *y, const double *z, cudaStream_t st)
{
    if (b.total <= 0) return NB_OK;
    uint64_t *keys = nullptr;
    uint32_t *vals = nullptr;
    NB_TRY(bh_sort_buffers(b.sorter, b.total, &keys, &vals));
    batch_geom_kernel<<<b.num_sys, 256, 0, st>>>(d_sys, x, y, z, b.geom.as<double4>());
    NB_LAUNCH_CHECK();
    batch_key_kernel<<<(b.total + 255) / 256, 256, 0, st>>>(
        x, y, z, b.body_sys.as<int>(), b.geom.as<double4>(), b.total, b.key_shift, keys, vals);
    NB_LAUNCH_CHECK();
    return bh_sort_keys(b.sorter, b.total, b.first_shift, st, &b.order);
}

nb_status batch_sorted_forces(BatchSorted &b, const double *x, const double *y, const double *z,
                              const double *m, const BatchQueue &q, double G, double eps2,
                              float4 *hi, float4 *lo, double *ax, double *ay, double *az,
                              cudaStream_t st, const KernelTimer *timer)
{
    if (!b.order) return fail(NB_ERR_NOT_LOADED, "sorted batch: no order (sort first)");
    batch_split_sorted_kernel<<<(2 * b.num_tiles + 7) / 8, 256, 0, st>>>(
        b.order, x, y, z, m, b.tiles.as<int4>(), b.num_tiles, b.geom.as<double4>(), b.total, hi,
        lo, b.boxes.as<float4>());
    NB_LAUNCH_CHECK();
    return launch_batch(hi, lo, b.boxes.as<float4>(), q, G, eps2, b.order, ax, ay, az, b.total,
                        b.num_tiles, st, timer);
}
} // namespace nb
