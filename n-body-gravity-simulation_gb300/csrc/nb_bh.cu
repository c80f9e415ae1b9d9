// nb_bh.cu -- Barnes-Hut on sm_103a: 63-bit Morton encode, LSD radix sort,
// a parallel octree build read off the sorted codes, monopoles from FP64 prefix
// sums, and a warp-cooperative walk over child groups.
//
// Replaces BarnesHutForceCalculator (CUDA/src/force_calculator_barnes_hut.cu):
// six CUB min/max passes (:108-173), a 30-bit Morton code (:217-251), a CUB pair
// sort (:254-273), a level-by-level octree build with a host round trip and a
// cudaMalloc/cudaFree set per level (:294-492), ten per-level COM launches
// (:494-578) and a per-thread 50-entry stack walk that silently falls back to a
// monopole when the stack is full (:15-91).
//
// Tree rule.  The octree is the reference CPU tree's set of non-empty cells
// (CPU/src/force_calculator_barnes_hut_optimized.cpp): root cube centred on the
// bounding box with side max extent + 1e-9 (:105-124); a cell splits while it
// holds more than leaf_capacity bodies and its half side is >= 1e-9 (:138-173,
// :206-211), here also at most 21 levels (63-bit codes).  A body's code is the
// sequence of octants it falls into, computed with the CPU tree's own FP64
// comparisons and child-centre additions, so codes, sort order and topology
// equal the CPU restatement bit for bit.  Digits are x-high (x=4, y=2, z=1),
// the Morton order of force_calculator_barnes_hut.cu:243-248.
//
// Build.  After the sort, body i starts a node at depth d exactly when its
// depth-d cell begins at i and that cell's parent holds more than
// leaf_capacity bodies.  The nodes starting at i form a chain of consecutive
// depths that ends at the first leaf; one thread per body finds its chain from
// the depths that its code shares with its neighbours', an exclusive scan of the chain lengths
// numbers every node in preorder (depth-first, children in Morton order), and
// the node after a cell's subtree -- its skip pointer -- is simply the first
// node of the body that follows the cell.  Masses and centres of mass come
// from FP64 prefix sums of (m, m x, m y, m z) over the sorted bodies (positions
// relative to the root centre), so no level-by-level pass is needed.
//
// Walk.  A walk serves 64 consecutive sorted bodies, two per lane of each warp that
// shares it.  At each node every body applies the reference's opening test (open
// when size^2 >= theta^2 d^2 to the COM, or when the node holds the body); the
// node is opened if any body does (so each body gets a refinement of its own walk,
// never a coarser one).  The children of every node are stored together (a
// group): a warp decides the nodes of four groups at once, lists the monopoles of
// the nodes no body opens and the bodies of opened leaves for evaluation, and
// pushes the groups of opened internal nodes on the CTA's stack, which holds the
// deepest tree's groups (group_walk_kernel).  Up to 524,288 bodies, and always under the
// reference's opening rule, every body's terms are added in the order of a serial walk,
// by serial_walk_kernel or by the ordered walk, which many warps share.  The stackless
// preorder walk over skip pointers finds the same interactions (NB_BH_WALK=preorder).  Accelerations are scattered back
// to the original order in FP64, multiplied by G.
#include "nb_internal.h"
#include "nb_after.cuh"
#include "nb_check.cuh"
#include "nb_curve.cuh"
#include "nb_pair.cuh"

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <vector>

namespace nb {

namespace {

constexpr int kMaxLevels = 21;

struct alignas(32) D4 {
    double x, y, z, w;
};

__host__ __device__ __forceinline__ D4 d4_add(const D4 &a, const D4 &b)
{
    return D4{a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w};
}

struct BHRoot {
    double cx, cy, cz, size;        // root cube (bh_*_order hand out &cx: centre, then side)
    double off[kMaxLevels];         // child-centre offset below depth l: size * 2^-(l+2)
    float size2[kMaxLevels + 1];    // squared side of a depth-d cell (opening test)
    int levels;                     // depths the root may split into (<= 21)
    float margin;                   // encode_kernel: distance from a grid line, in cells
    double scale;                   // 2^21 / size
    double lo[3], grid_lo[3];       // the cube's lower corner; kGridBase - that times scale
};

// A leaf is the node whose skip pointer is the next node (no subtree).
struct alignas(32) BHNode {
    float4 com_mass;  // centre of mass relative to the root centre, mass
    int first;        // first sorted body
    int count;        // bodies in the cell
    int skip;         // next node (preorder) outside this subtree
    float size2;      // squared side of the cell (the opening test's size^2)
};
static_assert(sizeof(BHNode) == 32, "node layout");

struct BHStats {
    unsigned long long m2p, p2p;  // terms of the last walk (reset by every build/refit)
    int leaves, max_depth;
    unsigned long long total;     // terms of every walk of this tree object (never reset)
};

// Added to a position in cells of the 2^21 grid (grid_index).
constexpr double kGridBase = 402653184.0;  // 1.5 * 2^28
constexpr unsigned long long kGridBits = 0x41B8000000000000ull;

// ------------------------------------------------------------ bounding box
__global__ void __launch_bounds__(256)
bbox_partial_kernel(const double *__restrict__ x, const double *__restrict__ y,
                    const double *__restrict__ z, int n, long long *__restrict__ part)
{
    constexpr long long kMax = 0x7fffffffffffffffll, kMin = -kMax - 1;
    __shared__ long long sh[6][8];
    long long v[6] = {kMax, kMax, kMax, kMin, kMin, kMin};
    const double *ax[3] = {x, y, z};
    // four grid strides per iteration: twelve loads in flight per thread
    const int stride = gridDim.x * 256;
    int i = blockIdx.x * 256 + threadIdx.x;
    for (; i + 3 * stride < n; i += 4 * stride) {
        double p[3][4];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int u = 0; u < 4; ++u) p[c][u] = ax[c][i + u * stride];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                v[c] = min(v[c], order_key(p[c][u], kMax));
                v[c + 3] = max(v[c + 3], order_key(p[c][u], kMin));
            }
    }
    for (; i < n; i += stride)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double q = ax[c][i];
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
    if (threadIdx.x < 6) {
        const int c = threadIdx.x;
        long long r = sh[c][0];
        for (int w = 1; w < 8; ++w) r = c < 3 ? min(r, sh[c][w]) : max(r, sh[c][w]);
        part[blockIdx.x * 6 + c] = r;  // the neutral key if it saw only NaN (or nothing)
    }
}

// One block: reduce the partials' keys, then one warp derives the root cube by the
// CPU tree's rule (force_calculator_barnes_hut_optimized.cpp:112-124,
// std::max(a,b) = a<b?b:a), a lane per level: halving is exact, so size * 2^-l is
// the side after l halvings.  Min and max are exact, so the order of the
// reduction does not matter.  What encode_kernel's blocks share of the cube is
// derived here, once.  Latency alone: FP64 min/max in shared memory and one thread
// for the 21 levels took 10.4 us.
__global__ void __launch_bounds__(256)
bbox_final_kernel(const long long *__restrict__ part, int nparts, BHRoot *root)
{
    __shared__ long long sh[6][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long v[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) v[k] = order_key(k < 3 ? 1e308 : -1e308, 0);
    for (int b = threadIdx.x; b < nparts; b += 256)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            v[k] = min(v[k], part[b * 6 + k]);
            v[k + 3] = max(v[k + 3], part[b * 6 + k + 3]);
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            v[k] = min(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
            v[k + 3] = max(v[k + 3], __shfl_xor_sync(0xffffffffu, v[k + 3], o));
        }
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < 6; ++k) sh[k][warp] = v[k];
    __syncthreads();
    if (warp > 0) return;
    double e[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        long long r = sh[k][0];
#pragma unroll
        for (int w = 1; w < 8; ++w) r = k < 3 ? min(r, sh[k][w]) : max(r, sh[k][w]);
        e[k] = key_value(r);
    }
    const double ex = e[3] - e[0], ey = e[4] - e[1], ez = e[5] - e[2];
    const double eyz = (ey < ez) ? ez : ey;
    const double size = ((ex < eyz) ? eyz : ex) + 1e-9;
    if (lane <= kMaxLevels) {
        const double side = size * double_of((long long)(1023 - lane) << 52);
        root->size2[lane] = (float)(side * side);
        if (lane < kMaxLevels) root->off[lane] = side / 4.0;
        // levels: halvings until the half falls below 1e-9
        const bool splits = lane < kMaxLevels && !(side / 2.0 < 1e-9);
        const unsigned vote = __ballot_sync((2u << kMaxLevels) - 1u, splits);
        if (lane == 0) root->levels = __ffs(~vote) - 1;
    }
    const double scale = 2097152.0 / size;
    double cmax = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double c = (e[k] + e[k + 3]) / 2, lo = c - size / 2;
        cmax = fmax(cmax, fabs(c));
        if (lane == k) {
            (&root->cx)[k] = c;
            root->lo[k] = lo;
            root->grid_lo[k] = kGridBase - lo * scale;
        }
    }
    if (lane != 0) return;
    root->size = size;
    root->scale = scale;
    // Running centres accumulate at most 21 roundings of half an ulp of
    // |centre| <= cmax + size; the fast index adds a few more roundings
    // (of |p| * scale and of lo * scale: 2^-52 (cmax + size) scale each).
    // Positions farther than this from every grid line index exactly.
    const double u_c = ldexp(1.0, ilogb(cmax + size) - 52);
    const double u_s = ldexp(1.0, ilogb(size) - 52);
    root->margin = (float)((32.0 * u_c + 4.0 * u_s) * scale + 1e-6);
}

// ------------------------------------------------------------ Morton encode
// Fast path of one axis: the cell index on the ideal 2^21 grid of the root
// cube and whether the position is far enough from every grid line that the
// CPU tree's rounded running centres cannot compare differently.  f carries a
// few roundings of ~2^-31 grid cells; the margin (>= 1e-6 cells) covers them.
// One FP64 operation (the FP64 pipe bounds this kernel): the index f + kGridBase has
// an ulp of 2^-24 cells, so its bits less kGridBase's are the index in fixed point,
// 24 bits of it the fraction (two more roundings of 2^-25 cells, far below the
// margin).  With f, its floor and its fraction in FP64 the kernel took 34 us at
// N = 2^20, 14 now.
__device__ __forceinline__ bool grid_index(double p, double lo, double scale, float margin,
                                           uint64_t *q)
{
    const unsigned long long f = (unsigned long long)bits_of(fma(p, scale, lo)) - kGridBits;
    *q = f >> 24;
    const float frac = (float)((unsigned)f & 0xFFFFFFu) * 5.9604644775390625e-8f;
    return f < 1ull << 45 && frac > margin && frac < 1.0f - margin;
}

__global__ void __launch_bounds__(256)
encode_kernel(const double *__restrict__ x, const double *__restrict__ y,
              const double *__restrict__ z, int n, const BHRoot *__restrict__ root,
              uint64_t *__restrict__ keys, uint32_t *__restrict__ vals)
{
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const double scale = root->scale;
    const float margin = root->margin;
    const int levels = root->levels;
    const double px = x[i], py = y[i], pz = z[i];
    uint64_t qx, qy, qz;
    const bool okx = grid_index(px, root->grid_lo[0], scale, margin, &qx);
    const bool oky = grid_index(py, root->grid_lo[1], scale, margin, &qy);
    const bool okz = grid_index(pz, root->grid_lo[2], scale, margin, &qz);
    if (okx && oky && okz) {
        uint64_t code = (spread21(qx) << 2) | (spread21(qy) << 1) | spread21(qz);
        const int drop = 3 * (kMaxLevels - levels);  // digits below the split limit are 0
        if (drop >= 63) code = 0;
        else code = (code >> drop) << drop;
        keys[i] = code;
        vals[i] = (uint32_t)i;
        return;
    }
    // Exact path: the CPU tree's own comparisons and child-centre additions.
    double cx = root->cx, cy = root->cy, cz = root->cz;
    uint64_t code = 0;
    for (int l = 0; l < kMaxLevels; ++l) {
        uint64_t d = 0;
        if (l < levels) {
            const bool bx = px >= cx, by = py >= cy, bz = pz >= cz;
            d = ((uint64_t)bx << 2) | ((uint64_t)by << 1) | (uint64_t)bz;
            const double o = root->off[l];
            cx = __dadd_rn(cx, bx ? o : -o);
            cy = __dadd_rn(cy, by ? o : -o);
            cz = __dadd_rn(cz, bz ? o : -o);
        }
        code = (code << 3) | d;
    }
    keys[i] = code;
    vals[i] = (uint32_t)i;
}

// ------------------------------------------------------------ Hilbert encode
// keys[i] = the 30-bit Hilbert index of body i in bits 33..62 (the bits a
// 10-level Morton sort orders by), vals[i] = i.
__global__ void __launch_bounds__(256)
hilbert_kernel(const double *__restrict__ x, const double *__restrict__ y,
               const double *__restrict__ z, int n, const BHRoot *__restrict__ root,
               uint64_t *__restrict__ keys, uint32_t *__restrict__ vals)
{
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const double scale = root->scale * (1.0 / 2048);  // 1024 / size
    const double p[3] = {x[i], y[i], z[i]};
    uint32_t g[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double f = floor((p[k] - root->lo[k]) * scale);
        g[k] = (uint32_t)fmin(fmax(f, 0.0), 1023.0);
    }
    keys[i] = (uint64_t)hilbert_index30(g[0], g[1], g[2]) << 33;
    vals[i] = (uint32_t)i;
}

// ------------------------------------------------------------ scans (fixed order)
template <class T> struct Add;
template <> struct Add<int> {
    __device__ static int zero() { return 0; }
    __device__ static int op(int a, int b) { return a + b; }
};
template <> struct Add<D4> {
    __device__ static D4 zero() { return D4{0.0, 0.0, 0.0, 0.0}; }
    __device__ static D4 op(const D4 &a, const D4 &b) { return d4_add(a, b); }
};

// Elements per thread of the scans: more for the FP64 moments, whose warp
// and block steps run on GB300's narrow FP64 pipe, so fewer of them per
// element pays.
template <class T> struct ScanItems { static constexpr int n = 4; };
template <> struct ScanItems<D4> { static constexpr int n = 8; };
template <class T> __host__ __device__ constexpr int scan_tile() { return 256 * ScanItems<T>::n; }

__device__ __forceinline__ int shfl_up(int v, int d) { return __shfl_up_sync(0xffffffffu, v, d); }
__device__ __forceinline__ D4 shfl_up(const D4 &v, int d)
{
    return D4{__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d),
              __shfl_up_sync(0xffffffffu, v.z, d), __shfl_up_sync(0xffffffffu, v.w, d)};
}

// Inclusive scan of one value per lane over a warp (shuffles).
template <class T>
__device__ __forceinline__ T warp_inclusive(T v, int lane)
{
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const T u = shfl_up(v, off);
        if (lane >= off) v = Add<T>::op(u, v);
    }
    return v;
}

// Exclusive scan of one value per thread over a block of NW warps: each warp
// scans its lanes, warp 0 scans the warp totals (the FP64 pipe is narrow, so
// no thread adds up all of them itself), and *total receives the block's
// sum.  Every thread of the block must call it; warp_sums holds NW + 1.
template <class T, int NW>
__device__ __forceinline__ T block_exclusive(T s, T *warp_sums, T *total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const T inc = warp_inclusive(s, lane);
    if (lane == 31) warp_sums[warp] = inc;
    T excl = shfl_up(inc, 1);
    if (lane == 0) excl = Add<T>::zero();
    __syncthreads();
    if (warp == 0) {
        const T w = lane < NW ? warp_sums[lane] : Add<T>::zero();
        const T wi = warp_inclusive(w, lane);
        T we = shfl_up(wi, 1);
        if (lane == 0) we = Add<T>::zero();
        __syncwarp();
        if (lane < NW) warp_sums[lane] = we;
        if (lane == NW - 1) warp_sums[NW] = wi;
    }
    __syncthreads();
    *total = warp_sums[NW];
    return Add<T>::op(warp_sums[warp], excl);
}

// sums[b] = the sum of tile b (scan_tile<T>() elements): a tree in shared memory,
// whose idle warps skip their steps (fewer FP64 adds than a shuffle
// reduction, in which every lane adds at every step).
template <class T>
__global__ void __launch_bounds__(256)
scan_reduce_kernel(const T *__restrict__ in, int n, T *__restrict__ sums)
{
    constexpr int kItems = ScanItems<T>::n;
    __shared__ T sh[256];
    const int base = blockIdx.x * scan_tile<T>() + threadIdx.x * kItems;
    T s = Add<T>::zero();
#pragma unroll
    for (int k = 0; k < kItems; ++k)
        if (base + k < n) s = Add<T>::op(s, in[base + k]);
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w) sh[threadIdx.x] = Add<T>::op(sh[threadIdx.x], sh[threadIdx.x + w]);
        __syncthreads();
    }
    if (threadIdx.x == 0) sums[blockIdx.x] = sh[0];
}

// Exclusive scan of the tile sums in place, one block of up to 1024 threads
// (a warp per 32 sums: the FP64 steps of a block scan run on one SM's narrow
// FP64 pipe, so idle warps would only cost time).
template <class T>
__global__ void __launch_bounds__(1024) scan_top_kernel(T *__restrict__ a, int len)
{
    __shared__ T warp_sums[33];
    const int t = threadIdx.x;
    if (t < 33) warp_sums[t] = Add<T>::zero();  // the warps the block lacks add nothing
    __syncthreads();
    const int chunk = (len + (int)blockDim.x - 1) / (int)blockDim.x;
    const int b = t * chunk, e = min(len, b + chunk);
    T s = Add<T>::zero();
    for (int k = b; k < e; ++k) s = Add<T>::op(s, a[k]);
    T total;
    T run = block_exclusive<T, 32>(s, warp_sums, &total);
    for (int k = b; k < e; ++k) {
        const T v = a[k];
        a[k] = run;
        run = Add<T>::op(run, v);
    }
}

// out[i] = sum_{k<i} in[k] for i in [0, n], out has n+1 entries.
template <class T>
__global__ void __launch_bounds__(256)
scan_apply_kernel(const T *__restrict__ in, int n, const T *__restrict__ block_off,
                  T *__restrict__ out)
{
    constexpr int kItems = ScanItems<T>::n;
    __shared__ T warp_sums[9];
    const int base = blockIdx.x * scan_tile<T>() + threadIdx.x * kItems;
    T s = Add<T>::zero();
#pragma unroll
    for (int k = 0; k < kItems; ++k)
        if (base + k < n) s = Add<T>::op(s, in[base + k]);
    T total;
    T run = Add<T>::op(block_off[blockIdx.x], block_exclusive<T, 8>(s, warp_sums, &total));
#pragma unroll
    for (int k = 0; k < kItems; ++k) {  // the thread's elements again (L1)
        if (base + k < n) {
            const T v = in[base + k];
            out[base + k] = run;
            run = Add<T>::op(run, v);
        }
        if (base + k == n - 1) out[n] = run;
    }
}

// ------------------------------------------------------------ radix sort
constexpr int kSortWarps = 8;
constexpr int kSortRounds = 8;
constexpr int kSortTile = kSortWarps * 32 * kSortRounds;  // 2048 keys
// Up to this many tiles (n <= 262,144) a scatter block sums the per-tile digit
// counts itself instead of a separate scan pass.
constexpr int kSortDirectTiles = 128;
// Up to this many tiles (n <= 131,072) the scatter also counts the next pass's
// digits (a global atomic per key), so passes after the first need no
// histogram launch; above it the atomics cost more than the launch saves.
constexpr int kSortFusedTiles = 64;

__global__ void __launch_bounds__(256)
radix_hist_kernel(const uint64_t *__restrict__ keys, int n, int shift, int *__restrict__ counts,
                  int digit_stride, int tile_stride)
{
    __shared__ int h[kSortWarps][256];
    const int warp = threadIdx.x >> 5;
    for (int k = threadIdx.x; k < kSortWarps * 256; k += 256) (&h[0][0])[k] = 0;
    __syncthreads();
    const int base = blockIdx.x * kSortTile;
    for (int k = threadIdx.x; k < kSortTile; k += 256) {
        const int idx = base + k;
        if (idx < n) atomicAdd(&h[warp][(int)((keys[idx] >> shift) & 0xFF)], 1);
    }
    __syncthreads();
    int c = 0;
    for (int w = 0; w < kSortWarps; ++w) c += h[w][threadIdx.x];
    counts[threadIdx.x * digit_stride + blockIdx.x * tile_stride] = c;
}

// Exclusive scan of a digit's counts over the tiles, in place, a block per digit, and the
// digit's total (the scatter scans the totals): one launch where a scan of the whole
// table took three, 3 for 9.2 us of a pass at N = 2^20.
__global__ void __launch_bounds__(256)
digit_scan_kernel(int *__restrict__ counts, int num_tiles, int *__restrict__ totals)
{
    __shared__ int warp_sums[kSortWarps + 1];
    int *row = counts + (size_t)blockIdx.x * num_tiles;
    int before = 0;
    for (int t0 = 0; t0 < num_tiles; t0 += 1024) {
        int v[4], sum = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int t = t0 + 4 * threadIdx.x + k;
            v[k] = t < num_tiles ? row[t] : 0;
            sum += v[k];
        }
        int all;
        int run = before + block_exclusive<int, kSortWarps>(sum, warp_sums, &all);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int t = t0 + 4 * threadIdx.x + k;
            if (t < num_tiles) row[t] = run;
            run += v[k];
        }
        before += all;
        __syncthreads();  // warp_sums are reused
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = before;
}

// Stable scatter of one 8-bit digit.  Warp w of the block ranks keys
// [tile + w*256, +256) in rounds of 32 (lane order), so ranks follow the input
// order; per-warp digit counts are turned into per-warp offsets.  The tile is
// then put in digit order in shared memory and written out by consecutive
// threads, so each digit's run of the tile goes to consecutive addresses.  The
// tile's global offset per digit is the digit's count in the earlier tiles plus all
// keys of smaller digits: from the scanned counts (digit_scan_kernel) and the
// digits' totals, or, when totals is null (few tiles), from the per-tile counts.
// next_counts (not for the last pass) receives the next pass's per-tile
// histogram, counted as the keys land (integer adds: any order gives the same
// counts), so that pass needs no histogram launch; each block also clears its
// column of zero_counts, the buffer the pass after next counts into.
__global__ void __launch_bounds__(256)
radix_scatter_kernel(const uint64_t *__restrict__ kin, const uint32_t *__restrict__ vin,
                     uint64_t *__restrict__ kout, uint32_t *__restrict__ vout, int n, int shift,
                     const int *__restrict__ counts, const int *__restrict__ totals,
                     int *__restrict__ next_counts, int *__restrict__ zero_counts, int num_tiles)
{
    __shared__ int wh[kSortWarps][256];
    __shared__ int toff[256];    // global position of the tile's first key of digit d
    __shared__ int tstart[256];  // position in the tile of its first key of digit d
    __shared__ int wsum[kSortWarps];
    __shared__ int dsum[kSortWarps + 1];
    __shared__ uint64_t skey[kSortTile];
    __shared__ uint32_t sval[kSortTile];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile0 = blockIdx.x * kSortTile;
    const int base = tile0 + warp * 32 * kSortRounds;
    uint64_t key[kSortRounds];
    uint32_t val[kSortRounds];
    int rank[kSortRounds], dig[kSortRounds];
    // every load before the first barrier: one round trip to memory, not one per round
#pragma unroll
    for (int r = 0; r < kSortRounds; ++r) {
        const int idx = base + r * 32 + lane;
        key[r] = idx < n ? kin[idx] : 0ull;
        val[r] = idx < n ? vin[idx] : 0u;
    }
    for (int k = threadIdx.x; k < kSortWarps * 256; k += 256) (&wh[0][0])[k] = 0;
    int before = 0, all = 0;
    if (totals) {
        before = counts[threadIdx.x * num_tiles + blockIdx.x];
        all = totals[threadIdx.x];
    } else {
#pragma unroll 16
        for (int tl = 0; tl < num_tiles; ++tl) {
            const int c = counts[tl * 256 + threadIdx.x];
            all += c;
            if (tl < (int)blockIdx.x) before += c;
        }
    }
    int keys;
    toff[threadIdx.x] = block_exclusive<int, kSortWarps>(all, dsum, &keys) + before;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortRounds; ++r) {
        const bool valid = base + r * 32 + lane < n;
        const int d = valid ? (int)((key[r] >> shift) & 0xFF) : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const int before = __popc(peers & ((1u << lane) - 1u));
        const int leader = 31 - __clz(peers);
        const int b = valid ? wh[warp][d] : 0;
        __syncwarp();
        if (valid && lane == leader) wh[warp][d] = b + __popc(peers);
        __syncwarp();
        rank[r] = b + before;
        dig[r] = d;
    }
    __syncthreads();
    {
        // per-warp offsets within the digit, and the tile's digit starts
        // (exclusive scan of the digit totals: warp shuffles, then warp sums)
        const int d = threadIdx.x;
        int run = 0;
        for (int w = 0; w < kSortWarps; ++w) {
            const int c = wh[w][d];
            wh[w][d] = run;
            run += c;
        }
        int inc = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        if (lane == 31) wsum[warp] = inc;
        __syncthreads();
        int before = 0;
        for (int w = 0; w < warp; ++w) before += wsum[w];
        tstart[d] = before + inc - run;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortRounds; ++r) {
        const int d = dig[r];
        if (d >= 0) {
            const int lpos = tstart[d] + wh[warp][d] + rank[r];
            skey[lpos] = key[r];
            sval[lpos] = val[r];
        }
    }
    __syncthreads();
    const int count = min(kSortTile, n - tile0);
    for (int j = threadIdx.x; j < count; j += 256) {
        const uint64_t k = skey[j];
        const int d = (int)((k >> shift) & 0xFF);
        const int pos = toff[d] + (j - tstart[d]);
        if (!NB_IN_RANGE(pos, n)) continue;
        kout[pos] = k;
        vout[pos] = sval[j];
        if (next_counts)
            atomicAdd(&next_counts[pos / kSortTile * 256 + (int)((k >> (shift + 8)) & 0xFF)], 1);
    }
    if (zero_counts) zero_counts[blockIdx.x * 256 + threadIdx.x] = 0;
}

// ------------------------------------------------------------ gather
__global__ void __launch_bounds__(256)
gather_kernel(const uint32_t *__restrict__ order, const double *__restrict__ x,
              const double *__restrict__ y, const double *__restrict__ z,
              const double *__restrict__ m, int n, const BHRoot *__restrict__ root,
              float4 *__restrict__ body, D4 *__restrict__ moments)
{
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const uint32_t o = order[i];
    if (!NB_IN_RANGE(o, n)) return;
    const double rx = x[o] - root->cx, ry = y[o] - root->cy, rz = z[o] - root->cz;
    const double mm = m[o];
    body[i] = make_float4((float)rx, (float)ry, (float)rz, (float)mm);
    moments[i] = D4{mm, mm * rx, mm * ry, mm * rz};
}

// Second moments m x x^T (relative to the root centre) of every sorted body,
// for the quadrupoles: a = (m x x, m y y, m z z, m x y), b = (m x z, m y z, 0, 0).
__global__ void __launch_bounds__(256)
gather2_kernel(const uint32_t *__restrict__ order, const double *__restrict__ x,
               const double *__restrict__ y, const double *__restrict__ z,
               const double *__restrict__ m, int n, const BHRoot *__restrict__ root,
               D4 *__restrict__ ma, D4 *__restrict__ mb)
{
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const uint32_t o = order[i];
    const double rx = x[o] - root->cx, ry = y[o] - root->cy, rz = z[o] - root->cz;
    const double mm = m[o];
    ma[i] = D4{mm * rx * rx, mm * ry * ry, mm * rz * rz, mm * rx * ry};
    mb[i] = D4{mm * rx * rz, mm * ry * rz, 0.0, 0.0};
}

// One past the last body of the depth-d cell of body i, its first: several probes per
// round trip to memory, first the next eight bodies (which ends the search of a leaf),
// then at distances 8^k, then within the bracket.
__device__ __forceinline__ int cell_end(const uint64_t *__restrict__ c, int n, int i, int d)
{
    if (d == 0) return n;
    const int sh = 63 - 3 * d;
    const uint64_t p = c[i] >> sh;
    const long limit = n - i;
    auto inside = [&](long k) { return k < limit && (c[i + k] >> sh) == p; };
    bool in[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) in[k] = inside(k + 1);
    long lo = 0, hi;  // lo inside, hi not
#pragma unroll
    for (int k = 0; k < 8; ++k) lo += in[k];
    if (lo < 8) return i + (int)lo + 1;
#pragma unroll
    for (int k = 2; k < 8; ++k) in[k] = inside(1l << 3 * k);
    hi = 64;
#pragma unroll
    for (int k = 2; k < 8; ++k)
        if (in[k]) {
            lo = 1l << 3 * k;
            hi = 8 * lo;
        }
    while (in[7] && inside(hi)) {  // beyond 8^7
        lo = hi;
        hi = 8 * lo;
    }
    hi = hi < limit ? hi : limit;
    while (hi - lo > 1) {
        const long step = (hi - lo + 7) / 8, from = lo;
#pragma unroll
        for (int k = 1; k < 8; ++k) in[k] = k * step < hi - from && inside(from + k * step);
#pragma unroll
        for (int k = 1; k < 8; ++k)
            if (in[k]) lo = from + k * step;
        hi = hi < lo + step ? hi : lo + step;
    }
    return i + (int)lo + 1;
}

// First index of the depth-d cell that contains body i (galloping: most of the
// searches are short).
__device__ __forceinline__ int cell_start(const uint64_t *__restrict__ c, int i, int d)
{
    if (d == 0) return 0;
    const int sh = 63 - 3 * d;
    const uint64_t p = c[i] >> sh;
    int hi = i, lo, step = 1;
    while (true) {
        lo = hi - step;
        if (lo < 0) {
            lo = -1;
            break;
        }
        if ((c[lo] >> sh) != p) break;
        hi = lo;
        step <<= 1;
    }
    while (hi - lo > 1) {
        const int mid = lo + (hi - lo) / 2;
        if ((c[mid] >> sh) == p) hi = mid;
        else lo = mid;
    }
    return hi;
}

// The depth down to which two codes lie in the same cell.
__device__ __forceinline__ int common_levels(uint64_t a, uint64_t b)
{
    const uint64_t x = a ^ b;
    return (x == 0 ? 63 : __clzll((long long)x) - 1) / 3;
}

// Depth of the first node starting at body i and the length of its chain
// (0 when no node starts at i); pstart[i]: the first body of that node's
// parent cell (when i starts a chain below the root).
__global__ void __launch_bounds__(256)
chain_kernel(const uint64_t *__restrict__ c, int n, int cap, const BHRoot *__restrict__ root,
             int *__restrict__ chain_len, int *__restrict__ chain_depth, int *__restrict__ pstart)
{
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const int levels = root->levels;
    int a = 0, L = 0;
    bool starts = true;
    if (i > 0) {
        const int s = min(common_levels(c[i], c[i - 1]), levels);
        if (s >= levels) {
            starts = false;
        } else {
            a = s + 1;
            const int ps = cell_start(c, i, s);
            starts = cap < n - ps && common_levels(c[ps + cap], c[i]) >= s;  // more than cap
            pstart[i] = ps;
        }
    }
    if (starts) {
        // the first depth from a on at which the cell holds cap bodies at most: body
        // i + cap is in body i's cells down to the depth their codes share
        const int t = cap < n - i ? common_levels(c[i], c[i + cap]) : -1;
        L = min(levels, max(a, t + 1)) - a + 1;
    }
    chain_len[i] = L;
    chain_depth[i] = a;
}

// (centre of mass, mass) of the bodies between two prefix sums of
// (m, m x, m y, m z): the differences in FP64 (exact enough: the sums are
// FP64), the division in FP32 (two roundings more than an FP64 division
// rounded to FP32, ~1e-7 of the position; the FP64 pipe is a small fraction
// of the FP32 one and three FP64 divisions per node dominated this kernel).
__device__ __forceinline__ float4 monopole(const D4 &lo, const D4 &hi)
{
    const double mass = hi.x - lo.x;
    if (!(mass > 0.0)) return make_float4(0.f, 0.f, 0.f, 0.f);
    const float m = (float)mass;
    if (m > 1e-30f && m < 1e30f) {
        const float r = 1.0f / m;
        return make_float4((float)(hi.y - lo.y) * r, (float)(hi.z - lo.z) * r,
                           (float)(hi.w - lo.w) * r, m);
    }
    return make_float4((float)((hi.y - lo.y) / mass), (float)((hi.z - lo.z) / mass),
                       (float)((hi.w - lo.w) / mass), m);  // outside FP32's comfortable range
}

// The centre of a depth-d cell's parent, relative to the root centre (the
// frame of the walk's bodies), and the cell's octant in that parent (bit 0 x,
// bit 1 y, bit 2 z: the high side), in .w as an int; the root (d = 0), which
// has no parent, gets 8.  The cell is read off the Morton code of any of its
// bodies: digit k (x high) of the 3d-bit prefix halves the cube along each axis.
__device__ __forceinline__ float4 parent_centre(uint64_t code, int d, const BHRoot *root)
{
    if (d == 0) return make_float4(0.f, 0.f, 0.f, __int_as_float(8));
    const uint64_t pfx = code >> (63 - 3 * d);
    const int dig = (int)(pfx & 7u);
    uint32_t ix = 0, iy = 0, iz = 0;
    for (int k = 0; k < d - 1; ++k) {
        const int g = (int)((pfx >> (3 * (d - 1 - k))) & 7u);
        ix = 2 * ix + ((g >> 2) & 1);
        iy = 2 * iy + ((g >> 1) & 1);
        iz = 2 * iz + (g & 1);
    }
    const double side = ldexp(root->size, -(d - 1));  // the parent's side
    const double h = 0.5 * root->size;
    const int oct = ((dig >> 2) & 1) | (((dig >> 1) & 1) << 1) | ((dig & 1) << 2);
    return make_float4((float)(((double)ix + 0.5) * side - h), (float)(((double)iy + 0.5) * side - h),
                       (float)(((double)iz + 0.5) * side - h), __int_as_float(oct));
}

// The nodes' first bodies and depths, by the bodies their chains start at, and what
// node_kernel adds to at zero (a memset each was a launch).
__global__ void __launch_bounds__(256)
place_kernel(int n, const int *__restrict__ chain_len, const int *__restrict__ chain_depth,
             const int *__restrict__ offsets, BHNode *__restrict__ nodes,
             unsigned char *__restrict__ node_depth, unsigned long long *__restrict__ kidrows,
             BHStats *__restrict__ stats, int node_cap)
{
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i == 0) {
        stats->m2p = stats->p2p = 0;
        stats->leaves = stats->max_depth = 0;
    }
    if (i >= n) return;
    const int L = chain_len[i];
    if (L == 0) return;
    const int a = chain_depth[i], id0 = offsets[i];
    for (int k = 0; k < L; ++k) {
        if (!NB_IN_RANGE(id0 + k, node_cap)) break;
        kidrows[id0 + k] = 0;
        nodes[id0 + k].first = i;
        node_depth[id0 + k] = (unsigned char)(a + k);
    }
}

// The rest of every node, a thread per node.  By body, a thread writing its chain,
// the longest chain was the critical path, and few lanes of a warp had the FP64 work:
// 79 us at N = 2^20, 31 at 100,000; 43 and 20 now, with place_kernel.
__global__ void __launch_bounds__(256)
node_kernel(const uint64_t *__restrict__ c, int n, const BHRoot *__restrict__ root,
            const int *__restrict__ total, const int *__restrict__ chain_depth,
            const int *__restrict__ offsets, const D4 *__restrict__ P,
            BHNode *__restrict__ nodes, const unsigned char *__restrict__ node_depth,
            const int *__restrict__ pstart, int *__restrict__ parent,
            unsigned char *__restrict__ octant, unsigned char *__restrict__ kidflag,
            BHStats *__restrict__ stats, int node_cap)
{
    const int num = *total;
    int leaves = 0, deepest = 0;
    for (int k = blockIdx.x * 256 + threadIdx.x; k < num; k += gridDim.x * 256) {
        if (!NB_IN_RANGE(k, node_cap)) break;
        BHNode nd;
        const int i = nd.first = nodes[k].first, d = node_depth[k];
        const int end = cell_end(c, n, i, d);
        if (!NB_IN_RANGE(i, n) || !NB_IN_RANGE(end, n + 1)) continue;
        nd.com_mass = monopole(P[i], P[end]);
        nd.count = end - i;
        nd.skip = offsets[end];
        nd.size2 = root->size2[d];
        nodes[k] = nd;
        if (d > 0) {  // the parent: the previous node of the chain, or the one holding it
            int par = k - 1;
            if (k == offsets[i]) {
                const int j = pstart[i];
                par = offsets[j] + (d - 1 - chain_depth[j]);
            }
            const int oct = (int)((c[i] >> (63 - 3 * d)) & 7u);
            parent[k] = par;
            octant[k] = (unsigned char)oct;
            if (NB_IN_RANGE(par, node_cap)) kidflag[(size_t)par * 8 + oct] = 1;
        }
        leaves += nd.skip == k + 1;
        deepest = max(deepest, d);
    }
    leaves = __reduce_add_sync(0xffffffffu, leaves);
    deepest = __reduce_max_sync(0xffffffffu, deepest);
    if ((threadIdx.x & 31) == 0 && leaves > 0) {
        atomicAdd(&stats->leaves, leaves);
        atomicMax(&stats->max_depth, deepest);
    }
}

// Parent centres and octants of every node (parent_centre), for the walk
// under the reference's opening rule only: read off the Morton code of the
// node's first body and its depth.
__global__ void __launch_bounds__(256)
pcen_kernel(const uint64_t *__restrict__ c, const BHNode *__restrict__ nodes,
            const unsigned char *__restrict__ node_depth, const int *__restrict__ total,
            const BHRoot *__restrict__ root, float4 *__restrict__ pcen)
{
    const int num = *total;
    for (int k = blockIdx.x * 256 + threadIdx.x; k < num; k += gridDim.x * 256)
        pcen[k] = parent_centre(c[nodes[k].first], node_depth[k], root);
}

// ------------------------------------------------------------ refit
// Tree reuse: the topology and body order of the last build are kept while
// the bodies move; every evaluation in between recomputes the monopoles from
// the bodies' current positions and replaces each cell's side by the larger of
// its cube side and the extent of its bodies' bounding box, so a drifted cell
// is opened at least as readily as a freshly built one would be.
__device__ __forceinline__ float box_ext2(float4 lo, float4 hi)
{
    const float e = fmaxf(hi.x - lo.x, fmaxf(hi.y - lo.y, hi.z - lo.z));
    return e * e;
}

// Monopoles of every node; bounding boxes and sides of the leaves.
__global__ void __launch_bounds__(256)
refit_kernel(BHNode *__restrict__ nodes, const int *__restrict__ total,
             const unsigned char *__restrict__ node_depth, const D4 *__restrict__ P,
             const BHRoot *__restrict__ root, const float4 *__restrict__ body,
             float4 *__restrict__ boxes)
{
    const int k = blockIdx.x * 256 + threadIdx.x;
    if (k >= *total) return;
    BHNode nd = nodes[k];
    nd.com_mass = monopole(P[nd.first], P[nd.first + nd.count]);
    if (nd.skip == k + 1) {  // leaf
        float4 mn = body[nd.first], mx = mn;
        for (int b = nd.first + 1; b < nd.first + nd.count; ++b) {
            const float4 q = body[b];
            mn = make_float4(fminf(mn.x, q.x), fminf(mn.y, q.y), fminf(mn.z, q.z), 0.f);
            mx = make_float4(fmaxf(mx.x, q.x), fmaxf(mx.y, q.y), fmaxf(mx.z, q.z), 0.f);
        }
        boxes[2 * k] = mn;
        boxes[2 * k + 1] = mx;
        nd.size2 = fmaxf(root->size2[node_depth[k]], box_ext2(mn, mx));
    }
    nodes[k] = nd;
}

// Internal nodes of depth d: box = union of the children's boxes (children:
// node + 1, then each child's skip pointer up to the node's own).
__global__ void __launch_bounds__(256)
refit_level_kernel(BHNode *__restrict__ nodes, const int *__restrict__ total,
                   const unsigned char *__restrict__ node_depth, int d,
                   const BHRoot *__restrict__ root, float4 *__restrict__ boxes)
{
    const int k = blockIdx.x * 256 + threadIdx.x;
    if (k >= *total || node_depth[k] != d) return;
    const int skip = nodes[k].skip;
    if (skip == k + 1) return;  // leaf: done by refit_kernel
    float4 mn = make_float4(3.0e38f, 3.0e38f, 3.0e38f, 0.f);
    float4 mx = make_float4(-3.0e38f, -3.0e38f, -3.0e38f, 0.f);
    for (int c = k + 1; c < skip; c = nodes[c].skip) {
        const float4 a = boxes[2 * c], b = boxes[2 * c + 1];
        mn = make_float4(fminf(mn.x, a.x), fminf(mn.y, a.y), fminf(mn.z, a.z), 0.f);
        mx = make_float4(fmaxf(mx.x, b.x), fmaxf(mx.y, b.y), fmaxf(mx.z, b.z), 0.f);
    }
    boxes[2 * k] = mn;
    boxes[2 * k + 1] = mx;
    nodes[k].size2 = fmaxf(root->size2[d], box_ext2(mn, mx));
}

// ------------------------------------------------------------ quadrupoles
// Traceless quadrupole of every node about its centre of mass, from the FP64
// prefix sums of the moments: with S = sum m x x^T - M c c^T (positions
// relative to the root centre, c the centre of mass),
// Q = 3 S - tr(S) I; stored as (Qxx, Qyy, Qzz, Qxy), (Qxz, Qyz, 0, 0).
__global__ void __launch_bounds__(256)
quad_kernel(const BHNode *__restrict__ nodes, const int *__restrict__ total, const D4 *__restrict__ P,
            const D4 *__restrict__ PA, const D4 *__restrict__ PB, float4 *__restrict__ quad)
{
    const int k = blockIdx.x * 256 + threadIdx.x;
    if (k >= *total) return;
    const int a = nodes[k].first, b = a + nodes[k].count;
    const double M = P[b].x - P[a].x;
    float4 q0 = make_float4(0.f, 0.f, 0.f, 0.f), q1 = q0;
    if (M > 0.0) {
        const double cx = (P[b].y - P[a].y) / M, cy = (P[b].z - P[a].z) / M,
                     cz = (P[b].w - P[a].w) / M;
        const double sxx = (PA[b].x - PA[a].x) - M * cx * cx;
        const double syy = (PA[b].y - PA[a].y) - M * cy * cy;
        const double szz = (PA[b].z - PA[a].z) - M * cz * cz;
        const double sxy = (PA[b].w - PA[a].w) - M * cx * cy;
        const double sxz = (PB[b].x - PB[a].x) - M * cx * cz;
        const double syz = (PB[b].y - PB[a].y) - M * cy * cz;
        const double tr = sxx + syy + szz;
        q0 = make_float4((float)(3.0 * sxx - tr), (float)(3.0 * syy - tr),
                         (float)(3.0 * szz - tr), (float)(3.0 * sxy));
        q1 = make_float4((float)(3.0 * sxz), (float)(3.0 * syz), 0.f, 0.f);
    }
    quad[2 * k] = q0;
    quad[2 * k + 1] = q1;
}

// ------------------------------------------------------------ walk
constexpr int kWalkBlock = 128;

// ZERO_SOFT: eps2 == 0, where the lane's own body (r2 == 0) contributes 0.
// QUAD: accepted cells act as monopole + quadrupole, a = G M r / |r|^3 +
// G (5/2 (r.Q r) r / |r|^2 - Q r) / |r|^5 with r from the body to the centre
// of mass (softened |r| throughout).
// The reference's opening rule (NB_FLAG_BH_REFERENCE_OPENING;
// CPU/src/force_calculator_barnes_hut_optimized.cpp and
// CUDA/src/force_calculator_barnes_hut.cu:60-73): of every node a walk opens,
// the child in the body's octant (relative to the node's centre) is opened
// too, whether or not it holds the body; the opening test applies to the
// other children.  A node is reached only after its parent was opened, so
// the walk asks, per node, whether the body lies on the node's side of its
// parent's centre on all three axes (pc from parent_centre).
__device__ __forceinline__ bool toward_body(float4 pc, float x, float y, float z)
{
    const int oct = __float_as_int(pc.w);
    return oct < 8 && ((x >= pc.x) == ((oct & 1) != 0)) && ((y >= pc.y) == ((oct & 2) != 0)) &&
           ((z >= pc.z) == ((oct & 4) != 0));
}

template <bool ZERO_SOFT, bool QUAD, bool DIR>
__global__ void __launch_bounds__(kWalkBlock)
walk_kernel(const BHNode *__restrict__ nodes, const int *__restrict__ total,
            const float4 *__restrict__ body, const uint32_t *__restrict__ order, int n,
            float theta2, float eps2, double G, double *__restrict__ ax,
            double *__restrict__ ay, double *__restrict__ az, BHStats *__restrict__ stats,
            const float4 *__restrict__ quad, const float4 *__restrict__ pcen)
{
    const int num_nodes = *total;
    const int lane = threadIdx.x & 31;
    const int warp0 = (blockIdx.x * kWalkBlock + threadIdx.x) - lane;
    if (warp0 >= n) return;  // whole warp past the end
    const int i = warp0 + lane;
    const bool valid = i < n;
    const float4 p = body[valid ? i : n - 1];
    const float2 npx = dup2(-p.x), npy = dup2(-p.y), npz = dup2(-p.z), e2 = dup2(eps2);
    float fx = 0.f, fy = 0.f, fz = 0.f;                         // monopoles, odd bodies
    float2 gx = dup2(0.f), gy = dup2(0.f), gz = dup2(0.f);     // leaf bodies in pairs
    unsigned m2p = 0, p2p = 0;
    int node = 0;
    while (node < num_nodes) {
        const BHNode nd = nodes[node];
        const float dx = nd.com_mass.x - p.x;
        const float dy = nd.com_mass.y - p.y;
        const float dz = nd.com_mass.z - p.z;
        const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
        const bool mine = (unsigned)(i - nd.first) < (unsigned)nd.count;
        bool open = valid && (mine || nd.size2 >= theta2 * d2);
        if (DIR) open = open || (valid && toward_body(pcen[node], p.x, p.y, p.z));
        if (__any_sync(0xffffffffu, open)) {
            if (nd.skip != node + 1) {  // internal: descend
                ++node;
                continue;
            }
            // leaf: its bodies, two per f32x2 instruction
            const int e = NB_IN_RANGE(nd.first, n) && NB_IN_RANGE(nd.first + nd.count - 1, n)
                              ? nd.first + nd.count
                              : nd.first;
            int b = nd.first;
            for (; b + 1 < e; b += 2) {
                const float4 q0 = body[b], q1 = body[b + 1];
                const float2 rx = add2(make_float2(q0.x, q1.x), npx);
                const float2 ry = add2(make_float2(q0.y, q1.y), npy);
                const float2 rz = add2(make_float2(q0.z, q1.z), npz);
                const float2 r2 = fma2(rz, rz, fma2(ry, ry, fma2(rx, rx, e2)));
                float2 inv = make_float2(rsqrt_mufu(r2.x), rsqrt_mufu(r2.y));
                if (ZERO_SOFT) {
                    inv.x = r2.x > 0.f ? inv.x : 0.f;
                    inv.y = r2.y > 0.f ? inv.y : 0.f;
                }
                const float2 s = mul2(mul2(make_float2(q0.w, q1.w), inv), mul2(inv, inv));
                gx = fma2(rx, s, gx);
                gy = fma2(ry, s, gy);
                gz = fma2(rz, s, gz);
            }
            if (b < e) {
                const float4 q = body[b];
                const float rx = q.x - p.x, ry = q.y - p.y, rz = q.z - p.z;
                const float r2 = fmaf(rz, rz, fmaf(ry, ry, fmaf(rx, rx, eps2)));
                float inv = rsqrt_mufu(r2);
                if (ZERO_SOFT) inv = r2 > 0.f ? inv : 0.f;
                const float s = (q.w * inv) * (inv * inv);
                fx = fmaf(rx, s, fx);
                fy = fmaf(ry, s, fy);
                fz = fmaf(rz, s, fz);
            }
            p2p += nd.count;
        } else {
            const float inv = rsqrt_mufu(d2 + eps2);
            const float inv2 = inv * inv;
            const float s = (nd.com_mass.w * inv) * inv2;
            fx = fmaf(dx, s, fx);
            fy = fmaf(dy, s, fy);
            fz = fmaf(dz, s, fz);
            if (QUAD) {
                const float4 q0 = quad[2 * node], q1 = quad[2 * node + 1];
                const float qx = fmaf(q0.x, dx, fmaf(q0.w, dy, q1.x * dz));
                const float qy = fmaf(q0.w, dx, fmaf(q0.y, dy, q1.y * dz));
                const float qz = fmaf(q1.x, dx, fmaf(q1.y, dy, q0.z * dz));
                const float rqr = fmaf(dx, qx, fmaf(dy, qy, dz * qz));
                const float inv5 = (inv * inv2) * inv2;  // |r|^-5
                const float f = 2.5f * rqr * inv2;
                fx = fmaf(inv5, fmaf(f, dx, -qx), fx);
                fy = fmaf(inv5, fmaf(f, dy, -qy), fy);
                fz = fmaf(inv5, fmaf(f, dz, -qz), fz);
            }
            ++m2p;
        }
        if (!NB_IN_RANGE(nd.skip - node - 1, num_nodes)) break;  // skips only go forward
        node = nd.skip;
    }
    if (valid) {
        const uint32_t o = order[i];
        ax[o] = G * ((double)fx + ((double)gx.x + (double)gx.y));
        ay[o] = G * ((double)fy + ((double)gy.x + (double)gy.y));
        az[o] = G * ((double)fz + ((double)gz.x + (double)gz.y));
    }
    // every lane ran the same interactions: count once per valid lane
    const unsigned nv = __popc(__ballot_sync(0xffffffffu, valid));
    if (lane == 0) {
        atomicAdd(&stats->m2p, (unsigned long long)m2p * nv);
        atomicAdd(&stats->p2p, (unsigned long long)p2p * nv);
        atomicAdd(&stats->total, (unsigned long long)(m2p + p2p) * nv);
    }
}

// The same walk for 64 * NP consecutive sorted bodies per warp, 2 * NP per
// lane (body w0 + 32 k + lane for k < 2 NP, held as NP packed pairs): one node
// load, vote and branch serve them all, and their MAC, monopole and leaf terms
// run as f32x2 pairs.  The warp opens a node if any of its bodies does --
// never a coarser walk than any body's own.
template <bool ZERO_SOFT, bool QUAD, int NP, bool DIR>
__global__ void __launch_bounds__(kWalkBlock)
walk2_kernel(const BHNode *__restrict__ nodes, const int *__restrict__ total,
             const float4 *__restrict__ body, const uint32_t *__restrict__ order, int n,
             float theta2, float eps2, double G, double *__restrict__ ax,
             double *__restrict__ ay, double *__restrict__ az, BHStats *__restrict__ stats,
             const float4 *__restrict__ quad, const float4 *__restrict__ pcen)
{
    const int num_nodes = *total;
    constexpr int kPer = 64 * NP;  // bodies per warp
    const int lane = threadIdx.x & 31;
    const int w0 = ((blockIdx.x * kWalkBlock + threadIdx.x) >> 5) * kPer;
    if (w0 >= n) return;  // whole warp past the end
    int ia[NP], ib[NP];
    bool va[NP], vb[NP];
    float2 npx[NP], npy[NP], npz[NP], fx[NP], fy[NP], fz[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) {
        ia[k] = w0 + 64 * k + lane;
        ib[k] = ia[k] + 32;
        va[k] = ia[k] < n;
        vb[k] = ib[k] < n;
        const float4 pa = body[va[k] ? ia[k] : n - 1], pb = body[vb[k] ? ib[k] : n - 1];
        npx[k] = make_float2(-pa.x, -pb.x);
        npy[k] = make_float2(-pa.y, -pb.y);
        npz[k] = make_float2(-pa.z, -pb.z);
        fx[k] = fy[k] = fz[k] = dup2(0.f);
    }
    const float2 e2 = dup2(eps2), t2 = dup2(theta2);
    unsigned m2p = 0, p2p = 0;
    int node = 0;
    while (node < num_nodes) {
        const BHNode nd = nodes[node];
        const float4 pc = DIR ? pcen[node] : make_float4(0.f, 0.f, 0.f, 0.f);
        float2 dx[NP], dy[NP], dz[NP], d2[NP];
        bool open = false;
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            dx[k] = add2(dup2(nd.com_mass.x), npx[k]);
            dy[k] = add2(dup2(nd.com_mass.y), npy[k]);
            dz[k] = add2(dup2(nd.com_mass.z), npz[k]);
            d2[k] = fma2(dz[k], dz[k], fma2(dy[k], dy[k], mul2(dx[k], dx[k])));
            const float2 td2 = mul2(t2, d2[k]);
            const bool oa = va[k] & (((unsigned)(ia[k] - nd.first) < (unsigned)nd.count) |
                                     (nd.size2 >= td2.x));
            const bool ob = vb[k] & (((unsigned)(ib[k] - nd.first) < (unsigned)nd.count) |
                                     (nd.size2 >= td2.y));
            open = open | oa | ob;
            if (DIR)
                open = open | (va[k] & toward_body(pc, -npx[k].x, -npy[k].x, -npz[k].x)) |
                       (vb[k] & toward_body(pc, -npx[k].y, -npy[k].y, -npz[k].y));
        }
        if (__any_sync(0xffffffffu, open)) {
            if (nd.skip != node + 1) {  // internal: descend
                ++node;
                continue;
            }
            const int e = NB_IN_RANGE(nd.first, n) && NB_IN_RANGE(nd.first + nd.count - 1, n)
                              ? nd.first + nd.count
                              : nd.first;
            for (int b = nd.first; b < e; ++b) {
                const float4 q = body[b];
#pragma unroll
                for (int k = 0; k < NP; ++k) {
                    const float2 rx = add2(dup2(q.x), npx[k]);
                    const float2 ry = add2(dup2(q.y), npy[k]);
                    const float2 rz = add2(dup2(q.z), npz[k]);
                    const float2 r2 = fma2(rz, rz, fma2(ry, ry, fma2(rx, rx, e2)));
                    float2 inv = make_float2(rsqrt_mufu(r2.x), rsqrt_mufu(r2.y));
                    if (ZERO_SOFT) {
                        inv.x = r2.x > 0.f ? inv.x : 0.f;
                        inv.y = r2.y > 0.f ? inv.y : 0.f;
                    }
                    const float2 s = mul2(mul2(dup2(q.w), inv), mul2(inv, inv));
                    fx[k] = fma2(rx, s, fx[k]);
                    fy[k] = fma2(ry, s, fy[k]);
                    fz[k] = fma2(rz, s, fz[k]);
                }
            }
            p2p += nd.count;
        } else {
            float4 q0, q1;
            if (QUAD) {
                q0 = quad[2 * node];
                q1 = quad[2 * node + 1];
            }
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                const float2 r2 = add2(d2[k], e2);
                const float2 inv = make_float2(rsqrt_mufu(r2.x), rsqrt_mufu(r2.y));
                const float2 inv2 = mul2(inv, inv);
                const float2 s = mul2(mul2(dup2(nd.com_mass.w), inv), inv2);
                fx[k] = fma2(dx[k], s, fx[k]);
                fy[k] = fma2(dy[k], s, fy[k]);
                fz[k] = fma2(dz[k], s, fz[k]);
                if (QUAD) {
                    const float2 qx = fma2(dup2(q0.x), dx[k],
                                           fma2(dup2(q0.w), dy[k], mul2(dup2(q1.x), dz[k])));
                    const float2 qy = fma2(dup2(q0.w), dx[k],
                                           fma2(dup2(q0.y), dy[k], mul2(dup2(q1.y), dz[k])));
                    const float2 qz = fma2(dup2(q1.x), dx[k],
                                           fma2(dup2(q1.y), dy[k], mul2(dup2(q0.z), dz[k])));
                    const float2 rqr = fma2(dx[k], qx, fma2(dy[k], qy, mul2(dz[k], qz)));
                    const float2 inv5 = mul2(mul2(inv, inv2), inv2);
                    const float2 f = mul2(mul2(dup2(2.5f), rqr), inv2);
                    fx[k] = fma2(inv5, fma2(f, dx[k], make_float2(-qx.x, -qx.y)), fx[k]);
                    fy[k] = fma2(inv5, fma2(f, dy[k], make_float2(-qy.x, -qy.y)), fy[k]);
                    fz[k] = fma2(inv5, fma2(f, dz[k], make_float2(-qz.x, -qz.y)), fz[k]);
                }
            }
            ++m2p;
        }
        if (!NB_IN_RANGE(nd.skip - node - 1, num_nodes)) break;  // skips only go forward
        node = nd.skip;
    }
    unsigned nv = 0;
#pragma unroll
    for (int k = 0; k < NP; ++k) {
        if (va[k]) {
            const uint32_t o = order[ia[k]];
            ax[o] = G * (double)fx[k].x;
            ay[o] = G * (double)fy[k].x;
            az[o] = G * (double)fz[k].x;
        }
        if (vb[k]) {
            const uint32_t o = order[ib[k]];
            ax[o] = G * (double)fx[k].y;
            ay[o] = G * (double)fy[k].y;
            az[o] = G * (double)fz[k].y;
        }
        nv += __popc(__ballot_sync(0xffffffffu, va[k])) + __popc(__ballot_sync(0xffffffffu, vb[k]));
    }
    if (lane == 0) {
        atomicAdd(&stats->m2p, (unsigned long long)m2p * nv);
        atomicAdd(&stats->p2p, (unsigned long long)p2p * nv);
        atomicAdd(&stats->total, (unsigned long long)(m2p + p2p) * nv);
    }
}

// ------------------------------------------------------------ child groups
// The group walk reads the children of a node together: gnodes holds, for
// every internal node, its children's records contiguously and in Morton order
// (a group), and group 0 is the root alone.  node_kernel records every node's
// parent and octant and marks byte (parent, octant) of an 8-byte row per node
// (each child its own byte: no atomics); alloc_groups_kernel packs a row into
// the node's octant mask and claims a place for each group from a counter (every node
// but the root is the child of exactly one node, so there are as many records
// as nodes; where a group lands changes no result, since the walk's arithmetic
// follows the groups' contents), and group_kernel writes each record with its
// children count, its parent centre and, for the quadrupole walk, its
// quadrupole beside it.  Both run over the node count read on the device.
struct alignas(32) BHGNode {
    float4 com_mass;  // as BHNode
    float size2;
    int first, count;
    int kids;         // the record of the node's first child (-1: a leaf)
};
static_assert(sizeof(BHGNode) == 32, "group record layout");

// A place for the group of every node with children (occ: the mask of its
// non-empty octants, packed from its row of kidflag): a block numbers its
// nodes' groups by a scan and claims their span from the counter with one
// atomic.
__global__ void __launch_bounds__(256)
alloc_groups_kernel(const unsigned char *__restrict__ kidflag, const int *__restrict__ total,
                    unsigned *__restrict__ occ, int *__restrict__ base, int *__restrict__ next)
{
    __shared__ int warp_sums[9];
    __shared__ int span0;
    const int num = *total;
    for (int k0 = blockIdx.x * 256; k0 < num; k0 += gridDim.x * 256) {
        const int k = k0 + threadIdx.x;
        unsigned o = 0;
        if (k < num) {
            const uint2 f = reinterpret_cast<const uint2 *>(kidflag)[k];
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                o |= ((f.x >> (8 * b)) & 0xFFu) ? 1u << b : 0u;
                o |= ((f.y >> (8 * b)) & 0xFFu) ? 1u << (b + 4) : 0u;
            }
            occ[k] = o;
        }
        const int nk = __popc(o);
        int span;
        const int off = block_exclusive<int, 8>(nk, warp_sums, &span);
        if (threadIdx.x == 0) span0 = atomicAdd(next, span);
        __syncthreads();
        if (nk > 0) base[k] = span0 + off;
        __syncthreads();  // span0 and warp_sums are reused by the next round
    }
}

// Every node's record: the root at 0, a child at its parent's group place
// plus its rank among the parent's non-empty octants (Morton order).
__global__ void __launch_bounds__(256)
group_kernel(const BHNode *__restrict__ nodes, const int *__restrict__ total,
             const unsigned *__restrict__ occ, const int *__restrict__ base,
             const int *__restrict__ parent, const unsigned char *__restrict__ octant,
             const float4 *__restrict__ pcen, const float4 *__restrict__ quad,
             BHGNode *__restrict__ gnodes, unsigned char *__restrict__ gnk,
             float4 *__restrict__ gpcen, float4 *__restrict__ gquad,
             const unsigned char *__restrict__ node_depth, unsigned *__restrict__ gkey,
             unsigned long long *__restrict__ log_next)
{
    if (log_next && blockIdx.x == 0 && threadIdx.x == 0) *log_next = 0;  // a walk follows
    const int num = *total;
    for (int k = blockIdx.x * 256 + threadIdx.x; k < num; k += gridDim.x * 256) {
        int pos = 0;
        if (k > 0) {
            const int par = parent[k];
            if (!NB_IN_RANGE(par, num)) continue;
            pos = 1 + base[par] + __popc(occ[par] & ((1u << octant[k]) - 1u));
        }
        if (!NB_IN_RANGE(pos, num)) continue;
        const BHNode nd = nodes[k];
        const unsigned o = occ[k];
        BHGNode g;
        g.com_mass = nd.com_mass;
        g.size2 = nd.size2;
        g.first = nd.first;
        g.count = nd.count;
        g.kids = o ? 1 + base[k] : -1;
        gnodes[pos] = g;
        gnk[pos] = (unsigned char)__popc(o);
        if (pcen) gpcen[pos] = pcen[k];
        if (gkey) gkey[pos] = 1u + (unsigned)(num + node_depth[k] - nd.skip);
        if (quad) {
            gquad[2 * pos] = quad[2 * k];
            gquad[2 * pos + 1] = quad[2 * k + 1];
        }
    }
}

// ------------------------------------------------------------ group walk
// One CTA walks for 64 NP consecutive sorted bodies, 2 NP per lane of each of its
// W warps.  A warp decides 32 nodes at a time, one per lane, and only then
// computes.  In each round
//   - warp w takes the groups w, W + w, 2 W + w, 3 W + w below the top of the
//     CTA's stack, and every lane loads one node's record;
//   - a lane closes its node when no body can open it, or opens it when some
//     body must, by the bounding boxes of the 32-body chunks; the few nodes in
//     between are tested against every body, two nodes at a time.  The distances
//     to a box are computed as those to a body are, operation by operation, so
//     rounding keeps their order and the decisions are those of testing every
//     body;
//   - closed nodes and the bodies of opened leaves are appended to the warp's
//     list in shared memory, two side by side, and the groups of opened internal
//     nodes go onto the stack; a long enough list is evaluated as f32x2 pairs of
//     list entries.
// The interactions are those of walk2_kernel; only their order differs, and it is
// a function of the tree, n and W alone.
//
// Bound by dispatch.  Testing each node by all bodies, one round trip to memory
// per group, took 2.32 ms at N = 2^20 (theta 0.5), 3.67 ms at N = 100,000 under
// the reference's opening rule (ten warps per SM, each a serial walk, the longest
// five times the mean); this takes 1.73 ms with one warp per walk and 0.55 ms with
// sixteen.  Of the 1.73 ms, about 1.2 are the 15.5 dispatch cycles per interaction
// of the evaluation, the rest the decisions (2,600 nodes per walk, a fifth of them
// undecided).
//
// Stack bound: the groups pushed by one round (at most 32 W) are children of
// nodes at or below the lowest level of the groups it took, so the lowest
// levels of the rounds on the stack strictly increase: 32 W per level.
constexpr int kWalkWarps = 16;                     // at most
constexpr int kWalkStack = 32 * (kMaxLevels + 1);  // per warp
constexpr int kListPairs = 32;                     // list capacity: 64 entries
constexpr int kListFlush = 2 * kListPairs - 32;    // evaluate from here on

// Lists of one warp; entry e lies in half e & 1 of pair e >> 1.
struct WalkList {
    float4 a[kListPairs];  // (x_0, x_1, y_0, y_1)
    float4 b[kListPairs];  // (z_0, z_1, m_0, m_1)
};
struct WalkQuads {
    float4 q[kListPairs][3];  // (xx, yy), (zz, xy), (xz, yz) of both entries
};
// Shared memory of a CTA: W of these, then its stack of W * kWalkStack groups
// (int first records, then unsigned char record counts).
template <bool QUAD>
struct WalkShared {
    float4 test[32];  // (com, size2) of the batch's nodes
    float4 side[32];  // their parents' centres (DIR)
    WalkList list;
};
template <>
struct WalkShared<true> : WalkShared<false> {
    WalkList bodies;  // leaf bodies apart: they have no quadrupole
    WalkQuads quads;
};
template <bool QUAD>
constexpr size_t walk_shared_bytes(int warps)
{
    return warps * (sizeof(WalkShared<QUAD>) + kWalkStack * (sizeof(int) + 1));
}

__device__ __forceinline__ void list_put(WalkList &l, int e, float x, float y, float z, float m)
{
    float *a = reinterpret_cast<float *>(&l.a[e >> 1]) + (e & 1);
    float *b = reinterpret_cast<float *>(&l.b[e >> 1]) + (e & 1);
    a[0] = x;
    a[2] = y;
    b[0] = z;
    b[2] = m;
}

// The lane's K bodies, negated and duplicated, and their sums (over the even
// and the odd list entries).
template <int K>
struct WalkBodies {
    float2 nx[K], ny[K], nz[K];
    float2 fx[K], fy[K], fz[K];
};

// Pairs [0, pairs) of a list, pairs a multiple of 4.
template <bool ZERO_SOFT, bool QUAD, int K>
__device__ __forceinline__ void list_eval(const WalkList &l, const WalkQuads *quads, int pairs,
                                          float2 e2, WalkBodies<K> &wb)
{
#pragma unroll 4
    for (int p = 0; p < pairs; ++p) {
        const float4 A = l.a[p], B = l.b[p];
        float2 qxx, qyy, qzz, qxy, qxz, qyz;
        if (QUAD) {
            const float4 Q0 = quads->q[p][0], Q1 = quads->q[p][1], Q2 = quads->q[p][2];
            qxx = make_float2(Q0.x, Q0.y); qyy = make_float2(Q0.z, Q0.w);
            qzz = make_float2(Q1.x, Q1.y); qxy = make_float2(Q1.z, Q1.w);
            qxz = make_float2(Q2.x, Q2.y); qyz = make_float2(Q2.z, Q2.w);
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const float2 dx = add2(make_float2(A.x, A.y), wb.nx[k]);
            const float2 dy = add2(make_float2(A.z, A.w), wb.ny[k]);
            const float2 dz = add2(make_float2(B.x, B.y), wb.nz[k]);
            const float2 r2 = fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, e2)));
            float2 inv = make_float2(rsqrt_mufu(r2.x), rsqrt_mufu(r2.y));
            if (ZERO_SOFT) {
                inv.x = r2.x > 0.f ? inv.x : 0.f;
                inv.y = r2.y > 0.f ? inv.y : 0.f;
            }
            const float2 inv2 = mul2(inv, inv);
            const float2 s = mul2(mul2(make_float2(B.z, B.w), inv), inv2);
            wb.fx[k] = fma2(dx, s, wb.fx[k]);
            wb.fy[k] = fma2(dy, s, wb.fy[k]);
            wb.fz[k] = fma2(dz, s, wb.fz[k]);
            if (QUAD) {
                const float2 qx = fma2(qxx, dx, fma2(qxy, dy, mul2(qxz, dz)));
                const float2 qy = fma2(qxy, dx, fma2(qyy, dy, mul2(qyz, dz)));
                const float2 qz = fma2(qxz, dx, fma2(qyz, dy, mul2(qzz, dz)));
                const float2 rqr = fma2(dx, qx, fma2(dy, qy, mul2(dz, qz)));
                const float2 inv5 = mul2(mul2(inv, inv2), inv2);
                const float2 f = mul2(mul2(dup2(2.5f), rqr), inv2);
                wb.fx[k] = fma2(inv5, fma2(f, dx, make_float2(-qx.x, -qx.y)), wb.fx[k]);
                wb.fy[k] = fma2(inv5, fma2(f, dy, make_float2(-qy.x, -qy.y)), wb.fy[k]);
                wb.fz[k] = fma2(inv5, fma2(f, dz, make_float2(-qz.x, -qz.y)), wb.fz[k]);
            }
        }
    }
}

// Evaluates the list down to its last 0 .. 7 entries, which move to the front;
// all: those too (padded with massless far bodies).
template <bool ZERO_SOFT, bool QUAD, int K>
__device__ __forceinline__ int list_flush(WalkList &l, WalkQuads *quads, int count, bool all,
                                          float2 e2, WalkBodies<K> &wb)
{
    const int lane = threadIdx.x & 31;
    const int full = all ? (count + 7) & ~7 : count & ~7, rest = all ? 0 : count - full;
    if (all && count + lane < full) {
        list_put(l, count + lane, 1.0e18f, 1.0e18f, 1.0e18f, 0.f);
        if (QUAD)
            for (int c = 0; c < 6; ++c)
                reinterpret_cast<float *>(&quads->q[(count + lane) >> 1][c >> 1])
                    [2 * (c & 1) + ((count + lane) & 1)] = 0.f;
    }
    __syncwarp();
    list_eval<ZERO_SOFT, QUAD, K>(l, quads, full / 2, e2, wb);
    __syncwarp();
    if (full > 0 && lane < (rest + 1) / 2) {  // full is even: whole pairs move
        l.a[lane] = l.a[full / 2 + lane];
        l.b[lane] = l.b[full / 2 + lane];
        if (QUAD)
            for (int c = 0; c < 3; ++c) quads->q[lane][c] = quads->q[full / 2 + lane][c];
    }
    __syncwarp();
    return rest;
}

// The boxes of the CTA's 32-body chunks.
template <int K>
struct WalkBoxes {
    float mn[K][3], mx[K][3];
};
// Bounds of the squared distance from a point to the nearest body: the distance
// to the nearest box, and that to the farthest point of the nearest face of a
// box (on each face of a box lies one of its bodies).  The first box starts them.
__device__ __forceinline__ void box_distances(const float (&mn)[3], const float (&mx)[3],
                                              const float (&c)[3], bool starts, float &least,
                                              float &most)
{
    float out[3], face[3], far[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float lo = mn[d] - c[d], hi = c[d] - mx[d];
        out[d] = fmaxf(0.f, fmaxf(lo, hi));
        face[d] = fminf(fabsf(lo), fabsf(hi));
        far[d] = fmaxf(fabsf(lo), fabsf(hi));
    }
    const float near2 = fmaf(out[2], out[2], fmaf(out[1], out[1], out[0] * out[0]));
    const float xy = fmaf(far[1], far[1], far[0] * far[0]);
    const float fx = fmaf(far[2], far[2], fmaf(far[1], far[1], face[0] * face[0]));
    const float fy = fmaf(far[2], far[2], fmaf(face[1], face[1], far[0] * far[0]));
    const float fz = fmaf(face[2], face[2], xy);
    const float face2 = fminf(fx, fminf(fy, fz));
    least = starts ? near2 : fminf(least, near2);
    most = starts ? face2 : fminf(most, face2);
}
// toward_body for a box's bodies: whether some body may lie on the node's side of
// its parent's centre (some), and whether all of them do (all); or-ed.
__device__ __forceinline__ void toward_box(const float (&mn)[3], const float (&mx)[3], float4 pc,
                                           bool &some, bool &all)
{
    const int oct = __float_as_int(pc.w);
    const float p[3] = {pc.x, pc.y, pc.z};
    bool may = oct < 8, must = oct < 8;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const bool high = (oct >> d & 1) != 0;
        may = may && (high ? mx[d] >= p[d] : mn[d] < p[d]);
        must = must && (high ? mn[d] >= p[d] : mx[d] < p[d]);
    }
    some = some || may;
    all = all || must;
}

// Chunk k's box.
template <int K>
__device__ __forceinline__ void load_box(const float (&p)[3], int k, WalkBoxes<K> &box)
{
    float mn[3] = {p[0], p[1], p[2]}, mx[3] = {p[0], p[1], p[2]};
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            mn[d] = fminf(mn[d], __shfl_xor_sync(0xffffffffu, mn[d], o));
            mx[d] = fmaxf(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], o));
        }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        box.mn[k][d] = mn[d];
        box.mx[k][d] = mx[d];
    }
}

// Whether some body of the CTA opens the lane's node (have: it holds one); the
// whole warp calls it.
template <int K, bool DIR>
__device__ __forceinline__ bool opened_nodes(const BHGNode &nd, bool have, float4 pc,
                                             const WalkBoxes<K> &box, const float (&p)[K][3],
                                             float theta2, int w0, int wend, float4 *test,
                                             float4 *side)
{
    const int lane = threadIdx.x & 31;
    const float c[3] = {nd.com_mass.x, nd.com_mass.y, nd.com_mass.z};
    float least = 0.f, most = 0.f;
    bool some = false, all = false;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        box_distances(box.mn[k], box.mx[k], c, k == 0, least, most);
        if (DIR) toward_box(box.mn[k], box.mx[k], pc, some, all);
    }
    // a node that holds one of the CTA's bodies is opened (each body's own cell)
    bool open = nd.first < wend && nd.first + nd.count > w0;
    open = open || nd.size2 >= theta2 * most || all;
    const bool by_distance = !(nd.size2 < theta2 * least), by_side = DIR && some;
    unsigned left = __ballot_sync(0xffffffffu, have && !open && (by_distance || by_side));
    if (!left) return open;
    // where the boxes do not decide, every body, two nodes at a time: the distance first,
    left = __ballot_sync(0xffffffffu, have && !open && by_distance);
    test[lane] = make_float4(c[0], c[1], c[2], nd.size2);
    if (DIR) side[lane] = pc;
    __syncwarp();
    while (left) {
        const int q0 = __ffs(left) - 1;
        left &= left - 1u;
        const int q1 = left ? __ffs(left) - 1 : q0;
        left &= left - 1u;
        const float4 t0 = test[q0], t1 = test[q1];
        bool any0 = false, any1 = false;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const float dx0 = t0.x - p[k][0], dx1 = t1.x - p[k][0];
            const float dy0 = t0.y - p[k][1], dy1 = t1.y - p[k][1];
            const float dz0 = t0.z - p[k][2], dz1 = t1.z - p[k][2];
            any0 |= t0.w >= theta2 * fmaf(dz0, dz0, fmaf(dy0, dy0, dx0 * dx0));
            any1 |= t1.w >= theta2 * fmaf(dz1, dz1, fmaf(dy1, dy1, dx1 * dx1));
        }
        any0 = __any_sync(0xffffffffu, any0);
        any1 = __any_sync(0xffffffffu, any1);
        if (lane == q0) open = any0;
        if (lane == q1) open = any1;
    }
    if (DIR) {  // then the side
        left = __ballot_sync(0xffffffffu, have && !open && by_side);
        while (left) {
            const int q0 = __ffs(left) - 1;
            left &= left - 1u;
            const int q1 = left ? __ffs(left) - 1 : q0;
            left &= left - 1u;
            const float4 c0 = side[q0], c1 = side[q1];
            bool any0 = false, any1 = false;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                any0 |= toward_body(c0, p[k][0], p[k][1], p[k][2]);
                any1 |= toward_body(c1, p[k][0], p[k][1], p[k][2]);
            }
            any0 = __any_sync(0xffffffffu, any0);
            any1 = __any_sync(0xffffffffu, any1);
            if (lane == q0) open = any0;
            if (lane == q1) open = any1;
        }
    }
    __syncwarp();
    return open;
}

template <bool ZERO_SOFT, bool QUAD, int NP, bool DIR>
__global__ void __maxnreg__(QUAD || NP > 1 ? 128 : DIR ? 64 : 80)
group_walk_kernel(const BHGNode *__restrict__ gnodes, const unsigned char *__restrict__ gnk,
                  const int *__restrict__ total, const float4 *__restrict__ body,
                  const uint32_t *__restrict__ order, int n, float theta2, float eps2, double G,
                  double *__restrict__ ax, double *__restrict__ ay, double *__restrict__ az,
                  BHStats *__restrict__ stats, const float4 *__restrict__ gquad,
                  const float4 *__restrict__ gpcen, const AfterForce after)
{
    extern __shared__ __align__(16) unsigned char walk_shared[];
    using Shared = WalkShared<QUAD>;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, W = blockDim.x >> 5;
    constexpr int K = 2 * NP;
    __shared__ int s_push[kWalkWarps];  // groups pushed in this round
    Shared &sh = reinterpret_cast<Shared *>(walk_shared)[w];
    int *s_first = reinterpret_cast<int *>(reinterpret_cast<Shared *>(walk_shared) + W);
    unsigned char *s_kids = reinterpret_cast<unsigned char *>(s_first + W * kWalkStack);
    [[maybe_unused]] const int num_nodes = *total;  // bounds checked builds only
    const int w0 = blockIdx.x * 32 * K;
    const int wend = min(n, w0 + 32 * K);  // the CTA's bodies: [w0, wend)
    const float2 e2 = dup2(eps2);

    WalkBodies<K> wb;
    WalkBoxes<K> box;
    float p[K][3];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        // a slot past n walks with body w0: its tests repeat that body's
        const int i = w0 + 32 * k + lane;
        const float4 q = body[i < n ? i : w0];
        p[k][0] = q.x; p[k][1] = q.y; p[k][2] = q.z;
        wb.nx[k] = dup2(-q.x); wb.ny[k] = dup2(-q.y); wb.nz[k] = dup2(-q.z);
        wb.fx[k] = wb.fy[k] = wb.fz[k] = dup2(0.f);
        load_box(p[k], k, box);
    }

    unsigned m2p = 0, p2p = 0;
    int count = 0, bcount = 0;  // list entries (bcount: the body list, QUAD only)
    int sp = 1;
    if (threadIdx.x == 0) {
        s_first[0] = 0;
        s_kids[0] = 1;
    }
    while (sp > 0) {
        __syncthreads();
        if (W > 1 && w >= sp) {  // a narrow round: no group for this warp
            if (lane == 0) s_push[w] = 0;
            __syncthreads();
            sp = 0;
            for (int v = 0; v < W; ++v) sp += s_push[v];
            continue;
        }
        // one node per lane: child lane & 7 of the warp's group lane >> 3
        const int e = sp - 1 - (w + W * (lane >> 3));
        const int kids = e >= 0 ? s_kids[e] : 0;
        const bool have = (lane & 7) < kids;
        const int id = have ? s_first[e] + (lane & 7) : 0;
        sp = max(0, sp - 4 * W);
        const BHGNode nd = gnodes[NB_IN_RANGE(id, num_nodes) ? id : 0];
        const float4 pc = DIR ? gpcen[id] : make_float4(0.f, 0.f, 0.f, 0.f);
        const bool open = opened_nodes<K, DIR>(nd, have, pc, box, p, theta2, w0, wend, sh.test,
                                               sh.side);

        // push the groups of the opened internal nodes
        const bool inner = have && open && nd.kids >= 0;
        const unsigned push = __ballot_sync(0xffffffffu, inner);
        const unsigned below = (1u << lane) - 1u;
        int top = sp;
        if (W > 1) {
            if (lane == 0) s_push[w] = __popc(push);
            __syncthreads();  // every warp has read its groups, too
            for (int v = 0; v < W; ++v) {
                if (v < w) top += s_push[v];
                sp += s_push[v];
            }
        } else {
            __syncwarp();
            sp += __popc(push);
        }
        if (inner) {
            const int to = top + __popc(push & below);
            if (NB_IN_RANGE(to, W * kWalkStack)) {
                s_first[to] = nd.kids;
                s_kids[to] = gnk[id];
            }
        }

        // closed nodes to the list
        const bool add = have && !open;
        const unsigned adds = __ballot_sync(0xffffffffu, add);
        if (add) {
            const int to = count + __popc(adds & below);
            list_put(sh.list, to, nd.com_mass.x, nd.com_mass.y, nd.com_mass.z, nd.com_mass.w);
            if constexpr (QUAD) {
                const float4 q0 = gquad[2 * id], q1 = gquad[2 * id + 1];
                const float v[6] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y};
#pragma unroll
                for (int d = 0; d < 6; ++d)
                    reinterpret_cast<float *>(&sh.quads.q[to >> 1][d >> 1])
                        [2 * (d & 1) + (to & 1)] = v[d];
            }
        }
        count += __popc(adds);
        m2p += __popc(adds);
        if constexpr (QUAD) {
            if (count >= kListFlush)
                count = list_flush<ZERO_SOFT, true, K>(sh.list, &sh.quads, count, false, e2, wb);
        } else if (count >= kListFlush) {
            count = list_flush<ZERO_SOFT, false, K>(sh.list, nullptr, count, false, e2, wb);
        }

        // the bodies of opened leaves: entry t of the batch's leaf bodies lies in
        // the leaf whose range of the running count holds t
        const int lc = have && open && nd.kids < 0 ? nd.count : 0;
        if (!__any_sync(0xffffffffu, lc > 0)) continue;
        int lincl = lc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, lincl, o);
            if (lane >= o) lincl += t;
        }
        const int leaf_bodies = __shfl_sync(0xffffffffu, lincl, 31);
        p2p += leaf_bodies;
        for (int t0 = 0; t0 < leaf_bodies; t0 += 32) {
            const int t = t0 + lane;
            int leaf = 0;  // the number of lanes whose running count is at most t
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const int v = __shfl_sync(0xffffffffu, lincl, leaf + o - 1);
                if (v <= t) leaf += o;
            }
            const int b0 = __shfl_sync(0xffffffffu, nd.first + lc - lincl, leaf & 31);
            const bool put = t < leaf_bodies;
            WalkList *list = &sh.list;
            int at = count;
            if constexpr (QUAD) {
                list = &sh.bodies;
                at = bcount;
            }
            if (put && NB_IN_RANGE(b0 + t, n)) {
                const float4 q = body[b0 + t];
                list_put(*list, at + lane, q.x, q.y, q.z, q.w);
            }
            const int got = min(32, leaf_bodies - t0);
            if constexpr (QUAD) {
                bcount += got;
                if (bcount >= kListFlush)
                    bcount = list_flush<ZERO_SOFT, false, K>(sh.bodies, nullptr, bcount, false, e2,
                                                          wb);
            } else {
                count += got;
                if (count >= kListFlush)
                    count = list_flush<ZERO_SOFT, false, K>(sh.list, nullptr, count, false, e2, wb);
            }
        }
        __syncwarp();
    }
    if constexpr (QUAD) {
        list_flush<ZERO_SOFT, true, K>(sh.list, &sh.quads, count, true, e2, wb);
        list_flush<ZERO_SOFT, false, K>(sh.bodies, nullptr, bcount, true, e2, wb);
    } else {
        list_flush<ZERO_SOFT, false, K>(sh.list, nullptr, count, true, e2, wb);
    }

    if (lane == 0) {
        const unsigned long long nv = wend - w0;
        atomicAdd(&stats->m2p, m2p * nv);
        atomicAdd(&stats->p2p, p2p * nv);
        atomicAdd(&stats->total, (m2p + p2p) * nv);
    }
    double f[K][3];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        f[k][0] = (double)wb.fx[k].x + (double)wb.fx[k].y;
        f[k][1] = (double)wb.fy[k].x + (double)wb.fy[k].y;
        f[k][2] = (double)wb.fz[k].x + (double)wb.fz[k].y;
    }
    if (W > 1) {
        __syncthreads();  // every warp is done with its lists
        double *part = reinterpret_cast<double *>(walk_shared);  // [W][3 K][32]
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
            for (int d = 0; d < 3; ++d) part[(w * 3 * K + 3 * k + d) * 32 + lane] = f[k][d];
        __syncthreads();
        if (w > 0) return;
        for (int v = 1; v < W; ++v)
#pragma unroll
            for (int k = 0; k < K; ++k)
#pragma unroll
                for (int d = 0; d < 3; ++d) f[k][d] += part[(v * 3 * K + 3 * k + d) * 32 + lane];
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int i = w0 + 32 * k + lane;
        if (i >= n) continue;
        const uint32_t o = order[i];
        double *out[3] = {ax, ay, az};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double a = G * f[k][d];
            out[d][o] = a;
            after_force(after, d, (int)o, a);
        }
    }
}

// ------------------------------------------------------------ serial walk
// One warp walks for 64 consecutive sorted bodies, two per lane (a packed pair):
// one round trip to memory brings a group's records into shared memory, and the
// warp tests the children one after the other, adding the monopoles of the children
// that no body opens and opened leaves' bodies in that order, and pushing the groups of
// opened internal children onto its stack.  The interactions are those of
// walk2_kernel; only their order differs.
// Bound by dispatch when the walks fill the chip (it spends least on a walk: no list, no
// sort), by each walk's chain of trips to memory when they do not.  The ordered walk
// below adds the same terms in the same order, so the two give the same bits and any
// walk may go by either.
//
// A depth-first walk over groups keeps, per level of its current path, at most
// 7 groups of unvisited siblings, plus the at most 8 groups the last group
// pushed; groups lie at levels 0 .. kMaxLevels.
constexpr int kSerialStack = 8 * (kMaxLevels + 1);

template <bool ZERO_SOFT, bool QUAD, bool DIR>
__global__ void __launch_bounds__(32)
serial_walk_kernel(const BHGNode *__restrict__ gnodes, const unsigned char *__restrict__ gnk,
                   const int *__restrict__ total, const float4 *__restrict__ body,
                   const uint32_t *__restrict__ order, int n, float theta2, float eps2, double G,
                   double *__restrict__ ax, double *__restrict__ ay, double *__restrict__ az,
                   BHStats *__restrict__ stats, const float4 *__restrict__ gquad,
                   const float4 *__restrict__ gpcen, const int2 *__restrict__ logged,
                   const AfterForce after)
{
    // logged: the walks with a log (its count not negative) are done already
    if (logged && logged[blockIdx.x].y >= 0) return;
    __shared__ BHGNode s_rec[8];
    __shared__ float4 s_quad[QUAD ? 16 : 1];
    __shared__ float4 s_pc[DIR ? 8 : 1];
    __shared__ int2 s_stack[kSerialStack];
    [[maybe_unused]] const int num_nodes = *total;  // bounds checked builds only
    const int lane = threadIdx.x;
    const int w0 = blockIdx.x * 64, wend = min(n, w0 + 64);  // the warp's bodies: [w0, wend)
    const int ia = w0 + lane, ib = ia + 32;
    // a slot past n walks with body w0: its tests repeat that body's
    const float4 pa = body[ia < n ? ia : w0], pb = body[ib < n ? ib : w0];
    const float2 npx = make_float2(-pa.x, -pb.x), npy = make_float2(-pa.y, -pb.y),
                 npz = make_float2(-pa.z, -pb.z);
    float2 fx = dup2(0.f), fy = dup2(0.f), fz = dup2(0.f);
    const float2 e2 = dup2(eps2), t2 = dup2(theta2);
    unsigned m2p = 0, p2p = 0;
    int sp = 1;
    if (lane == 0) s_stack[0] = make_int2(0, 1);
    while (sp > 0) {
        __syncwarp();
        const int2 g = s_stack[--sp];
        if (!NB_IN_RANGE(g.x + g.y - 1, num_nodes)) break;
        int mynk = 0;
        if (lane < g.y) {
            s_rec[lane] = gnodes[g.x + lane];
            mynk = gnk[g.x + lane];
            if (DIR) s_pc[lane] = gpcen[g.x + lane];
        }
        if (QUAD && lane < 2 * g.y) s_quad[lane] = gquad[2 * g.x + lane];
        __syncwarp();
        for (int c = 0; c < g.y; ++c) {
            const BHGNode nd = s_rec[c];
            const float2 dx = add2(dup2(nd.com_mass.x), npx), dy = add2(dup2(nd.com_mass.y), npy),
                         dz = add2(dup2(nd.com_mass.z), npz);
            const float2 d2 = fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));
            const float2 td2 = mul2(t2, d2);
            // a node that holds one of the warp's bodies is opened (each body's
            // own cell); the others by the opening test of any body
            bool open = nd.first < wend && nd.first + nd.count > w0;
            open = open | (nd.size2 >= td2.x) | (nd.size2 >= td2.y);
            if (DIR) {
                const float4 pc = s_pc[c];
                open = open | toward_body(pc, -npx.x, -npy.x, -npz.x) |
                       toward_body(pc, -npx.y, -npy.y, -npz.y);
            }
            if (__any_sync(0xffffffffu, open)) {
                if (nd.kids >= 0) {  // internal: its children's group, later
                    const int nk = __shfl_sync(0xffffffffu, mynk, c);
                    if (NB_IN_RANGE(sp, kSerialStack)) {
                        if (lane == 0) s_stack[sp] = make_int2(nd.kids, nk);
                        ++sp;
                    }
                    continue;
                }
                const int e = NB_IN_RANGE(nd.first, n) && NB_IN_RANGE(nd.first + nd.count - 1, n)
                                  ? nd.first + nd.count
                                  : nd.first;
#pragma unroll 2
                for (int b = nd.first; b < e; ++b) {
                    const float4 q = body[b];
                    const float2 rx = add2(dup2(q.x), npx), ry = add2(dup2(q.y), npy),
                                 rz = add2(dup2(q.z), npz);
                    const float2 r2 = fma2(rz, rz, fma2(ry, ry, fma2(rx, rx, e2)));
                    float2 inv = make_float2(rsqrt_mufu(r2.x), rsqrt_mufu(r2.y));
                    if (ZERO_SOFT) {
                        inv.x = r2.x > 0.f ? inv.x : 0.f;
                        inv.y = r2.y > 0.f ? inv.y : 0.f;
                    }
                    const float2 s = mul2(mul2(dup2(q.w), inv), mul2(inv, inv));
                    fx = fma2(rx, s, fx);
                    fy = fma2(ry, s, fy);
                    fz = fma2(rz, s, fz);
                }
                p2p += nd.count;
            } else {
                const float2 r2 = add2(d2, e2);
                const float2 inv = make_float2(rsqrt_mufu(r2.x), rsqrt_mufu(r2.y));
                const float2 inv2 = mul2(inv, inv);
                const float2 s = mul2(mul2(dup2(nd.com_mass.w), inv), inv2);
                fx = fma2(dx, s, fx);
                fy = fma2(dy, s, fy);
                fz = fma2(dz, s, fz);
                if (QUAD) {
                    const float4 q0 = s_quad[2 * c], q1 = s_quad[2 * c + 1];
                    const float2 qx =
                        fma2(dup2(q0.x), dx, fma2(dup2(q0.w), dy, mul2(dup2(q1.x), dz)));
                    const float2 qy =
                        fma2(dup2(q0.w), dx, fma2(dup2(q0.y), dy, mul2(dup2(q1.y), dz)));
                    const float2 qz =
                        fma2(dup2(q1.x), dx, fma2(dup2(q1.y), dy, mul2(dup2(q0.z), dz)));
                    const float2 rqr = fma2(dx, qx, fma2(dy, qy, mul2(dz, qz)));
                    const float2 inv5 = mul2(mul2(inv, inv2), inv2);
                    const float2 f = mul2(mul2(dup2(2.5f), rqr), inv2);
                    fx = fma2(inv5, fma2(f, dx, make_float2(-qx.x, -qx.y)), fx);
                    fy = fma2(inv5, fma2(f, dy, make_float2(-qy.x, -qy.y)), fy);
                    fz = fma2(inv5, fma2(f, dz, make_float2(-qz.x, -qz.y)), fz);
                }
                ++m2p;
            }
        }
    }
    double *const out[3] = {ax, ay, az};
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int i = w0 + 32 * k + lane;
        if (i >= n) continue;
        const uint32_t o = order[i];
        const float f[3] = {k ? fx.y : fx.x, k ? fy.y : fy.x, k ? fz.y : fz.x};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double a = G * (double)f[d];
            out[d][o] = a;
            after_force(after, d, (int)o, a);
        }
    }
    if (lane == 0) {
        const unsigned long long nv = wend - w0;
        atomicAdd(&stats->m2p, m2p * nv);
        atomicAdd(&stats->p2p, p2p * nv);
        atomicAdd(&stats->total, (m2p + p2p) * nv);
    }
}

// ---------------------------------------------------------- ordered walk
// An FP32 sum of thousands of terms depends on their order in the fifth digit (walks
// under the reference's opening rule have up to 20,000 at n = 100,000, theta 0.5,
// disk galaxy), and a trajectory with it.  This walk adds each body's terms one after
// the other in the order of the serial walk, in two kernels:
//   - decide_kernel finds the groups that the walk visits and which of their records
//     are opened, in any order, by many warps (as group_walk_kernel), and sorts
//     the groups by their place in the serial walk of the whole tree: the rank
//     of the group's parent v in a preorder with children reversed, which is
//     depth(v) - skip(v) but for a constant;
//   - log_eval_kernel goes through a walk's groups in that order: four warps list the
//     terms in shared memory, two add them up, a body per lane.
// The stack is kept in the serial walk's order, so whatever sorts before its top is
// complete: a CTA that has no room for more groups moves those to the pool and goes on
// (a walk under the reference's rule visits up to 4,900 at n = 400,000, theta 0.5, and
// 18,000 with one body per leaf).  A walk that the pool has no room for (which ones
// depends on scheduling), or whose stack is full, is left to serial_walk_kernel, which
// gives the same bits but takes 9 ms for that one.
//
// A force evaluation by serial_walk_kernel / this walk, disk galaxy, in us:
//                        theta 0.5        0.3             0.5, reference's rule
//   n =  16,384        564 /  272     892 /  315        1817 /  426
//   n = 100,000       1001 /  503    1921 /  782        3910 / 1048
//   n = 400,000       1342 / 1227    3091 / 2410       11208 / 3598
// Up to kOrderedBodies, and always under the reference's rule, results are the serial
// walk's bit for bit.  That has its price: by group_walk_kernel, in another order, an
// evaluation takes about 0.8 times as long at every size (serial / ordered / group, disk,
// theta 0.5):
//   n =   200,000     936 /  722 /  602      with quadrupoles  1305 / 1140 /  991
//   n =   400,000    1350 / 1227 /  993                        1917 / 2035 / 1697
//   n =   524,288    1591 / 1570 / 1263                        2379 / 2657 / 2084
//   n =   800,000    2087 / 2253 / 1689                        3236 / 3866 / 2923
//   n = 1,048,576    2900 / 3083 / 2296                        4518 / 5424 / 4100
// Summed in another order, velocities after a few steps of 1e-3 moved by up to 9e-8 of
// their scale for trees of 16,000 to 200,000 bodies.  The line lies where the ordered walk
// is no faster than the serial one; beyond, walks are of similar length and the order shows
// at 1e-8.
constexpr int kOrderedBodies = 524288;
// Up to this many walks 16 warps decide one, above it 4 (16 / 4 warps at 256, 512 and
// 1024 walks: 314 / 332, 320 / 318, 406 / 380 us).  Under the reference's rule always 16,
// with room for 4096 groups: its longest walks, not the number of walks, take the time.
constexpr int kFewWalks = 400;
constexpr int kLogSegments = 16;  // times a walk's groups may move to the pool
// Beyond this many pool entries per body the serial walk is taken (log_per_body).
constexpr double kMostLogPerBody = 64.0;
constexpr int kLogChunk = 256;    // terms per list
constexpr int kLogListers = 128;  // threads of log_eval_kernel that list terms

template <bool DIR, int WARPS, int GROUPS>
struct LogShared {
    static_assert(GROUPS <= 4096, "a slot has 12 bits");
    static_assert(GROUPS % (32 * WARPS) == 0 && (GROUPS & (GROUPS - 1)) == 0, "log_flush");
    static constexpr int kStack = 3 * GROUPS / 4;
    unsigned long long sorted[GROUPS];  // key, slot (12 bits), records (4), opened ones (8)
    int first[GROUPS];                  // by slot: the group's first record
    static constexpr int kKeep = GROUPS / (32 * WARPS);
    float4 test[WARPS][32], side[DIR ? WARPS : 1][32];
    int s_first[kStack];  // the stack: as group_walk_kernel's, and the groups' keys
    unsigned s_key[kStack];
    unsigned char s_kids[kStack];
};

// Sorts the CTA's groups and moves the complete ones, those before `key` in the serial
// order (all: every one), to the pool, as segment `seg` of the walk; the rest take the
// first slots.  Returns how many stay, or -1 where there is no room.
template <class Shared>
__device__ __forceinline__ int log_flush(Shared &sh, int groups, bool all, unsigned key, int seg,
                                         int2 *__restrict__ segs, uint2 *__restrict__ pool,
                                         int pool_size, unsigned long long *__restrict__ pool_next,
                                         int before, int *s_at)
{
    __syncthreads();
    // bitonic sort, padded to a power of two
    int size = 1;
    while (size < groups) size <<= 1;
    for (int k = groups + (int)threadIdx.x; k < size; k += blockDim.x) sh.sorted[k] = ~0ull;
    for (int k = 2; k <= size; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            __syncthreads();
            for (int t = threadIdx.x; t < size / 2; t += blockDim.x) {
                const int lo = ((t & ~(j - 1)) << 1) | (t & (j - 1)), hi = lo | j;
                const unsigned long long a = sh.sorted[lo], b = sh.sorted[hi];
                if ((a > b) == ((lo & k) == 0)) {
                    sh.sorted[lo] = b;
                    sh.sorted[hi] = a;
                }
            }
        }
    __syncthreads();
    int done = groups;
    if (!all) {  // the number of groups before key
        int lo = -1;
        while (done - lo > 1) {
            const int mid = (lo + done) / 2;
            if ((unsigned)(sh.sorted[mid] >> 24) < key) lo = mid;
            else done = mid;
        }
    }
    if (threadIdx.x == 0) {
        const unsigned long long at = atomicAdd(pool_next, (unsigned long long)done);
        const bool room = seg < kLogSegments &&
                          at + done <= (unsigned long long)pool_size;
        *s_at = room ? (int)at : -1;
        if (room) segs[seg] = make_int2((int)at, before + done);
    }
    __syncthreads();
    const int at = *s_at;
    if (at < 0) return -1;
    for (int k = threadIdx.x; k < done; k += blockDim.x) {
        const unsigned low = (unsigned)sh.sorted[k];
        pool[at + k] = make_uint2((unsigned)sh.first[(low >> 12) & 0xFFFu], low & 0xFFFu);
    }
    if (all) return 0;
    unsigned long long kept[Shared::kKeep];
    int first[Shared::kKeep];
#pragma unroll
    for (int u = 0; u < Shared::kKeep; ++u) {
        const int k = done + (int)threadIdx.x + u * (int)blockDim.x;
        kept[u] = k < groups ? sh.sorted[k] : 0ull;
        first[u] = k < groups ? sh.first[(unsigned)(kept[u] >> 12) & 0xFFFu] : 0;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < Shared::kKeep; ++u) {
        const int to = (int)threadIdx.x + u * (int)blockDim.x;
        if (done + to < groups) {
            sh.sorted[to] = (kept[u] & ~0xFFF000ull) | (unsigned)to << 12;
            sh.first[to] = first[u];
        }
    }
    __syncthreads();
    return groups - done;
}

// Bound by dispatch; under the reference's rule, with 0.35 ms at n = 100,000 (theta
// 0.5, disk galaxy), by that of the longest walk (1,939 groups in 35 rounds of up to 64, of 10,000 cycles each with
// every node undecided by the boxes).  Tighter boxes (8 bodies each) and a pass over
// the bodies per batch instead of one per node pair cost as much as they saved;
// 8 warps took 0.12 ms longer, 4 warps for short walks with a second launch for the
// rest 0.15.
template <bool DIR, int WARPS, int GROUPS>
__global__ void __launch_bounds__(32 * WARPS, 32 / WARPS)
decide_kernel(const BHGNode *__restrict__ gnodes, const unsigned char *__restrict__ gnk,
              const unsigned *__restrict__ gkey, const float4 *__restrict__ gpcen,
              const int *__restrict__ total, const float4 *__restrict__ body, int n, float theta2,
              BHStats *__restrict__ stats, int2 *__restrict__ walks, int2 *__restrict__ segs,
              uint2 *__restrict__ pool, int pool_size,
              unsigned long long *__restrict__ pool_next)
{
    constexpr int W = WARPS;
    extern __shared__ __align__(16) unsigned char walk_shared[];
    __shared__ int s_push[W];
    __shared__ unsigned s_m2p, s_p2p;
    __shared__ int s_at;
    using Shared = LogShared<DIR, WARPS, GROUPS>;
    Shared &sh = *reinterpret_cast<Shared *>(walk_shared);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    [[maybe_unused]] const int num_nodes = *total;  // bounds checked builds only
    const int w0 = blockIdx.x * 64, wend = min(n, w0 + 64);
    WalkBoxes<2> box;
    float p[2][3];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        // a slot past n walks with body w0: its tests repeat that body's
        const int i = w0 + 32 * k + lane;
        const float4 q = body[i < n ? i : w0];
        p[k][0] = q.x; p[k][1] = q.y; p[k][2] = q.z;
        load_box(p[k], k, box);
    }
    if (threadIdx.x == 0) {
        sh.s_first[0] = 0;  // the root's group comes first: key 0
        sh.s_kids[0] = 1;
        sh.s_key[0] = 0;
        s_m2p = s_p2p = 0;
    }
    segs += (size_t)blockIdx.x * kLogSegments;
    unsigned m2p = 0, p2p = 0;  // per lane
    int sp = 1, groups = 0, moved = 0, seg = 0;  // moved: groups in the pool
    bool fits = true;
    while (sp > 0) {
        __syncthreads();
        const int take = min(sp, 4 * W);
        if (groups + take > GROUPS) {
            const int stay = log_flush(sh, groups, false, sh.s_key[sp - 1], seg++, segs, pool,
                                       pool_size, pool_next, moved, &s_at);
            moved += groups - stay;
            groups = stay;
            fits = stay >= 0 && stay + take <= GROUPS;
            if (!fits) break;
        }
        // the first groups to the first warps: in a narrow round the others have none
        const int j = 4 * w + (lane >> 3), e = sp - 1 - j;
        const bool busy = 4 * w < take;
        sp -= take;
        bool inner = false;
        unsigned push = 0;
        int id = 0;
        BHGNode nd;
        if (busy) {
            const int kids = e >= 0 ? sh.s_kids[e] : 0;
            const bool have = (lane & 7) < kids;
            id = have ? sh.s_first[e] + (lane & 7) : 0;
            const unsigned key = e >= 0 ? sh.s_key[e] : 0;
            nd = gnodes[NB_IN_RANGE(id, num_nodes) ? id : 0];
            const float4 pc = DIR ? gpcen[id] : make_float4(0.f, 0.f, 0.f, 0.f);
            const bool open = opened_nodes<2, DIR>(nd, have, pc, box, p, theta2, w0, wend,
                                                   sh.test[w], sh.side[DIR ? w : 0]);
            const unsigned opened = __ballot_sync(0xffffffffu, have && open);
            if (have) {
                if (!open) ++m2p;
                else if (nd.kids < 0) p2p += nd.count;
            }
            if (kids > 0 && (lane & 7) == 0) {
                const int slot = groups + j;
                sh.first[slot] = id;
                sh.sorted[slot] = (unsigned long long)key << 24 | (unsigned)slot << 12 |
                                  (unsigned)kids << 8 | ((opened >> lane) & 0xFFu);
            }
            inner = have && open && nd.kids >= 0;
            push = __ballot_sync(0xffffffffu, inner);
        }
        groups += take;
        if (lane == 0) s_push[w] = __popc(push);
        __syncthreads();  // every warp has read its groups, too
        // in the serial order: the first group's children on top, the last child first
        int top = sp;
        for (int v = 0; v < W; ++v) {
            if (v > w) top += s_push[v];
            sp += s_push[v];
        }
        fits = sp <= Shared::kStack;
        if (!fits) break;
        if (inner) {
            const unsigned mine = 0xFFu << (lane & 24), later = ~(mine | (mine - 1u));
            const int to = top + __popc(push & (later | (mine & ((1u << lane) - 1u))));
            sh.s_first[to] = nd.kids;
            sh.s_kids[to] = gnk[id];
            sh.s_key[to] = gkey[id];
        }
    }
    if (fits)
        fits = log_flush(sh, groups, true, 0u, seg++, segs, pool, pool_size, pool_next, moved,
                         &s_at) == 0;
    if (threadIdx.x == 0) walks[blockIdx.x] = make_int2(seg, fits ? moved + groups : -1);
    if (!fits) return;
    m2p = __reduce_add_sync(0xffffffffu, m2p);
    p2p = __reduce_add_sync(0xffffffffu, p2p);
    if (lane == 0) {
        atomicAdd(&s_m2p, m2p);
        atomicAdd(&s_p2p, p2p);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned long long nv = wend - w0;
        atomicAdd(&stats->m2p, s_m2p * nv);
        atomicAdd(&stats->p2p, s_p2p * nv);
        atomicAdd(&stats->total, (s_m2p + s_p2p) * nv);
    }
}

__device__ __forceinline__ void list_barrier()
{
    asm volatile("bar.sync 1, %0;" ::"n"(kLogListers) : "memory");
}

// Bound by dispatch: a term costs a warp 19 cycles (13 FP32 instructions, the
// reciprocal root, two loads from shared memory), 0.2 ms in all at n = 100,000; with
// the longest walk, whose terms are a chain, 0.46 ms.  A batch's records are loaded a
// batch ahead (0.57 without), and a list is filled while the other is added up.
template <bool ZERO_SOFT, bool QUAD>
__global__ void __launch_bounds__(64 + kLogListers)
log_eval_kernel(const BHGNode *__restrict__ gnodes, const float4 *__restrict__ gquad,
                const float4 *__restrict__ body,
                const uint32_t *__restrict__ order, int n, float eps2, double G,
                double *__restrict__ ax, double *__restrict__ ay, double *__restrict__ az,
                const int2 *__restrict__ walks, const int2 *__restrict__ segs,
                const uint2 *__restrict__ pool, const AfterForce after)
{
    __shared__ float4 s_term[2][kLogChunk];  // position, mass
    __shared__ float2 s_soft[2][kLogChunk];  // eps^2, added before a body's r^2, after a node's
    __shared__ float4 s_quad[2][QUAD ? kLogChunk : 1][2];
    __shared__ unsigned char s_node[2][QUAD ? kLogChunk : 1];  // whether the term is a node's
    __shared__ int s_id[QUAD ? kLogListers : 1];
    __shared__ int s_count[2];
    // a batch of groups, a record per lister:
    __shared__ float4 s_com[kLogListers];  // its term as a node
    __shared__ int s_body[kLogListers];    // the first body of an opened leaf; -1: a node's term
    __shared__ int s_incl[kLogListers];    // running count of terms
    __shared__ int s_warp[kLogListers / 32];
    const int2 walk = walks[blockIdx.x];  // segments, groups
    if (walk.y < 0) return;
    const int w0 = blockIdx.x * 64;
    if (threadIdx.x < 64) {
        const int i = w0 + threadIdx.x;
        const float4 q = body[i < n ? i : w0];
        const float nx = -q.x, ny = -q.y, nz = -q.z;
        float fx = 0.f, fy = 0.f, fz = 0.f;
        for (int b = 0;; b ^= 1) {
            __syncthreads();
            const int count = s_count[b];
            if (count == 0) break;
#pragma unroll 8
            for (int k = 0; k < count; ++k) {
                const float4 t = s_term[b][k];
                const float2 soft = s_soft[b][k];
                const float dx = t.x + nx, dy = t.y + ny, dz = t.z + nz;
                const float r2 =
                    fmaf(dz, dz, fmaf(dy, dy, fmaf(dx, dx, soft.x))) + soft.y;
                float inv = rsqrt_mufu(r2);
                if (ZERO_SOFT) inv = r2 > 0.f ? inv : 0.f;
                const float s = __fmul_rn(__fmul_rn(t.w, inv), __fmul_rn(inv, inv));
                fx = fmaf(dx, s, fx);
                fy = fmaf(dy, s, fy);
                fz = fmaf(dz, s, fz);
                if (QUAD && s_node[b][k]) {
                    const float4 q0 = s_quad[b][k][0], q1 = s_quad[b][k][1];
                    const float qx = fmaf(q0.x, dx, fmaf(q0.w, dy, __fmul_rn(q1.x, dz)));
                    const float qy = fmaf(q0.w, dx, fmaf(q0.y, dy, __fmul_rn(q1.y, dz)));
                    const float qz = fmaf(q1.x, dx, fmaf(q1.y, dy, __fmul_rn(q0.z, dz)));
                    const float rqr = fmaf(dx, qx, fmaf(dy, qy, __fmul_rn(dz, qz)));
                    const float inv2 = __fmul_rn(inv, inv);
                    const float inv5 = __fmul_rn(__fmul_rn(inv, inv2), inv2);
                    const float f = __fmul_rn(__fmul_rn(2.5f, rqr), inv2);
                    fx = fmaf(inv5, fmaf(f, dx, -qx), fx);
                    fy = fmaf(inv5, fmaf(f, dy, -qy), fy);
                    fz = fmaf(inv5, fmaf(f, dz, -qz), fz);
                }
            }
        }
        if (i < n) {
            const uint32_t o = order[i];
            double *out[3] = {ax, ay, az};
            const double f[3] = {(double)fx, (double)fy, (double)fz};
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double a = G * f[d];
                out[d][o] = a;
                after_force(after, d, (int)o, a);
            }
        }
        return;
    }
    // A lister's record of a batch, loaded a batch ahead, and the log entry of the
    // batch after it: neither trip to memory waits for the other.
    const int q = threadIdx.x - 64, lane = q & 31, wq = q >> 5;
    const int child = q & 7;
    // the segment of the lister's next group (they only go up): its place in the pool, the
    // group after its last, and its first
    const int2 *seg = segs + (size_t)blockIdx.x * kLogSegments, *const last = seg + walk.x - 1;
    int2 in_seg = *seg;
    int seg0 = 0;
    auto load_log = [&](int g) {
        while (g >= in_seg.y && seg < last) {
            seg0 = in_seg.y;
            in_seg = *++seg;
        }
        return g < walk.y ? pool[in_seg.x + g - seg0] : make_uint2(0u, 0u);
    };
    auto load_node = [&](uint2 log) {
        return gnodes[child < (int)(log.y >> 8) ? log.x + child : 0];
    };
    constexpr int kBatch = kLogListers / 8;
    int next = 0;  // the next batch's first group
    uint2 log = load_log(q >> 3), log_ahead = load_log(kBatch + (q >> 3));
    BHGNode node_ahead = load_node(log);
    int terms = 0, t0 = 0;  // of this batch: how many, how many listed
    for (int b = 0;; b ^= 1) {
        int filled = 0;
        while (filled < kLogChunk) {
            if (t0 == terms) {
                if (next >= walk.y) break;
                next += kBatch;
                const BHGNode nd = node_ahead;
                const bool have = child < (int)(log.y >> 8), open = (log.y >> child & 1u) != 0;
                const int id = (int)log.x + child;
                const int count = !have ? 0 : (!open ? 1 : (nd.kids < 0 ? nd.count : 0));
                log = log_ahead;
                node_ahead = load_node(log);
                log_ahead = load_log(next + kBatch + (q >> 3));
                int incl = count;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += t;
                }
                list_barrier();  // the last batch's terms are read
                if (lane == 31) s_warp[wq] = incl;
                s_com[q] = nd.com_mass;
                if (QUAD) s_id[q] = id;
                s_body[q] = open ? nd.first : -1;
                list_barrier();
#pragma unroll
                for (int v = 0; v < kLogListers / 32 - 1; ++v)
                    if (v < wq) incl += s_warp[v];
                s_incl[q] = incl;
                list_barrier();
                terms = s_incl[kLogListers - 1];
                t0 = 0;
                continue;
            }
            const int take = min(kLogChunk - filled, terms - t0);
            for (int k = q; k < take; k += kLogListers) {
                const int t = t0 + k;
                int node = 0;  // the number of running counts at most t
#pragma unroll
                for (int o = kLogListers / 2; o > 0; o >>= 1)
                    if (s_incl[node + o - 1] <= t) node += o;
                const int before = node > 0 ? s_incl[node - 1] : 0;
                const int first = s_body[node];
                float4 term;
                if (QUAD) s_node[b][filled + k] = first < 0;
                if (first < 0) {
                    term = s_com[node];
                    if (QUAD) {
                        const int id = s_id[node];
                        s_quad[b][filled + k][0] = gquad[2 * id];
                        s_quad[b][filled + k][1] = gquad[2 * id + 1];
                    }
                } else term = body[NB_IN_RANGE(first + t - before, n) ? first + t - before : 0];
                s_term[b][filled + k] = term;
                s_soft[b][filled + k] = first < 0 ? make_float2(0.f, eps2) : make_float2(eps2, 0.f);
            }
            filled += take;
            t0 += take;
        }
        if (q == 0) s_count[b] = filled;
        __syncthreads();
        if (filled == 0) return;
    }
}

// How a walk is computed.  The serial and the ordered walk give the same bits.
enum class Walk { kPreorder, kGroup, kSerial, kOrdered };

// Body pairs per lane of the walk (0: the one-body-per-lane preorder walk);
// NB_BH_WALK_PAIRS overrides the default.
int walk_pairs()
{
    static const int np = [] {
        const char *e = std::getenv("NB_BH_WALK_PAIRS");
        const int v = e ? std::atoi(e) : 1;
        return v < 0 ? 0 : (v > 2 ? 2 : v);
    }();
    return np;
}

// Pool entries per body that an ordered walk is given, above the mean of the groups that
// walks visit divided by their 64 bodies.  Means of Plummer spheres (disks have half),
// per body, at theta 0.5 / 0.4 / 0.3 / 0.2:
//   n =    16,384    4.3 /  5.7 /  8.2 / 11.6    the reference's rule   6.1 /  7.6 /  9.6 / 12.5
//   n =   100,000    6.3 /  9.3 / 16.3 / 32.1                          10.9 / 15.1 / 23.0 / 39.7
//   n =   500,000    7.3 / 11.4 / 22.1 / 53.0                          15.6 / 22.7 / 38.4 / 78.9
//   n = 1,000,000                                                      17.5 / 25.7 / 45.4 / 98.5
// With one body per leaf 1.5 times as many, twice under the reference's rule.  Where
// that is more than kMostLogPerBody (512 bytes per body) the serial walk is taken: its
// walks fill the chip then, and what the ordered walk lists and sorts costs more.
double log_per_body(int n, double theta, int leaf_capacity, bool ref_open)
{
    const double base = ref_open ? 18.0 : 8.0, angle = 0.5 / std::max(theta, 1e-3);
    const double small = ref_open ? std::pow(n / 1e6, 0.30) : std::pow(n / 5e5, 0.35);
    const double more = std::max(0.0, std::pow(angle, ref_open ? 1.9 : 2.3) - 1.0);
    const double leaves = 1.0 + std::max(0, 8 - leaf_capacity) / (ref_open ? 7.0 : 14.0);
    return base * leaves * (1.0 + more * std::min(1.0, small));
}

// Entries of an ordered walk's log pool; 0: no such walk.
int log_pool_entries(int n, double theta, int leaf_capacity, bool ref_open)
{
    const double per_body = log_per_body(n, theta, leaf_capacity, ref_open);
    if ((!ref_open && n > kOrderedBodies) || per_body > kMostLogPerBody) return 0;
    return (int)std::min(per_body * n + 64.0, 2e9);
}

// The walk of n bodies: over child groups, or the stackless preorder walk
// (NB_BH_WALK=preorder, read at every walk; both find the same interactions).
// NB_BH_WALK=serial takes the serial walk where the ordered one is the default.
Walk choose_walk(int n, double theta, int leaf_capacity, bool ref_open)
{
    const char *e = std::getenv("NB_BH_WALK");
    if (walk_pairs() < 1 || (e && std::strcmp(e, "preorder") == 0)) return Walk::kPreorder;
    if (walk_pairs() > 1 || (!ref_open && n > kOrderedBodies)) return Walk::kGroup;
    if (e && std::strcmp(e, "serial") == 0) return Walk::kSerial;
    return log_pool_entries(n, theta, leaf_capacity, ref_open) > 0 ? Walk::kOrdered
                                                                   : Walk::kSerial;
}

int div_up(long a, long b) { return (int)((a + b - 1) / b); }

template <class T>
nb_status scan_exclusive(const T *in, int n, T *out, DevBuf &tmp, cudaStream_t st)
{
    const int nb = div_up(n, scan_tile<T>());
    NB_TRY(tmp.reserve(sizeof(T) * (size_t)std::max(nb, 1)));
    T *sums = tmp.as<T>();
    scan_reduce_kernel<T><<<nb, 256, 0, st>>>(in, n, sums);
    NB_LAUNCH_CHECK();
    scan_top_kernel<T><<<1, std::min(1024, 32 * div_up(nb, 32)), 0, st>>>(sums, nb);
    NB_LAUNCH_CHECK();
    scan_apply_kernel<T><<<nb, 256, 0, st>>>(in, n, sums, out);
    NB_LAUNCH_CHECK();
    return NB_OK;
}

} // namespace

struct BHTree {
    int n = 0;
    int num_nodes = -1;         // host copy of the node count (-1: not read back yet)
    int node_cap = 0;           // node slots reserved (an upper bound of the count)
    int *h_total = nullptr;     // pinned host copy of the count, filled asynchronously
    cudaEvent_t total_ready = nullptr;
    DevBuf part, root, keys0, keys1, vals0, vals1, hist, body, moments, chain_len,
        chain_depth, offsets, scan_tmp, nodes, node_depth, boxes, stats, moments2a, moments2b,
        prefix2a, prefix2b, quad, pcen, pstart, parent, octant, occ, kidflag, kbase, gnodes, gnk,
        gpcen, gquad, gkey, walks;
    bool with_quad = false;     // the nodes carry quadrupoles (quad, 2 float4 per node)
    bool ref_open = false;      // the reference's opening rule (the child toward the body too)
    bool prefer_serial = false; // the serial walk where the ordered one would be taken
    Walk walk = Walk::kGroup;   // the next walk's kernels (ordered: gkey is set)
    int log_pool = 0;           // entries of the log pool
    bool pcen_valid = false;    // pcen holds the parent centres of the current topology
    const uint64_t *sorted_codes = nullptr;
    const uint32_t *order = nullptr;
    bool tree_valid = false;    // nodes/order describe a build of these bodies' count
    int evals_since_build = 0;  // walks on the current topology
};

void bh_invalidate(BHTree *t)
{
    if (t) t->tree_valid = false;
}

void bh_mark_count_stale(BHTree *t)
{
    if (t) t->num_nodes = -1;
}

void bh_prefer_serial(BHTree *t, bool serial) { t->prefer_serial = serial; }

BHTree *bh_create() { return new BHTree(); }

nb_status bh_restart(BHTree *t, cudaStream_t st)
{
    t->tree_valid = false;
    if (t->stats.ptr) NB_CUDA_TRY(cudaMemsetAsync(t->stats.ptr, 0, sizeof(BHStats), st));
    return NB_OK;
}

void bh_destroy(BHTree *t)
{
    if (!t) return;
    DevBuf *bufs[] = {&t->part, &t->root, &t->keys0, &t->keys1, &t->vals0, &t->vals1,
                      &t->hist, &t->body, &t->moments, &t->chain_len,
                      &t->chain_depth, &t->offsets, &t->scan_tmp, &t->nodes, &t->node_depth,
                      &t->boxes, &t->stats, &t->moments2a, &t->moments2b, &t->prefix2a,
                      &t->prefix2b, &t->quad, &t->pcen, &t->pstart, &t->parent, &t->octant,
                      &t->occ, &t->kidflag, &t->kbase, &t->gnodes,
                      &t->gnk, &t->gpcen, &t->gquad, &t->gkey, &t->walks};
    for (DevBuf *b : bufs) b->release();
    if (t->h_total) cudaFreeHost(t->h_total);
    if (t->total_ready) cudaEventDestroy(t->total_ready);
    delete t;
}

// The moments buffer: the bodies' moments, then their prefix sums, which nothing reads
// once the nodes and their quadrupoles are made; the walk's log pool takes their place
// (its counter first), until the next evaluation.
static D4 *prefix_sums(const BHTree *t, int n) { return t->moments.as<D4>() + n; }
static size_t moments_bytes(int n, int log_pool)
{
    return std::max(sizeof(D4) * (2 * (size_t)n + 1), sizeof(uint2) * ((size_t)log_pool + 1));
}

// The device copy of the node count of the last build (scan total).
static const int *d_total(const BHTree *t) { return t->offsets.as<int>() + t->n; }

// Nodes to launch over: the count if it has been read back, else the bound.
static int launch_nodes(const BHTree *t) { return t->num_nodes >= 0 ? t->num_nodes : t->node_cap; }

// The node count on the host (waits for its asynchronous read-back).
static nb_status known_nodes(BHTree *t, int *count)
{
    if (t->num_nodes < 0) {
        NB_CUDA_TRY(cudaEventSynchronize(t->total_ready));
        t->num_nodes = *t->h_total;
    }
    *count = t->num_nodes;
    return NB_OK;
}

// An upper bound of the node count of n bodies: the cells of one depth that
// split are disjoint and hold more than leaf_capacity bodies each (and there
// are at most 8^d of them); every leaf holds a body.
static size_t node_bound(int n, int leaf_capacity)
{
    const size_t per_level = (size_t)n / (size_t)(std::max(leaf_capacity, 0) + 1);
    size_t total = (size_t)n, cells = 1;
    for (int d = 0; d < kMaxLevels; ++d) {
        total += std::min(cells, per_level);
        cells = std::min(cells * 8, (size_t)1 << 40);
    }
    return total;
}

// Root cube, 63-bit codes and the stable LSD sort of the code bits
// [first_shift, 64) (first_shift 0: the full code).  Leaves the sorted codes
// and the permutation (sorted index -> original index) in t.
size_t bh_bytes(int n, double theta, int leaf_capacity)
{
    const size_t N = (size_t)n, cap = node_bound(n, leaf_capacity);
    const size_t sort = 2 * (sizeof(uint64_t) + sizeof(uint32_t)) * N +
                        sizeof(int) * (3 * (256 * (size_t)div_up(n, kSortTile) + 1) + 256);
    const size_t bodies =
        sizeof(float4) * N + moments_bytes(n, log_pool_entries(n, theta, leaf_capacity, false)) +
        sizeof(int) * (4 * N + 1) + sizeof(D4) * (N / 1024 + 1);
    // nodes and node_depth, parent, octant, occ, kidflag, kbase, gnodes and gnk, gkey
    const size_t nodes = (sizeof(BHNode) + 1 + 4 + 1 + 4 + 8 + 4 + sizeof(BHGNode) + 1 + 4) * cap;
    const size_t walks = sizeof(int2) * (1 + kLogSegments) * (size_t)div_up(n, 64);
    const size_t rest = sizeof(long long) * 6 * 4 * (size_t)device_props().num_sms +
                        sizeof(BHRoot) + sizeof(BHStats) + 64;
    return sort + bodies + nodes + walks + rest;
}

// Key/value ping-pong buffers and digit histograms for n entries.
static nb_status reserve_sort(BHTree *t, int n)
{
    const size_t N = (size_t)n;
    const int num_tiles = div_up(n, kSortTile);
    NB_TRY(t->keys0.reserve(sizeof(uint64_t) * N));
    NB_TRY(t->keys1.reserve(sizeof(uint64_t) * N));
    NB_TRY(t->vals0.reserve(sizeof(uint32_t) * N));
    NB_TRY(t->vals1.reserve(sizeof(uint32_t) * N));
    // three rotating digit-count buffers per tile, then their exclusive scan
    // (256 * tiles + 1 each)
    NB_TRY(t->hist.reserve(sizeof(int) * (3 * (256 * (size_t)num_tiles + 1) + 256)));
    return NB_OK;
}

// Stable LSD radix sort of (keys0, vals0) by the key bits [first_shift, 64),
// 8 bits per pass; leaves the sorted keys and values in t.
static nb_status radix_passes(BHTree *t, int n, int first_shift, cudaStream_t st)
{
    const int num_tiles = div_up(n, kSortTile);
    uint64_t *kin = t->keys0.as<uint64_t>(), *kout = t->keys1.as<uint64_t>();
    uint32_t *vin = t->vals0.as<uint32_t>(), *vout = t->vals1.as<uint32_t>();
    // pass p reads counts cnt[p % 3], counts the next digit into cnt[(p + 1) % 3]
    // and clears cnt[(p + 2) % 3] (read by pass p - 1) for pass p + 1
    const size_t stride = 256 * (size_t)num_tiles + 1;
    int *cnt[3] = {t->hist.as<int>(), t->hist.as<int>() + stride, t->hist.as<int>() + 2 * stride};
    int *totals = t->hist.as<int>() + 3 * stride;  // by digit
    const bool direct = num_tiles <= kSortDirectTiles;  // the scatter adds up the counts
    const bool fused = num_tiles <= kSortFusedTiles;    // next histogram in the scatter
    if (fused) NB_CUDA_TRY(cudaMemsetAsync(cnt[1], 0, sizeof(int) * 256 * (size_t)num_tiles, st));
    int p = 0;
    for (int shift = first_shift; shift < 64; shift += 8, ++p) {
        const bool last = shift + 8 >= 64;
        int *cur = fused ? cnt[p % 3] : cnt[0];
        if (!fused || p == 0) {
            radix_hist_kernel<<<num_tiles, 256, 0, st>>>(kin, n, shift, cur, direct ? 1 : num_tiles,
                                                         direct ? 256 : 1);
            NB_LAUNCH_CHECK();
        }
        if (!direct) {
            digit_scan_kernel<<<256, 256, 0, st>>>(cur, num_tiles, totals);
            NB_LAUNCH_CHECK();
        }
        const bool next = fused && !last;
        radix_scatter_kernel<<<num_tiles, 256, 0, st>>>(
            kin, vin, kout, vout, n, shift, cur, direct ? nullptr : totals,
            next ? cnt[(p + 1) % 3] : nullptr, next ? cnt[(p + 2) % 3] : nullptr, num_tiles);
        NB_LAUNCH_CHECK();
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
    t->sorted_codes = kin;
    t->order = vin;
    return NB_OK;
}

// Root cube, 63-bit codes and the stable LSD sort of the code bits
// [first_shift, 64) (first_shift 0: the full code).  Leaves the sorted codes
// and the permutation (sorted index -> original index) in t.
static nb_status morton_sort(BHTree *t, const double *x, const double *y, const double *z,
                             int n, int first_shift, cudaStream_t st, bool hilbert = false)
{
    const int nparts = std::min(div_up(n, 1024), 4 * device_props().num_sms);
    NB_TRY(t->part.reserve(sizeof(long long) * 6 * nparts));
    NB_TRY(t->root.reserve(sizeof(BHRoot)));
    NB_TRY(reserve_sort(t, n));
    BHRoot *root = t->root.as<BHRoot>();

    bbox_partial_kernel<<<nparts, 256, 0, st>>>(x, y, z, n, t->part.as<long long>());
    NB_LAUNCH_CHECK();
    bbox_final_kernel<<<1, 256, 0, st>>>(t->part.as<long long>(), nparts, root);
    NB_LAUNCH_CHECK();
    if (hilbert)
        hilbert_kernel<<<div_up(n, 256), 256, 0, st>>>(x, y, z, n, root, t->keys0.as<uint64_t>(),
                                                        t->vals0.as<uint32_t>());
    else
        encode_kernel<<<div_up(n, 256), 256, 0, st>>>(x, y, z, n, root,
                                                       t->keys0.as<uint64_t>(),
                                                       t->vals0.as<uint32_t>());
    NB_LAUNCH_CHECK();
    return radix_passes(t, n, first_shift, st);
}

nb_status bh_sort_buffers(BHTree *t, int n, uint64_t **keys, uint32_t **vals)
{
    NB_TRY(reserve_sort(t, std::max(n, 1)));
    *keys = t->keys0.as<uint64_t>();
    *vals = t->vals0.as<uint32_t>();
    return NB_OK;
}

nb_status bh_sort_keys(BHTree *t, int n, int first_shift, cudaStream_t st,
                       const uint32_t **order)
{
    if (n > 0) NB_TRY(radix_passes(t, n, first_shift, st));
    *order = t->order;
    t->tree_valid = false;
    return NB_OK;
}

nb_status bh_hilbert_order(BHTree *t, const double *x, const double *y, const double *z, int n,
                           cudaStream_t st, const uint32_t **order, const double **root_centre)
{
    if (n <= 0) return NB_OK;
    NB_TRY(morton_sort(t, x, y, z, n, 32, st, true));  // key bits 32..63
    *order = t->order;
    *root_centre = &t->root.as<BHRoot>()->cx;
    t->tree_valid = false;
    return NB_OK;
}

// Warps that share the group walk of one CTA's bodies: doubled while there are no more
// than 110 per SM, up to 8.  Fewer CTAs than fill the chip leave it to the longest
// walks, which more warps shorten; with enough CTAs the rounds' barriers and the
// shorter lists only cost.  A whole force evaluation took, with 1 / 2 / 4 / 8 / 16
// warps (theta 0.5, disk galaxy), in us:
//   n =    16,384    501 /  402 /  335 /  303 /  300
//   n =   100,000    598 /  511 /  463 /  459 /  522
//   n =   262,144    999 /  928 /  881 /  913 / 1111
//   n =   524,288   1380 / 1347 / 1364 / 1479 / 1887
//   n = 1,048,576   2368 / 2395 / 2501 / 2725 / 3606
// The reference's rule opens far more for some bodies than
// for others (the longest walk at n = 100,000 has 20,270 interactions, the mean 3,891),
// so three times as many, up to 16:
//   n =   100,000   3141 / 1925 / 1196 /  922 /  830
//   n =   400,000   7618 / 4921 / 3417 / 2928 / 3036
// Quadrupoles hold more registers, so half as many:
//   n =   100,000    766 /  726 /  665 /  685 /  806
//   n =   500,000   2132 / 2169 / 2324 / 2666 / 3400
template <bool D>
constexpr int most_walk_warps()
{
    return D ? kWalkWarps : kWalkWarps / 2;
}
template <bool Q, bool D>
int walk_warps(int ctas)
{
    const long sought = (Q ? 55L : 110L) * (D ? 3 : 1) * device_props().num_sms;
    int w = 1;
    while (w < most_walk_warps<D>() && 2L * w * ctas <= sought) w *= 2;
    return w;
}

// Every launch is checked before the next: a kernel that did not run leaves walks and
// logs of an earlier evaluation, which the next would follow.
template <bool ZS, bool Q, bool D>
nb_status walk_launch(BHTree *t, int n, float theta2, float eps2, double G, double *ax,
                      double *ay, double *az, cudaStream_t st, const AfterForce &after)
{
    const int np = walk_pairs();
    const float4 *pc = t->pcen.as<float4>();
    const BHGNode *gn = t->gnodes.as<BHGNode>();
    const unsigned char *gk = t->gnk.as<unsigned char>();
    const float4 *gq = t->gquad.as<float4>(), *gp = t->gpcen.as<float4>();
    if (t->walk == Walk::kOrdered || t->walk == Walk::kSerial) {
        const int ctas = div_up(n, 64);
        const int2 *logged = nullptr;
        if (t->walk == Walk::kOrdered) {
            // logs: the pool's counter, then the pool
            unsigned long long *next = t->moments.as<unsigned long long>();
            uint2 *pool = reinterpret_cast<uint2 *>(next + 1);
            int2 *walks = t->walks.as<int2>(), *segs = walks + ctas;
            auto decide = [&](auto *kernel, int threads, size_t shared) -> nb_status {
                NB_CUDA_TRY(cudaFuncSetAttribute(
                    kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared));
                kernel<<<ctas, threads, shared, st>>>(
                    gn, gk, t->gkey.as<unsigned>(), gp, d_total(t), t->body.as<float4>(), n,
                    theta2, t->stats.as<BHStats>(), walks, segs, pool, t->log_pool, next);
                NB_LAUNCH_CHECK();
                return NB_OK;
            };
            if (D || ctas <= kFewWalks)
                NB_TRY(decide(decide_kernel<D, 16, D ? 4096 : 1024>, 512,
                              sizeof(LogShared<D, 16, D ? 4096 : 1024>)));
            else
                NB_TRY(decide(decide_kernel<D, 4, 1024>, 128, sizeof(LogShared<D, 4, 1024>)));
            log_eval_kernel<ZS, Q><<<ctas, 64 + kLogListers, 0, st>>>(
                gn, gq, t->body.as<float4>(), t->order, n, eps2, G, ax, ay, az, walks, segs, pool,
                after);
            NB_LAUNCH_CHECK();
            logged = walks;  // mostly none are left: a launch that only looks
        }
        serial_walk_kernel<ZS, Q, D><<<ctas, 32, 0, st>>>(
            gn, gk, d_total(t), t->body.as<float4>(), t->order, n, theta2, eps2, G, ax, ay, az,
            t->stats.as<BHStats>(), gq, gp, logged, after);
    } else if (t->walk == Walk::kGroup) {
        const int ctas = div_up(n, 64 * np), warps = walk_warps<Q, D>(ctas);
        // one pair per lane: never under the reference's rule (choose_walk)
        auto *kernel = np == 2 ? group_walk_kernel<ZS, Q, 2, D> : group_walk_kernel<ZS, Q, 1, false>;
        const size_t shared = walk_shared_bytes<Q>(warps);
        // what the most warps need, not these: the attribute is the function's, and
        // another thread's launch may come between this call and the launch below
        NB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)walk_shared_bytes<Q>(most_walk_warps<D>())));
        kernel<<<ctas, 32 * warps, shared, st>>>(
            gn, gk, d_total(t), t->body.as<float4>(), t->order, n, theta2, eps2, G, ax, ay, az,
            t->stats.as<BHStats>(), gq, gp, after);
    } else if (np == 2)
        walk2_kernel<ZS, Q, 2, D><<<div_up(n, 4 * kWalkBlock), kWalkBlock, 0, st>>>(
            t->nodes.as<BHNode>(), d_total(t), t->body.as<float4>(), t->order, n, theta2,
            eps2, G, ax, ay, az, t->stats.as<BHStats>(), t->quad.as<float4>(), pc);
    else if (np == 1)
        walk2_kernel<ZS, Q, 1, D><<<div_up(n, 2 * kWalkBlock), kWalkBlock, 0, st>>>(
            t->nodes.as<BHNode>(), d_total(t), t->body.as<float4>(), t->order, n, theta2,
            eps2, G, ax, ay, az, t->stats.as<BHStats>(), t->quad.as<float4>(), pc);
    else
        walk_kernel<ZS, Q, D><<<div_up(n, kWalkBlock), kWalkBlock, 0, st>>>(
            t->nodes.as<BHNode>(), d_total(t), t->body.as<float4>(), t->order, n, theta2,
            eps2, G, ax, ay, az, t->stats.as<BHStats>(), t->quad.as<float4>(), pc);
    NB_LAUNCH_CHECK();
    return NB_OK;
}

template <bool ZS, bool Q>
nb_status walk_launch_rule(BHTree *t, int n, float theta2, float eps2, double G, double *ax,
                           double *ay, double *az, cudaStream_t st, const AfterForce &after)
{
    return t->ref_open ? walk_launch<ZS, Q, true>(t, n, theta2, eps2, G, ax, ay, az, st, after)
                       : walk_launch<ZS, Q, false>(t, n, theta2, eps2, G, ax, ay, az, st, after);
}

static nb_status launch_walk(BHTree *t, int n, double G, double eps2, double theta, double *ax,
                             double *ay, double *az, cudaStream_t st, const KernelTimer *timer,
                             const AfterForce &after)
{
    NvtxRange range("bh_walk");
    const float th2 = (float)(theta * theta), e2 = (float)eps2;
    if (timer && timer->start) NB_CUDA_TRY(cudaEventRecord(timer->start, st));
    const bool zero = !(eps2 > 0.0);
    auto *launch = t->with_quad
                       ? (zero ? walk_launch_rule<true, true> : walk_launch_rule<false, true>)
                       : (zero ? walk_launch_rule<true, false> : walk_launch_rule<false, false>);
    NB_TRY(launch(t, n, th2, zero ? 0.0f : e2, G, ax, ay, az, st, after));
    if (timer && timer->stop) NB_CUDA_TRY(cudaEventRecord(timer->stop, st));
    // the child-group walks apply the update, the preorder walks do not
    if (t->walk == Walk::kPreorder) return apply_after(after, n, ax, ay, az, st);
    return NB_OK;
}

// Quadrupoles of every node of the current tree (after its monopole pass).
static nb_status compute_quads(BHTree *t, const double *x, const double *y, const double *z,
                               const double *m, int n, cudaStream_t st)
{
    const size_t N = (size_t)n;
    const int nn = launch_nodes(t);
    NB_TRY(t->moments2a.reserve(sizeof(D4) * N));
    NB_TRY(t->moments2b.reserve(sizeof(D4) * N));
    NB_TRY(t->prefix2a.reserve(sizeof(D4) * (N + 1)));
    NB_TRY(t->prefix2b.reserve(sizeof(D4) * (N + 1)));
    NB_TRY(t->quad.reserve(sizeof(float4) * 2 * (size_t)nn));
    gather2_kernel<<<div_up(n, 256), 256, 0, st>>>(t->order, x, y, z, m, n,
                                                   t->root.as<BHRoot>(), t->moments2a.as<D4>(),
                                                   t->moments2b.as<D4>());
    NB_LAUNCH_CHECK();
    NB_TRY(scan_exclusive<D4>(t->moments2a.as<D4>(), n, t->prefix2a.as<D4>(), t->scan_tmp, st));
    NB_TRY(scan_exclusive<D4>(t->moments2b.as<D4>(), n, t->prefix2b.as<D4>(), t->scan_tmp, st));
    quad_kernel<<<div_up(nn, 256), 256, 0, st>>>(t->nodes.as<BHNode>(), d_total(t), prefix_sums(t, n),
                                                 t->prefix2a.as<D4>(), t->prefix2b.as<D4>(),
                                                 t->quad.as<float4>());
    NB_LAUNCH_CHECK();
    return NB_OK;
}

// The parent centres the reference's opening rule needs, once per topology.
static nb_status ensure_pcen(BHTree *t, cudaStream_t st)
{
    if (!t->ref_open || t->pcen_valid) return NB_OK;
    const int slots = launch_nodes(t);
    NB_TRY(t->pcen.reserve(sizeof(float4) * (size_t)slots));
    const int grid = std::max(1, std::min(div_up(slots, 256), 8 * device_props().num_sms));
    pcen_kernel<<<grid, 256, 0, st>>>(t->sorted_codes, t->nodes.as<BHNode>(),
                                      t->node_depth.as<unsigned char>(), d_total(t),
                                      t->root.as<BHRoot>(), t->pcen.as<float4>());
    NB_LAUNCH_CHECK();
    t->pcen_valid = true;
    return NB_OK;
}

// The child-group records of the current tree (after its monopoles, sides
// and quadrupoles); recount: a new topology (children counts and group
// places), else only the records are rewritten.
static nb_status group_nodes(BHTree *t, cudaStream_t st, bool recount)
{
    const int slots = launch_nodes(t);
    const int grid = std::max(1, std::min(div_up(slots, 256), 8 * device_props().num_sms));
    if (recount) {
        NB_TRY(t->kbase.reserve(sizeof(int) * ((size_t)slots + 1)));
        int *next = t->kbase.as<int>() + slots;  // the group counter (group 0: the root)
        NB_CUDA_TRY(cudaMemsetAsync(next, 0, sizeof(int), st));
        alloc_groups_kernel<<<grid, 256, 0, st>>>(t->kidflag.as<unsigned char>(), d_total(t),
                                                  t->occ.as<unsigned>(), t->kbase.as<int>(), next);
        NB_LAUNCH_CHECK();
    }
    NB_TRY(t->gnodes.reserve(sizeof(BHGNode) * (size_t)slots));
    NB_TRY(t->gnk.reserve((size_t)slots));
    if (t->ref_open) NB_TRY(t->gpcen.reserve(sizeof(float4) * (size_t)slots));
    if (t->with_quad) NB_TRY(t->gquad.reserve(sizeof(float4) * 2 * (size_t)slots));
    if (t->walk == Walk::kOrdered) {
        NB_TRY(t->gkey.reserve(sizeof(unsigned) * (size_t)slots));
        NB_TRY(t->walks.reserve(sizeof(int2) * (1 + kLogSegments) * (size_t)div_up(t->n, 64)));
        NB_TRY(t->moments.reserve(moments_bytes(t->n, t->log_pool)));  // done with, now
    }
    group_kernel<<<grid, 256, 0, st>>>(
        t->nodes.as<BHNode>(), d_total(t), t->occ.as<unsigned>(), t->kbase.as<int>(),
        t->parent.as<int>(), t->octant.as<unsigned char>(),
        t->ref_open ? t->pcen.as<float4>() : nullptr,
        t->with_quad ? t->quad.as<float4>() : nullptr, t->gnodes.as<BHGNode>(),
        t->gnk.as<unsigned char>(), t->gpcen.as<float4>(),
        t->with_quad ? t->gquad.as<float4>() : nullptr, t->node_depth.as<unsigned char>(),
        t->walk == Walk::kOrdered ? t->gkey.as<unsigned>() : nullptr,
        t->walk == Walk::kOrdered ? t->moments.as<unsigned long long>() : nullptr);
    NB_LAUNCH_CHECK();
    return NB_OK;
}

// Monopoles and cell sides of the kept topology for the current positions.
static nb_status refit(BHTree *t, const double *x, const double *y, const double *z,
                       const double *m, int n, cudaStream_t st)
{
    const BHRoot *root = t->root.as<BHRoot>();
    int nn = 0;
    NB_TRY(known_nodes(t, &nn));  // read back during an earlier evaluation
    NB_TRY(t->boxes.reserve(sizeof(float4) * 2 * (size_t)nn));
    gather_kernel<<<div_up(n, 256), 256, 0, st>>>(t->order, x, y, z, m, n, root,
                                                  t->body.as<float4>(), t->moments.as<D4>());
    NB_LAUNCH_CHECK();
    NB_TRY(scan_exclusive<D4>(t->moments.as<D4>(), n, prefix_sums(t, n), t->scan_tmp, st));
    refit_kernel<<<div_up(nn, 256), 256, 0, st>>>(t->nodes.as<BHNode>(), d_total(t),
                                                  t->node_depth.as<unsigned char>(),
                                                  prefix_sums(t, n), root, t->body.as<float4>(),
                                                  t->boxes.as<float4>());
    NB_LAUNCH_CHECK();
    // internal nodes, deepest first (an internal node is shallower than the
    // deepest possible level)
    for (int d = kMaxLevels - 1; d >= 0; --d) {
        refit_level_kernel<<<div_up(nn, 256), 256, 0, st>>>(
            t->nodes.as<BHNode>(), d_total(t), t->node_depth.as<unsigned char>(), d, root,
            t->boxes.as<float4>());
        NB_LAUNCH_CHECK();
    }
    // this walk's interaction counts (the tree's leaf and depth figures stay)
    NB_CUDA_TRY(cudaMemsetAsync(t->stats.ptr, 0, 2 * sizeof(unsigned long long), st));
    return NB_OK;
}

nb_status bh_compute(BHTree *t, const double *x, const double *y, const double *z,
                     const double *m, int n, double G, double eps2, double theta,
                     int leaf_capacity, double *ax, double *ay, double *az, cudaStream_t st,
                     const KernelTimer *timer, int reuse, bool quad, bool ref_open,
                     const AfterForce &after)
{
    if (n <= 0) return NB_OK;
    t->with_quad = quad;
    t->ref_open = ref_open;
    t->walk = choose_walk(n, theta, leaf_capacity, ref_open);
    if (t->walk == Walk::kOrdered && t->prefer_serial) t->walk = Walk::kSerial;
    t->log_pool = log_pool_entries(n, theta, leaf_capacity, ref_open);
    if (ax && reuse > 1 && t->tree_valid && t->n == n && t->evals_since_build < reuse) {
        NB_TRY(refit(t, x, y, z, m, n, st));
        if (quad) NB_TRY(compute_quads(t, x, y, z, m, n, st));
        NB_TRY(ensure_pcen(t, st));
        NB_TRY(group_nodes(t, st, false));
        ++t->evals_since_build;
        return launch_walk(t, n, G, eps2, theta, ax, ay, az, st, timer, after);
    }
    t->tree_valid = false;
    NvtxRange range("bh_build");
    const size_t N = (size_t)n;
    NB_TRY(t->body.reserve(sizeof(float4) * N));
    NB_TRY(t->moments.reserve(moments_bytes(n, t->log_pool)));
    NB_TRY(t->chain_len.reserve(sizeof(int) * N));
    NB_TRY(t->chain_depth.reserve(sizeof(int) * N));
    NB_TRY(t->offsets.reserve(sizeof(int) * (N + 1)));
    NB_TRY(t->pstart.reserve(sizeof(int) * N));
    if (!t->stats.ptr) {
        NB_TRY(t->stats.reserve(sizeof(BHStats)));
        NB_CUDA_TRY(cudaMemsetAsync(t->stats.ptr, 0, sizeof(BHStats), st));
    }
    NB_TRY(morton_sort(t, x, y, z, n, 0, st));
    BHRoot *root = t->root.as<BHRoot>();
    BHStats *stats = t->stats.as<BHStats>();
    uint64_t *kin = const_cast<uint64_t *>(t->sorted_codes);
    uint32_t *vin = const_cast<uint32_t *>(t->order);

    gather_kernel<<<div_up(n, 256), 256, 0, st>>>(vin, x, y, z, m, n, root,
                                                  t->body.as<float4>(), t->moments.as<D4>());
    NB_LAUNCH_CHECK();
    NB_TRY(scan_exclusive<D4>(t->moments.as<D4>(), n, prefix_sums(t, n), t->scan_tmp, st));
    chain_kernel<<<div_up(n, 256), 256, 0, st>>>(kin, n, leaf_capacity, root,
                                                 t->chain_len.as<int>(),
                                                 t->chain_depth.as<int>(), t->pstart.as<int>());
    NB_LAUNCH_CHECK();
    NB_TRY(scan_exclusive<int>(t->chain_len.as<int>(), n, t->offsets.as<int>(), t->scan_tmp,
                               st));
    // No host read of the node count before the walk: node storage is sized
    // for the bound, the kernels read the count on the device, and the count
    // comes back to the host asynchronously for later launches and queries.
    const size_t cap = node_bound(n, leaf_capacity);
    NB_TRY(t->nodes.reserve(sizeof(BHNode) * cap));
    NB_TRY(t->node_depth.reserve(cap));
    NB_TRY(t->parent.reserve(sizeof(int) * cap));
    NB_TRY(t->octant.reserve(cap));
    NB_TRY(t->occ.reserve(sizeof(unsigned) * cap));
    NB_TRY(t->kidflag.reserve(8 * cap));
    if (!t->h_total) NB_CUDA_TRY(cudaMallocHost(&t->h_total, sizeof(int)));
    if (!t->total_ready) NB_CUDA_TRY(cudaEventCreateWithFlags(&t->total_ready,
                                                              cudaEventDisableTiming));
    NB_CUDA_TRY(cudaMemcpyAsync(t->h_total, t->offsets.as<int>() + n, sizeof(int),
                                cudaMemcpyDeviceToHost, st));
    // inside a captured step graph the record must be an external event node
    // (recorded by every replay) for the host to be able to wait for the count
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    NB_CUDA_TRY(cudaStreamIsCapturing(st, &capturing));
    if (capturing == cudaStreamCaptureStatusActive)
        NB_CUDA_TRY(cudaEventRecordWithFlags(t->total_ready, st, cudaEventRecordExternal));
    else
        NB_CUDA_TRY(cudaEventRecord(t->total_ready, st));
    t->node_cap = (int)std::min(cap, (size_t)INT32_MAX);
    t->num_nodes = -1;
    t->n = n;
    place_kernel<<<div_up(n, 256), 256, 0, st>>>(n, t->chain_len.as<int>(),
                                                 t->chain_depth.as<int>(), t->offsets.as<int>(),
                                                 t->nodes.as<BHNode>(),
                                                 t->node_depth.as<unsigned char>(),
                                                 t->kidflag.as<unsigned long long>(), stats,
                                                 t->node_cap);
    NB_LAUNCH_CHECK();
    const int node_grid = std::min(div_up(launch_nodes(t), 256), 8 * device_props().num_sms);
    node_kernel<<<std::max(1, node_grid), 256, 0, st>>>(
        kin, n, root, d_total(t), t->chain_depth.as<int>(), t->offsets.as<int>(),
        prefix_sums(t, n), t->nodes.as<BHNode>(), t->node_depth.as<unsigned char>(),
        t->pstart.as<int>(), t->parent.as<int>(), t->octant.as<unsigned char>(),
        t->kidflag.as<unsigned char>(), stats, t->node_cap);
    NB_LAUNCH_CHECK();
    if (quad) NB_TRY(compute_quads(t, x, y, z, m, n, st));
    t->pcen_valid = false;
    NB_TRY(ensure_pcen(t, st));
    NB_TRY(group_nodes(t, st, true));
    t->tree_valid = true;
    t->evals_since_build = 0;
    if (!ax) return NB_OK;
    t->evals_since_build = 1;
    return launch_walk(t, n, G, eps2, theta, ax, ay, az, st, timer, after);
}

nb_status bh_info(BHTree *t, cudaStream_t st, nb_bh_info *info)
{
    if (!t->n) return fail(NB_ERR_NOT_LOADED, "no Barnes-Hut tree built");
    BHRoot r;
    BHStats s;
    NB_CUDA_TRY(cudaMemcpyAsync(&r, t->root.ptr, sizeof(r), cudaMemcpyDeviceToHost, st));
    NB_CUDA_TRY(cudaMemcpyAsync(&s, t->stats.ptr, sizeof(s), cudaMemcpyDeviceToHost, st));
    NB_CUDA_TRY(cudaStreamSynchronize(st));
    int nn = 0;
    NB_TRY(known_nodes(t, &nn));
    info->num_nodes = nn;
    info->num_leaves = s.leaves;
    info->max_depth = s.max_depth;
    info->split_levels = r.levels;
    info->root[0] = r.cx;
    info->root[1] = r.cy;
    info->root[2] = r.cz;
    info->root[3] = r.size;
    info->interactions_m2p = s.m2p;
    info->interactions_p2p = s.p2p;
    info->interactions_total = s.total;
    return NB_OK;
}

nb_status bh_read_order(BHTree *t, cudaStream_t st, uint64_t *codes, uint32_t *order)
{
    if (!t->n) return fail(NB_ERR_NOT_LOADED, "no Barnes-Hut tree built");
    if (codes)
        NB_CUDA_TRY(cudaMemcpyAsync(codes, t->sorted_codes, sizeof(uint64_t) * t->n,
                                    cudaMemcpyDeviceToHost, st));
    if (order)
        NB_CUDA_TRY(cudaMemcpyAsync(order, t->order, sizeof(uint32_t) * t->n,
                                    cudaMemcpyDeviceToHost, st));
    NB_CUDA_TRY(cudaStreamSynchronize(st));
    return NB_OK;
}

nb_status bh_read_nodes(BHTree *t, cudaStream_t st, int max_nodes, int *depth,
                        uint64_t *prefix, int *first, int *count, int *is_leaf, int *skip,
                        float *com_mass)
{
    if (!t->n) return fail(NB_ERR_NOT_LOADED, "no Barnes-Hut tree built");
    int nn = 0;
    NB_TRY(known_nodes(t, &nn));
    if (max_nodes < nn) return fail(NB_ERR_CAPACITY, "max_nodes is smaller than the node count");
    std::vector<BHNode> h(nn);
    std::vector<unsigned char> dep(nn);
    std::vector<uint64_t> codes(t->n);
    BHRoot r;
    NB_CUDA_TRY(cudaMemcpyAsync(h.data(), t->nodes.ptr, sizeof(BHNode) * h.size(),
                                cudaMemcpyDeviceToHost, st));
    NB_CUDA_TRY(cudaMemcpyAsync(dep.data(), t->node_depth.ptr, dep.size(),
                                cudaMemcpyDeviceToHost, st));
    NB_CUDA_TRY(cudaMemcpyAsync(codes.data(), t->sorted_codes, sizeof(uint64_t) * t->n,
                                cudaMemcpyDeviceToHost, st));
    NB_CUDA_TRY(cudaMemcpyAsync(&r, t->root.ptr, sizeof(r), cudaMemcpyDeviceToHost, st));
    NB_CUDA_TRY(cudaStreamSynchronize(st));
    for (int k = 0; k < nn; ++k) {
        const BHNode &nd = h[k];
        const int d = dep[k];
        if (depth) depth[k] = d;
        if (prefix) prefix[k] = d == 0 ? 0 : codes[nd.first] >> (63 - 3 * d);
        if (first) first[k] = nd.first;
        if (count) count[k] = nd.count;
        if (is_leaf) is_leaf[k] = nd.skip == k + 1;
        if (skip) skip[k] = nd.skip;
        if (com_mass) {
            com_mass[4 * k + 0] = (float)(r.cx + (double)nd.com_mass.x);
            com_mass[4 * k + 1] = (float)(r.cy + (double)nd.com_mass.y);
            com_mass[4 * k + 2] = (float)(r.cz + (double)nd.com_mass.z);
            com_mass[4 * k + 3] = nd.com_mass.w;
        }
    }
    return NB_OK;
}

} // namespace nb
