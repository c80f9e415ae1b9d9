// nb_diag.cu -- energy and momentum diagnostics reduced on the GPU in FP64.
//
// Replaces the host loops of CUDA/src/test_common.cpp:63-182 (and
// CPU/include/tests_common.hpp:33-75), which needed a full device-to-host copy
// of the state every step and an O(N^2) host loop for the potential.
//   - per-body sums (kinetic energy, angular momentum, centre of mass, linear
//     momentum, mass): one HBM-bound pass (56 B per body), block partials in a
//     fixed tree order, then one block that adds the partials in index order;
//   - potential energy: an O(N^2 / 2) FP64 pass over unordered pairs, unsoftened
//     and softened together, reduced like the above.
// All reductions have a fixed order, so results do not depend on scheduling.
#include "nb_internal.h"
#include "nb_fp64pair.cuh"

#include <algorithm>

namespace nb {
namespace {

constexpr int kRed = 256;     // threads per reduction block
constexpr int kNSum = 11;     // KE, Lx, Ly, Lz, Mx, My, Mz, Px, Py, Pz, M

template <int NV>
__device__ __forceinline__ void block_reduce(double (&v)[NV], double *sh /* [NV][kRed] */)
{
    const int t = threadIdx.x;
#pragma unroll
    for (int c = 0; c < NV; ++c) sh[c * kRed + t] = v[c];
    __syncthreads();
    for (int w = kRed / 2; w > 0; w >>= 1) {
        if (t < w) {
#pragma unroll
            for (int c = 0; c < NV; ++c) sh[c * kRed + t] += sh[c * kRed + t + w];
        }
        __syncthreads();
    }
#pragma unroll
    for (int c = 0; c < NV; ++c) v[c] = sh[c * kRed];
}

__global__ void __launch_bounds__(kRed)
body_sums_kernel(const double *__restrict__ x, const double *__restrict__ y,
                 const double *__restrict__ z, const double *__restrict__ vx,
                 const double *__restrict__ vy, const double *__restrict__ vz,
                 const double *__restrict__ m, int n, double *__restrict__ part)
{
    __shared__ double sh[kNSum * kRed];
    double acc[kNSum];
#pragma unroll
    for (int c = 0; c < kNSum; ++c) acc[c] = 0.0;
    for (int i = blockIdx.x * kRed + threadIdx.x; i < n; i += gridDim.x * kRed) {
        const double X = x[i], Y = y[i], Z = z[i];
        const double U = vx[i], V = vy[i], W = vz[i], M = m[i];
        acc[0] += 0.5 * M * (U * U + V * V + W * W);
        acc[1] += (Y * W - Z * V) * M;
        acc[2] += (Z * U - X * W) * M;
        acc[3] += (X * V - Y * U) * M;
        acc[4] += X * M;
        acc[5] += Y * M;
        acc[6] += Z * M;
        acc[7] += U * M;
        acc[8] += V * M;
        acc[9] += W * M;
        acc[10] += M;
    }
    block_reduce<kNSum>(acc, sh);
    if (threadIdx.x == 0)
        for (int c = 0; c < kNSum; ++c) part[blockIdx.x * kNSum + c] = acc[c];
}

// Potential sums over unordered pairs, unsoftened and softened: the warp of
// block pair (p, a) holds 32 bodies of the first block in its lanes and rotates
// the tiles of the second through them (the schedule of nb_fp64pair.cuh), so
// each pair is met once.  Per pair 19 FP64 operations (13 without softening,
// where the two sums are equal); the seed's integer work is free beside them.
// Warps take block pairs in strides of the grid, a fixed assignment:
// part[2 w], part[2 w + 1] = warp w's sums.  One-warp CTAs: with four warps a
// CTA's slowest warp holds the others' places (8.31 ms instead of 7.70 at
// n = 20,000).  Bound by the FP64 pipe, 84 % busy (the per-body rows that this
// replaces, each pair met twice with a square root and a division a term: 56.2).
template <bool SOFT>
__global__ void __launch_bounds__(32)
potential_pairs_kernel(const double *__restrict__ x, const double *__restrict__ y,
                       const double *__restrict__ z, const double *__restrict__ m, int n,
                       double eps2, int blocks, int T, long items, double *__restrict__ part)
{
    const int lane = threadIdx.x, next = (lane + 1) & 31;
    const int width = 32 * T;
    double tu = 0.0, ts = 0.0;
    for (long it = blockIdx.x; it < items; it += gridDim.x) {
        const int a = (int)(it % blocks), p = (int)(it / blocks);
        if (!pair_first(p, a, blocks)) continue;
        const int b = (a + p) % blocks;
        const int ta = min(T, (n - a * width + 31) / 32), tb = min(T, (n - b * width + 31) / 32);
        for (int u = 0; u < ta; ++u) {
            const int i = a * width + 32 * u + lane;
            const bool iv = i < n;
            const double xi = iv ? x[i] : 0.0, yi = iv ? y[i] : 0.0, zi = iv ? z[i] : 0.0;
            double su = 0.0, ss = 0.0;
            for (int v = p == 0 ? u : 0; v < tb; ++v) {
                const bool self = p == 0 && u == v;
                const int j0 = b * width + 32 * v;
                // a tile with itself: steps 1 .. 15 meet a pair once, step 16
                // from both sides (the lower half of the lanes takes it)
                const int s0 = self ? 1 : 0, s1 = self ? 17 : 32;
                const int j = j0 + ((lane + s0) & 31);
                double xj = j < n ? x[j] : 0.0, yj = j < n ? y[j] : 0.0, zj = j < n ? z[j] : 0.0,
                       mj = j < n ? m[j] : 0.0;
                for (int s = s0; s < s1; ++s) {
                    const bool valid = iv && j0 + ((lane + s) & 31) < n &&
                                       !(self && s == 16 && lane >= 16);
                    const double dx = xj - xi, dy = yj - yi, dz = zj - zi;
                    const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
                    const double qu = inv_sqrt(r2);
                    su = fma(valid ? mj : 0.0, valid ? qu : 0.0, su);
                    if (SOFT) {
                        const double qs = inv_sqrt(r2 + eps2);
                        ss = fma(valid ? mj : 0.0, valid ? qs : 0.0, ss);
                    }
                    xj = __shfl_sync(0xffffffffu, xj, next);
                    yj = __shfl_sync(0xffffffffu, yj, next);
                    zj = __shfl_sync(0xffffffffu, zj, next);
                    mj = __shfl_sync(0xffffffffu, mj, next);
                }
            }
            if (iv) {
                const double mi = m[i];
                tu = fma(mi, su, tu);
                if (SOFT) ts = fma(mi, ss, ts);
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        tu += __shfl_xor_sync(0xffffffffu, tu, o);
        ts += __shfl_xor_sync(0xffffffffu, ts, o);
    }
    if (lane == 0) {
        part[2 * (size_t)blockIdx.x] = tu;
        part[2 * (size_t)blockIdx.x + 1] = SOFT ? ts : tu;
    }
}

// Final pass, one block: warp c adds the partials of sum c (kNSum body sums,
// then the two potential sums), lanes in strides and a fixed tree.
__global__ void __launch_bounds__(32 * (kNSum + 2))
finish_kernel(const double *__restrict__ part, int nparts, const double *__restrict__ pot,
              int npot, double *__restrict__ out)
{
    const int c = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool body = c < kNSum;
    const double *src = body ? part + c : pot + (c - kNSum);
    const int count = body ? nparts : npot, stride = body ? kNSum : 2;
    // four running sums: the FP64 add latency, not the loads, sets the time
    double r[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
    for (int k = lane; k < count; k += 128)
#pragma unroll
        for (int u = 0; u < 4; ++u)
            r[u] += k + 32 * u < count ? src[(size_t)(k + 32 * u) * stride] : 0.0;
    double s = (r[0] + r[1]) + (r[2] + r[3]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) out[c] = s;
}

// FP32 pipe rate probe: every thread runs kFmaRounds rounds of kFmaChains
// independent packed FMAs on register values (no memory traffic in the loop)
// and stores one sum, so that nothing is optimised away.
constexpr int kFmaChains = 8, kFmaRounds = 4096;
__global__ void __launch_bounds__(256) fma_rate_kernel(float seed, float *__restrict__ out)
{
    float2 a[kFmaChains];
    const float2 m = make_float2(0.9999999f, 0.9999998f), c = make_float2(1e-7f, 2e-7f);
#pragma unroll
    for (int k = 0; k < kFmaChains; ++k)
        a[k] = make_float2(seed + (float)(threadIdx.x + k), seed - (float)k);
    for (int r = 0; r < kFmaRounds; ++r)
#pragma unroll
        for (int k = 0; k < kFmaChains; ++k) a[k] = __ffma2_rn(a[k], m, c);
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < kFmaChains; ++k) sum += a[k].x + a[k].y;
    out[blockIdx.x * 256 + threadIdx.x] = sum;
}

} // namespace

nb_status fp32_rate(double *lane_ops_per_s)
{
    const int blocks = 8 * device_props().num_sms;
    DevBuf out;
    NB_TRY(out.reserve(sizeof(float) * 256 * (size_t)blocks));
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    NB_CUDA_TRY(cudaEventCreate(&e0));
    NB_CUDA_TRY(cudaEventCreate(&e1));
    float best = 1e30f;
    nb_status st = NB_OK;
    for (int r = 0; r < 4 && st == NB_OK; ++r) {  // the first launch warms up
        cudaEventRecord(e0, 0);
        fma_rate_kernel<<<blocks, 256>>>(1.0f + r, out.as<float>());
        const cudaError_t launched = cudaGetLastError();
        cudaEventRecord(e1, 0);
        if (launched != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess)
            st = fail(NB_ERR_CUDA, "fp32 rate probe");
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        if (r > 0) best = std::min(best, ms);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    out.release();
    NB_TRY(st);
    const double ops = (double)blocks * 256.0 * kFmaRounds * kFmaChains * 2.0;
    *lane_ops_per_s = ops / (best * 1e-3);
    return NB_OK;
}

nb_status diagnostics(const double *x, const double *y, const double *z, const double *vx,
                      const double *vy, const double *vz, const double *m, int n, double G,
                      double eps2, DevBuf &scratch, cudaStream_t st, nb_diag *out)
{
    if (n <= 0) return fail(NB_ERR_NOT_LOADED, "diagnostics: no bodies");
    const int nparts = std::min((n + kRed - 1) / kRed, 4 * device_props().num_sms);
    // blocks of up to 8 tiles while the block pairs fill the FP64 pipes evenly
    int T = 1;
    auto block_pairs = [&](int t) {
        const long M = (n + 32 * t - 1) / (32 * t);
        return M * (M / 2 + 1);
    };
    while (T < 8 && block_pairs(2 * T) >= 12 * device_props().num_sms) T *= 2;
    const int blocks = (n + 32 * T - 1) / (32 * T);
    const long items = block_pairs(T);
    const int npot = (int)std::min<long>(items, 32 * device_props().num_sms);
    const size_t bytes = sizeof(double) * ((size_t)nparts * kNSum + 2 * (size_t)npot + 16);
    NB_TRY(scratch.reserve(bytes));
    double *part = scratch.as<double>();
    double *pot = part + (size_t)nparts * kNSum;
    double *res = pot + 2 * (size_t)npot;
    body_sums_kernel<<<nparts, kRed, 0, st>>>(x, y, z, vx, vy, vz, m, n, part);
    NB_LAUNCH_CHECK();
    if (eps2 > 0.0)
        potential_pairs_kernel<true><<<npot, 32, 0, st>>>(x, y, z, m, n, eps2, blocks,
                                                                     T, items, pot);
    else
        potential_pairs_kernel<false><<<npot, 32, 0, st>>>(x, y, z, m, n, 0.0, blocks,
                                                                      T, items, pot);
    NB_LAUNCH_CHECK();
    finish_kernel<<<1, 32 * (kNSum + 2), 0, st>>>(part, nparts, pot, npot, res);
    NB_LAUNCH_CHECK();
    double h[kNSum + 2];
    NB_CUDA_TRY(cudaMemcpyAsync(h, res, sizeof(h), cudaMemcpyDeviceToHost, st));
    NB_CUDA_TRY(cudaStreamSynchronize(st));
    out->kinetic = h[0];
    out->angular_momentum[0] = h[1];
    out->angular_momentum[1] = h[2];
    out->angular_momentum[2] = h[3];
    out->mass = h[10];
    for (int c = 0; c < 3; ++c) {
        out->center_of_mass[c] = h[4 + c] / h[10];
        out->momentum[c] = h[7 + c];
    }
    out->potential = -G * h[kNSum + 0];
    out->potential_softened = -G * h[kNSum + 1];
    out->total = out->kinetic + out->potential;
    out->total_softened = out->kinetic + out->potential_softened;
    return NB_OK;
}

} // namespace nb
