// nb_fp64pair.cuh -- FP64 building blocks of the all-pairs kernels: a reciprocal
// square root seeded on the MUFU pipe.
//
// GB300 issues two FP64 lane operations per clock and SM, a 64th of its FP32
// rate, so an FP64 all-pairs kernel is bound by the number of FP64 operations
// alone: integer, FP32, shuffle and shared-memory work beside them is free as
// long as a few warps are resident.  Hence the two rules here: spend integer
// operations to save FP64 ones (the seed below), and evaluate a pair once for
// both of its bodies.
#pragma once

#include "nb_pair.cuh"

namespace nb {

// y ~ r2^(-1/2) to about 2^-22, a 24-bit value (so y * y is exact in FP64), for
// r2 in [2^-320, 2^321); false outside (zero, subnormal, infinite, NaN and
// extreme r2: the caller takes the library rsqrt).  r2 = f 4^k with f in [1, 4)
// truncated to FP32; exponents move by integer arithmetic, so the range of FP32
// does not matter and no FP64 operation is spent.
__device__ __forceinline__ bool rsqrt_seed(double r2, double &y)
{
    const int hi = __double2hiint(r2), lo = __double2loint(r2);
    const int e = (int)((unsigned)hi >> 20) - 1023;
    const int k = e >> 1;
    const unsigned f = ((unsigned)(127 + e - 2 * k) << 23) |
                       (__funnelshift_l((unsigned)lo, (unsigned)hi, 3) & 0x7fffffu);
    const unsigned b = __float_as_uint(rsqrt_mufu(__uint_as_float(f)));
    y = __hiloint2double((int)((b >> 3) + ((unsigned)(1023 - 127 - k) << 20)), (int)(b << 29));
    return (unsigned)(e + 320) <= 640u;
}

// r2^(-3/2): with y = seed and e = 1 - r2 y^2 (|e| < 2^-21), r2^(-3/2) =
// y^3 (1 + 3/2 e + 15/8 e^2 + O(e^3)), the dropped term below 2^-62.  Six FP64
// operations, one unit in the last place; r2 outside the seed's range takes
// the library rsqrt, and r2 == 0 gives 0 when ZERO_SOFT (a body on itself or
// on another).
template <bool ZERO_SOFT>
__device__ __forceinline__ double inv_cube(double r2)
{
    double y;
    if (rsqrt_seed(r2, y)) {
        const double z = y * y;  // exact
        const double e = fma(-r2, z, 1.0);
        const double y3 = z * y;
        return fma(y3 * e, fma(e, 1.875, 1.5), y3);
    }
    double inv = rsqrt(r2);
    if (ZERO_SOFT) inv = r2 > 0.0 ? inv : 0.0;
    return inv * inv * inv;
}

// r2^(-1/2): y (1 + e/2 + 3/8 e^2), five FP64 operations.
__device__ __forceinline__ double inv_sqrt(double r2)
{
    double y;
    if (rsqrt_seed(r2, y)) {
        const double e = fma(-r2, y * y, 1.0);
        return fma(y * e, fma(e, 0.375, 0.5), y);
    }
    return 1.0 / sqrt(r2);
}

} // namespace nb
