// nb_after.cuh -- what a force kernel does with a body's acceleration once it
// has it: the integrator's next update of that body (AfterForce, nb_internal.h).
//
// An update reads and writes one body, so the thread that finishes an
// acceleration can apply it, and the launch of its own that it took, with the gap
// before it and its trip to memory, goes.  Those launches bound the smallest
// systems: a velocity-Verlet step at n = 1000 went from 32.5 to 30.7 us, an
// RK4 step at n = 5003 from 139 to 109 us, a leapfrog step in FP64 at n = 100 / 1024
// from 17.1 / 43.0 to 14.9 / 38.9 us.
// The updates restate the reference's with its operation order (nb_integrate.cu)
// in round-to-nearest operations that no compiler fuses.
#pragma once

#include "nb_internal.h"

namespace nb {

// One component of a body's position, split for the mixed kernels (split_kernel).
__device__ __forceinline__ void split_component(float4 *hi, float4 *lo, const double *m, int c,
                                                int i, double v)
{
    const float h = __double2float_rn(v);
    reinterpret_cast<float *>(hi + i)[c] = h;
    reinterpret_cast<float *>(lo + i)[c] = __double2float_rn(v - (double)h);
    if (c == 0) {
        hi[i].w = __double2float_rn(m[i]);
        lo[i].w = 0.0f;
    }
}

// Component c of body i has acceleration a (already stored).
__device__ __forceinline__ void after_force(const AfterForce &t, int c, int i, double a)
{
    switch (t.kind) {
    case AfterForce::kKick:  // v += a dt/2
        t.v[c][i] = __dadd_rn(t.v[c][i], __dmul_rn(a, t.h));
        break;
    case AfterForce::kKickMean:  // v += (a_old + a) * (0.5 dt)
        t.v[c][i] = __dadd_rn(t.v[c][i], __dmul_rn(__dadd_rn(t.a0[c][i], a), t.h));
        break;
    case AfterForce::kStage: {  // pos = x + kv*h ; vel = v + ka*h
        const double p = __dadd_rn(t.x0[c][i], __dmul_rn(t.kv[c][i], t.h));
        t.x[c][i] = p;
        t.v[c][i] = __dadd_rn(t.v0[c][i], __dmul_rn(a, t.h));
        if (t.hi) split_component(t.hi, t.lo, t.m, c, i, p);
        break;
    }
    case AfterForce::kFinish: {  // rk4_combine_kernel; a is the last stage's
        const double v = t.v[c][i];
        const double sv =
            __dadd_rn(__dadd_rn(__dadd_rn(v, __dmul_rn(t.k2[(3 + c) * t.ps + i], 2.0)),
                                __dmul_rn(t.k3[(3 + c) * t.ps + i], 2.0)),
                      t.kv[c][i]);
        const double sa =
            __dadd_rn(__dadd_rn(__dadd_rn(t.a0[c][i], __dmul_rn(t.k2[(6 + c) * t.ps + i], 2.0)),
                                __dmul_rn(t.k3[(6 + c) * t.ps + i], 2.0)),
                      a);
        t.x[c][i] = __dadd_rn(t.x[c][i], __dmul_rn(sv, t.h));
        t.v[c][i] = __dadd_rn(v, __dmul_rn(sa, t.h));
        break;
    }
    default: break;
    }
}

} // namespace nb
