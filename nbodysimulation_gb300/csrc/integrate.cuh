// integrate.cuh -- the integrators, applied to one body by the kernels that
// finish its acceleration (kernels/brute_force_update.cl:62-104,
// kernels/calculate_forces.cl:152-181).
#pragma once
#include "nbgb_internal.cuh"

namespace nbgb {

template <int kMethod>
__device__ __forceinline__ void integrate_body(const DevSim &s, const StepParams &p, int b, const float4 P, float ax,
                                               float ay, float az) {
    const float dt = p.dt;
    const float4 v = s.vel[b];
    float4 x = P, vo = v;
    if constexpr (kMethod == 2) {  // Euler (calculate_forces.cl:168-181)
        vo.x = __fadd_rn(v.x, __fmul_rn(ax, dt));
        vo.y = __fadd_rn(v.y, __fmul_rn(ay, dt));
        vo.z = __fadd_rn(v.z, __fmul_rn(az, dt));
        x.x = __fadd_rn(P.x, __fmul_rn(vo.x, dt));
        x.y = __fadd_rn(P.y, __fmul_rn(vo.y, dt));
        x.z = __fadd_rn(P.z, __fmul_rn(vo.z, dt));
        s.acc[b] = make_float4(ax, ay, az, 0.0f);
    } else if constexpr (kMethod == 1) {  // "Leapfrog" as written (:152-167): acc read, not written
        const float4 ap = s.acc[b];
        const float hx = __fadd_rn(v.x, __fmul_rn(__fmul_rn(ap.x, dt), 0.5f));
        const float hy = __fadd_rn(v.y, __fmul_rn(__fmul_rn(ap.y, dt), 0.5f));
        const float hz = __fadd_rn(v.z, __fmul_rn(__fmul_rn(ap.z, dt), 0.5f));
        x.x = __fadd_rn(P.x, __fmul_rn(hx, dt));
        x.y = __fadd_rn(P.y, __fmul_rn(hy, dt));
        x.z = __fadd_rn(P.z, __fmul_rn(hz, dt));
        vo.x = __fadd_rn(hx, __fmul_rn(__fmul_rn(ax, dt), 0.5f));
        vo.y = __fadd_rn(hy, __fmul_rn(__fmul_rn(ay, dt), 0.5f));
        vo.z = __fadd_rn(hz, __fmul_rn(__fmul_rn(az, dt), 0.5f));
    } else if constexpr (kMethod == 3) {  // kick-drift-kick, velocities at half steps
        const float h = p.kdk_primed ? dt : __fmul_rn(dt, 0.5f);
        vo.x = __fadd_rn(v.x, __fmul_rn(ax, h));
        vo.y = __fadd_rn(v.y, __fmul_rn(ay, h));
        vo.z = __fadd_rn(v.z, __fmul_rn(az, h));
        x.x = __fadd_rn(P.x, __fmul_rn(vo.x, dt));
        x.y = __fadd_rn(P.y, __fmul_rn(vo.y, dt));
        x.z = __fadd_rn(P.z, __fmul_rn(vo.z, dt));
        s.acc[b] = make_float4(ax, ay, az, 0.0f);
    } else {  // any other method value moves nothing (the as-wired reference)
    }
    s.vel[b] = vo;
    s.body_next[b] = x;
}

// the same with the method chosen at run time (epilogues that run once a body)
__device__ __forceinline__ void integrate_any(const DevSim &s, const StepParams &p, int b, const float4 P, float ax,
                                              float ay, float az) {
    switch (p.method) {
    case 1: integrate_body<1>(s, p, b, P, ax, ay, az); break;
    case 2: integrate_body<2>(s, p, b, P, ax, ay, az); break;
    case 3: integrate_body<3>(s, p, b, P, ax, ay, az); break;
    default: integrate_body<0>(s, p, b, P, ax, ay, az); break;
    }
}

}  // namespace nbgb
