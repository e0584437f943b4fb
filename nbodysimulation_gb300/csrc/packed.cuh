// packed.cuh -- packed FP32 arithmetic (add / mul / fma.rn.f32x2: two FP32
// operations per instruction, each rounded as the scalar one) for the pair
// sums of the force walk and the direct sums.
//
// Throughput measured on a GB300 in issue cycles per warp: packed add or
// multiply 2.03, packed FMA 2.01 with two different register pairs, 2.86 with
// three (the register file delivers one pair a cycle), 2.4 when consecutive
// ones share an operand; scalar FADD 1.08, FFMA 1.08 to 1.41 by the same
// count.  Packing saves issue slots for the rest of a loop, not FP32 pipe
// cycles.
#pragma once
#include "nbgb_internal.cuh"

namespace nbgb {

__device__ __forceinline__ float2 dup(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 lo2(const float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4 v) { return make_float2(v.z, v.w); }

__device__ __forceinline__ float2 pair_dist2(const float2 dx, const float2 dy, const float2 dz, float2 eps2) {
    return __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, eps2)));
}

}  // namespace nbgb
