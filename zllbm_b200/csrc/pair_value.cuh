// A pair of nodes' values in packed FP32 registers (fma.rn.f32x2 and friends, sm_100): the second value
// type of fused_collide.cuh.
#pragma once
#include "fused_collide.cuh"

namespace zl {

struct F2 {
    float2 v;
};
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return {__fadd2_rn(a.v, b.v)}; }
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return {__ffma2_rn(b.v, make_float2(-1.f, -1.f), a.v)}; }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return {__fmul2_rn(a.v, b.v)}; }
__device__ __forceinline__ F2 vfma(F2 a, F2 b, F2 c) { return {__ffma2_rn(a.v, b.v, c.v)}; }

__device__ __forceinline__ F2 neg(F2 a) { return F2{make_float2(0.f, 0.f)} - a; }  // (0 - a: a zero's sign aside)

template <> __device__ __forceinline__ F2 splat_as<F2>(float s) { return {make_float2(s, s)}; }
__device__ __forceinline__ F2 splat(float s) { return splat_as<F2>(s); }

// fn applied to every element
template <class Fn> __device__ __forceinline__ F2 each(F2 a, Fn fn) { return {make_float2(fn(a.v.x), fn(a.v.y))}; }

__device__ __forceinline__ F2 smag_omega(F2 pi2, F2 c, float tau0) {
    return {make_float2(smag_omega(pi2.v.x, c.v.x, tau0), smag_omega(pi2.v.y, c.v.y, tau0))};
}

}  // namespace zl
