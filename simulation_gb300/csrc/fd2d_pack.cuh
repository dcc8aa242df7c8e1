// Four cells of a lane as two packed FP32 pairs (f32x2 instructions: two
// operations to an issue slot, each rounded as the scalar one), for the 2D
// kernels that hold four columns per lane.
#pragma once

#include <cuda_runtime.h>

namespace fdtd {
namespace {

// A packed product is not added with add4: the compiler joins the two to one
// fma, which rounds a subnormal 0.5*x differently.  x + 0.5*y is written
// sub4(x, mul4(-0.5f, y)).
struct F4 {  // four cells of a lane as two packed pairs
  float2 a, b;
};
__device__ __forceinline__ float2 bc2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 sub2(float2 x, float2 y) { return __ffma2_rn(y, bc2(-1.f), x); }  // x - y, rounded once
__device__ __forceinline__ F4 f4(float4 v) { return {make_float2(v.x, v.y), make_float2(v.z, v.w)}; }
__device__ __forceinline__ float4 to4(const F4& v) { return make_float4(v.a.x, v.a.y, v.b.x, v.b.y); }
__device__ __forceinline__ F4 sub4(const F4& x, const F4& y) { return {sub2(x.a, y.a), sub2(x.b, y.b)}; }
__device__ __forceinline__ F4 add4(const F4& x, const F4& y) { return {__fadd2_rn(x.a, y.a), __fadd2_rn(x.b, y.b)}; }
__device__ __forceinline__ F4 mul4(const F4& x, const F4& y) { return {__fmul2_rn(x.a, y.a), __fmul2_rn(x.b, y.b)}; }
__device__ __forceinline__ F4 mul4(float s, const F4& y) { return {__fmul2_rn(bc2(s), y.a), __fmul2_rn(bc2(s), y.b)}; }
__device__ __forceinline__ F4 fma4(const F4& x, const F4& y, const F4& z) {
  return {__ffma2_rn(x.a, y.a, z.a), __ffma2_rn(x.b, y.b, z.b)};
}
__device__ __forceinline__ F4 mul4(float2 s, const F4& y) { return {__fmul2_rn(s, y.a), __fmul2_rn(s, y.b)}; }
__device__ __forceinline__ F4 fma4(float2 s, const F4& y, const F4& z) {
  return {__ffma2_rn(s, y.a, z.a), __ffma2_rn(s, y.b, z.b)};
}
__device__ __forceinline__ F4 fma4(float s, const F4& y, const F4& z) {
  return {__ffma2_rn(bc2(s), y.a, z.a), __ffma2_rn(bc2(s), y.b, z.b)};
}

}  // namespace
}  // namespace fdtd
