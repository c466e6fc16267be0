// Four neighbouring floats at a time: loads, stores and the few operations the recurrences' tiles are made of.
#pragma once
#include <cuda_runtime.h>

namespace mdma {

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }
// c + a b, two numbers at a time: one instruction for two multiply-adds, each rounded as fmaf rounds it
__device__ __forceinline__ float2 fma2(const float2& a, const float2& b, const float2& c) {
    float2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(reinterpret_cast<unsigned long long&>(r))
        : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)), "l"(reinterpret_cast<const unsigned long long&>(c)));
    return r;
}
__device__ __forceinline__ void fma4(float4& acc, float a, const float4& b) {
    const float2 aa = make_float2(a, a), lo = fma2(aa, make_float2(b.x, b.y), make_float2(acc.x, acc.y)),
                 hi = fma2(aa, make_float2(b.z, b.w), make_float2(acc.z, acc.w));
    acc = make_float4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ void scale4(float4& v, float a) { v.x *= a; v.y *= a; v.z *= a; v.w *= a; }
__device__ __forceinline__ float dot4(const float4& a, const float4& b, float acc) {
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc))));
}
// the same as two sums, of the even and of the odd places
__device__ __forceinline__ void dot4(float2& acc, const float4& a, const float4& b) {
    acc = fma2(make_float2(a.z, a.w), make_float2(b.z, b.w), fma2(make_float2(a.x, a.y), make_float2(b.x, b.y), acc));
}

}  // namespace mdma
