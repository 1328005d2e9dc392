// ff.cuh -- float-float arithmetic: a value is an FP32 pair hi + lo with |lo| <= ulp(hi)/2,
// about 48 significant bits, formed with error-free FP32 transformations. Compiled
// without contraction (the FMAs are explicit); the CPU compiles it too
// (tests/ff_host.cpp).
#pragma once

namespace falcon {
namespace sv {

__device__ __forceinline__ float2 ff_quick(float s, float e) {
    const float h = s + e;
    return make_float2(h, e - (h - s));
}
__device__ __forceinline__ float2 ff_two_sum(float a, float b) {
    const float s = a + b;
    const float bb = s - a;
    return make_float2(s, (a - (s - bb)) + (b - bb));
}
__device__ __forceinline__ float2 ff_add(float2 a, float2 b) {
    float2 s = ff_two_sum(a.x, b.x);
    const float2 t = ff_two_sum(a.y, b.y);
    s.y += t.x;
    s = ff_quick(s.x, s.y);
    s.y += t.y;
    return ff_quick(s.x, s.y);
}
__device__ __forceinline__ float2 ff_mul(float2 a, float2 b) {
    const float p = a.x * b.x;
    float e = fmaf(a.x, b.x, -p);
    e = fmaf(a.x, b.y, e);
    e = fmaf(a.y, b.x, e);
    return ff_quick(p, e);
}
__device__ __forceinline__ float2 ff_neg(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 ff_from(double v) {   // a few FP64 operations: per thread, not per cell
    const float h = (float)v;
    return make_float2(h, (float)(v - (double)h));
}
__device__ __forceinline__ double ff_to(float2 a) { return (double)a.x + (double)a.y; }

// Sums of products. Compensated sums (Ogita, Rump and Oishi's Dot2) take a third of the
// instructions, but lose up to five times as much: their error term is one FP32 number.
// In the operator and the dot products they gained 0.1 of 11.9 ms of a 6.3M-cell solve.
struct FFSum {
    float2 v = make_float2(0.f, 0.f);
    __device__ __forceinline__ void add(float2 a, float2 b) { v = ff_add(v, ff_mul(a, b)); }
    __device__ __forceinline__ float2 value() const { return v; }
};

}  // namespace sv
}  // namespace falcon
