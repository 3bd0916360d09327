// Scalar and complex arithmetic shared by the stencil and nonlocal kernels.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace lynxb {

template <typename T> struct ScalarOf;
template <> struct ScalarOf<double> { using type = double; static constexpr bool cplx = false; };
template <> struct ScalarOf<float> { using type = float; static constexpr bool cplx = false; };
template <> struct ScalarOf<double2> { using type = double; static constexpr bool cplx = true; };
template <> struct ScalarOf<float2> { using type = float; static constexpr bool cplx = true; };

__device__ __forceinline__ double vzero(double) { return 0.0; }
__device__ __forceinline__ float vzero(float) { return 0.0f; }
__device__ __forceinline__ double2 vzero(double2) { return make_double2(0.0, 0.0); }
__device__ __forceinline__ float2 vzero(float2) { return make_float2(0.0f, 0.0f); }

// acc + c * v  (c real)
__device__ __forceinline__ double fmac(double acc, double c, double v) { return fma(c, v, acc); }
__device__ __forceinline__ float fmac(float acc, float c, float v) { return fmaf(c, v, acc); }
__device__ __forceinline__ double2 fmac(double2 acc, double c, double2 v) {
    return make_double2(fma(c, v.x, acc.x), fma(c, v.y, acc.y));
}
__device__ __forceinline__ float2 fmac(float2 acc, float c, float2 v) {
    return make_float2(fmaf(c, v.x, acc.x), fmaf(c, v.y, acc.y));
}
__device__ __forceinline__ double vadd(double a, double b) { return a + b; }
__device__ __forceinline__ float vadd(float a, float b) { return a + b; }
__device__ __forceinline__ double2 vadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double vscale(double c, double v) { return c * v; }
__device__ __forceinline__ float vscale(float c, float v) { return c * v; }
__device__ __forceinline__ double2 vscale(double c, double2 v) { return make_double2(c * v.x, c * v.y); }
__device__ __forceinline__ float2 vscale(float c, float2 v) { return make_float2(c * v.x, c * v.y); }
// v * ph: real phase for real data, complex product for complex data.
__device__ __forceinline__ double pmul(double v, double ph) { return v * ph; }
__device__ __forceinline__ float pmul(float v, float ph) { return v * ph; }
__device__ __forceinline__ double2 pmul(double2 v, double2 ph) {
    return make_double2(v.x * ph.x - v.y * ph.y, v.x * ph.y + v.y * ph.x);
}
__device__ __forceinline__ float2 pmul(float2 v, float2 ph) {
    return make_float2(v.x * ph.x - v.y * ph.y, v.x * ph.y + v.y * ph.x);
}

}  // namespace lynxb
