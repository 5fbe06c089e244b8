// Arithmetic on 8-byte lanes: one column in FP64, two neighbouring columns in FP32 (the .f32x2
// instructions: one issue slot for both, each rounded as the scalar operation).
#pragma once

namespace a43g {

template <typename T> struct LaneOf;
template <> struct LaneOf<double> { using V = double; };
template <> struct LaneOf<float> { using V = unsigned long long; };

__device__ __forceinline__ double vfma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ unsigned long long vfma(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ double vmul(double a, double b) { return a*b; }
__device__ __forceinline__ unsigned long long vmul(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ double vadd(double a, double b) { return a + b; }
__device__ __forceinline__ unsigned long long vadd(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ double vdup(double a) { return a; }
__device__ __forceinline__ unsigned long long vdup(float a) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(a));
    return d;
}

} // namespace a43g
