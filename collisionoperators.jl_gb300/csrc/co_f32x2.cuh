// co_f32x2.cuh -- packed FP32 arithmetic (two FP32 operations per instruction).
// Each half is rounded as the scalar instruction rounds it. Note that the compiler
// contracts a mul.rn.f32x2 whose result enters an add.rn.f32x2.
#pragma once

typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    return (f32x2)__float_as_uint(lo) | ((f32x2)__float_as_uint(hi) << 32);
}
__device__ __forceinline__ f32x2 dup2(float a) { return pack2(a, a); }
__device__ __forceinline__ float lo2(f32x2 a) { return __uint_as_float((unsigned)a); }
__device__ __forceinline__ float hi2(f32x2 a) { return __uint_as_float((unsigned)(a >> 32)); }
// 1/sqrt of a normal number (rsqrtf without its scaling of subnormal arguments)
__device__ __forceinline__ float rsqrt_normal(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// 1/|d| of both halves, 0 where |d|^2 < 1e-24
__device__ __forceinline__ f32x2 rsqrt_guard2(f32x2 r2) {
    const float a = lo2(r2), b = hi2(r2);
    const float ya = rsqrt_normal(a), yb = rsqrt_normal(b);
    return pack2(a >= 1e-24f ? ya : 0.f, b >= 1e-24f ? yb : 0.f);
}
__device__ __forceinline__ f32x2 neg2(f32x2 a) { return a ^ 0x8000000080000000ull; }
