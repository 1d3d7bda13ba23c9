// co_pair_fixed.cuh -- the Landau pair term in 64-bit fixed point.
//
// Formats (see co_pair_fixed.cu for the scaling that produces them):
//   coordinate  X = x' 2^61, |x'| < 1           (two's complement, 64 bits)
//   gradient    G = G' 2^60 = gh 2^31 + gl,     |G'| < 1, |gl| <= 2^30
//   weight      w = w' 2^61, |w'| <= 1
// A 64-bit product's high part comes from 32 x 32 -> 64 multiply-adds (one
// IMAD.WIDE each) on limbs of base 2^31, whose cross terms fit a signed 64-bit
// sum without a carry. Right shifts of cross terms round to nearest: the added
// half unit is the constant the first multiply-add starts from.
#pragma once
#include <stdint.h>
#ifdef __CUDACC__
#define FXF __host__ __device__ __forceinline__
#else
#define FXF static inline
#endif

typedef long long fx64;
typedef unsigned long long fxu64;

FXF fx64 fx_mad(int32_t a, int32_t b, fx64 c) { return (fx64)a * b + c; }
FXF fxu64 fx_madu(uint32_t a, uint32_t b, fxu64 c) { return (fxu64)a * b + c; }
FXF int32_t fx_hi(fx64 a) { return (int32_t)(a >> 32); }
FXF uint32_t fx_lo(fx64 a) { return (uint32_t)a; }
// bits [n, n + 32) of a, 0 < n < 32
FXF int32_t fx_mid(fx64 a, int n) {
#ifdef __CUDA_ARCH__
    return (int32_t)__funnelshift_r(fx_lo(a), (uint32_t)fx_hi(a), n);
#else
    return (int32_t)(a >> n);
#endif
}
// base-2^31 limbs of a 64-bit value below 2^62
struct fx_limb {
    int32_t h, l;   // value = h 2^31 + l, 0 <= l < 2^31
};
FXF fx_limb fx_split(fx64 a) { return {fx_mid(a, 31), (int32_t)(fx_lo(a) & 0x7fffffffu)}; }
// a b 2^-62, rounded to within one unit. The product of the low limbs is left out:
// between 0 and 1 unit, 1/4 on average, which the rounding constant carries (left
// uncorrected, the offset of S shows as 3e-16 in sums with unequal weights)
FXF fx64 fx_mul(fx_limb a, fx_limb b) {
    fx64 x = fx_mad(a.h, b.l, (1ll << 30) + (1ll << 29));
    x = fx_mad(a.l, b.h, x);
    return fx_mad(fx_mid(x, 31), 1, fx_mad(a.h, b.h, 0));
}
// limbs of 2^k a, for a below 2^(62 - k): k more significant bits in the product
template <int k>
FXF fx_limb fx_split_up(fx64 a) {
    return {fx_mid(a, 31 - k), (int32_t)((fx_lo(a) << k) & 0x7fffffffu)};
}
// a (64 bits, unsigned) times b (32 bits) 2^-32, plus c 2^-32
FXF fxu64 fx_mulu(fxu64 a, uint32_t b, fxu64 c) {
    return fx_madu((uint32_t)(a >> 32), b, fx_madu((uint32_t)a, b, c) >> 32);
}

// float of an int and the seed of 1/sqrt, as the device forms them
FXF float fx_i2f(int32_t a) { return (float)a; }
FXF uint32_t fx_seed(int32_t rhi) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"((float)rhi));
    return __float2uint_rn(y * 0x1p44f);
#else
    return (uint32_t)lrintf(1.0f / sqrtf((float)rhi) * 0x1p44f);
#endif
}

// D = X_a - X_g shifted left until its larger component fills 61 bits
struct fx_dist {
    fx_limb d1, d2;   // normalised, base 2^31, half the shifted value
    int s;            // the shift
    float m;          // size of the unshifted larger component (2^29 for |D'| = 1)
};
FXF fx_limb fx_shl(fx64 d, int s) {
#ifdef __CUDA_ARCH__
    uint32_t l;   // defined for every s (the shift of a close pair is not used)
    asm("shl.b32 %0, %1, %2;" : "=r"(l) : "r"(fx_lo(d)), "r"(s));
    return {(int32_t)__funnelshift_l(fx_lo(d), (uint32_t)fx_hi(d), s), (int32_t)(l >> 1)};
#else
    const fx64 x = (fx64)((fxu64)d << s);
    return {fx_hi(x), (int32_t)(fx_lo(x) >> 1)};
#endif
}
FXF fx_dist fx_norm(fx64 D1, fx64 D2) {
    fx_dist r;
    const float f1 = fx_i2f(fx_hi(D1)), f2 = fx_i2f(fx_hi(D2));
    r.m = fmaxf(fabsf(f1), fabsf(f2));
#ifdef __CUDA_ARCH__
    r.s = (int)((0x4e7fffffu - __float_as_uint(r.m)) >> 23);   // 29 - exponent
#else
    uint32_t b;
    memcpy(&b, &r.m, 4);
    r.s = (int)((0x4e7fffffu - b) >> 23);
#endif
    r.d1 = fx_shl(D1, r.s);
    r.d2 = fx_shl(D2, r.s);
    return r;
}

// y3 = |d|^-3 of the normalised distance: y^3 2^58 (y = r^-1/2, r = d1^2 + d2^2
// of the normalised components in [1/4, 2))
FXF fx_limb fx_invcube(const fx_limb &d1, const fx_limb &d2) {
    // R = r 2^60
    fx64 x = fx_mad(d1.h, d1.l, 1ll << 31);
    x = fx_mad(d2.h, d2.l, x);
    fx64 R = fx_mad(d1.h, d1.h, 0);
    R = fx_mad(d2.h, d2.h, R);
    R = fx_mad(fx_hi(x), 4, R);
    const uint32_t Y = fx_seed(fx_hi(R));               // y 2^30, relative error 2^-22.7
    const fxu64 V = fx_mulu((fxu64)R, Y, 0);            // sqrt(r) 2^58
    const fxu64 W = fx_mulu(V, Y, 0x8c0000000ull);      // r Y^2: (1 + e) 2^56 + 8.75
    const int32_t e = fx_mid((fx64)W, 4);               // e 2^52, |e| < 2^-21.6
    // y^3 (1 + e)^-3/2 = y^3 (1 + c), c = e (-3/2 + 15/8 e) + O(e^3 ~ 2^-64)
    const int32_t P = fx_hi(fx_mad(e, 1920, -(3ll << 61)));       // (-3/2 + 15/8 e) 2^30
    const int32_t c = fx_mid(fx_mad(e, P, 1ll << 29), 30);         // c 2^52
    const fxu64 Q = fx_madu(Y, Y, 0);
    const fx64 Y3 = (fx64)fx_mulu(Q, Y, 0);             // Y^3 2^-32
    const fx64 w = fx_mad(fx_mid(Y3, 31), c, 1ll << 20);
    return fx_split(Y3 + (w >> 21));
}

// C = K1 D2 + nK2 D1 (nK2 = G_g2 - G_a2), times 2^-62
FXF fx64 fx_cross(int32_t k1h, int32_t k1l, int32_t k2h, int32_t k2l, const fx_limb &d1,
                  const fx_limb &d2) {
    fx64 x = fx_mad(k1h, d2.l, 1ll << 30);
    x = fx_mad(k1l, d2.h, x);
    x = fx_mad(k2h, d1.l, x);
    x = fx_mad(k2l, d1.h, x);
    fx64 C = fx_mad(k1h, d2.h, 0);
    C = fx_mad(k2h, d1.h, C);
    return fx_mad(fx_hi(x), 2, C);
}
