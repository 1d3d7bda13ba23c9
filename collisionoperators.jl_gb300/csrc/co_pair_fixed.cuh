// co_pair_fixed.cuh -- the Landau pair term in 64-bit fixed point.
//
// Formats (see co_pair_fixed.cu for the scaling that produces them):
//   coordinate  X = x' 2^61, |x'| < 1           (two's complement, 64 bits)
//   gradient    G = G' 2^60 = gh 2^31 + gl,     |G'| < 1, |gl| <= 2^30
//   weight      w = w' 2^61, |w'| <= 1
// and what the rounding of X and G left, in units of 2^-32 of theirs (32 bits)
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

// A difference (of coordinates or gradients) shifted left until its larger component
// fills 61 bits
struct fx_diff {
    fx_limb c1, c2;   // normalised, base 2^31, half the shifted value
    int s;            // the shift
    float m;          // size of the unshifted larger component (2^29 for 2^61)
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
FXF int fx_shift_of(float m) {   // 29 - exponent
#ifdef __CUDA_ARCH__
    const uint32_t b = __float_as_uint(m);
#else
    uint32_t b;
    memcpy(&b, &m, 4);
#endif
    return (int)((0x4e7fffffu - b) >> 23);
}
FXF float fx_size(fx64 D1, fx64 D2) {
    return fmaxf(fabsf(fx_i2f(fx_hi(D1))), fabsf(fx_i2f(fx_hi(D2))));
}
FXF fx_diff fx_norm(fx64 D1, fx64 D2) {
    const float m = fx_size(D1, D2);
    const int s = fx_shift_of(m);
    return {fx_shl(D1, s), fx_shl(D2, s), s, m};
}

// 96-bit value h + l 2^-32
struct fx96 {
    fx64 h;
    uint32_t l;
};
// difference of the rounded words and of what their rounding left
FXF fx96 fx_sub96(fx64 D, int32_t ra, int32_t rg) {
    const fx64 r = (fx64)ra - rg;
    return {D + (r >> 32), fx_lo(r)};
}
FXF fx_limb fx_shl(fx96 d, int s) {   // 0 <= s < 32
#ifdef __CUDA_ARCH__
    const uint32_t l = __funnelshift_l(d.l, fx_lo(d.h), s);
    return {(int32_t)__funnelshift_l(fx_lo(d.h), (uint32_t)fx_hi(d.h), s), (int32_t)(l >> 1)};
#else
    const fxu64 x = ((fxu64)d.h << s) | (((fxu64)d.l << s) >> 32);
    return {fx_hi((fx64)x), (int32_t)(fx_lo((fx64)x) >> 1)};
#endif
}
FXF fx_diff fx_norm(fx96 D1, fx96 D2) {
    const float m = fx_size(D1.h, D2.h);
    const int s = fx_shift_of(m);
    return {fx_shl(D1, s), fx_shl(D2, s), s, m};
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
    const int32_t P = fx_hi(fx_mad(e, 1920, (1ll << 31) - (3ll << 61)));       // (-3/2 + 15/8 e) 2^30
    const int32_t c = fx_mid(fx_mad(e, P, 1ll << 29), 30);         // c 2^52
    // y (1 + c), then times y^2: c enters at y, which has all its bits in 31 (taken to the
    // upper half of y^3, 26 bits where that is small, it left errors of up to 55 units of
    // 2^-53; 3.3 so, 1.1 in the mean)
    const fxu64 T = ((fxu64)Y << 32) + (fxu64)(fx_mad((int32_t)(Y >> 1), c, 0) >> 19);
    const fxu64 Q = fx_madu(Y, Y, 0);
    const fxu64 q = fx_madu((uint32_t)(Q >> 32), (uint32_t)T, 0);
    return fx_split((fx64)fx_mulu(Q, (uint32_t)(T >> 32), q));
}

// C = K1 D2 + nK2 D1 (nK2 = G_g2 - G_a2), times 2^-62
FXF fx64 fx_cross(const fx_limb &k1, const fx_limb &k2, const fx_limb &d1, const fx_limb &d2) {
    fx64 x = fx_mad(k1.h, d2.l, 1ll << 30);
    x = fx_mad(k1.l, d2.h, x);
    x = fx_mad(k2.h, d1.l, x);
    x = fx_mad(k2.l, d1.h, x);
    fx64 C = fx_mad(k1.h, d2.h, 0);
    C = fx_mad(k2.h, d1.h, C);
    return fx_mad(fx_hi(x), 2, C);
}
// -2^n <= a, b < 2^n
FXF bool fx_within(int32_t a, int32_t b, int n) {
    return (((uint32_t)(a + (1 << n)) | (uint32_t)(b + (1 << n))) >> (n + 1)) == 0;
}
// |wa| or |wt| below 2^-8
FXF bool fx_light(fx64 wa, fx64 wt) {
    return (uint32_t)(fx_hi(wa) + (1 << 21)) < (1u << 22) ||
           (uint32_t)(fx_hi(wt) + (1 << 21)) < (1u << 22);
}
FXF fx64 fx_join(const fx_limb &a) { return ((fx64)a.h << 31) + a.l; }

// A pair's differences from all 96 bits, K normalised like D, so that the error of its
// terms is relative to its own |d| and |g|. K's shift stays below D's, sf = d.s + 1 - it:
// terms are then no finer than the unit their sums have, 2^-57 of the scales.
struct fx_fine {
    fx_diff d;
    fx_limb k1, k2;
    int sf;   // shift of the terms of S
};
FXF fx_fine fx_refine(fx96 D1, fx96 D2, fx96 K1, fx96 K2) {
    fx_fine p;
    p.d = fx_norm(D1, D2);
    const int k = fx_shift_of(fx_size(K1.h, K2.h)), s = k < p.d.s + 1 ? k : p.d.s + 1;
    p.k1 = fx_shl(K1, s);
    p.k2 = fx_shl(K2, s);
    p.sf = p.d.s + 1 - s;
    return p;
}
// the same from the rounded words alone
FXF fx_fine fx_plain(fx64 D1, fx64 D2, const fx_limb &k1, const fx_limb &k2) {
    const fx_diff d = fx_norm(D1, D2);
    return {d, k1, k2, d.s};
}
