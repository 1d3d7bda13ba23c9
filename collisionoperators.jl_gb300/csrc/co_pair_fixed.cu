// co_pair_fixed.cu -- the Landau pair sum (functions.jl:205-237) at FP64 accuracy
// on the integer pipes.
//
// GB300 issues FP64 at 1/64 of the FP32 rate: the 20 FP64 instructions of a pair
// take 10 clocks of an SM per lane. 32 x 32 -> 64-bit multiply-adds run at 64
// lanes per clock, beside 128 lanes of 32-bit adds, so the pair term is evaluated
// in 64-bit fixed point (co_pair_fixed.cuh): 35 wide multiply-adds, which issue at
// about 32 lanes per clock where they have distinct operands, and some 140 adds,
// shifts and moves. What bounds it is that multiply pipe (78 % busy) with the issue
// slots (64 %): 2.0 clocks per pair and SM lane. At 131,072 markers (8.6e9 pairs) the
// sum takes 59 ms against 352 for the FP64 kernel it replaces, at 16,384 0.97 against
// 6.4; F with the metric at 10,000 markers 0.71 against 6.4 (one-sided FP64).
// Measured error of vdot and of the metric (2-norm, against 80-bit sums): 1.1e-16 to
// 1.2e-16 for 600 to 10,000 markers, the rounding of the results; the FP64 kernels' is
// 2.8e-16 to 5.6e-16 for vdot and 2.3e-16 to 4.6e-16 for the metric.
//
// Operands (k_pair_fixed_pack). Exact scalings by powers of two bring every
// coordinate below 1 in units of 2^-61 and every G in units of 2^-60; what that
// rounding leaves of a value (any of its bits may lie below) is kept in a third word.
// Differences are exact integer subtractions.
//
// Pair term. In two dimensions the projection of g = G_a - G_g off
// d = x_g - x_a is c (d2, -d1) / |d|^2 with c = g1 d2 - g2 d1, so the term is
// s (d2, -d1) with s = c / |d|^3: the same as functions.jl:221-231 in exact
// arithmetic. d is shifted left until it fills its word (float exponent of the
// larger component); 1/|d|^3 starts from the MUFU seed y of 1/sqrt(r) and takes
// y^3 (1 - 3e/2 + 15 e^2/8), e = r y^2 - 1, in integers. A term carries an error
// of about 1.2e-16 of |g|/|d| (4e-16 at most; FP64 arithmetic: 2-3e-16), unbiased, and the
// sums of terms are exact integers, converted to FP64 once per tile pair.
//
// Small differences: the rounding of the two-word operands is 2^-53 of a difference that
// is 2^-8 of the scale. A pair with |d| below 2^-9 of the scaled domain or |g| below
// 2^-9 of the largest G is taken from all three words, g shifted left like d
// (fx_refine), so that its error is relative to its own |d| and |g|: less than one pair
// in a hundred in the distributions of the performance cases. The bounds of 32 targets and
// 32 sources pick one of three loops: neither can be small (80 % of the group pairs for a
// smooth G, 2 to 20 % where the largest G is 25 to 40 times the median), only |g| can, or
// |d| can, the only one with the FP64 form. 131,072 markers: 57.9 ms; 58.7 with two words
// for every pair, 62.3 with the test in every loop, 67.2 with three words for every pair
// (59.0 now, with c at y in fx_invcube).
// A map of 16,384 markers with strong outliers in G: 1.13 ms with two words for every pair,
// 1.19 with one loop for both kinds of small pairs, 1.18 now.
//
// Close pairs: |d| < 2^-22 of the scaled domain (a few 1e-6 for [-6, 6]^2) take
// the FP64 form from the FP64 operands, including the |d|^2 < 1e-24 guard of
// functions.jl:224; that covers coincident markers. So do pairs with |d| below 2^-9 of it
// where a weight is below 2^-8 of the largest.
//
// The metric A = sum_a w_a U(v_g - v_a) of functions.jl:249-290 comes from the same
// evaluation: U = (d2, -d1) (d2, -d1)^T / |d|^3.
//
// Range: where the operands of a launch span too much for one scale (fixed_wide), the
// same tiles run the FP64 pair term (co_pair64.cuh) instead, on the device's own decision:
// 16,384 markers 5.8 ms, with the metric 9.2.
//
// Tiling: tiles of TS = 32 W sorted markers, W warps, one target per lane; tile
// pairs (I, I + k mod nt), k = 0..nt/2, so each unordered tile pair appears once
// and one evaluation serves both markers (Newton's third law). Within a warp,
// lane l meets source (l + q) mod 32 of a 32-source group at step q, and the
// source's accumulators pass to lane l - 1 by shuffles. Partials go to fixed slots
// and are added in a fixed order: bitwise reproducible.
#include "co_f32x2.cuh"
#include "co_internal.cuh"
#include "co_pair64.cuh"
#include "co_pair_fixed.cuh"

// 96-bit sum of terms T 2^s
struct fx_acc {
    uint32_t w0, w1, w2;
};
__device__ __forceinline__ void fx_acc_add(fx_acc &a, const fx_acc &t) {
    asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
        : "+r"(a.w0), "+r"(a.w1), "+r"(a.w2)
        : "r"(t.w0), "r"(t.w1), "r"(t.w2));
}
// T 2^s, 0 <= s < 32, rs = 32 - s
__device__ __forceinline__ fx_acc fx_shift96(fx64 T, int s, int rs) {
    fx_acc a;
    asm("shl.b32 %0, %1, %2;" : "=r"(a.w0) : "r"(fx_lo(T)), "r"(s));
    a.w1 = __funnelshift_l(fx_lo(T), (uint32_t)fx_hi(T), s);
    asm("shr.s32 %0, %1, %2;" : "=r"(a.w2) : "r"(fx_hi(T)), "r"(rs));
    return a;
}
__device__ __forceinline__ double fx_to_double(const fx_acc &a) {
    const fx64 hi = ((fx64)(int32_t)a.w2 << 32) | a.w1;
    return fma((double)hi, 4294967296.0, (double)a.w0);
}

// FP64 pair term of close pairs: u = U(d) g / |d| (0 for |d|^2 < 1e-24) and, for
// the metric, U(d) / |d|
struct close_term {
    double u1, u2, a11, a12, a22;
};
__device__ __forceinline__ close_term pair_close64(double2 xg, double2 Gg, double2 xa,
                                                   double2 Ga) {
    const double d1 = xg.x - xa.x, d2 = xg.y - xa.y;
    const double g1 = Ga.x - Gg.x, g2 = Ga.y - Gg.y;
    const double r2 = fma(d2, d2, d1 * d1);
    close_term t = {0.0, 0.0, 0.0, 0.0, 0.0};
    if (r2 < 1e-24) return t;
    const double ir = rsqrt(r2), ir2 = ir * ir, c = fma(d2, g2, d1 * g1) * ir2;
    t.u1 = fma(-d1, c, g1) * ir;
    t.u2 = fma(-d2, c, g2) * ir;
    t.a11 = fma(-d1 * d1, ir2, 1.0) * ir;
    t.a12 = -d1 * d2 * ir2 * ir;
    t.a22 = fma(-d2 * d2, ir2, 1.0) * ir;
    return t;
}

// T 2^s in units of 2^-58 (sums of s (d2, d1)) and 2^-59 (metric)
#define FX_UNIT_F 0x1p-58
#define FX_UNIT_A 0x1p-59

// Differences below 2^n in units of the high word (x: 2^29 is 1; G: 2^29 is 1): from
// three words
#define FX_SMALL_D 20
#define FX_SMALL_G 20

template <int W, int NC>
struct fixed_smem {
    longlong2 x[32 * W];
    int4 g[32 * W];            // g1h g1l g2h g2l
    fx64 w[32 * W];
    double acc[NC][32 * W];    // source-side sums of the tile pair
};

// the lane's target
struct fixed_target {
    longlong2 x;
    int4 g;
    fx64 w;
};

// The NC sums' terms of one pair, unsigned: S d2, S d1 and, for NC = 5, y3 d2 d2,
// y3 d1 d2, y3 d1 d1; S = C y3 with the weight of the pair's other marker unless
// UNI (all weights equal: the factor enters with the fold)
template <int NC, bool UNI>
__device__ __forceinline__ void fixed_terms(fx64 S, const fx_limb &y3, fx_limb w,
                                            const fx_diff &d, fx64 (&T)[NC]) {
    const fx_limb s = UNI ? fx_split_up<3>(S) : fx_split_up<1>(fx_mul(fx_split_up<3>(S), w));
    T[0] = fx_mul(s, d.c2);
    T[1] = fx_mul(s, d.c1);
    if (NC == 5) {
        const fx_limb yw = UNI ? y3 : fx_split_up<1>(fx_mul(y3, w));
        const fx_limb m2 = fx_split_up<2>(fx_mul(yw, d.c2));
        const fx_limb m1 = fx_split_up<2>(fx_mul(yw, d.c1));
        T[2] = fx_mul(m2, d.c2);
        T[3] = fx_mul(m2, d.c1);
        T[NC - 1] = fx_mul(m1, d.c1);
    }
}

// Whether any of 32 targets and 32 sources may differ by little, from the bounds of the high
// words (their difference is that of the values, or one less): 2 in x, 1 in G alone, 0 no
__device__ __forceinline__ int fixed_near(const co_fixed_ops &o, int gt, int gs) {
    const int4 l = o.box[2 * gt], h = o.box[2 * gt + 1], sl = o.box[2 * gs], sh = o.box[2 * gs + 1];
    const int x = max(max(sl.x - h.x, l.x - sh.x), max(sl.y - h.y, l.y - sh.y));
    const int g = max(max(sl.z - h.z, l.z - sh.z), max(sl.w - h.w, l.w - sh.w));
    return x < o.x_near ? 2 : g < (1 << FX_SMALL_G);
}

// 32 rotation steps: this warp's 32 targets against the 32 sources of group grp of
// tile J; SRC: the sources' sums too; NEAR: small differences among them (fixed_near).
// Signs are applied when the sums are written.
template <int W, int NC, bool SRC, bool UNI, int NEAR>
__device__ __forceinline__ void fixed_group(fixed_smem<W, NC> &sm, const co_fixed_ops &o,
                                            const fixed_target &t, int ig, int J, int grp,
                                            int lane, const double (&tf)[2], fx_acc (&a)[NC],
                                            double (&gd)[NC]) {
    constexpr int TS = 32 * W;
    fx_acc b[NC];
#pragma unroll
    for (int i = 0; i < NC; i++) b[i] = {0, 0, 0};
#pragma unroll 1
    for (int q = 0; q < 32; q++) {
        const int j = grp * 32 + ((lane + q) & 31);
        const longlong2 xa = sm.x[j];
        const int4 ga = sm.g[j];
        const fx_limb k1 = {ga.x - t.g.x, ga.y - t.g.y}, k2 = {t.g.z - ga.z, t.g.w - ga.w};
        fx_fine p = fx_plain(xa.x - t.x.x, xa.y - t.x.y, k1, k2);
        bool close = false;
        if (NEAR && ((NEAR == 2 && p.d.m < o.m_small) || fx_within(k1.h, k2.h, FX_SMALL_G))) {
            const int ia = J * TS + j;
            // a light weight's product is rounded to 2^-61 of the heaviest over |d|
            close = NEAR == 2 && (p.d.m < o.m_close ||
                                  (!UNI && p.d.m < o.m_small && fx_light(sm.w[j], t.w)));
            if (close) {
                const close_term c = pair_close64(o.px[ig], o.pg[ig], o.px[ia], o.pg[ia]);
                const double uf = o.unit[0], ua = o.unit[2];   // into scaled units
                const double v[5] = {c.u1 * uf, -c.u2 * uf, c.a11 * ua, -c.a12 * ua, c.a22 * ua};
#pragma unroll
                for (int i = 0; i < NC; i++) {
                    gd[i] = fma(v[i], o.pwn[ia], gd[i]);
                    if (SRC) sm.acc[i][j] = fma(v[i], o.pwn[ig], sm.acc[i][j]);
                }
            } else {
                const int4 ra = o.rest[ia], rt = o.rest[ig];
                p = fx_refine(fx_sub96(xa.x - t.x.x, ra.x, rt.x), fx_sub96(xa.y - t.x.y, ra.y, rt.y),
                              fx_sub96(fx_join(k1), ra.z, rt.z), fx_sub96(fx_join(k2), rt.w, ra.w));
            }
        }
        // the source's sum passes on: lane - 1 may add to it in the next step, and the
        // shuffles below do not order shared memory between lanes
        if (SRC && NEAR == 2) __syncwarp();
        const fx_limb y3 = fx_invcube(p.d.c1, p.d.c2);
        const fx64 S = fx_mul(fx_split(fx_cross(p.k1, p.k2, p.d.c1, p.d.c2)), y3);
        fx64 T[NC], U[NC];
        if (UNI) {
            fixed_terms<NC, true>(S, y3, {0, 0}, p.d, T);
        } else {   // T: times the source's weight, U: times the target's
            fixed_terms<NC, false>(S, y3, fx_split(sm.w[j]), p.d, T);
            if (SRC) fixed_terms<NC, false>(S, y3, fx_split(t.w), p.d, U);
        }
        const int src = (lane + 1) & 31;
#pragma unroll
        for (int i = 0; i < NC; i++) {
            const int s = i < 2 ? p.sf : p.d.s;
            const fx_acc q = fx_shift96(close ? 0 : T[i], s, 32 - s);
            fx_acc_add(a[i], q);
            if (SRC) {
                fx_acc_add(b[i], UNI ? q : fx_shift96(close ? 0 : U[i], s, 32 - s));
                b[i].w0 = __shfl_sync(0xffffffffu, b[i].w0, src);
                b[i].w1 = __shfl_sync(0xffffffffu, b[i].w1, src);
                b[i].w2 = __shfl_sync(0xffffffffu, b[i].w2, src);
            }
        }
    }
    if (SRC) {
        const int k = grp * 32 + lane;
#pragma unroll
        for (int i = 0; i < NC; i++) sm.acc[i][k] = fma(tf[i > 1], fx_to_double(b[i]), sm.acc[i][k]);
    }
}

// sign of sum i in the target's and the source's result
__device__ __forceinline__ double fixed_sign(int i, bool src) {
    return i == 0 ? (src ? -1.0 : 1.0) : i == 1 ? (src ? 1.0 : -1.0) : i == 3 ? -1.0 : 1.0;
}

// tile I against tiles I + k, k0 <= k < k1
template <int W, int NC>
__device__ __forceinline__ void fixed_item(fixed_smem<W, NC> &sm, const co_fixed_ops &o,
                                           const fixed_target &t, int nt, int H, int I, int k0,
                                           int k1, int ka, double *__restrict__ gp,
                                           double *__restrict__ apart) {
    constexpr int TS = 32 * W;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ig = I * TS + tid;
    // the equal-weight loop serves tile pairs whose markers all carry weight w0
    const fx64 w0 = o.w[(size_t)I * TS];
    const bool own = w0 != 0 && t.w == w0;
    double gd[NC];
#pragma unroll
    for (int i = 0; i < NC; i++) gd[i] = 0.0;
#pragma unroll 1
    for (int k = k0; k < k1; k++) {
        if (sym_skip(nt, H, I, k)) continue;
        int J = I + k;
        if (J >= nt) J -= nt;
        __syncthreads();
        sm.x[tid] = o.x[(size_t)J * TS + tid];
        sm.g[tid] = o.g[(size_t)J * TS + tid];
        const fx64 wj = o.w[(size_t)J * TS + tid];
        sm.w[tid] = wj;
#pragma unroll
        for (int i = 0; i < NC; i++) sm.acc[i][tid] = 0.0;
        const bool uni = __syncthreads_and(own && wj == w0) != 0;
        const double f = uni ? (double)w0 * 0x1p-61 : 1.0;
        const double tf[2] = {f * FX_UNIT_F, f * FX_UNIT_A};
        fx_acc a[NC];
#pragma unroll
        for (int i = 0; i < NC; i++) a[i] = {0, 0, 0};
        // diagonal tile (k = 0): every ordered pair, target side only
#pragma unroll 1
        for (int rr = 0; rr < W; rr++) {
            const int grp = (warp + rr) & (W - 1);
            if (k == 0) {
                if (uni) fixed_group<W, NC, false, true, 2>(sm, o, t, ig, J, grp, lane, tf, a, gd);
                else fixed_group<W, NC, false, false, 2>(sm, o, t, ig, J, grp, lane, tf, a, gd);
            } else {
                const int near = fixed_near(o, I * W + warp, J * W + grp);
                if (near == 2) {
                    if (uni) fixed_group<W, NC, true, true, 2>(sm, o, t, ig, J, grp, lane, tf, a, gd);
                    else fixed_group<W, NC, true, false, 2>(sm, o, t, ig, J, grp, lane, tf, a, gd);
                } else if (near) {
                    if (uni) fixed_group<W, NC, true, true, 1>(sm, o, t, ig, J, grp, lane, tf, a, gd);
                    else fixed_group<W, NC, true, false, 1>(sm, o, t, ig, J, grp, lane, tf, a, gd);
                } else {
                    if (uni) fixed_group<W, NC, true, true, 0>(sm, o, t, ig, J, grp, lane, tf, a, gd);
                    else fixed_group<W, NC, true, false, 0>(sm, o, t, ig, J, grp, lane, tf, a, gd);
                }
                __syncthreads();
            }
        }
        if (k > 0) {
            double *ap = apart + ((size_t)(k - ka) * nt + J) * NC * TS;
#pragma unroll
            for (int i = 0; i < NC; i++) ap[i * TS + tid] = fixed_sign(i, true) * sm.acc[i][tid];
        }
#pragma unroll
        for (int i = 0; i < NC; i++) gd[i] = fma(tf[i > 1], fx_to_double(a[i]), gd[i]);
    }
#pragma unroll
    for (int i = 0; i < NC; i++) gp[i * TS + tid] = fixed_sign(i, false) * gd[i];
}

template <int W, int NC>
__global__ void __launch_bounds__(32 * W, NC == 2 ? (W == 4 ? 7 : 25) : 16 / W)
k_pair_fixed_sym(const co_fixed_ops o, int nt, int H, int KC, int kb, int ke,
                 double *__restrict__ gpart, double *__restrict__ apart) {
    co_grid_wait();
    __shared__ union {
        fixed_smem<W, NC> f;
        sym64_smem<W, NC> d;
    } sm;
    const int I = blockIdx.x % nt, chunk = blockIdx.x / nt;
    const int k0 = kb + chunk * KC, k1 = min(ke, k0 + KC), ka = max(kb, 1);
    double *gp = gpart + ((size_t)chunk * nt + I) * 32 * W * NC;
    const int ig = I * 32 * W + threadIdx.x;
    const fixed_target t = {o.x[ig], o.g[ig], o.w[ig]};
    if (*o.wide) sym64_item<W, NC>(sm.d, o.px, o.pg, o.pw, nt, H, I, k0, k1, ka, gp, apart);
    else fixed_item<W, NC>(sm.f, o, t, nt, H, I, k0, k1, ka, gp, apart);
}

// The sums of the packed positions: the target-side partials of every chunk and
// the source-side partials of ka <= k < ke, in a fixed order, times the unit of the
// scaled operands; components 0, 1 to vdot and 2.. to A, added to what is there where
// add is set. FIXED_SL threads share a
// position (a slice of the rows each), so a small launch does not wait on one
// chain of loads, and the FP64 rounding of the sum grows with the slice's length
// instead of the row count.
#define FIXED_SL 8
template <int NC>
__global__ void __launch_bounds__(32 * FIXED_SL)
k_fixed_reduce(const double *__restrict__ gpart, const double *__restrict__ apart, int nt, int H,
               int nchunk, int ka, int ke, int TS, const double *__restrict__ unit,
               const int *__restrict__ wide, int add, double *__restrict__ pdot,
               double *__restrict__ pA, size_t ld) {
    co_grid_wait();
    __shared__ double sh[NC][FIXED_SL][33];
    const int lane = threadIdx.x & 31, sl = threadIdx.x >> 5;
    const int p = blockIdx.x * 32 + lane;          // TS is a multiple of 32
    const int K = p / TS, t = p - K * TS;
    // FP64 sums have no scale
    const double u = sl >= NC || *wide ? 1.0 : unit[sl < 2 ? 1 : 3];
    double s[NC];
#pragma unroll
    for (int i = 0; i < NC; i++) s[i] = 0.0;
    for (int c = sl; c < nchunk; c += FIXED_SL) {
        const double *gp = gpart + ((size_t)c * nt + K) * NC * TS + t;
#pragma unroll
        for (int i = 0; i < NC; i++) s[i] += gp[i * TS];
    }
#pragma unroll 4
    for (int k = ka + sl; k < ke; k += FIXED_SL) {
        int I = K - k;
        if (I < 0) I += nt;
        if (sym_skip(nt, H, I, k)) continue;
        const double *ap = apart + ((size_t)(k - ka) * nt + K) * NC * TS + t;
#pragma unroll
        for (int i = 0; i < NC; i++) s[i] += ap[i * TS];
    }
#pragma unroll
    for (int i = 0; i < NC; i++) sh[i][sl][lane] = s[i];
    __syncthreads();
    if (sl < NC) {
        double r = sh[sl][0][lane];
#pragma unroll
        for (int i = 1; i < FIXED_SL; i++) r += sh[sl][i][lane];
        double *d = sl < 2 ? pdot + (size_t)sl * ld + p : pA + (size_t)(sl - 2) * ld + p;
        *d = add ? fma(r, u, *d) : r * u;
    }
}

// ------------------------------------------------------------------ operands

// exponent E with x < 2^E (0 for x = 0), kept where 2^-E is a normal number
__device__ __forceinline__ int scale_exp(double x) {
    if (!(x > 0.0)) return 0;
    const int e = ilogb(x) + 1;
    return e < -1000 ? -1000 : (e > 1000 ? 1000 : e);
}

// Whether the fixed-point sums of a marker would be less accurate than FP64 ones. Their
// terms w |g| / |d| are accurate relative to |g| / |d|, but rounded to 2^-57 of the largest
// G and to 2^-61 of the largest weight, so one marker of a huge G, or of a weight far
// above the others', costs the sums of all others digits. Against that stands the sum
// itself, estimated from 64 of the sorted markers (scaled: largest G and weight about 1;
// 1/|d| counts up to 64, so that one close sample does not decide). The fixed-point form
// stays while w |g| / |d| is on average above 2^-6 of what the units stand for: its error
// is then below that of FP64 arithmetic for every marker (a weightless marker of |G| 2^k
// times the others: 2^-2 to 2^-5.5 and 0.1 to 0.7 times FP64's error for k = 0 to 5, 2^-6.4
// and 1.2 times for k = 6). Thermal distributions with the solver's own G: 2^-4 and more.
// Markers so close together in their domain that most pairs would be close ones are left
// to the FP64 loop too (half-width 1e6 for thermal width 1).
#define FIXED_SAMPLES 64
__device__ __forceinline__ bool fixed_wide(const float4 *sv, const float *swt, float x1, float x2,
                                           float G1, float G2, bool force) {
    float num = 0.f, gr = 0.f, wr = 0.f, rr = 0.f;
    int near = 0;
#pragma unroll 4
    for (int s = 0; s < FIXED_SAMPLES; s++) {
        const float4 v = sv[s];
        const float d1 = x1 - v.x, d2 = x2 - v.y, g1 = G1 - v.z, g2 = G2 - v.w;
        const float r2 = fmaf(d2, d2, d1 * d1);
        near += r2 < 0x1p-40f;
        const float r = r2 > 0.f ? fminf(rsqrt_normal(r2), 64.f) : 0.f;   // 0: the marker itself
        const float q = fmaxf(fabsf(g1), fabsf(g2)) * r;
        num = fmaf(swt[s], q, num);
        gr += q;
        wr = fmaf(swt[s], r, wr);
        rr += r;
    }
    const bool ok = (!force || num >= 0x1p-6f * (gr + FIXED_SAMPLES)) && wr >= 0x1p-6f * rr;
    return !ok || near > FIXED_SAMPLES / 8;
}

// a rounded to an integer, and what that leaves in units of 2^-32
__device__ __forceinline__ fx64 fx_round(double a, int &rest) {
    const double r = rint(a);
    rest = __double2int_rn((a - r) * 0x1p32);   // 2^31 saturates
    return __double2ll_rn(r);
}

// Fixed-point operands of the sorted markers from the FP64 packed arrays. Every
// block takes the maxima of |G| and |w| from the pack kernel's block partials
// (max is order-free), so the scales are one set for the launch. A non-finite operand (maximum inf) makes every
// vdot NaN, as the FP64 sum does. unit[0], unit[2]: FP64 terms of F and A into
// scaled units; unit[1], unit[3]: scaled sums back to vdot and A.
// Threads: the 60 FP64 operations and conversions of a marker queue on its SM's FP64 pipe, so
// blocks are small: at 2,048 markers 11.2 us with 256 threads, 7.7 with 64 (ncu, cold).
#define FIXED_PACK 64
static_assert(FIXED_PACK == FIXED_SAMPLES, "a sample per thread");
__global__ void __launch_bounds__(FIXED_PACK)
k_pair_fixed_pack(const double2 *__restrict__ px, const double2 *__restrict__ pg,
                  const double *__restrict__ pw, const int *__restrict__ Mp,
                  const double2 *__restrict__ part, int npart, int ex, double c1, double c2,
                  longlong2 *__restrict__ ox, int4 *__restrict__ og, int4 *__restrict__ rest,
                  int4 *__restrict__ box, fx64 *__restrict__ ow, double *__restrict__ pwn,
                  double *__restrict__ unit, int *__restrict__ wide) {
    co_grid_wait();
    __shared__ double shg[FIXED_PACK / 32], shw[FIXED_PACK / 32];
    __shared__ float4 sv[FIXED_SAMPLES];   // x1 x2 g1 g2, scaled
    __shared__ float swt[FIXED_SAMPLES];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // all loads first: their latency passes with that of the maxima
    const int M = *Mp;
    const int p = blockIdx.x * blockDim.x + tid;   // below Mpad: the blocks are whole
    const double2 zero = make_double2(0.0, 0.0);
    const double2 x = p < M ? px[p] : zero, G = p < M ? pg[p] : zero;
    const double w = p < M ? pw[p] : 0.0;
    double2 xs = zero, Gs = zero;
    double ws = 0.0;
    if (M > 0) {
        const int q = (int)((long long)tid * M / FIXED_SAMPLES);
        xs = px[q];
        Gs = pg[q];
        ws = pw[q];
    }
    double gm = 0.0, wm = 0.0;
    for (int i = tid; i < npart; i += blockDim.x) {
        const double2 q = part[i];
        gm = fmax(gm, q.x);
        wm = fmax(wm, q.y);
    }
    for (int s = 16; s > 0; s >>= 1) {
        gm = fmax(gm, __shfl_xor_sync(0xffffffffu, gm, s));
        wm = fmax(wm, __shfl_xor_sync(0xffffffffu, wm, s));
    }
    if (lane == 0) {
        shg[warp] = gm;
        shw[warp] = wm;
    }
    __syncthreads();
    for (int i = 0; i < FIXED_PACK / 32; i++) {
        gm = fmax(gm, shg[i]);
        wm = fmax(wm, shw[i]);
    }
    const int eg = scale_exp(gm), ew = scale_exp(wm);
    const double sg = ldexp(1.0, -eg), sx = ldexp(1.0, -ex), sw = ldexp(1.0, -ew);
    if (blockIdx.x == 0 && tid == 0) {
        const bool ok = isfinite(gm) && isfinite(wm);
        unit[0] = ldexp(1.0, ex - eg);
        unit[1] = ok ? ldexp(1.0, ew + eg - ex) : nan("");
        unit[2] = ldexp(1.0, ex);
        unit[3] = ok ? ldexp(1.0, ew - ex) : nan("");
    }
    sv[tid] = make_float4((float)((xs.x - c1) * sx), (float)((xs.y - c2) * sx), (float)(Gs.x * sg),
                          (float)(Gs.y * sg));
    swt[tid] = (float)fabs(ws * sw);
    // padding: outside the scaled domain (coordinates stay below 1/2), weight 0
    double x1 = 0.96875, x2 = 0.96875, G1 = 0.0, G2 = 0.0, wn = 0.0;
    if (p < M) {
        x1 = (x.x - c1) * sx;
        x2 = (x.y - c2) * sx;
        G1 = G.x * sg;
        G2 = G.y * sg;
        wn = w * sw;
    }
    int4 r;
    const fx64 V1 = fx_round(G1 * 0x1p60, r.z), V2 = fx_round(G2 * 0x1p60, r.w);
    const int h1 = (int)((V1 + (1ll << 30)) >> 31), h2 = (int)((V2 + (1ll << 30)) >> 31);
    const fx64 X1 = fx_round(x1 * 0x1p61, r.x), X2 = fx_round(x2 * 0x1p61, r.y);
    ox[p] = make_longlong2(X1, X2);
    rest[p] = r;
    // bounds of 32 markers: min, max of the high words of x1 x2 g1 g2 (the blocks are whole)
    const int hw[4] = {fx_hi(X1), fx_hi(X2), h1, h2};
    int4 lo, hi;
    lo.x = __reduce_min_sync(0xffffffffu, hw[0]), hi.x = __reduce_max_sync(0xffffffffu, hw[0]);
    lo.y = __reduce_min_sync(0xffffffffu, hw[1]), hi.y = __reduce_max_sync(0xffffffffu, hw[1]);
    lo.z = __reduce_min_sync(0xffffffffu, hw[2]), hi.z = __reduce_max_sync(0xffffffffu, hw[2]);
    lo.w = __reduce_min_sync(0xffffffffu, hw[3]), hi.w = __reduce_max_sync(0xffffffffu, hw[3]);
    if (lane < 2) box[2 * (p >> 5) + lane] = lane ? hi : lo;
    __syncthreads();
    const bool bad = p < M && fixed_wide(sv, swt, (float)x1, (float)x2, (float)G1, (float)G2, gm > 0.0);
    if (__syncthreads_or(bad) && tid == 0) *wide = 1;   // every writer writes the same
    og[p] = make_int4(h1, (int)(V1 - ((fx64)h1 << 31)), h2, (int)(V2 - ((fx64)h2 << 31)));
    ow[p] = __double2ll_rn(wn * 0x1p61);
    pwn[p] = wn;
}

// ------------------------------------------------------------------ host

// The domain's scale and origin (exact in FP64): coordinates below 1/2 after
// (x - c) 2^-ex. A domain that lies far to one side of 0 is taken from its
// centre, exact by Sterbenz's lemma when hi <= 2 lo; any other from 0.
static double fixed_centre(double lo, double hi) {
    if (lo > 0.0 && hi <= 2.0 * lo) return 0.5 * (lo + hi);
    if (hi < 0.0 && lo >= 2.0 * hi) return 0.5 * (lo + hi);
    return 0.0;
}

int co_pair_fixed_pack(co_ctx *c, int Mub, int npart) {
    co_bufs &b = c->mb;
    const double c1 = fixed_centre(c->lo1, c->hi1), c2 = fixed_centre(c->lo2, c->hi2);
    const double big = fmax(fmax(fabs(c->lo1 - c1), fabs(c->hi1 - c1)),
                            fmax(fabs(c->lo2 - c2), fabs(c->hi2 - c2)));
    const int ex = ilogb(big) + 2;
    c->fixed_ex = ex;
    const int Mpad = co_cdiv(Mub, 256) * 256;
    co_launch(c, k_pair_fixed_pack, Mpad / FIXED_PACK, FIXED_PACK, 0, b.px, b.pg, b.pw, b.cstart + c->n_el,
              b.gwmax, npart, ex, c1, c2, (longlong2 *)b.fx_x, b.fx_g, b.fx_rest,
              b.fx_box, b.fx_w, b.pwn, b.unit, &c->st->wide);
    c->launches++;
    CO_CK(cudaGetLastError());
    return CO_OK;
}

co_fixed_ops co_fixed_operands(co_ctx *c) {
    co_bufs &b = c->mb;
    co_fixed_ops o;
    o.x = (const longlong2 *)b.fx_x;
    o.g = b.fx_g;
    o.rest = b.fx_rest;
    o.box = b.fx_box;
    o.w = b.fx_w;
    o.px = b.px;
    o.pg = b.pg;
    o.pw = b.pw;
    o.pwn = b.pwn;
    o.wide = &c->st->wide;
    o.unit = b.unit;
    // |d| < 2^-22 in scaled units, and at least the 1e-12 guard distance, in units
    // of the coordinates' high words (2^29 for 1)
    o.m_close = (float)(0x1p29 * fmax(0x1p-22, 1.001e-12 * exp2(-(double)c->fixed_ex)));
    o.m_small = fmaxf(o.m_close, (float)(1 << FX_SMALL_D));
    o.x_near = (int)fminf(o.m_small, 0x1p30f) + 2;   // differences of bounds are below 2^30
    return o;
}

// Tile width and chunk. An item (one tile pair) is (32 W)^2 pairs. 152 SMs hold
// eight blocks of four warps each, so tiles of 128 leave the last wave less than a
// quarter of the time from four waves of items on (12,600 markers); below, one-warp
// items balance better: 358 against 386 us at 10,000 markers, 27 against 45 at
// 2,048 (at 16,384: 932 against 947, but 134 MB of partials to add up). Chunks of
// up to eight tile pairs keep the target-side partials few where items abound.
// Two targets per lane (half the source loads and shuffles) were 3-5 % slower at
// every size: 122 registers leave half the warps.
static void fixed_shape(co_ctx *c, int Mub, int *W, int *KC) {
    const long long nt = co_cdiv(Mub, 128), items = nt * (nt / 2 + 1);
    *W = items >= 32LL * c->nsm ? 4 : 1;
    int kc = 1;
    if (*W == 4)
        while (kc < 8 && items / (2 * kc) >= 48LL * c->nsm) kc *= 2;
    *KC = kc;
}

// Source-side partials take a slot per marker and k, N^2 / 256 in all (F with the metric
// of 131,072 markers: 2.7 GB, of 2^20: 172). From FIXED_PART bytes on, the sum goes in
// bands of k that fit, one after another on the same buffer.
#define FIXED_PART (1ull << 30)
template <int W, int NC>
static int fixed_run(co_ctx *c, int Mub, int KC, int prof_kind) {
    const int TS = 32 * W, nt = co_cdiv(Mub, TS), H = nt / 2;
    const size_t row = (size_t)nt * NC * TS;   // slots of one k
    const size_t fit = FIXED_PART / (8 * row) / KC * KC;
    const int band = (size_t)H <= fit ? H + 1 : (int)(fit > 0 ? fit : KC);
    const size_t gsz = co_cdiv(band, KC) * row;
    int rc = co_ensure_part(c, gsz + (size_t)(band > H ? (H > 0 ? H : 1) : band) * row);
    if (rc) return rc;
    double *gpart = c->mb.part, *apart = c->mb.part + gsz;
    co_prof_begin(c, prof_kind);
    for (int kb = 0; kb <= H; kb += band) {
        const int ke = kb + band < H + 1 ? kb + band : H + 1, nchunk = co_cdiv(ke - kb, KC);
        co_launch(c, k_pair_fixed_sym<W, NC>, nt * nchunk, TS, 0, co_fixed_operands(c), nt, H, KC,
                  kb, ke, gpart, apart);
        if (ke == H + 1) co_prof_end(c);
        co_launch(c, k_fixed_reduce<NC>, nt * W, 32 * FIXED_SL, 0, gpart, apart, nt, H, nchunk,
                  kb > 0 ? kb : 1, ke, TS, c->mb.unit, &c->st->wide, (int)(kb > 0), c->mb.pdot,
                  c->mb.pA, (size_t)c->mb.cap);
        c->launches += 2;
    }
    CO_CK(cudaGetLastError());
    return CO_OK;
}

// vdot (and, with metric, A) of the packed markers
int co_pair_fixed_sum(co_ctx *c, int Mub, int metric, int prof_kind) {
    int W, KC;
    fixed_shape(c, Mub, &W, &KC);
    if (metric) return W == 4 ? fixed_run<4, 5>(c, Mub, KC, prof_kind) : fixed_run<1, 5>(c, Mub, KC, prof_kind);
    return W == 4 ? fixed_run<4, 2>(c, Mub, KC, prof_kind) : fixed_run<1, 2>(c, Mub, KC, prof_kind);
}
