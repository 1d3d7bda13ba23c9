// co_pair.cu -- the O(N^2) Landau pair sum (functions.jl:205-237) on sm_103a.
//
// N-body layout: the in-domain markers are compacted and cell-sorted by the
// spline stage; the pack kernel lays their operands out contiguously (px, pg,
// pw). A block owns a tile of targets gamma (one per thread) and streams the
// sources alpha through shared memory in tiles; the alpha range can be split
// into slices whose partial sums are added afterwards in slice order, so
// results are bitwise reproducible for a given N.
//
// Calls that evaluate the Float64 sum once run on the fixed-point kernels of
// co_pair_fixed.cu, as do the first iterations of step_anderson!. The FP64 arithmetic
// below (its symmetric loop in co_pair64.cuh) serves the solves, the predictor, the batch
// engine, the one-sided kernels (CO_FLAG_ONESIDED, fewer than 385 markers) and operands
// whose range is too wide for fixed point. On GB300 FP64 issues at 1/64 of the FP32
// rate, so the per-pair FP64 instruction count is what sets its time. The pair body
// is 20 FP64 instructions:
//   d (2), |d|^2 (2), 1/|d| refinement (5), G difference (2), d.g (2),
//   1/|d|^2 and (d.g)/|d|^2 (2), projection (2), w/|d| (1), accumulate (2).
// 1/|d| starts from a single-precision seed built from the FP64 bit pattern
// with integer operations (no FP64 conversion instructions) and MUFU.RSQ, then
// one third-order Newton step y += y e (1/2 + 3/8 e), e = 1 - x y^2, which
// takes the ~2^-20 seed error to below 2^-53 (the same idea as the
// reference's f32 seed + two Newton steps, collision_gpu.jl:36-44, with one
// higher-order step in place of two quadratic ones). The |d|^2 < 1e-24 guard
// (functions.jl:224) is an integer compare on the bit pattern.
//
// Mixed form (the precision form of the solver): the pair arithmetic runs in FP32 on
// FP64-centred differences -- each coordinate is split into an FP32 head and
// tail (x = xh + xl), so d = (xh_g - xh_a) + (xl_g - xl_a) is accurate to an
// FP32 rounding of d itself even for close pairs -- and the per-tile FP32
// partial sums are accumulated in FP64.
#include "co_f32x2.cuh"
#include "co_internal.cuh"
#include "co_pair64.cuh"
#include "co_reduce.cuh"

#define PAIR_TPB 128

__device__ __forceinline__ void pair64(double xg1, double xg2, double Gg1, double Gg2,
                                       double xa1, double xa2, double Ga1, double Ga2,
                                       double wa, double &acc1, double &acc2) {
    double d1 = xg1 - xa1;
    double d2 = xg2 - xa2;
    double r2 = d1 * d1;
    r2 = fma(d2, d2, r2);
    bool ok = __double_as_longlong(r2) >= CO_R2_MIN_BITS;
    double xr = ok ? r2 : 1.0;
    double y = rsqrt_seed64(xr);
    double t = xr * y;
    double e = fma(-t, y, 1.0);
    double p = fma(0.375, e, 0.5);
    double ye = y * e;
    y = fma(ye, p, y);
    double g1 = Ga1 - Gg1;
    double g2 = Ga2 - Gg2;
    double dg = d1 * g1;
    dg = fma(d2, g2, dg);
    double y2 = y * y;
    double cc = dg * y2;
    double t1 = fma(-d1, cc, g1);
    double t2 = fma(-d2, cc, g2);
    double s = wa * y;
    s = ok ? s : 0.0;
    acc1 = fma(s, t1, acc1);
    acc2 = fma(s, t2, acc2);
}

// F and the metric A (functions.jl:249-290 / collision_gpu.jl:289-339)
__device__ __forceinline__ void pair64_metric(double xg1, double xg2, double Gg1, double Gg2,
                                              double xa1, double xa2, double Ga1, double Ga2,
                                              double wa, double &acc1, double &acc2,
                                              double &a11, double &a12, double &a22) {
    double d1 = xg1 - xa1;
    double d2 = xg2 - xa2;
    double q11 = d1 * d1, q22 = d2 * d2;
    double r2 = q11 + q22;
    bool ok = __double_as_longlong(r2) >= CO_R2_MIN_BITS;
    double xr = ok ? r2 : 1.0;
    double y = rsqrt_seed64(xr);
    double t = xr * y;
    double e = fma(-t, y, 1.0);
    double p = fma(0.375, e, 0.5);
    double ye = y * e;
    y = fma(ye, p, y);
    double g1 = Ga1 - Gg1;
    double g2 = Ga2 - Gg2;
    double dg = d1 * g1;
    dg = fma(d2, g2, dg);
    double y2 = y * y;
    double cc = dg * y2;
    double t1 = fma(-d1, cc, g1);
    double t2 = fma(-d2, cc, g2);
    double s = wa * y;
    s = ok ? s : 0.0;
    acc1 = fma(s, t1, acc1);
    acc2 = fma(s, t2, acc2);
    a11 = fma(s, fma(-q11, y2, 1.0), a11);
    a12 = fma(-s, (d1 * d2) * y2, a12);
    a22 = fma(s, fma(-q22, y2, 1.0), a22);
}

// out layout: partial[slice][comp][M] with stride ld
template <bool METRIC>
__global__ void __launch_bounds__(PAIR_TPB)
k_pair64(const double2 *__restrict__ px, const double2 *__restrict__ pg,
         const double *__restrict__ pw, const int *__restrict__ Mp, int slice_len,
         double *__restrict__ out, size_t ld) {
    __shared__ double2 sx[PAIR_TPB];
    __shared__ double2 sg[PAIR_TPB];
    __shared__ double sw[PAIR_TPB];
    const int M = *Mp;
    const int g0 = blockIdx.x * PAIR_TPB;
    if (g0 >= M) return;
    const int g = g0 + threadIdx.x;
    const int sl = blockIdx.y;
    const int a0 = sl * slice_len;
    const int a1 = min(M, a0 + slice_len);
    double2 xg = make_double2(0.0, 0.0), Gg = make_double2(0.0, 0.0);
    if (g < M) {
        xg = px[g];
        Gg = pg[g];
    }
    double acc1 = 0.0, acc2 = 0.0, a11 = 0.0, a12 = 0.0, a22 = 0.0;
    for (int base = a0; base < a1; base += PAIR_TPB) {
        int a = base + threadIdx.x;
        if (a < a1) {
            sx[threadIdx.x] = px[a];
            sg[threadIdx.x] = pg[a];
            sw[threadIdx.x] = pw[a];
        } else {  // inert padding: far away, zero weight
            sx[threadIdx.x] = make_double2(1e3, 1e3);
            sg[threadIdx.x] = make_double2(0.0, 0.0);
            sw[threadIdx.x] = 0.0;
        }
        __syncthreads();
#pragma unroll 4
        for (int k = 0; k < PAIR_TPB; k++) {
            double2 xa = sx[k], Ga = sg[k];
            if (METRIC)
                pair64_metric(xg.x, xg.y, Gg.x, Gg.y, xa.x, xa.y, Ga.x, Ga.y, sw[k], acc1, acc2,
                              a11, a12, a22);
            else
                pair64(xg.x, xg.y, Gg.x, Gg.y, xa.x, xa.y, Ga.x, Ga.y, sw[k], acc1, acc2);
        }
        __syncthreads();
    }
    if (g < M) {
        const int nc = METRIC ? 5 : 2;
        double *o = out + (size_t)sl * nc * ld;
        o[g] = acc1;
        o[ld + g] = acc2;
        if (METRIC) {
            o[2 * ld + g] = a11;
            o[3 * ld + g] = a12;
            o[4 * ld + g] = a22;
        }
    }
}

// FP32 pair body on head/tail-split operands
__device__ __forceinline__ void pair32(const float4 &xg, const float4 &Gg, const float4 &xa,
                                       const float4 &Ga, float wa, float &acc1, float &acc2) {
    float d1 = (xg.x - xa.x) + (xg.z - xa.z);
    float d2 = (xg.y - xa.y) + (xg.w - xa.w);
    float g1 = (Ga.x - Gg.x) + (Ga.z - Gg.z);
    float g2 = (Ga.y - Gg.y) + (Ga.w - Gg.w);
    float r2 = d1 * d1;
    r2 = fmaf(d2, d2, r2);
    float y = rsqrtf(r2);
    y = r2 >= 1e-24f ? y : 0.0f;
    float dg = d1 * g1;
    dg = fmaf(d2, g2, dg);
    float y2 = y * y;
    float cc = dg * y2;
    float t1 = fmaf(-d1, cc, g1);
    float t2 = fmaf(-d2, cc, g2);
    float s = wa * y;
    acc1 = fmaf(s, t1, acc1);
    acc2 = fmaf(s, t2, acc2);
}

#define PAIR32_TILE 256
__global__ void __launch_bounds__(PAIR_TPB)
k_pair32(const float4 *__restrict__ pfx, const float4 *__restrict__ pfg,
         const float *__restrict__ pfw, const int *__restrict__ Mp, int slice_len,
         double *__restrict__ out, size_t ld) {
    __shared__ float4 sx[PAIR32_TILE];
    __shared__ float4 sg[PAIR32_TILE];
    __shared__ float sw[PAIR32_TILE];
    const int M = *Mp;
    const int g0 = blockIdx.x * PAIR_TPB;
    if (g0 >= M) return;
    const int g = g0 + threadIdx.x;
    const int sl = blockIdx.y;
    const int a0 = sl * slice_len;
    const int a1 = min(M, a0 + slice_len);
    float4 xg = make_float4(0.f, 0.f, 0.f, 0.f), Gg = xg;
    if (g < M) {
        xg = pfx[g];
        Gg = pfg[g];
    }
    double acc1 = 0.0, acc2 = 0.0;
    for (int base = a0; base < a1; base += PAIR32_TILE) {
        for (int k = threadIdx.x; k < PAIR32_TILE; k += PAIR_TPB) {
            int a = base + k;
            if (a < a1) {
                sx[k] = pfx[a];
                sg[k] = pfg[a];
                sw[k] = pfw[a];
            } else {
                sx[k] = make_float4(1e3f, 1e3f, 0.f, 0.f);
                sg[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                sw[k] = 0.f;
            }
        }
        __syncthreads();
        float t1 = 0.f, t2 = 0.f;
#pragma unroll 8
        for (int k = 0; k < PAIR32_TILE; k++) pair32(xg, Gg, sx[k], sg[k], sw[k], t1, t2);
        acc1 += (double)t1;
        acc2 += (double)t2;
        __syncthreads();
    }
    if (g < M) {
        double *o = out + (size_t)sl * 2 * ld;
        o[g] = acc1;
        o[ld + g] = acc2;
    }
}

// ------------------------------------------------------------------ metric (FP32)
//
// A_g = sum_a w_a U(v_g - v_a), U(z) = (I - z z^T/|z|^2)/|z|  (functions.jl:278-281),
// evaluated in FP32 on the head parts of the packed operands. Used only as the
// frozen metric of the defect-correction inner model (solver.jl:585-595), where
// it shapes the convergence rate but not the fixed point: the outer residual is
// always an FP64 (or, in the mixed form, FP32-then-FP64) Picard map.
__global__ void __launch_bounds__(PAIR_TPB)
k_metric32(const float4 *__restrict__ pfx, const float *__restrict__ pfw,
           const int *__restrict__ Mp, double *__restrict__ out, size_t ld) {
    __shared__ float2 sx[PAIR32_TILE];
    __shared__ float sw[PAIR32_TILE];
    const int M = *Mp;
    const int g0 = blockIdx.x * PAIR_TPB;
    if (g0 >= M) return;
    const int g = g0 + threadIdx.x;
    float2 xg = make_float2(0.f, 0.f);
    if (g < M) {
        float4 t = pfx[g];
        xg = make_float2(t.x + t.z, t.y + t.w);
    }
    double A11 = 0.0, A12 = 0.0, A22 = 0.0;
    for (int base = 0; base < M; base += PAIR32_TILE) {
        for (int k = threadIdx.x; k < PAIR32_TILE; k += PAIR_TPB) {
            int a = base + k;
            if (a < M) {
                float4 t = pfx[a];
                sx[k] = make_float2(t.x + t.z, t.y + t.w);
                sw[k] = pfw[a];
            } else {
                sx[k] = make_float2(1e3f, 1e3f);
                sw[k] = 0.f;
            }
        }
        __syncthreads();
        float a11 = 0.f, a12 = 0.f, a22 = 0.f;
#pragma unroll 8
        for (int k = 0; k < PAIR32_TILE; k++) {
            float d1 = xg.x - sx[k].x, d2 = xg.y - sx[k].y;
            float r2 = fmaf(d2, d2, d1 * d1);
            float y = rsqrtf(r2);
            y = r2 >= 1e-24f ? y : 0.f;
            float s = sw[k] * y;
            float y2 = y * y;
            a11 = fmaf(s, fmaf(-d1 * d1, y2, 1.f), a11);
            a12 = fmaf(-s, d1 * d2 * y2, a12);
            a22 = fmaf(s, fmaf(-d2 * d2, y2, 1.f), a22);
        }
        A11 += (double)a11;
        A12 += (double)a12;
        A22 += (double)a22;
        __syncthreads();
    }
    if (g < M) {
        out[g] = A11;
        out[ld + g] = A12;
        out[2 * ld + g] = A22;
    }
}

// ------------------------------------------------------------------ symmetric
//
// Newton's third law for the pair sum: with d = v_g - v_a and g = G_a - G_g,
// the ordered pair (a, g) sees d' = -d and g' = -g, so its term is
// w_g U(d)(-g)/|d| = -w_g u with u = U(d) g / |d| the unweighted term of
// (g, a). One evaluation of u serves both targets.
//
// Tiles of ST = 128 sorted markers; tile pairs (I, J = I + k mod nt) for
// k = 0..H (H = nt/2; for even nt the k = H pairs are taken once, I < nt/2),
// so every unordered tile pair appears exactly once and every row I has the
// same work. A block owns I and a chunk of KC consecutive k. Inside a tile
// pair the 4 warps take the 4 source sub-tiles in rotation (one warp per
// sub-tile per round); within a warp, lane l pairs its target with source
// (l + q) mod 32 at step q and passes the source's accumulator to lane l - 1
// with a shuffle, so each source accumulator has one owner at every step. The
// target side accumulates in registers across the chunk (gpart); the source
// side of each tile pair is written to its own slot (apart) and everything is
// summed afterwards in a fixed order: bitwise reproducible.
//
// FP64 body: 19 FP64 instructions for u + 4 FMAs for the two accumulations =
// 23 per unordered pair, 11.5 per ordered pair (20 in k_pair64).
#define ST 128

// The FP64 pair sum of solves and predictors; batch instances run the same arithmetic in
// k_pair64_sym_batch. Bound by the FP64 pipe (89 % of its peak; 10,000 markers 2.1 ms
// against 0.36 of the fixed-point form).
__global__ void __launch_bounds__(ST)
k_pair64_sym(const double2 *__restrict__ px, const double2 *__restrict__ pg,
             const double *__restrict__ pw, int nt, int H, int KC,
             double *__restrict__ gpart, double *__restrict__ apart) {
    __shared__ sym64_smem<4, 2> sm;
    const int I = blockIdx.x % nt, chunk = blockIdx.x / nt, k0 = chunk * KC;
    sym64_item<4, 2>(sm, px, pg, pw, nt, H, I, k0, min(H + 1, k0 + KC), 1,
                     gpart + ((size_t)chunk * nt + I) * 2 * ST, apart);
}

// FP32 body on head/tail operands: returns the unweighted term u
__device__ __forceinline__ void pair_u32(const float4 &xg, const float4 &Gg, const float4 &xa,
                                         const float4 &Ga, float &u1, float &u2) {
    float d1 = (xg.x - xa.x) + (xg.z - xa.z);
    float d2 = (xg.y - xa.y) + (xg.w - xa.w);
    float g1 = (Ga.x - Gg.x) + (Ga.z - Gg.z);
    float g2 = (Ga.y - Gg.y) + (Ga.w - Gg.w);
    float r2 = d1 * d1;
    r2 = fmaf(d2, d2, r2);
    float y = rsqrtf(r2);
    y = r2 >= 1e-24f ? y : 0.0f;
    float dg = d1 * g1;
    dg = fmaf(d2, g2, dg);
    float y2 = y * y;
    float cc = dg * y2;
    u1 = fmaf(-d1, cc, g1) * y;
    u2 = fmaf(-d2, cc, g2) * y;
}

// Two consecutive tile pairs (I, J), (I, J') of a row in the halves of packed
// registers: their sums are independent (the target side of each is folded into
// FP64 before the next, the source sides are different tiles), so every half sees
// the operations of one tile pair in its order. `next_pair` returns the k after the
// pair that starts at k (k >= 1) and whether the second half is in use; an unused
// half holds inert operands and is not written.
__device__ __forceinline__ int next_pair(int nt, int H, int I, int k, int k1, bool &two) {
    two = k + 1 < k1 && !sym_skip(nt, H, I, k + 1);
    return k + 2;
}

// FP32 symmetric kernel: each of the ST threads holds R = 2 targets (t, t + ST) of a
// TS = 256 tile and meets the same source of two tiles per step, so a source loaded
// from shared memory and a shuffle of the rotating source accumulators serve two
// pair evaluations, and an instruction two of them. Source tiles are handled in
// NG = TS / 32 groups of 32: in round rr warp w takes group (w + rr) mod NG, so each
// group meets each warp once and its accumulators pass from warp to warp through
// sacc between rounds (fixed order, deterministic). 26 FP32 operations per pair in 13
// instructions; what bounds it is the FMA pipe, which issues packed operations with
// three distinct register operands at two thirds of its rate. Bit-identical to the
// scalar form it replaces: 50,021 markers 1.92 -> 1.55 ms a call.
template <int R>
struct pair32_smem {
    float4 x[2][R * ST], g[2][R * ST];   // heads: {c1 J, c1 J', c2 J, c2 J'}; tails
    float2 w[R * ST];
    float4 acc[R * ST];                  // {a1 J, a1 J', a2 J, a2 J'}
};

template <int R>
__global__ void __launch_bounds__(ST)
k_pair32_sym(const float4 *__restrict__ pfx, const float4 *__restrict__ pfg,
             const float *__restrict__ pfw, int nt, int H, int KC,
             double *__restrict__ gpart, float *__restrict__ apart) {
    constexpr int TS = R * ST, NG = TS / 32;
    __shared__ pair32_smem<R> sm;
    const int I = blockIdx.x % nt, chunk = blockIdx.x / nt;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double ga1[R], ga2[R];
#pragma unroll
    for (int r = 0; r < R; r++) ga1[r] = ga2[r] = 0.0;
    const int k0 = chunk * KC, k1 = min(H + 1, k0 + KC);
    int k = k0;
    if (k == 0) {  // diagonal tile: ordered pairs, self excluded by the guard
        float4 xg[R], Gg[R];
        float t1[R], t2[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int t = r * ST + tid;
            xg[r] = pfx[I * TS + t];
            Gg[r] = pfg[I * TS + t];
            sm.x[0][t] = xg[r];
            sm.g[0][t] = Gg[r];
            sm.w[t].x = pfw[I * TS + t];
            t1[r] = t2[r] = 0.f;
        }
        __syncthreads();
#pragma unroll 4
        for (int a = 0; a < TS; a++) {
            const float4 xa = sm.x[0][a], Ga = sm.g[0][a];
            const float wa = sm.w[a].x;
#pragma unroll
            for (int r = 0; r < R; r++) {
                float u1, u2;
                pair_u32(xg[r], Gg[r], xa, Ga, u1, u2);
                t1[r] = fmaf(wa, u1, t1[r]);
                t2[r] = fmaf(wa, u2, t2[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < R; r++) {
            ga1[r] += (double)t1[r];
            ga2[r] += (double)t2[r];
        }
        k = 1;
    }
    f32x2 xg[R][4], Gg[R][4], nw[R];   // dup'd halves: heads c1 c2, tails c1 c2; -weight
#pragma unroll
    for (int r = 0; r < R; r++) {
        const float4 x = pfx[I * TS + r * ST + tid], g = pfg[I * TS + r * ST + tid];
        const float wv = pfw[I * TS + r * ST + tid];
        xg[r][0] = dup2(x.x), xg[r][1] = dup2(x.y), xg[r][2] = dup2(x.z), xg[r][3] = dup2(x.w);
        Gg[r][0] = dup2(g.x), Gg[r][1] = dup2(g.y), Gg[r][2] = dup2(g.z), Gg[r][3] = dup2(g.w);
        nw[r] = dup2(-wv);
    }
    while (k < k1) {
        if (sym_skip(nt, H, I, k)) break;   // k = H, the last one
        bool two;
        const int kn = next_pair(nt, H, I, k, k1, two);
        const int Ja = (I + k) % nt, Jb = (I + k + 1) % nt;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int t = r * ST + tid;
            const float4 xa = pfx[Ja * TS + t], ga = pfg[Ja * TS + t];
            const float wa = pfw[Ja * TS + t];
            float4 xb = make_float4(1e3f, 1e3f, 0.f, 0.f), gb = make_float4(0.f, 0.f, 0.f, 0.f);
            float wb = 0.f;
            if (two) {
                xb = pfx[Jb * TS + t];
                gb = pfg[Jb * TS + t];
                wb = pfw[Jb * TS + t];
            }
            sm.x[0][t] = make_float4(xa.x, xb.x, xa.y, xb.y);
            sm.x[1][t] = make_float4(xa.z, xb.z, xa.w, xb.w);
            sm.g[0][t] = make_float4(ga.x, gb.x, ga.y, gb.y);
            sm.g[1][t] = make_float4(ga.z, gb.z, ga.w, gb.w);
            sm.w[t] = make_float2(wa, wb);
            sm.acc[t] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncthreads();
        f32x2 t1[R], t2[R];
#pragma unroll
        for (int r = 0; r < R; r++) t1[r] = t2[r] = 0;
        for (int rr = 0; rr < NG; rr++) {
            const int base = ((warp + rr) % NG) * 32;
            const ulonglong2 a0 = *reinterpret_cast<const ulonglong2 *>(&sm.acc[base + lane]);
            f32x2 a1 = a0.x, a2 = a0.y;
#pragma unroll 2
            for (int q = 0; q < 32; q++) {
                const int ai = base + ((lane + q) & 31);
                const ulonglong2 xh = *reinterpret_cast<const ulonglong2 *>(&sm.x[0][ai]);
                const ulonglong2 xl = *reinterpret_cast<const ulonglong2 *>(&sm.x[1][ai]);
                const ulonglong2 gh = *reinterpret_cast<const ulonglong2 *>(&sm.g[0][ai]);
                const ulonglong2 gl = *reinterpret_cast<const ulonglong2 *>(&sm.g[1][ai]);
                const f32x2 wa = *reinterpret_cast<const f32x2 *>(&sm.w[ai]);
#pragma unroll
                for (int r = 0; r < R; r++) {   // pair_u32 on both halves
                    const f32x2 d1 = add2(sub2(xg[r][0], xh.x), sub2(xg[r][2], xl.x));
                    const f32x2 d2 = add2(sub2(xg[r][1], xh.y), sub2(xg[r][3], xl.y));
                    const f32x2 g1 = add2(sub2(gh.x, Gg[r][0]), sub2(gl.x, Gg[r][2]));
                    const f32x2 g2 = add2(sub2(gh.y, Gg[r][1]), sub2(gl.y, Gg[r][3]));
                    const f32x2 y = rsqrt_guard2(fma2(d2, d2, mul2(d1, d1)));
                    const f32x2 dg = fma2(d2, g2, mul2(d1, g1));
                    const f32x2 nc = mul2(dg, mul2(y, neg2(y)));   // -(d.g) / |d|^2
                    const f32x2 u1 = mul2(fma2(d1, nc, g1), y), u2 = mul2(fma2(d2, nc, g2), y);
                    t1[r] = fma2(wa, u1, t1[r]);
                    t2[r] = fma2(wa, u2, t2[r]);
                    a1 = fma2(nw[r], u1, a1);
                    a2 = fma2(nw[r], u2, a2);
                }
                a1 = __shfl_sync(0xffffffffu, a1, (lane + 1) & 31);
                a2 = __shfl_sync(0xffffffffu, a2, (lane + 1) & 31);
            }
            *reinterpret_cast<ulonglong2 *>(&sm.acc[base + lane]) = make_ulonglong2(a1, a2);
            __syncthreads();
        }
#pragma unroll
        for (int r = 0; r < R; r++) {
            ga1[r] += (double)lo2(t1[r]);
            ga2[r] += (double)lo2(t2[r]);
            if (two) {
                ga1[r] += (double)hi2(t1[r]);
                ga2[r] += (double)hi2(t2[r]);
            }
        }
        float *ap = apart + ((size_t)(k - 1) * nt + Ja) * 2 * TS;
        float *bp = apart + ((size_t)k * nt + Jb) * 2 * TS;
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int t = r * ST + tid;
            const float4 v = sm.acc[t];
            ap[t] = v.x;
            ap[TS + t] = v.z;
            if (two) {
                bp[t] = v.y;
                bp[TS + t] = v.w;
            }
        }
        k = kn;
    }
    double *gp = gpart + ((size_t)chunk * nt + I) * 2 * TS;
#pragma unroll
    for (int r = 0; r < R; r++) {
        gp[r * ST + tid] = ga1[r];
        gp[TS + r * ST + tid] = ga2[r];
    }
}

// ------------------------------------------------------------------ double-single
//
// The same symmetric pair sum in double-single arithmetic: every value is an
// unevaluated sum hi + lo of two FP32 numbers (about 44 significant bits), built
// from the error-free transformations of Dekker (1971) and Knuth (TAOCP vol. 2):
// two_sum (6 adds), fast_two_sum (3), two_prod via FMA (2). The scalar form serves the
// diagonal tiles, the packed form below it all other tile pairs. The intrinsics
// __fadd_rn/__fsub_rn/__fmul_rn/__fmaf_rn keep the compiler from contracting
// these sequences. Each unordered pair (both orders) costs 137 FP32 operations at
// ~1e-13 relative accuracy per term; momentum stays
// exact to the accumulation round-off because each pair's term is computed once
// and added with both signs. Used for the FP64 stage of the mixed precision form.
struct dsf {
    float h, l;
};

__device__ __forceinline__ dsf ds_two_sum(float a, float b) {
    float s = __fadd_rn(a, b);
    float bb = __fsub_rn(s, a);
    float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    return {s, e};
}
__device__ __forceinline__ dsf ds_fast(float a, float b) {
    float s = __fadd_rn(a, b);
    return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
// Unnormalised double-single values: an intermediate that only feeds a
// product or a sum is kept as an exact pair (h, l) whose l may exceed
// ulp(h)/2 by a few ulps; the value h + l carries the same ~2^-44 accuracy,
// and skipping the renormalising fast_two_sum saves 3 instructions each time.
// The products drop the l*l term, so a factor whose l can be large relative to
// h (a difference of nearly equal inputs) is renormalised first.
__device__ __forceinline__ dsf ds_mul_u(dsf a, dsf b) {   // a b, unnormalised
    float p = __fmul_rn(a.h, b.h);
    float e = __fmaf_rn(a.h, b.h, -p);
    e = __fmaf_rn(a.h, b.l, e);
    e = __fmaf_rn(a.l, b.h, e);
    return {p, e};
}
__device__ __forceinline__ dsf ds_sqr_u(dsf a) {          // a^2, unnormalised
    float p = __fmul_rn(a.h, a.h);
    float e = __fmaf_rn(a.h, a.h, -p);
    e = __fmaf_rn(__fadd_rn(a.h, a.h), a.l, e);
    return {p, e};
}
__device__ __forceinline__ dsf ds_add_u(dsf a, dsf b) {   // a + b, unnormalised
    dsf s = ds_two_sum(a.h, b.h);
    return {s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l))};
}
__device__ __forceinline__ dsf ds_norm(dsf a) { return ds_fast(a.h, a.l); }
// acc += x with acc kept unnormalised (renormalised by the caller every 32 terms)
__device__ __forceinline__ void ds_acc(dsf &acc, dsf x) {
    dsf s = ds_two_sum(acc.h, x.h);
    acc.h = s.h;
    acc.l = __fadd_rn(acc.l, __fadd_rn(x.l, s.l));
}

// Pair term of the symmetric sum in double-single. In two dimensions the
// projection of g = G_a - G_g off d = x_g - x_a is
//   g - d (d.g)/|d|^2 = c (d2, -d1) / |d|^2,   c = g1 d2 - g2 d1,
// so u = U(d) g / |d| = s (d2, -d1) with s = c / |d|^3 (the same term as
// functions.jl:221-231 in exact arithmetic; c carries the cancellation that
// g - d (d.g)/|d|^2 carries when g is nearly parallel to d). Returns d1, d2 and
// s (0 for |d|^2 < 1e-24). The target gets w_a s (d2, -d1), the source the
// same with -w_g.
__device__ __forceinline__ void pair_s_ds(const float4 &xg, const float4 &Gg, const float4 &xa,
                                          const float4 &Ga, dsf &d1, dsf &d2, dsf &s) {
    // differences are renormalised: for close markers the heads cancel exactly
    // and the tail difference would otherwise be a large l (the products drop l*l)
    d1 = ds_norm(ds_add_u({xg.x, xg.z}, {-xa.x, -xa.z}));
    d2 = ds_norm(ds_add_u({xg.y, xg.w}, {-xa.y, -xa.w}));
    dsf r2 = ds_add_u(ds_sqr_u(d1), ds_sqr_u(d2));
    const bool ok = r2.h >= 1e-24f;
    if (!ok) r2 = {1.f, 0.f};
    // 1/|d|^3 from the MUFU seed y0 ~ 1/sqrt(r2): with e = 1 - r2 y0^2 (~1e-7),
    // 1/|d|^3 = y0^3 (1 - e)^{-3/2} = y0^3 (1 + 3e/2 + 15e^2/8 + O(e^3)). y0^2
    // and y0^3 are formed as exact double-single products and e from them, so
    // the result carries ~1e-14 relative error, as a Newton step on y0 followed
    // by double-single cubing does, in 18 instructions instead of 25.
    const float y0 = rsqrtf(r2.h);
    const float p2 = __fmul_rn(y0, y0);
    const float e2 = __fmaf_rn(y0, y0, -p2);       // y0^2 = p2 + e2 exactly
    float q = __fmul_rn(r2.h, p2);
    float qe = __fmaf_rn(r2.h, p2, -q);
    qe = __fmaf_rn(r2.h, e2, qe);
    qe = __fmaf_rn(r2.l, p2, qe);                  // r2 y0^2 = q + qe
    const float e = __fsub_rn(__fsub_rn(1.0f, q), qe);
    const float p3 = __fmul_rn(p2, y0);
    float e3 = __fmaf_rn(p2, y0, -p3);
    e3 = __fmaf_rn(e2, y0, e3);                    // y0^3 = p3 + e3
    const float corr = __fmul_rn(e, __fmaf_rn(1.875f, e, 1.5f));
    const dsf y3 = {p3, __fmaf_rn(p3, corr, e3)};
    const dsf g1 = ds_norm(ds_add_u({Ga.x, Ga.z}, {-Gg.x, -Gg.z}));
    const dsf g2 = ds_norm(ds_add_u({Ga.y, Ga.w}, {-Gg.y, -Gg.w}));
    const dsf m2 = ds_mul_u(g2, d1);
    const dsf c = ds_norm(ds_add_u(ds_mul_u(g1, d2), {-m2.h, -m2.l}));
    s = ds_mul_u(c, y3);
    if (!ok) s = {0.f, 0.f};
}

// Double-single values of two tile pairs in the halves of packed registers, operation
// for operation as above: each half is rounded as the scalar form rounds it. A product
// whose value enters a sum is an FMA with a -0 the compiler cannot see (nz), because a
// packed product and the sum it enters would be contracted into one FMA.
struct ds2 {
    f32x2 h, l;
};
__device__ __forceinline__ ds2 ds2_norm(f32x2 h, f32x2 l) {
    const f32x2 s = add2(h, l);
    return {s, sub2(l, sub2(s, h))};
}
// a - b, unnormalised
__device__ __forceinline__ ds2 ds2_sub(ds2 a, ds2 b) {
    const f32x2 s = sub2(a.h, b.h);
    const f32x2 bb = sub2(s, a.h);
    const f32x2 e = sub2(sub2(a.h, sub2(s, bb)), add2(b.h, bb));
    return {s, add2(e, sub2(a.l, b.l))};
}
__device__ __forceinline__ ds2 ds2_sqr(ds2 a, f32x2 nz) {
    const f32x2 p = fma2(a.h, a.h, nz);
    return {p, fma2(add2(a.h, a.h), a.l, fma2(a.h, a.h, neg2(p)))};
}
// a b, unnormalised; SUM: the head enters a sum
template <bool SUM>
__device__ __forceinline__ ds2 ds2_mul(ds2 a, ds2 b, f32x2 nz) {
    const f32x2 p = SUM ? fma2(a.h, b.h, nz) : mul2(a.h, b.h);
    f32x2 e = fma2(a.h, b.h, neg2(p));
    e = fma2(a.h, b.l, e);
    e = fma2(a.l, b.h, e);
    return {p, e};
}
__device__ __forceinline__ void ds2_acc(ds2 &acc, ds2 x) {
    const f32x2 s = add2(acc.h, x.h);
    const f32x2 bb = sub2(s, acc.h);
    const f32x2 e = add2(sub2(acc.h, sub2(s, bb)), sub2(x.h, bb));
    acc.h = s;
    acc.l = add2(acc.l, add2(x.l, e));
}
// pair_s_ds of both halves; the sources' operands as {h of both, l of both}
__device__ __forceinline__ void pair_s_ds2(const ds2 (&xg)[2], const ds2 (&Gg)[2], ds2 xa1, ds2 xa2,
                                           ds2 Ga1, ds2 Ga2, f32x2 nz, ds2 &d1, ds2 &d2, ds2 &s) {
    d1 = ds2_sub(xg[0], xa1);
    d1 = ds2_norm(d1.h, d1.l);
    d2 = ds2_sub(xg[1], xa2);
    d2 = ds2_norm(d2.h, d2.l);
    const ds2 q1 = ds2_sqr(d1, nz), q2 = ds2_sqr(d2, nz);
    const f32x2 rh = add2(q1.h, q2.h);
    const f32x2 rb = sub2(rh, q1.h);
    const f32x2 re = add2(sub2(q1.h, sub2(rh, rb)), sub2(q2.h, rb));
    const f32x2 rl = add2(re, add2(q1.l, q2.l));
    const float ra = lo2(rh), rc = hi2(rh);
    const f32x2 y0 = pack2(rsqrt_normal(ra), rsqrt_normal(rc));
    const f32x2 p2 = mul2(y0, y0);
    const f32x2 e2 = fma2(y0, y0, neg2(p2));
    const f32x2 q = fma2(rh, p2, nz);
    f32x2 qe = fma2(rh, p2, neg2(q));
    qe = fma2(rh, e2, qe);
    qe = fma2(rl, p2, qe);
    const f32x2 e = sub2(sub2(dup2(1.0f), q), qe);
    const f32x2 p3 = mul2(p2, y0);
    f32x2 e3 = fma2(p2, y0, neg2(p3));
    e3 = fma2(e2, y0, e3);
    const f32x2 corr = mul2(e, fma2(dup2(1.875f), e, dup2(1.5f)));
    const ds2 y3 = {p3, fma2(p3, corr, e3)};
    ds2 g1 = ds2_sub(Ga1, Gg[0]);
    g1 = ds2_norm(g1.h, g1.l);
    ds2 g2 = ds2_sub(Ga2, Gg[1]);
    g2 = ds2_norm(g2.h, g2.l);
    ds2 c = ds2_sub(ds2_mul<true>(g1, d2, nz), ds2_mul<true>(g2, d1, nz));
    c = ds2_norm(c.h, c.l);
    s = ds2_mul<false>(c, y3, nz);
    // the guard acts on s alone: what a discarded half computed does not spread
    const bool oka = ra >= 1e-24f, okc = rc >= 1e-24f;
    s.h = pack2(oka ? lo2(s.h) : 0.f, okc ? hi2(s.h) : 0.f);
    s.l = pack2(oka ? lo2(s.l) : 0.f, okc ? hi2(s.l) : 0.f);
}

struct ds_smem {
    ulonglong2 xh[ST], xl[ST], gh[ST], gl[ST];   // {component 1 of both tiles, component 2}
    ulonglong2 w[ST];                            // weights {heads, tails}
    ulonglong2 a1[ST], a2[ST];                   // source sums {heads, tails}
};

// Warp w's targets against the two tiles in sm, off the diagonal: in round r it meets
// the sources of group (w + r) mod 4, whose sums rotate with the lanes and pass from
// warp to warp through sm between rounds. UNI: the unweighted terms s (d2, -d1) on
// both sides. The second components are summed without their sign.
template <bool UNI>
__device__ __forceinline__ void ds_tiles(ds_smem &sm, const ds2 (&xg)[2], const ds2 (&Gg)[2], ds2 wg,
                                         f32x2 nz, int lane, int warp, ds2 &ga1, ds2 &ga2) {
#pragma unroll 1
    for (int r = 0; r < 4; r++) {
        const int base = ((warp + r) & 3) * 32;
        ds2 a1 = {sm.a1[base + lane].x, sm.a1[base + lane].y};
        ds2 a2 = {sm.a2[base + lane].x, sm.a2[base + lane].y};
#pragma unroll 1
        for (int q = 0; q < 32; q++) {
            const int ai = base + ((lane + q) & 31);
            const ulonglong2 xh = sm.xh[ai], xl = sm.xl[ai], gh = sm.gh[ai], gl = sm.gl[ai];
            ds2 d1, d2, s;
            pair_s_ds2(xg, Gg, {xh.x, xl.x}, {xh.y, xl.y}, {gh.x, gl.x}, {gh.y, gl.y}, nz, d1, d2, s);
            if (UNI) {
                const ds2 t1 = ds2_mul<true>(s, d2, nz), t2 = ds2_mul<true>(s, d1, nz);
                ds2_acc(ga1, t1);
                ds2_acc(ga2, t2);
                ds2_acc(a1, t1);
                ds2_acc(a2, t2);
            } else {
                const ulonglong2 wa = sm.w[ai];
                const ds2 ws = ds2_mul<false>({wa.x, wa.y}, s, nz);   // w_a s
                const ds2 wn = ds2_mul<false>(wg, s, nz);             // -w_g s
                ds2_acc(ga1, ds2_mul<true>(ws, d2, nz));
                ds2_acc(ga2, ds2_mul<true>(ws, d1, nz));
                ds2_acc(a1, ds2_mul<true>(wn, d2, nz));
                ds2_acc(a2, ds2_mul<true>(wn, d1, nz));
            }
            const int src = (lane + 1) & 31;
            a1.h = __shfl_sync(0xffffffffu, a1.h, src);
            a1.l = __shfl_sync(0xffffffffu, a1.l, src);
            a2.h = __shfl_sync(0xffffffffu, a2.h, src);
            a2.l = __shfl_sync(0xffffffffu, a2.l, src);
        }
        a1 = ds2_norm(a1.h, a1.l);
        a2 = ds2_norm(a2.h, a2.l);
        ga1 = ds2_norm(ga1.h, ga1.l);
        ga2 = ds2_norm(ga2.h, ga2.l);
        sm.a1[base + lane] = make_ulonglong2(a1.h, a1.l);
        sm.a2[base + lane] = make_ulonglong2(a2.h, a2.l);
        __syncthreads();
    }
}

// Two consecutive tile pairs of a row in the halves of packed registers, as in
// k_pair32_sym. Tile pairs whose 2 x 128 markers all carry one weight w0 (the common
// case: equal-weight markers) take the unweighted loop: the terms s (d2, -d1) are
// summed without the per-pair weight products and w0 multiplies the FP64 fold. A block
// vote on the loaded tiles decides; padding (weight 0) and unequal weights take the
// weighted loop. Two tiles that differ in this take a pass each, the first tile's first.
// 137 FP32 operations a pair in packed instructions. What bounds it is the FMA pipe,
// which issues packed operations with three distinct register operands at two thirds of
// its rate: 2.35 of the 2.56 clocks that two pairs take on an SM. 90 registers, five
// blocks per SM (six: 1 % slower). Bit-identical to the scalar form it replaces: 131,072
// markers 41.7 -> 37.7 ms a map, 47.9 -> 43.2 with unequal weights.
__global__ void __launch_bounds__(ST, 5)
k_pair_ds_sym(const float4 *__restrict__ pfx, const float4 *__restrict__ pfg,
              const float *__restrict__ pfw, const float *__restrict__ pfwl, int nt, int H,
              int KC, double *__restrict__ gpart, double *__restrict__ apart, f32x2 nz) {
    __shared__ ds_smem sm;
    const int I = blockIdx.x % nt, chunk = blockIdx.x / nt;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float2 w0 = make_float2(pfw[I * ST], pfwl[I * ST]);
    const double w0d = (double)w0.x + (double)w0.y;
    double gd1 = 0.0, gd2 = 0.0;
    const int k0 = chunk * KC, k1 = min(H + 1, k0 + KC);
    int k = k0;
    const float4 x = pfx[I * ST + tid], g = pfg[I * ST + tid];
    const dsf w = {pfw[I * ST + tid], pfwl[I * ST + tid]};
    const bool own_same = w.h == w0.x && w.l == w0.y && w0.x != 0.f;
    if (k == 0) {   // diagonal tile: ordered pairs, self excluded by the guard
        float4 *sx = reinterpret_cast<float4 *>(sm.xh), *sg = reinterpret_cast<float4 *>(sm.gh);
        float2 *sw = reinterpret_cast<float2 *>(sm.w);
        sx[tid] = x;
        sg[tid] = g;
        sw[tid] = make_float2(w.h, w.l);
        const bool uni = __syncthreads_and(own_same) != 0;
        dsf t1 = {0.f, 0.f}, t2 = {0.f, 0.f};
        for (int a = 0; a < ST; a++) {
            dsf d1, d2, s;
            pair_s_ds(x, g, sx[a], sg[a], d1, d2, s);
            if (!uni) s = ds_mul_u({sw[a].x, sw[a].y}, s);
            ds_acc(t1, ds_mul_u(s, d2));
            ds_acc(t2, ds_mul_u(s, {-d1.h, -d1.l}));
            if ((a & 31) == 31) {
                t1 = ds_norm(t1);
                t2 = ds_norm(t2);
            }
        }
        const double tf = uni ? w0d : 1.0;
        gd1 += tf * ((double)t1.h + (double)t1.l);
        gd2 += tf * ((double)t2.h + (double)t2.l);
        k = 1;
    }
    const ds2 xg[2] = {{dup2(x.x), dup2(x.z)}, {dup2(x.y), dup2(x.w)}};
    const ds2 Gg[2] = {{dup2(g.x), dup2(g.z)}, {dup2(g.y), dup2(g.w)}};
    const ds2 wg = {dup2(-w.h), dup2(-w.l)};
    while (k < k1) {
        if (sym_skip(nt, H, I, k)) break;   // k = H, the last one
        bool two;
        const int kn = next_pair(nt, H, I, k, k1, two);
        const int J[2] = {(I + k) % nt, (I + k + 1) % nt};
        __syncthreads();
        const float4 xa = pfx[J[0] * ST + tid], ga = pfg[J[0] * ST + tid];
        const float2 wa = make_float2(pfw[J[0] * ST + tid], pfwl[J[0] * ST + tid]);
        float4 xb = make_float4(1e3f, 1e3f, 0.f, 0.f), gb = make_float4(0.f, 0.f, 0.f, 0.f);
        float2 wb = wa;
        if (two) {
            xb = pfx[J[1] * ST + tid];
            gb = pfg[J[1] * ST + tid];
            wb = make_float2(pfw[J[1] * ST + tid], pfwl[J[1] * ST + tid]);
        }
        sm.xh[tid] = make_ulonglong2(pack2(xa.x, xb.x), pack2(xa.y, xb.y));
        sm.xl[tid] = make_ulonglong2(pack2(xa.z, xb.z), pack2(xa.w, xb.w));
        sm.gh[tid] = make_ulonglong2(pack2(ga.x, gb.x), pack2(ga.y, gb.y));
        sm.gl[tid] = make_ulonglong2(pack2(ga.z, gb.z), pack2(ga.w, gb.w));
        sm.w[tid] = make_ulonglong2(pack2(wa.x, wb.x), pack2(wa.y, wb.y));
        sm.a1[tid] = sm.a2[tid] = make_ulonglong2(0, 0);
        const bool ua = __syncthreads_and(own_same && wa.x == w0.x && wa.y == w0.y) != 0;
        const bool ub = __syncthreads_and(own_same && wb.x == w0.x && wb.y == w0.y) != 0;
        for (int pass = 0; pass < (ua == ub ? 1 : 2); pass++) {
            const bool uni = pass ? ub : ua;
            ds2 t1 = {0, 0}, t2 = {0, 0};
            if (pass) {
                sm.a1[tid] = sm.a2[tid] = make_ulonglong2(0, 0);
                __syncthreads();
            }
            if (uni) ds_tiles<true>(sm, xg, Gg, wg, nz, lane, warp, t1, t2);
            else ds_tiles<false>(sm, xg, Gg, wg, nz, lane, warp, t1, t2);
            // fold each tile pair's double-single sums into FP64
            const double tf = uni ? w0d : 1.0, sf = uni ? -w0d : 1.0;
            const ulonglong2 v1 = sm.a1[tid], v2 = sm.a2[tid];
            if (pass == 0) {
                double *ap = apart + ((size_t)(k - 1) * nt + J[0]) * 2 * ST;
                gd1 += tf * ((double)lo2(t1.h) + (double)lo2(t1.l));
                gd2 -= tf * ((double)lo2(t2.h) + (double)lo2(t2.l));
                ap[tid] = sf * ((double)lo2(v1.x) + (double)lo2(v1.y));
                ap[ST + tid] = -sf * ((double)lo2(v2.x) + (double)lo2(v2.y));
            }
            if (two && (pass == 1 || ua == ub)) {
                double *bp = apart + ((size_t)k * nt + J[1]) * 2 * ST;
                gd1 += tf * ((double)hi2(t1.h) + (double)hi2(t1.l));
                gd2 -= tf * ((double)hi2(t2.h) + (double)hi2(t2.l));
                bp[tid] = sf * ((double)hi2(v1.x) + (double)hi2(v1.y));
                bp[ST + tid] = -sf * ((double)hi2(v2.x) + (double)hi2(v2.y));
            }
        }
        k = kn;
    }
    double *gp = gpart + ((size_t)chunk * nt + I) * 2 * ST;
    gp[tid] = gd1;
    gp[ST + tid] = gd2;
}

// Symmetric FP32 metric: U(d) = (I - d d^T/|d|^2)/|d| is even in d, so one
// evaluation adds w_a U to A_g and w_g U to A_a (same tiling and rotation as
// k_pair32_sym; head+tail differences). Partials: 3 components.
__device__ __forceinline__ void metric_u32(const float4 &xg, const float4 &xa, float &u11,
                                           float &u12, float &u22) {
    float d1 = (xg.x - xa.x) + (xg.z - xa.z);
    float d2 = (xg.y - xa.y) + (xg.w - xa.w);
    float q11 = d1 * d1, q22 = d2 * d2;
    float r2 = q11 + q22;
    float y = rsqrtf(r2);
    y = r2 >= 1e-24f ? y : 0.0f;
    float y2 = y * y;
    u11 = y * fmaf(-q11, y2, 1.f);
    u12 = -y * (d1 * d2 * y2);
    u22 = y * fmaf(-q22, y2, 1.f);
}

// Two tile pairs of a row per step in packed halves, as in k_pair32_sym; the squares
// come from an FMA with a -0 the compiler cannot see (nz), so that their sum is not
// contracted (the results are those of the scalar form, bit for bit).
__global__ void __launch_bounds__(ST)
k_metric32_sym(const float4 *__restrict__ pfx, const float *__restrict__ pfw, int nt, int H,
               int KC, double *__restrict__ gpart, float *__restrict__ apart, f32x2 nz) {
    __shared__ float4 sx[2][ST];   // heads: {c1 J, c1 J', c2 J, c2 J'}; tails
    __shared__ float2 sw[ST];
    __shared__ float2 sacc[3][ST];
    const int I = blockIdx.x % nt, chunk = blockIdx.x / nt;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float4 x = pfx[I * ST + tid];
    const float wv = pfw[I * ST + tid];
    double g11 = 0.0, g12 = 0.0, g22 = 0.0;
    const int k0 = chunk * KC, k1 = min(H + 1, k0 + KC);
    int k = k0;
    if (k == 0) {
        sx[0][tid] = x;
        sw[tid].x = wv;
        __syncthreads();
        float t11 = 0.f, t12 = 0.f, t22 = 0.f;
#pragma unroll 8
        for (int a = 0; a < ST; a++) {
            float u11, u12, u22;
            metric_u32(x, sx[0][a], u11, u12, u22);
            t11 = fmaf(sw[a].x, u11, t11);
            t12 = fmaf(sw[a].x, u12, t12);
            t22 = fmaf(sw[a].x, u22, t22);
        }
        g11 += (double)t11;
        g12 += (double)t12;
        g22 += (double)t22;
        k = 1;
    }
    const f32x2 xg[4] = {dup2(x.x), dup2(x.y), dup2(x.z), dup2(x.w)}, wg = dup2(wv);
    const f32x2 one = dup2(1.f);
    while (k < k1) {
        if (sym_skip(nt, H, I, k)) break;
        bool two;
        const int kn = next_pair(nt, H, I, k, k1, two);
        const int Ja = (I + k) % nt, Jb = (I + k + 1) % nt;
        __syncthreads();
        const float4 xa = pfx[Ja * ST + tid];
        const float4 xb = two ? pfx[Jb * ST + tid] : make_float4(1e3f, 1e3f, 0.f, 0.f);
        sx[0][tid] = make_float4(xa.x, xb.x, xa.y, xb.y);
        sx[1][tid] = make_float4(xa.z, xb.z, xa.w, xb.w);
        sw[tid] = make_float2(pfw[Ja * ST + tid], two ? pfw[Jb * ST + tid] : 0.f);
        sacc[0][tid] = sacc[1][tid] = sacc[2][tid] = make_float2(0.f, 0.f);
        __syncthreads();
        f32x2 t11 = 0, t12 = 0, t22 = 0;
        for (int r = 0; r < 4; r++) {
            const int base = ((warp + r) & 3) * 32;
            f32x2 a11 = *reinterpret_cast<const f32x2 *>(&sacc[0][base + lane]);
            f32x2 a12 = *reinterpret_cast<const f32x2 *>(&sacc[1][base + lane]);
            f32x2 a22 = *reinterpret_cast<const f32x2 *>(&sacc[2][base + lane]);
#pragma unroll 4
            for (int q = 0; q < 32; q++) {   // metric_u32 on both halves
                const int ai = base + ((lane + q) & 31);
                const ulonglong2 xh = *reinterpret_cast<const ulonglong2 *>(&sx[0][ai]);
                const ulonglong2 xl = *reinterpret_cast<const ulonglong2 *>(&sx[1][ai]);
                const f32x2 wa = *reinterpret_cast<const f32x2 *>(&sw[ai]);
                const f32x2 d1 = add2(sub2(xg[0], xh.x), sub2(xg[2], xl.x));
                const f32x2 d2 = add2(sub2(xg[1], xh.y), sub2(xg[3], xl.y));
                const f32x2 q11 = fma2(d1, d1, nz), q22 = fma2(d2, d2, nz);
                const f32x2 y = rsqrt_guard2(add2(q11, q22));
                const f32x2 y2 = mul2(y, y);
                const f32x2 u11 = mul2(y, fma2(neg2(q11), y2, one));
                const f32x2 u12 = mul2(neg2(y), mul2(mul2(d1, d2), y2));
                const f32x2 u22 = mul2(y, fma2(neg2(q22), y2, one));
                t11 = fma2(wa, u11, t11);
                t12 = fma2(wa, u12, t12);
                t22 = fma2(wa, u22, t22);
                a11 = fma2(wg, u11, a11);
                a12 = fma2(wg, u12, a12);
                a22 = fma2(wg, u22, a22);
                const int src = (lane + 1) & 31;
                a11 = __shfl_sync(0xffffffffu, a11, src);
                a12 = __shfl_sync(0xffffffffu, a12, src);
                a22 = __shfl_sync(0xffffffffu, a22, src);
            }
            *reinterpret_cast<f32x2 *>(&sacc[0][base + lane]) = a11;
            *reinterpret_cast<f32x2 *>(&sacc[1][base + lane]) = a12;
            *reinterpret_cast<f32x2 *>(&sacc[2][base + lane]) = a22;
            __syncthreads();
        }
        g11 += (double)lo2(t11);
        g12 += (double)lo2(t12);
        g22 += (double)lo2(t22);
        float *ap = apart + ((size_t)(k - 1) * nt + Ja) * 3 * ST;
        for (int i = 0; i < 3; i++) ap[i * ST + tid] = sacc[i][tid].x;
        if (two) {
            g11 += (double)hi2(t11);
            g12 += (double)hi2(t12);
            g22 += (double)hi2(t22);
            float *bp = apart + ((size_t)k * nt + Jb) * 3 * ST;
            for (int i = 0; i < 3; i++) bp[i * ST + tid] = sacc[i][tid].y;
        }
        k = kn;
    }
    double *gp = gpart + ((size_t)chunk * nt + I) * 3 * ST;
    gp[tid] = g11;
    gp[ST + tid] = g12;
    gp[2 * ST + tid] = g22;
}

__global__ void k_metric_reduce(const double *__restrict__ gpart, const float *__restrict__ apart,
                                int nt, int H, int nchunk, double *__restrict__ dst, size_t ld) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nt * ST) return;
    int K = p / ST, t = p - K * ST;
    double s[3] = {0.0, 0.0, 0.0};
    for (int c = 0; c < nchunk; c++) {
        const double *gp = gpart + ((size_t)c * nt + K) * 3 * ST;
        for (int q = 0; q < 3; q++) s[q] += gp[q * ST + t];
    }
    for (int k = 1; k <= H; k++) {
        int I = (K - k + nt) % nt;
        if (sym_skip(nt, H, I, k)) continue;
        const float *ap = apart + ((size_t)(k - 1) * nt + K) * 3 * ST;
        for (int q = 0; q < 3; q++) s[q] += (double)ap[q * ST + t];
    }
    for (int q = 0; q < 3; q++) dst[(size_t)q * ld + p] = s[q];
}

// vdot[p] = sum over chunks of the target-side partials + sum over k of the
// source-side partials, in that fixed order
template <typename TA>
__global__ void k_sym_reduce(const double *__restrict__ gpart, const TA *__restrict__ apart,
                             int nt, int H, int nchunk, int TS, double *__restrict__ dst,
                             size_t ld) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nt * TS) return;
    int K = p / TS, t = p - K * TS;
    double s1 = 0.0, s2 = 0.0;
    for (int c = 0; c < nchunk; c++) {
        const double *gp = gpart + ((size_t)c * nt + K) * 2 * TS;
        s1 += gp[t];
        s2 += gp[TS + t];
    }
    for (int k = 1; k <= H; k++) {
        int I = (K - k + nt) % nt;
        if (sym_skip(nt, H, I, k)) continue;
        const TA *ap = apart + ((size_t)(k - 1) * nt + K) * 2 * TS;
        s1 += (double)ap[t];
        s2 += (double)ap[TS + t];
    }
    dst[p] = s1;
    dst[ld + p] = s2;
}

// sum the slice partials of components [c0, c0+nc) in slice order into
// dst (nc x ld); the partials hold ncomp components per slice
__global__ void k_slice_reduce(const double *__restrict__ part, int split, int ncomp, int c0,
                               int nc, size_t ld, const int *__restrict__ Mp,
                               double *__restrict__ dst) {
    int M = *Mp;
    int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= M) return;
    for (int c = 0; c < nc; c++) {
        double s = 0.0;
        for (int sl = 0; sl < split; sl++) s += part[((size_t)sl * ncomp + c0 + c) * ld + g];
        dst[(size_t)c * ld + g] = s;
    }
}

// Packed operands of one sorted position, by mode bit: 1 FP64, 2 FP32 head/tail.
// Positions M .. Mpad are inert padding up to the tile boundary: far away, zero
// weight.
struct co_pack_out {
    double2 *px, *pg;
    double *pw;
    float4 *pfx, *pfg;
    float *pfw, *pfwl;
    double2 *gwmax;   // block maxima of |G| and |w| (the fixed-point scales)
    int *wide;        // co_solver_state::wide, cleared for the fixed-point operands
};

__device__ __forceinline__ void pack_store(const co_pack_out &o, int mode, int p, bool in,
                                           double x1, double x2, double G1, double G2, double w) {
    if (mode & 2) {
        const float x1h = in ? (float)x1 : 1e3f, x2h = in ? (float)x2 : 1e3f;
        const float G1h = (float)G1, G2h = (float)G2;
        o.pfx[p] = make_float4(x1h, x2h, in ? (float)(x1 - (double)x1h) : 0.f,
                               in ? (float)(x2 - (double)x2h) : 0.f);
        o.pfg[p] = make_float4(G1h, G2h, (float)(G1 - (double)G1h), (float)(G2 - (double)G2h));
        const float wh = (float)w;
        o.pfw[p] = wh;
        o.pfwl[p] = (float)(w - (double)wh);
    }
    if (mode & 1) {
        o.px[p] = in ? make_double2(x1, x2) : make_double2(1e3, 1e3);
        o.pg[p] = make_double2(G1, G2);
        o.pw[p] = w;
    }
}

// block maxima of |G| and |w|; inf where an operand is not finite
__device__ __forceinline__ void pack_max(const co_pack_out &o, double x1, double x2, double G1,
                                         double G2, double w) {
    __shared__ double2 sh[8];
    double gm = fmax(fabs(G1), fabs(G2)), wm = fabs(w);
    if (!isfinite(x1 + x2) || !isfinite(G1) || !isfinite(G2) || !isfinite(w)) gm = INFINITY;
    for (int s = 16; s > 0; s >>= 1) {
        gm = fmax(gm, __shfl_xor_sync(0xffffffffu, gm, s));
        wm = fmax(wm, __shfl_xor_sync(0xffffffffu, wm, s));
    }
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = make_double2(gm, wm);
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < (int)(blockDim.x >> 5); i++) {
            gm = fmax(gm, sh[i].x);
            wm = fmax(wm, sh[i].y);
        }
        o.gwmax[blockIdx.x] = make_double2(gm, wm);
        if (blockIdx.x == 0) *o.wide = 0;
    }
}

// Landau pack: lambda from the device state, G_eff = -(dS + lambda dv)/w
// (solver.jl:107-111), operands in sorted order.
__global__ void __launch_bounds__(256)
k_pack_landau(const int *__restrict__ perm, const int *__restrict__ Mp, int Mpad, int N,
              const double *__restrict__ vmid, const double *__restrict__ dS,
              const double *__restrict__ dv, const double *__restrict__ w,
              const co_solver_state *__restrict__ st, int use_lambda, int mode, co_pack_out o) {
    co_grid_wait();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = p < *Mp;
    double x1 = 0.0, x2 = 0.0, G1 = 0.0, G2 = 0.0, wa = 0.0;
    if (in) {
        const int a = perm[p];
        const double lam = use_lambda ? st->lambda : 0.0;
        wa = w[a];
        const double iw = 1.0 / wa;
        x1 = vmid[a];
        x2 = vmid[N + a];
        G1 = -(dS[a] + lam * dv[a]) * iw;
        G2 = -(dS[N + a] + lam * dv[N + a]) * iw;
    }
    if (p < Mpad) pack_store(o, mode, p, in, x1, x2, G1, G2, wa);
    if (mode & 1) pack_max(o, x1, x2, G1, G2, wa);
}

// Hook pack: operands straight from (v, G, w) (COLLISION_FN semantics).
__global__ void __launch_bounds__(256)
k_pack_plain(const int *__restrict__ perm, const int *__restrict__ Mp, int Mpad, int N,
             const double *__restrict__ v, const double *__restrict__ G,
             const double *__restrict__ w, int mode, co_pack_out o) {
    co_grid_wait();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = p < *Mp;
    double x1 = 0.0, x2 = 0.0, G1 = 0.0, G2 = 0.0, wa = 0.0;
    if (in) {
        const int a = perm[p];
        x1 = v[a];
        x2 = v[N + a];
        G1 = G[a];
        G2 = G[N + a];
        wa = w[a];
    }
    if (p < Mpad) pack_store(o, mode, p, in, x1, x2, G1, G2, wa);
    if (mode & 1) pack_max(o, x1, x2, G1, G2, wa);
}

// Gv = v0 + dt * vdot (solver.jl:225), vdot unpacked from sorted order (0 for
// out-of-domain markers); optionally r = Gv - v1 and block partials of |r|^2,
// |v1|^2 for step_anderson! (solver.jl:339-349).
__global__ void __launch_bounds__(CO_RED_THREADS)
k_unpack_update(const int *__restrict__ inv, int N, const double *__restrict__ pdot, size_t ld,
                double dt, const double *__restrict__ v0, double *__restrict__ Gv,
                double *__restrict__ dotv, const double *__restrict__ v1, double *__restrict__ r,
                double *__restrict__ red) {
    co_grid_wait();
    __shared__ double sh[64];
    double sr = 0.0, sv = 0.0;
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < N; a += gridDim.x * blockDim.x) {
        int p = inv[a];
        double q1 = 0.0, q2 = 0.0;
        if (p >= 0) {
            q1 = pdot[p];
            q2 = pdot[ld + p];
        }
        if (dotv) {
            dotv[a] = q1;
            dotv[N + a] = q2;
        }
        if (Gv) {
            double g1 = v0[a] + dt * q1, g2 = v0[N + a] + dt * q2;
            Gv[a] = g1;
            Gv[N + a] = g2;
            if (r) {
                double x1 = v1[a], x2 = v1[N + a];
                double r1 = g1 - x1, r2 = g2 - x2;
                r[a] = r1;
                r[N + a] = r2;
                sr += r1 * r1 + r2 * r2;
                sv += x1 * x1 + x2 * x2;
            }
        }
    }
    if (red) {
        double s[2] = {sr, sv};
        co_block_sums<2>(s, sh);
        if (threadIdx.x == 0) {
            red[blockIdx.x * 2 + 0] = s[0];
            red[blockIdx.x * 2 + 1] = s[1];
        }
    }
}

// unpack A (3 comps) for COLLMETRIC_FN
__global__ void k_unpack_A(const int *__restrict__ inv, int N, const double *__restrict__ pA,
                           size_t ld, double *__restrict__ A) {
    int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= N) return;
    int p = inv[a];
    for (int c = 0; c < 3; c++) A[(size_t)c * N + a] = p >= 0 ? pA[(size_t)c * ld + p] : 0.0;
}

// ------------------------------------------------------------------ host

static int choose_split(co_ctx *c, int M, int tpb, int force) {
    if (force > 0) return force;
    int tiles = co_cdiv(M, tpb);
    if (tiles < 1) tiles = 1;
    int want = co_cdiv(4LL * c->nsm, tiles);
    int max_split = co_cdiv(M, 256);
    if (max_split < 1) max_split = 1;
    if (want > max_split) want = max_split;
    if (want < 1) want = 1;
    return want;
}

int co_ensure_part(co_ctx *c, size_t n) {
    if (n <= c->mb.part_cap) return CO_OK;
    if (c->mb.part) cudaFree(c->mb.part);
    c->mb.part = nullptr;
    c->mb.part_cap = 0;
    if (cudaMalloc(&c->mb.part, n * sizeof(double)) != cudaSuccess) return co_nomem();
    c->mb.part_cap = n;
    return CO_OK;
}

#define SYM_KC 8

// FP64 symmetric pair sum on the padded operands (solves and predictors)
static int pair64_sym(co_ctx *c, int Mub) {
    const int nt = co_cdiv(Mub, ST), H = nt / 2, KC = SYM_KC, nchunk = co_cdiv(H + 1, KC);
    const size_t gsz = (size_t)nchunk * nt * 2 * ST, asz = (size_t)(H > 0 ? H : 1) * nt * 2 * ST;
    int rc = co_ensure_part(c, gsz + asz);
    if (rc) return rc;
    double *gpart = c->mb.part, *apart = c->mb.part + gsz;
    co_prof_begin(c, 1);
    k_pair64_sym<<<nt * nchunk, ST, 0, c->stream>>>(c->mb.px, c->mb.pg, c->mb.pw, nt, H, KC, gpart,
                                                    apart);
    co_prof_end(c);
    k_sym_reduce<double><<<co_cdiv((long long)nt * ST, 256), 256, 0, c->stream>>>(
        gpart, apart, nt, H, nchunk, ST, c->mb.pdot, (size_t)c->mb.cap);
    c->launches += 2;
    CO_CK(cudaGetLastError());
    return CO_OK;
}

// M is an upper bound (N); the true count sits at cstart[n_el] on the device.
int co_pair_fp64(co_ctx *c, int Mub, int with_metric) {
    if (Mub <= 0) return CO_OK;
    if (co_use_fixed(c, Mub, CO_PREC_FP64)) return co_pair_fixed_sum(c, Mub, with_metric, 1);
    if (!with_metric && c->pair_symmetric && co_cdiv(Mub, ST) >= 4) return pair64_sym(c, Mub);
    const int *Mp = c->mb.cstart + c->n_el;
    size_t ld = (size_t)c->mb.cap;
    int split = choose_split(c, Mub, PAIR_TPB, c->pair_split_fp64);
    int slice = co_cdiv(Mub, split);
    slice = co_cdiv(slice, PAIR_TPB) * PAIR_TPB;
    split = co_cdiv(Mub, slice);
    int nc = with_metric ? 5 : 2;
    dim3 grid(co_cdiv(Mub, PAIR_TPB), split);
    double *dst = c->mb.pdot;
    if (split > 1 || with_metric) {
        int rc = co_ensure_part(c, (size_t)split * nc * ld);
        if (rc) return rc;
        dst = c->mb.part;
    }
    co_prof_begin(c, 1);
    if (with_metric)
        k_pair64<true><<<grid, PAIR_TPB, 0, c->stream>>>(c->mb.px, c->mb.pg, c->mb.pw, Mp, slice,
                                                         dst, ld);
    else
        k_pair64<false><<<grid, PAIR_TPB, 0, c->stream>>>(c->mb.px, c->mb.pg, c->mb.pw, Mp, slice,
                                                          dst, ld);
    co_prof_end(c);
    c->launches++;
    if (with_metric) {
        // components 0,1 -> pdot ; 2,3,4 -> pA
        k_slice_reduce<<<co_cdiv(Mub, 256), 256, 0, c->stream>>>(dst, split, 5, 0, 2, ld, Mp,
                                                                c->mb.pdot);
        k_slice_reduce<<<co_cdiv(Mub, 256), 256, 0, c->stream>>>(dst, split, 5, 2, 3, ld, Mp,
                                                                c->mb.pA);
        c->launches += 2;
    } else if (split > 1) {
        k_slice_reduce<<<co_cdiv(Mub, 256), 256, 0, c->stream>>>(dst, split, 2, 0, 2, ld, Mp,
                                                                c->mb.pdot);
        c->launches++;
    }
    CO_CK(cudaGetLastError());
    return CO_OK;
}

// FP32 symmetric pair sum: two targets per thread on 256-marker tiles (Mpad is a
// multiple of 256 and the tile count has been checked by the caller)
static int pair32_sym(co_ctx *c, int Mub) {
    constexpr int R32 = 2, TS32 = R32 * ST;
    const int KC = SYM_KC;
    const int nt = co_cdiv(Mub, TS32), H = nt / 2, nchunk = co_cdiv(H + 1, KC);
    const size_t gsz = (size_t)nchunk * nt * 2 * TS32;
    const size_t asz = (size_t)(H > 0 ? H : 1) * nt * 2 * TS32;   // floats
    int rc = co_ensure_part(c, gsz + (asz + 1) / 2);
    if (rc) return rc;
    double *gpart = c->mb.part;
    float *apart = (float *)(c->mb.part + gsz);
    co_prof_begin(c, 0);
    k_pair32_sym<R32><<<nt * nchunk, ST, 0, c->stream>>>(c->mb.pf_x, c->mb.pf_g, c->mb.pf_w, nt, H,
                                                         KC, gpart, apart);
    co_prof_end(c);
    k_sym_reduce<float><<<co_cdiv((long long)nt * TS32, 256), 256, 0, c->stream>>>(
        gpart, apart, nt, H, nchunk, TS32, c->mb.pdot, (size_t)c->mb.cap);
    c->launches += 2;
    CO_CK(cudaGetLastError());
    return CO_OK;
}

int co_pair_fp32(co_ctx *c, int Mub) {
    if (Mub <= 0) return CO_OK;
    if (c->pair_symmetric && co_cdiv(Mub, 2 * ST) >= 4) return pair32_sym(c, Mub);
    const int *Mp = c->mb.cstart + c->n_el;
    size_t ld = (size_t)c->mb.cap;
    int split = choose_split(c, Mub, PAIR_TPB, c->pair_split_fp32);
    int slice = co_cdiv(Mub, split);
    slice = co_cdiv(slice, PAIR32_TILE) * PAIR32_TILE;
    split = co_cdiv(Mub, slice);
    dim3 grid(co_cdiv(Mub, PAIR_TPB), split);
    double *dst = c->mb.pdot;
    if (split > 1) {
        int rc = co_ensure_part(c, (size_t)split * 2 * ld);
        if (rc) return rc;
        dst = c->mb.part;
    }
    co_prof_begin(c, 0);
    k_pair32<<<grid, PAIR_TPB, 0, c->stream>>>(c->mb.pf_x, c->mb.pf_g, c->mb.pf_w, Mp, slice, dst,
                                               ld);
    co_prof_end(c);
    c->launches++;
    if (split > 1) {
        k_slice_reduce<<<co_cdiv(Mub, 256), 256, 0, c->stream>>>(dst, split, 2, 0, 2, ld, Mp,
                                                                c->mb.pdot);
        c->launches++;
    }
    CO_CK(cudaGetLastError());
    return CO_OK;
}

static co_pack_out pack_out(co_ctx *c) {
    co_bufs &b = c->mb;
    return {b.px, b.pg, b.pw, b.pf_x, b.pf_g, b.pf_w, b.pf_wl, b.gwmax, &c->st->wide};
}

int co_pack_plain(co_ctx *c, int N, int Mub, int precision, const double *x, const double *G) {
    if (Mub <= 0) return CO_OK;
    const int *Mp = c->mb.cstart + c->n_el;
    co_bufs &b = c->mb;
    int Mpad = co_cdiv(Mub, 256) * 256;  // whole tiles of up to 256 markers
    co_launch(c, k_pack_plain, Mpad / 256, 256, 0, b.perm, Mp, Mpad, N, x, G, b.w,
              co_pack_mode(precision), pack_out(c));
    c->launches++;
    CO_CK(cudaGetLastError());
    return co_use_fixed(c, Mub, precision) ? co_pair_fixed_pack(c, Mub, Mpad / 256) : CO_OK;
}

int co_pack_landau(co_ctx *c, int N, int Mub, int precision, int gonzalez) {
    if (Mub <= 0) return CO_OK;
    const int *Mp = c->mb.cstart + c->n_el;
    co_bufs &b = c->mb;
    int Mpad = co_cdiv(Mub, 256) * 256;  // whole tiles of up to 256 markers
    co_launch(c, k_pack_landau, Mpad / 256, 256, 0, b.perm, Mp, Mpad, N, b.vmid, b.dS, b.dv, b.w,
              c->st, gonzalez, co_pack_mode(precision), pack_out(c));
    c->launches++;
    CO_CK(cudaGetLastError());
    return co_use_fixed(c, Mub, precision) ? co_pair_fixed_pack(c, Mub, Mpad / 256) : CO_OK;
}

int co_unpack_update(co_ctx *c, int N, double dt, double *Gv, const double *v0,
                     const double *v1, double *r, double *red) {
    if (N == 0) return CO_OK;
    int g = co_cdiv(N, CO_RED_THREADS);
    if (g > c->mb.red_cap) g = c->mb.red_cap;
    co_launch(c, k_unpack_update, g, CO_RED_THREADS, 0, c->mb.inv, N, c->mb.pdot,
              (size_t)c->mb.cap, dt, v0, Gv, c->mb.dotv, v1, r, red);
    c->launches++;
    CO_CK(cudaGetLastError());
    return CO_OK;
}

int co_unpack_A(co_ctx *c, int N, double *A) {
    if (N == 0) return CO_OK;
    k_unpack_A<<<co_cdiv(N, 256), 256, 0, c->stream>>>(c->mb.inv, N, c->mb.pA, (size_t)c->mb.cap,
                                                       A);
    c->launches++;
    CO_CK(cudaGetLastError());
    return CO_OK;
}

int co_metric32(co_ctx *c, int Mub) {
    if (Mub <= 0) return CO_OK;
    if (c->pair_symmetric && co_cdiv(Mub, ST) >= 4) {
        int nt = co_cdiv(Mub, ST), H = nt / 2, KC = SYM_KC, nchunk = co_cdiv(H + 1, KC);
        size_t gsz = (size_t)nchunk * nt * 3 * ST;
        size_t asz = (size_t)(H > 0 ? H : 1) * nt * 3 * ST;  // floats
        int rc = co_ensure_part(c, gsz + (asz + 1) / 2);
        if (rc) return rc;
        float *apart = (float *)(c->mb.part + gsz);
        k_metric32_sym<<<nt * nchunk, ST, 0, c->stream>>>(c->mb.pf_x, c->mb.pf_w, nt, H, KC,
                                                          c->mb.part, apart,
                                                          0x8000000080000000ull);
        k_metric_reduce<<<co_cdiv((long long)nt * ST, 256), 256, 0, c->stream>>>(
            c->mb.part, apart, nt, H, nchunk, c->mb.pA, (size_t)c->mb.cap);
        c->launches += 2;
        CO_CK(cudaGetLastError());
        return CO_OK;
    }
    const int *Mp = c->mb.cstart + c->n_el;
    k_metric32<<<co_cdiv(Mub, PAIR_TPB), PAIR_TPB, 0, c->stream>>>(c->mb.pf_x, c->mb.pf_w, Mp,
                                                                   c->mb.pA, (size_t)c->mb.cap);
    c->launches++;
    CO_CK(cudaGetLastError());
    return CO_OK;
}

// FP64-equivalent pair sum in double-single arithmetic (symmetric kernel); falls
// back to the FP64 kernel below 4 tiles
int co_pair_ds(co_ctx *c, int Mub) {
    if (Mub <= 0) return CO_OK;
    const int nt = co_cdiv(Mub, ST), H = nt / 2, KC = SYM_KC, nchunk = co_cdiv(H + 1, KC);
    if (nt < 4) return co_pair_fp64(c, Mub, 0);
    const size_t gsz = (size_t)nchunk * nt * 2 * ST, asz = (size_t)(H > 0 ? H : 1) * nt * 2 * ST;
    int rc = co_ensure_part(c, gsz + asz);
    if (rc) return rc;
    double *gpart = c->mb.part, *apart = c->mb.part + gsz;
    co_prof_begin(c, 2);
    k_pair_ds_sym<<<nt * nchunk, ST, 0, c->stream>>>(c->mb.pf_x, c->mb.pf_g, c->mb.pf_w,
                                                     c->mb.pf_wl, nt, H, KC, gpart, apart,
                                                     0x8000000080000000ull);
    co_prof_end(c);
    k_sym_reduce<double><<<co_cdiv((long long)nt * ST, 256), 256, 0, c->stream>>>(
        gpart, apart, nt, H, nchunk, ST, c->mb.pdot, (size_t)c->mb.cap);
    c->launches += 2;
    CO_CK(cudaGetLastError());
    return CO_OK;
}

// ================================================================== batched
//
// Many independent ensembles in one persistent launch: the work items of all
// Landau instances -- (instance, tile I, chunk of k) as in the symmetric form above, with a
// tile of T = 32 W markers -- are handed out through an atomic counter, so the
// grid size and the tile shape are free parameters (chosen by the autotuner of
// the batch engine). Items of instances whose solve has finished are skipped.
// Every item writes its own partial slots, so the result does not depend on
// which block ran which item.
template <int W>
__global__ void __launch_bounds__(32 * W)
k_pair64_sym_batch(const co_bwork *__restrict__ works, int n_inst, int total, int KC,
                   unsigned *__restrict__ counter) {
    __shared__ sym64_smem<W, 2> sm;
    __shared__ int s_item;
    for (;;) {
        if (threadIdx.x == 0) s_item = (int)atomicAdd(counter, 1u);
        __syncthreads();
        const int item = s_item;
        __syncthreads();
        if (item >= total) return;
        int lo = 0, hi = n_inst;
        while (hi - lo > 1) {
            int mid = (lo + hi) >> 1;
            if (works[mid].blk0 <= item) lo = mid; else hi = mid;
        }
        const co_bwork wk = works[lo];
        if (wk.st->done) continue;
        const int b = item - wk.blk0, nt = wk.nt, H = wk.H;
        const int I = b % nt, chunk = b / nt, k0 = chunk * KC;
        sym64_item<W, 2>(sm, wk.px, wk.pg, wk.pw, nt, H, I, k0, min(H + 1, k0 + KC), 1,
                         wk.gpart + ((size_t)chunk * nt + I) * 64 * W, wk.apart);
    }
}

// fixed-order reduction of every instance's partials (blockIdx.y = instance)
__global__ void k_sym_reduce_batch(const co_bwork *__restrict__ works, int T) {
    const co_bwork wk = works[blockIdx.y];
    if (wk.st->done) return;
    const int nt = wk.nt, H = wk.H;
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nt * T) return;
    int K = p / T, t = p - K * T;
    double s1 = 0.0, s2 = 0.0;
    for (int c = 0; c < wk.nchunk; c++) {
        const double *gp = wk.gpart + ((size_t)c * nt + K) * 2 * T;
        s1 += gp[t];
        s2 += gp[T + t];
    }
    for (int k = 1; k <= H; k++) {
        int I = (K - k + nt) % nt;
        if (sym_skip(nt, H, I, k)) continue;
        const double *ap = wk.apart + ((size_t)(k - 1) * nt + K) * 2 * T;
        s1 += ap[t];
        s2 += ap[T + t];
    }
    wk.pdot[p] = s1;
    wk.pdot[wk.ld + p] = s2;
}

// Fill the work table of a batch for tile width T = 32 W and chunk KC; makes
// sure every instance's partial buffer is large enough. Returns the number of
// work items.
int co_batch_work_table(co_ctx *const *ctxs, const co_solver_state *const *states, int n,
                        int W, int KC, co_bwork *tab, int *max_pos) {
    const int T = 32 * W;
    int blk = 0, mp = 0;
    for (int i = 0; i < n; i++) {
        co_ctx *c = ctxs[i];
        co_bwork &wk = tab[i];
        int N = c->batch_N;
        int nt = co_cdiv(N, T), H = nt / 2, nchunk = co_cdiv(H + 1, KC);
        size_t gsz = (size_t)nchunk * nt * 2 * T, asz = (size_t)(H > 0 ? H : 1) * nt * 2 * T;
        if (c->batch_landau) {
            int rc = co_ensure_part(c, gsz + asz);
            if (rc) return -rc;
        }
        wk.px = c->mb.px;
        wk.pg = c->mb.pg;
        wk.pw = c->mb.pw;
        wk.gpart = c->mb.part;
        wk.apart = c->mb.part + gsz;
        wk.pdot = c->mb.pdot;
        wk.ld = (size_t)c->mb.cap;
        wk.st = states[i];
        wk.nt = c->batch_landau ? nt : 0;   // LB instances have no pair sum
        wk.H = H;
        wk.nchunk = nchunk;
        wk.blk0 = blk;
        blk += c->batch_landau ? nt * nchunk : 0;
        if (c->batch_landau && nt * T > mp) mp = nt * T;
    }
    *max_pos = mp;
    return blk;
}

// one batched symmetric FP64 pair sum over all Landau instances
int co_pair64_batch(cudaStream_t s, const co_bwork *d_tab, int n, int total, int W, int KC,
                    int grid, unsigned *d_counter, int max_pos) {
    if (total <= 0) return CO_OK;
    CO_CK(cudaMemsetAsync(d_counter, 0, sizeof(unsigned), s));
    switch (W) {
        case 2: k_pair64_sym_batch<2><<<grid, 64, 0, s>>>(d_tab, n, total, KC, d_counter); break;
        case 4: k_pair64_sym_batch<4><<<grid, 128, 0, s>>>(d_tab, n, total, KC, d_counter); break;
        case 8: k_pair64_sym_batch<8><<<grid, 256, 0, s>>>(d_tab, n, total, KC, d_counter); break;
        default: return CO_ERR_ARG;
    }
    dim3 rg(co_cdiv(max_pos, 256), n);
    k_sym_reduce_batch<<<rg, 256, 0, s>>>(d_tab, 32 * W);
    CO_CK(cudaGetLastError());
    return CO_OK;
}
