// co_pair64.cuh -- the Landau pair term in FP64 and the symmetric tile loop on it: used
// by the FP64 kernels of solves and batches (co_pair.cu) and by the fixed-point kernels
// where the operands' range is too wide for them (co_pair_fixed.cu).
#pragma once

// bit pattern of 1e-24 (functions.jl:224 guard)
#define CO_R2_MIN_BITS 0x3AF357C299A88EA7LL

__device__ __forceinline__ double rsqrt_seed64(double x) {
    // FP32 value of x from its high word (x in [1e-30, 1e30], positive)
    int hi = __double2hiint(x);
    float xf = __int_as_float((hi - (896 << 20)) << 3);
    float yf = rsqrtf(xf);
    int fb = __float_as_int(yf);
    return __hiloint2double((fb >> 3) + (896 << 20), fb << 29);
}

// u[0], u[1]: U(d) g / |d|, 0 within the guard distance; NC = 5: u[2..4] the entries 11,
// 12, 22 of U(d) / |d| (functions.jl:278-281)
template <int NC>
__device__ __forceinline__ void pair_u64(double d1, double d2, double g1, double g2,
                                         double (&u)[NC]) {
    const double q11 = d1 * d1;
    const double r2 = fma(d2, d2, q11);
    bool ok = __double_as_longlong(r2) >= CO_R2_MIN_BITS;
    double xr = ok ? r2 : 1.0;
    double y = rsqrt_seed64(xr);
    double t = xr * y;
    double e = fma(-t, y, 1.0);
    double p = fma(0.375, e, 0.5);
    double ye = y * e;
    y = fma(ye, p, y);
    double dg = d1 * g1;
    dg = fma(d2, g2, dg);
    double y2 = y * y;
    double cc = dg * y2;
    double t1 = fma(-d1, cc, g1);
    double t2 = fma(-d2, cc, g2);
    double ym = ok ? y : 0.0;
    u[0] = t1 * ym;
    u[1] = t2 * ym;
    if (NC == 5) {
        u[2] = fma(-q11, y2, 1.0) * ym;
        u[3] = -(d1 * d2 * y2) * ym;
        u[NC - 1] = fma(-(d2 * d2), y2, 1.0) * ym;
    }
}

__device__ __forceinline__ bool sym_skip(int nt, int H, int I, int k) {
    return k > 0 && (nt & 1) == 0 && k == H && I >= nt / 2;
}

template <int W, int NC>
struct sym64_smem {
    double2 x[32 * W], g[32 * W];
    double w[32 * W];
    double acc[NC][32 * W];
};

// Tile I of T = 32 W markers against the tiles I + k, k0 <= k < k1, one target per
// thread: target sums to gp, the sources' to their slots in apart (the first is ka's)
template <int W, int NC>
__device__ __forceinline__ void sym64_item(sym64_smem<W, NC> &sm, const double2 *__restrict__ px,
                                           const double2 *__restrict__ pg,
                                           const double *__restrict__ pw, int nt, int H, int I,
                                           int k0, int k1, int ka, double *__restrict__ gp,
                                           double *__restrict__ apart) {
    constexpr int T = 32 * W;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double2 xg = px[I * T + tid], Gg = pg[I * T + tid];
    const double wg = pw[I * T + tid];
    double ga[NC];
#pragma unroll
    for (int i = 0; i < NC; i++) ga[i] = 0.0;
    for (int k = k0; k < k1; k++) {
        if (sym_skip(nt, H, I, k)) continue;
        const int J = (I + k) % nt;
        __syncthreads();
        sm.x[tid] = px[J * T + tid];
        sm.g[tid] = pg[J * T + tid];
        sm.w[tid] = pw[J * T + tid];
#pragma unroll
        for (int i = 0; i < NC; i++) sm.acc[i][tid] = 0.0;
        __syncthreads();
        if (k == 0) {  // diagonal tile: ordered pairs, self excluded by the guard
#pragma unroll 4
            for (int a = 0; a < T; a++) {
                double u[NC];
                const double2 xa = sm.x[a], Ga = sm.g[a];
                pair_u64(xg.x - xa.x, xg.y - xa.y, Ga.x - Gg.x, Ga.y - Gg.y, u);
#pragma unroll
                for (int i = 0; i < NC; i++) ga[i] = fma(sm.w[a], u[i], ga[i]);
            }
            continue;
        }
        for (int r = 0; r < W; r++) {
            const int base = ((warp + r) & (W - 1)) * 32;
            double b[NC];
#pragma unroll
            for (int i = 0; i < NC; i++) b[i] = sm.acc[i][base + lane];
#pragma unroll 4
            for (int q = 0; q < 32; q++) {
                const int ai = base + ((lane + q) & 31);
                const double2 xa = sm.x[ai], Ga = sm.g[ai];
                const double wa = sm.w[ai];
                double u[NC];
                pair_u64(xg.x - xa.x, xg.y - xa.y, Ga.x - Gg.x, Ga.y - Gg.y, u);
#pragma unroll
                for (int i = 0; i < NC; i++) {
                    ga[i] = fma(wa, u[i], ga[i]);
                    // F's terms change sign with the pair's order, the metric's do not
                    b[i] = fma(i < 2 ? -wg : wg, u[i], b[i]);
                    b[i] = __shfl_sync(0xffffffffu, b[i], (lane + 1) & 31);
                }
            }
#pragma unroll
            for (int i = 0; i < NC; i++) sm.acc[i][base + lane] = b[i];
            __syncthreads();
        }
        double *ap = apart + ((size_t)(k - ka) * nt + J) * NC * T;
#pragma unroll
        for (int i = 0; i < NC; i++) ap[i * T + tid] = sm.acc[i][tid];
    }
#pragma unroll
    for (int i = 0; i < NC; i++) gp[i * T + tid] = ga[i];
}
