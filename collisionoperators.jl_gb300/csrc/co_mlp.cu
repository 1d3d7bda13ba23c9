// co_mlp.cu -- the learned warm start: a small MLP trained and evaluated by
// this library's own kernels.
//
// Network: n_in -> 64 -> 64 -> 64 -> n_out, GELU (erf form) after the three
// hidden layers. The weight matrices are BF16 (the copy every kernel reads); an
// FP32 master copy and the Adam moments live beside them; biases are FP32.
// Every kernel converts the BF16 weights to FP32 in shared memory and
// accumulates in FP32. Loss: mean squared error over samples and outputs.
// Training is deterministic run to run: gradients are summed over a tile's
// samples in order, over a block's tiles, then over the blocks.
//
// Used as the warm start of the implicit step: the network maps per-marker
// features at the start of a step (velocity, entropy gradient, predictor
// velocity, log-density and its gradient) to the normalised correction
// (v_converged - v_Euler)/dt^2, in the spirit of the reference's planned
// "Euler + dt^2 * delta" correction (Parameters.jl:108-112). The solver keeps
// the last word: the caller keeps the plain predictor whenever the learned
// proposal's first residual is larger.
#include <cuda_bf16.h>
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <vector>

#include "co_internal.cuh"

#define MLP_H 64
#define MLP_MAX_IN 16
#define MLP_MAX_OUT 4

struct co_mlp {
    int device;
    int n_in, n_out;
    size_t P;                    // number of parameters
    float *master;               // FP32 parameters (layout below)
    __nv_bfloat16 *wbf;          // BF16 copy of all parameters (weights used in BF16)
    float *grad, *m1, *m2;       // gradient and Adam moments
    int step;
    // training scratch: a row of P gradients and an FP64 loss per block, then the loss
    float *part;
    double *lpart;
    int cap, nsm;
    // feature and output normalisation applied by co_mlp_forward (inference):
    // [mean (MLP_MAX_IN), 1/std (MLP_MAX_IN), out std (MLP_MAX_OUT), out mean
    // (MLP_MAX_OUT)]; NULL = none. Training kernels see normalised data as given.
    float *norm;
};
#define MLP_NORM_FLOATS (2 * MLP_MAX_IN + 2 * MLP_MAX_OUT)

// parameter offsets: W0 [H][n_in], b0 [H], W1 [H][H], b1 [H], W2 [H][H], b2 [H],
// W3 [n_out][H], b3 [n_out]
struct mlp_off {
    int W0, b0, W1, b1, W2, b2, W3, b3, P;
};
__host__ __device__ inline mlp_off mlp_offsets(int n_in, int n_out) {
    mlp_off o;
    o.W0 = 0;
    o.b0 = o.W0 + MLP_H * n_in;
    o.W1 = o.b0 + MLP_H;
    o.b1 = o.W1 + MLP_H * MLP_H;
    o.W2 = o.b1 + MLP_H;
    o.b2 = o.W2 + MLP_H * MLP_H;
    o.W3 = o.b2 + MLP_H;
    o.b3 = o.W3 + n_out * MLP_H;
    o.P = o.b3 + n_out;
    return o;
}

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_d(float x) {
    return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) +
           x * 0.39894228040143268f * expf(-0.5f * x * x);
}

// ---------------------------------------------------------------- tile kernels
//
// A block of 256 threads takes a tile of 64 samples through the network; the tile's
// activations and one layer's weights stay in shared memory. Every product is a
// 64 x 64 output with a 4 x 4 register block per thread (two 16-byte shared loads
// per 16 FMAs), FP32 accumulation in ascending order of the summed index.
// What bounds a training step is latency: one tile per SM at the usual minibatch
// (8,192 samples: 128 tiles), nine dependent products with barriers between them,
// 43 us, and 15 us to add up 128 gradient rows. Forward, loss and gradients as one
// launch instead of a thread per sample for each pass and a thread per parameter
// walking the minibatch: 2.05 ms -> 84 us a step with its loss on the host.
#define MLP_T 64            // samples of a tile
#define MLP_THREADS 256
#define MLP_LD 68           // row length of the tile arrays (64 + 4: conflict-free columns)
typedef float mlp_tile[64][MLP_LD];

// acc[r][c] += sum_k A[k][4 ty + r] B[k][4 tx + c], k < K
__device__ __forceinline__ void tile_mac(const mlp_tile &A, const mlp_tile &B, int K, int ty, int tx,
                                         float (&acc)[4][4]) {
#pragma unroll 4
    for (int k = 0; k < K; k++) {
        const float4 a = *reinterpret_cast<const float4 *>(&A[k][4 * ty]);
        const float4 b = *reinterpret_cast<const float4 *>(&B[k][4 * tx]);
        const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) acc[r][c] = fmaf(av[r], bv[c], acc[r][c]);
    }
}

// W (rows x cols, BF16, row-major) into shared memory: T[col][row] (transposed) or
// T[row][col]
__device__ __forceinline__ void load_weights(const __nv_bfloat16 *__restrict__ w, int rows, int cols,
                                             bool transposed, mlp_tile &T) {
    for (int i = threadIdx.x; i < rows * cols; i += MLP_THREADS) {
        const int r = i / cols, c = i - r * cols;
        const float v = __bfloat162float(w[i]);
        if (transposed) T[c][r] = v;
        else T[r][c] = v;
    }
}

// the tile's inputs, transposed (X[input][sample], 0 past the batch), normalised
// where norm is set
__device__ __forceinline__ void load_inputs(const float *__restrict__ X, int n_in, int s0, int B,
                                            const float *__restrict__ norm, mlp_tile &T) {
    for (int i = threadIdx.x; i < MLP_T * n_in; i += MLP_THREADS) {
        const int s = i / n_in, c = i - s * n_in;
        float x = 0.f;
        if (s0 + s < B) {
            x = X[(size_t)(s0 + s) * n_in + c];
            if (norm) x = (x - norm[c]) * norm[MLP_MAX_IN + c];
        }
        T[c][s] = x;
    }
}

// hidden layer: out[unit][sample] = gelu(z), z = bias + W in; with dout, gelu'(z)
__device__ __forceinline__ void hidden_layer(const mlp_tile &in, const mlp_tile &Wt, int K,
                                             const float *__restrict__ bias, int ty, int tx,
                                             mlp_tile &out, mlp_tile *dout) {
    float acc[4][4];   // [unit][sample]
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const float bv = bias[4 * ty + r];
#pragma unroll
        for (int c = 0; c < 4; c++) acc[r][c] = bv;
    }
    tile_mac(Wt, in, K, ty, tx, acc);
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
            out[4 * ty + r][4 * tx + c] = gelu(acc[r][c]);
            if (dout) (*dout)[4 * ty + r][4 * tx + c] = gelu_d(acc[r][c]);
        }
}

// y[k][sample] of the output layer: thread t takes sample t % 64 and output t / 64
__device__ __forceinline__ float output_layer(const mlp_tile &a, const __nv_bfloat16 *__restrict__ w3,
                                              const float *__restrict__ b3, int k, int s) {
    float v = b3[k];
#pragma unroll 8
    for (int i = 0; i < MLP_H; i++) v = fmaf(__bfloat162float(w3[k * MLP_H + i]), a[i][s], v);
    return v;
}

struct mlp_fwd_smem {
    mlp_tile x, a, b, w;
};

__global__ void __launch_bounds__(MLP_THREADS)
k_mlp_forward(const __nv_bfloat16 *__restrict__ wbf, const float *__restrict__ master, int n_in,
              int n_out, const float *__restrict__ X, int B, float *__restrict__ Y,
              const float *__restrict__ norm) {
    extern __shared__ __align__(16) unsigned char raw[];
    mlp_fwd_smem &sm = *reinterpret_cast<mlp_fwd_smem *>(raw);
    const mlp_off o = mlp_offsets(n_in, n_out);
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15, s0 = blockIdx.x * MLP_T;
    load_inputs(X, n_in, s0, B, norm, sm.x);
    load_weights(wbf + o.W0, MLP_H, n_in, true, sm.w);
    __syncthreads();
    hidden_layer(sm.x, sm.w, n_in, master + o.b0, ty, tx, sm.a, nullptr);
    __syncthreads();
    load_weights(wbf + o.W1, MLP_H, MLP_H, true, sm.w);
    __syncthreads();
    hidden_layer(sm.a, sm.w, MLP_H, master + o.b1, ty, tx, sm.b, nullptr);
    __syncthreads();
    load_weights(wbf + o.W2, MLP_H, MLP_H, true, sm.w);
    __syncthreads();
    hidden_layer(sm.b, sm.w, MLP_H, master + o.b2, ty, tx, sm.a, nullptr);
    __syncthreads();
    const int k = threadIdx.x >> 6, s = threadIdx.x & 63;
    if (k < n_out && s0 + s < B) {
        float y = output_layer(sm.a, wbf + o.W3, master + o.b3, k, s);
        if (norm) y = fmaf(y, norm[2 * MLP_MAX_IN + k], norm[2 * MLP_MAX_IN + MLP_MAX_OUT + k]);
        Y[(size_t)(s0 + s) * n_out + k] = y;
    }
}

// Forward, loss and gradients in one launch. A block walks tiles blockIdx.x,
// blockIdx.x + gridDim.x, ... and keeps the gradients of its tiles in registers
// (the two 64 x 64 matrices, a 4 x 4 block per thread) and shared memory (the
// rest); it writes one row of P partial gradients and its FP64 loss partial. The
// rows are added in block order by k_mlp_reduce: deterministic.
struct mlp_train_smem {
    mlp_tile x, a0, a1, a2;      // activations [unit][sample]
    mlp_tile g0, g1, g2;         // gelu'(z)
    mlp_tile w, d, t;            // weights; deltas [unit][sample]; transposed scratch
    float dy[MLP_MAX_OUT][MLP_T];
    float gW0[MLP_H * MLP_MAX_IN], gW3[MLP_MAX_OUT * MLP_H], gb[3][MLP_H], gb3[MLP_MAX_OUT];
    double loss[MLP_THREADS / 32];
};

// T[sample][unit] = A[unit][sample]
__device__ __forceinline__ void transpose_tile(const mlp_tile &A, mlp_tile &T) {
    for (int i = threadIdx.x; i < 64 * 64; i += MLP_THREADS) T[i & 63][i >> 6] = A[i >> 6][i & 63];
}

// dW[out][in] += sum_s delta[out][s] act[in][s]: both transposed first so that the
// sample is the summed row index; db[out] += sum_s delta[out][s]
__device__ __forceinline__ void weight_grad(const mlp_tile &act, mlp_tile &delta_t, mlp_tile &act_t,
                                            int ty, int tx, float (&acc)[4][4], float *db) {
    transpose_tile(act, act_t);
    __syncthreads();
    tile_mac(delta_t, act_t, MLP_T, ty, tx, acc);
    if (threadIdx.x < MLP_H) {
        float s = 0.f;
        for (int k = 0; k < MLP_T; k++) s += delta_t[k][threadIdx.x];
        db[threadIdx.x] += s;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(MLP_THREADS)
k_mlp_train(const __nv_bfloat16 *__restrict__ wbf, const float *__restrict__ master, int n_in,
            int n_out, const float *__restrict__ X, const float *__restrict__ T, int B,
            float *__restrict__ part, double *__restrict__ lpart) {
    extern __shared__ __align__(16) unsigned char raw[];
    mlp_train_smem &sm = *reinterpret_cast<mlp_train_smem *>(raw);
    const mlp_off o = mlp_offsets(n_in, n_out);
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const float scale = 2.0f / ((float)B * (float)n_out);
    for (int i = tid; i < MLP_H * MLP_MAX_IN; i += MLP_THREADS) sm.gW0[i] = 0.f;
    for (int i = tid; i < MLP_MAX_OUT * MLP_H; i += MLP_THREADS) sm.gW3[i] = 0.f;
    if (tid < 3 * MLP_H) sm.gb[tid / MLP_H][tid % MLP_H] = 0.f;
    if (tid < MLP_MAX_OUT) sm.gb3[tid] = 0.f;
    float gW1[4][4], gW2[4][4];
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int c = 0; c < 4; c++) gW1[r][c] = gW2[r][c] = 0.f;
    double loss = 0.0;
    const int tiles = (B - 1) / MLP_T + 1;   // counted in tiles: a sample index would overflow
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int s0 = tile * MLP_T;
        __syncthreads();
        load_inputs(X, n_in, s0, B, nullptr, sm.x);
        load_weights(wbf + o.W0, MLP_H, n_in, true, sm.w);
        __syncthreads();
        hidden_layer(sm.x, sm.w, n_in, master + o.b0, ty, tx, sm.a0, &sm.g0);
        __syncthreads();
        load_weights(wbf + o.W1, MLP_H, MLP_H, true, sm.w);
        __syncthreads();
        hidden_layer(sm.a0, sm.w, MLP_H, master + o.b1, ty, tx, sm.a1, &sm.g1);
        __syncthreads();
        load_weights(wbf + o.W2, MLP_H, MLP_H, true, sm.w);
        __syncthreads();
        hidden_layer(sm.a1, sm.w, MLP_H, master + o.b2, ty, tx, sm.a2, &sm.g2);
        __syncthreads();
        // output, loss and its gradient
        const int k = tid >> 6, s = tid & 63;
        float dy = 0.f;
        if (k < n_out && s0 + s < B) {
            const float e = output_layer(sm.a2, wbf + o.W3, master + o.b3, k, s) -
                            T[(size_t)(s0 + s) * n_out + k];
            dy = scale * e;
            loss += (double)e * (double)e;
        }
        sm.dy[k][s] = dy;
        __syncthreads();
        // W3: dy a2^T; d = W3^T dy * gelu'(z2)
        for (int i = tid; i < n_out * MLP_H; i += MLP_THREADS) {
            const int kk = i / MLP_H, j = i - kk * MLP_H;
            float v = 0.f;
            for (int q = 0; q < MLP_T; q++) v = fmaf(sm.dy[kk][q], sm.a2[j][q], v);
            sm.gW3[i] += v;
        }
        if (tid < n_out) {
            float v = 0.f;
            for (int q = 0; q < MLP_T; q++) v += sm.dy[tid][q];
            sm.gb3[tid] += v;
        }
        // deltas are kept transposed, t[sample][unit]: the row the gradients sum over
        for (int i = tid; i < 64 * 64; i += MLP_THREADS) {
            const int u = i & 63, q = i >> 6;
            float v = 0.f;
#pragma unroll
            for (int kk = 0; kk < MLP_MAX_OUT; kk++)
                if (kk < n_out) v = fmaf(__bfloat162float(wbf[o.W3 + kk * MLP_H + u]), sm.dy[kk][q], v);
            v *= sm.g2[u][q];
            sm.t[q][u] = v;
            sm.d[u][q] = v;
        }
        // layer 2 weights (not transposed): row = output unit, the index W^T delta sums
        load_weights(wbf + o.W2, MLP_H, MLP_H, false, sm.w);
        __syncthreads();
        weight_grad(sm.a1, sm.t, sm.a2, ty, tx, gW2, sm.gb[2]);
        // delta1[in][s] = sum_out W2[out][in] delta2[out][s] * gelu'(z1)
        float acc[4][4];
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) acc[r][c] = 0.f;
        tile_mac(sm.w, sm.d, MLP_H, ty, tx, acc);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const float v = acc[r][c] * sm.g1[4 * ty + r][4 * tx + c];
                sm.d[4 * ty + r][4 * tx + c] = v;
                sm.t[4 * tx + c][4 * ty + r] = v;
                acc[r][c] = 0.f;
            }
        load_weights(wbf + o.W1, MLP_H, MLP_H, false, sm.w);
        __syncthreads();
        weight_grad(sm.a0, sm.t, sm.a2, ty, tx, gW1, sm.gb[1]);
        tile_mac(sm.w, sm.d, MLP_H, ty, tx, acc);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 4; c++)
                sm.d[4 * ty + r][4 * tx + c] = acc[r][c] * sm.g0[4 * ty + r][4 * tx + c];
        __syncthreads();
        // W0: delta0 x^T and its bias
        for (int i = tid; i < MLP_H * n_in; i += MLP_THREADS) {
            const int j = i / n_in, c = i - j * n_in;
            float v = 0.f;
            for (int q = 0; q < MLP_T; q++) v = fmaf(sm.d[j][q], sm.x[c][q], v);
            sm.gW0[i] += v;
        }
        if (tid < MLP_H) {
            float v = 0.f;
            for (int q = 0; q < MLP_T; q++) v += sm.d[tid][q];
            sm.gb[0][tid] += v;
        }
    }
    __syncthreads();
    float *g = part + (size_t)blockIdx.x * o.P;
    for (int i = tid; i < MLP_H * n_in; i += MLP_THREADS) g[o.W0 + i] = sm.gW0[i];
    for (int i = tid; i < n_out * MLP_H; i += MLP_THREADS) g[o.W3 + i] = sm.gW3[i];
    if (tid < MLP_H) {
        g[o.b0 + tid] = sm.gb[0][tid];
        g[o.b1 + tid] = sm.gb[1][tid];
        g[o.b2 + tid] = sm.gb[2][tid];
    }
    if (tid < n_out) g[o.b3 + tid] = sm.gb3[tid];
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
            g[o.W1 + (4 * ty + r) * MLP_H + 4 * tx + c] = gW1[r][c];
            g[o.W2 + (4 * ty + r) * MLP_H + 4 * tx + c] = gW2[r][c];
        }
    for (int sft = 16; sft > 0; sft >>= 1) loss += __shfl_down_sync(0xffffffffu, loss, sft);
    if ((tid & 31) == 0) sm.loss[tid >> 5] = loss;
    __syncthreads();
    if (tid == 0) {
        for (int i = 1; i < MLP_THREADS / 32; i++) loss += sm.loss[i];
        lpart[blockIdx.x] = loss;
    }
}

// Gradient of every parameter from the block rows, in block order (eight rows in
// flight), and the mean squared error
__device__ __forceinline__ float grad_sum(const float *__restrict__ part, int nb, int P, int p) {
    float s = 0.f;
    int b = 0;
    for (; b + 8 <= nb; b += 8) {
        float t[8];
#pragma unroll
        for (int u = 0; u < 8; u++) t[u] = part[(size_t)(b + u) * P + p];
        s += ((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7]));
    }
    for (; b < nb; b++) s += part[(size_t)b * P + p];
    return s;
}
__device__ __forceinline__ void loss_sum(const double *__restrict__ lpart, int nb, double n,
                                         float *loss) {
    double s = 0.0;
    for (int b = 0; b < nb; b++) s += lpart[b];
    *loss = (float)(s / n);
}

__global__ void __launch_bounds__(64)
k_mlp_reduce(int P, int nb, const float *__restrict__ part, const double *__restrict__ lpart,
             double n, float *__restrict__ grad, float *__restrict__ loss) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < P) grad[p] = grad_sum(part, nb, P, p);
    if (p == 0) loss_sum(lpart, nb, n, loss);
}

// the gradient and one Adam update of every parameter
__global__ void __launch_bounds__(64)
k_mlp_adam(int P, int nb, const float *__restrict__ part, const double *__restrict__ lpart,
           double n, float *__restrict__ loss, float lr, float b1, float b2, float eps, int step,
           float *__restrict__ master, __nv_bfloat16 *__restrict__ wbf, float *__restrict__ grad,
           float *__restrict__ m1, float *__restrict__ m2) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p == 0) loss_sum(lpart, nb, n, loss);
    if (p >= P) return;
    const float g = grad_sum(part, nb, P, p);
    grad[p] = g;
    float a = b1 * m1[p] + (1.f - b1) * g;
    float v = b2 * m2[p] + (1.f - b2) * g * g;
    m1[p] = a;
    m2[p] = v;
    float ah = a / (1.f - powf(b1, (float)step));
    float vh = v / (1.f - powf(b2, (float)step));
    float w = master[p] - lr * ah / (sqrtf(vh) + eps);
    master[p] = w;
    wbf[p] = __float2bfloat16_rn(w);
}

__global__ void k_mlp_refresh(int P, const float *__restrict__ master, __nv_bfloat16 *__restrict__ wbf) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < P) wbf[p] = __float2bfloat16_rn(master[p]);
}

// ---------------------------------------------------------------- host

// block rows of the training kernel: one block per tile up to the SM count (a block
// fills an SM's shared memory)
static int mlp_grid(const co_mlp *m, int B) {
    const int t = co_cdiv(B, MLP_T);
    return t < m->nsm ? t : m->nsm;
}

static int mlp_ensure(co_mlp *m, int nb) {
    if (nb <= m->cap) return CO_OK;
    cudaFree(m->part);
    cudaFree(m->lpart);
    m->part = nullptr;
    m->lpart = nullptr;
    m->cap = 0;
    if (cudaMalloc(&m->part, sizeof(float) * (size_t)nb * m->P) != cudaSuccess ||
        cudaMalloc(&m->lpart, sizeof(double) * nb + sizeof(float)) != cudaSuccess)
        return co_nomem();
    m->cap = nb;
    return CO_OK;
}

extern "C" int co_mlp_create(int n_in, int n_out, unsigned seed, int device, co_mlp **out) {
    if (!out || n_in < 1 || n_in > MLP_MAX_IN || n_out < 1 || n_out > MLP_MAX_OUT)
        return CO_ERR_ARG;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return CO_ERR_NODEVICE;
    CO_CK(cudaSetDevice(device));
    co_mlp *m = (co_mlp *)calloc(1, sizeof(co_mlp));
    m->device = device;
    m->n_in = n_in;
    m->n_out = n_out;
    mlp_off o = mlp_offsets(n_in, n_out);
    m->P = o.P;
    // He-style init with a small LCG (deterministic from the seed)
    std::vector<float> h(o.P, 0.f);
    unsigned long long st = 0x9E3779B97F4A7C15ull ^ seed;
    auto unif = [&]() {
        st = st * 6364136223846793005ull + 1442695040888963407ull;
        return ((st >> 40) & 0xFFFFFF) / 16777216.0f * 2.f - 1.f;
    };
    for (int i = o.W0; i < o.b0; i++) h[i] = unif() * sqrtf(3.f * 2.f / n_in);
    for (int i = o.W1; i < o.b1; i++) h[i] = unif() * sqrtf(3.f * 2.f / MLP_H);
    for (int i = o.W2; i < o.b2; i++) h[i] = unif() * sqrtf(3.f * 2.f / MLP_H);
    for (int i = o.W3; i < o.b3; i++) h[i] = unif() * sqrtf(3.f / MLP_H) * 0.1f;
    if (cudaMalloc(&m->master, sizeof(float) * o.P) != cudaSuccess ||
        cudaMalloc(&m->wbf, sizeof(__nv_bfloat16) * o.P) != cudaSuccess ||
        cudaMalloc(&m->grad, sizeof(float) * o.P) != cudaSuccess ||
        cudaMalloc(&m->m1, sizeof(float) * o.P) != cudaSuccess ||
        cudaMalloc(&m->m2, sizeof(float) * o.P) != cudaSuccess) {
        co_mlp_destroy(m);
        return co_nomem();
    }
    cudaMemcpy(m->master, h.data(), sizeof(float) * o.P, cudaMemcpyHostToDevice);
    cudaMemset(m->m1, 0, sizeof(float) * o.P);
    cudaMemset(m->m2, 0, sizeof(float) * o.P);
    k_mlp_refresh<<<co_cdiv(o.P, 256), 256>>>((int)o.P, m->master, m->wbf);
    cudaFuncSetAttribute(k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(mlp_fwd_smem));
    cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(mlp_train_smem));
    if (cudaDeviceGetAttribute(&m->nsm, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
        co_mlp_destroy(m);
        return CO_ERR_CUDA;
    }
    if (cudaDeviceSynchronize() != cudaSuccess) {
        co_mlp_destroy(m);
        return CO_ERR_CUDA;
    }
    *out = m;
    return CO_OK;
}

extern "C" int co_mlp_destroy(co_mlp *m) {
    if (!m) return CO_ERR_ARG;
    cudaSetDevice(m->device);
    void *ptrs[] = {m->master, m->wbf, m->grad, m->m1, m->m2, m->part, m->lpart, m->norm};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    free(m);
    return CO_OK;
}

extern "C" int co_mlp_num_params(const co_mlp *m, int *P) {
    if (!m || !P) return CO_ERR_ARG;
    *P = (int)m->P;
    return CO_OK;
}

extern "C" int co_mlp_set_params(co_mlp *m, const float *host) {
    if (!m || !host) return CO_ERR_ARG;
    CO_CK(cudaSetDevice(m->device));
    CO_CK(cudaMemcpy(m->master, host, sizeof(float) * m->P, cudaMemcpyHostToDevice));
    CO_CK(cudaMemset(m->m1, 0, sizeof(float) * m->P));
    CO_CK(cudaMemset(m->m2, 0, sizeof(float) * m->P));
    m->step = 0;
    k_mlp_refresh<<<co_cdiv(m->P, 256), 256>>>((int)m->P, m->master, m->wbf);
    CO_CK(cudaDeviceSynchronize());
    return CO_OK;
}

extern "C" int co_mlp_get_params(const co_mlp *m, float *host) {
    if (!m || !host) return CO_ERR_ARG;
    CO_CK(cudaSetDevice(m->device));
    CO_CK(cudaMemcpy(host, m->master, sizeof(float) * m->P, cudaMemcpyDeviceToHost));
    return CO_OK;
}

extern "C" int co_mlp_set_normalization(co_mlp *m, const double *x_mean, const double *x_std,
                                        const double *y_mean, const double *y_std) {
    if (!m) return CO_ERR_ARG;
    CO_CK(cudaSetDevice(m->device));
    if (!x_mean) {
        if (m->norm) cudaFree(m->norm);
        m->norm = nullptr;
        return CO_OK;
    }
    if (!x_std || !y_mean || !y_std) return CO_ERR_ARG;
    float h[MLP_NORM_FLOATS] = {0.f};
    for (int i = 0; i < m->n_in; i++) {
        if (!(x_std[i] > 0.0) || !isfinite(x_mean[i])) return CO_ERR_ARG;
        h[i] = (float)x_mean[i];
        h[MLP_MAX_IN + i] = (float)(1.0 / x_std[i]);
    }
    for (int k = 0; k < m->n_out; k++) {
        if (!isfinite(y_std[k]) || !isfinite(y_mean[k])) return CO_ERR_ARG;
        h[2 * MLP_MAX_IN + k] = (float)y_std[k];
        h[2 * MLP_MAX_IN + MLP_MAX_OUT + k] = (float)y_mean[k];
    }
    if (!m->norm && cudaMalloc(&m->norm, sizeof(h)) != cudaSuccess) return co_nomem();
    CO_CK(cudaMemcpy(m->norm, h, sizeof(h), cudaMemcpyHostToDevice));
    return CO_OK;
}

// Y = net(X) for B samples (device pointers, row-major B x n_in / B x n_out),
// with the normalisation of co_mlp_set_normalization applied if set
extern "C" int co_mlp_forward(co_mlp *m, const float *X, int B, float *Y, void *stream) {
    if (!m || B < 0 || (B > 0 && (!X || !Y))) return CO_ERR_ARG;
    if (B == 0) return CO_OK;
    CO_CK(cudaSetDevice(m->device));
    k_mlp_forward<<<co_cdiv(B, MLP_T), MLP_THREADS, sizeof(mlp_fwd_smem), (cudaStream_t)stream>>>(
        m->wbf, m->master, m->n_in, m->n_out, X, B, Y, m->norm);
    CO_CK(cudaGetLastError());
    return CO_OK;
}

// block rows of the gradient and the loss; *nb rows
static int mlp_grad(co_mlp *m, const float *X, const float *T, int B, int *nb) {
    *nb = mlp_grid(m, B);
    int rc = mlp_ensure(m, *nb);
    if (rc) return rc;
    k_mlp_train<<<*nb, MLP_THREADS, sizeof(mlp_train_smem)>>>(m->wbf, m->master, m->n_in, m->n_out,
                                                            X, T, B, m->part, m->lpart);
    CO_CK(cudaGetLastError());
    return CO_OK;
}
static float *mlp_loss(const co_mlp *m) { return (float *)(m->lpart + m->cap); }

// gradients of the mean squared error w.r.t. all parameters (host array of P)
extern "C" int co_mlp_gradients(co_mlp *m, const float *X, const float *T, int B, float *grad,
                                float *loss) {
    if (!m || !X || !T || !grad || B < 1) return CO_ERR_ARG;
    CO_CK(cudaSetDevice(m->device));
    int nb = 0;
    int rc = mlp_grad(m, X, T, B, &nb);
    if (rc) return rc;
    k_mlp_reduce<<<co_cdiv(m->P, 64), 64>>>((int)m->P, nb, m->part, m->lpart,
                                           (double)B * m->n_out, m->grad, mlp_loss(m));
    CO_CK(cudaGetLastError());
    if (loss) CO_CK(cudaMemcpy(loss, mlp_loss(m), sizeof(float), cudaMemcpyDeviceToHost));
    CO_CK(cudaMemcpy(grad, m->grad, sizeof(float) * m->P, cudaMemcpyDeviceToHost));
    return CO_OK;
}

// one Adam step on a minibatch (device X: B x n_in, T: B x n_out)
extern "C" int co_mlp_train_step(co_mlp *m, const float *X, const float *T, int B, float lr,
                                 float *loss) {
    if (!m || !X || !T || B < 1) return CO_ERR_ARG;
    CO_CK(cudaSetDevice(m->device));
    int nb = 0;
    int rc = mlp_grad(m, X, T, B, &nb);
    if (rc) return rc;
    m->step += 1;
    k_mlp_adam<<<co_cdiv(m->P, 64), 64>>>((int)m->P, nb, m->part, m->lpart, (double)B * m->n_out,
                                         mlp_loss(m), lr, 0.9f, 0.999f, 1e-8f, m->step, m->master,
                                         m->wbf, m->grad, m->m1, m->m2);
    CO_CK(cudaGetLastError());
    if (loss) CO_CK(cudaMemcpy(loss, mlp_loss(m), sizeof(float), cudaMemcpyDeviceToHost));
    return CO_OK;
}
