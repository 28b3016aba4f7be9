// mlp.cuh -- the learned Newton guess of the exact Euler solver.
//
// Network: 6 -> 32 -> 32 -> 1, tanh hidden layers, linear output; inputs and
// output as in exact_euler::features (the guess is p0 * exp(w * y), p0 the
// adaptive PVRS guess, w = J^2/(1+J^2) a jump weight, so a weak wave keeps the
// accurate PVRS value).  Parameters (FP32, 1313): W1[32][6], b1[32],
// W2[32][32], b2[32], W3[32], b3.
//
// Training (all kernels of this file, FP32): k_gen_samples draws seeded
// Riemann problems and solves each to tol by FP64 Newton; k_train_epoch runs the
// minibatches of an epoch: forward and backward, each CTA's gradient sums in a row
// of a partial-sum array, then the sum of the rows and Adam.  k_train_grad and
// k_train_update are the same two halves as launches of their own (the gradient
// alone; devices without cooperative launches).
//
// Inference: k_mlp_guess_tc, one thread per grid site, evaluates the MLP for
// the x- and y-interface of the site (interfaces with a weak jump keep the
// PVRS guess) in BF16 on the tensor cores with FP32 accumulation --
// tcgen05.mma from shared-memory operands into TMEM accumulators, 128
// interfaces per MMA tile -- and writes the guesses that the step kernel's
// Newton iteration starts from.  k_mlp_guess is the same pass on the
// warp-level mma.sync.m16n8k16 (64 interfaces = 4 row tiles per warp; a
// layer's accumulator fragments are exactly the next layer's A fragments),
// kept as the comparison path (claw2_mlp_set_engine).
#pragma once

#include <cuda_bf16.h>

#include "riemann.cuh"

namespace claw2 {

constexpr int MLP_IN = 6, MLP_H = 32;
// Jump weight below which the learned correction is not applied (J^2 < 0.053).
constexpr double MLP_WMIN = 0.05;
constexpr int MLP_NPARAM = MLP_H * MLP_IN + MLP_H + MLP_H * MLP_H + MLP_H + MLP_H + 1;  // 1313
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + MLP_H * MLP_IN, OFF_W2 = OFF_B1 + MLP_H,
              OFF_B2 = OFF_W2 + MLP_H * MLP_H, OFF_W3 = OFF_B2 + MLP_H, OFF_B3 = OFF_W3 + MLP_H;

// ---- counter-based random numbers (splitmix64 finaliser of seed ^ index) ----
__host__ __device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__host__ __device__ __forceinline__ double u01(unsigned long long seed, unsigned long long i, int k) {
    const unsigned long long z = mix64(seed ^ mix64(i * 8ull + (unsigned long long)k));
    return (double)(z >> 11) * (1.0 / 9007199254740992.0);  // [0, 1)
}

// The training distribution: rho, p log-uniform in [1e-2, 1e2], u uniform in
// [-3, 3] on both sides.
__host__ __device__ __forceinline__ void draw_problem(unsigned long long seed, unsigned long long i, double& rl,
                                                      double& ul, double& pl, double& rr, double& ur, double& pr) {
    const double l10 = 2.302585092994046;
    rl = exp(l10 * (-2.0 + 4.0 * u01(seed, i, 0)));
    pl = exp(l10 * (-2.0 + 4.0 * u01(seed, i, 1)));
    ul = -3.0 + 6.0 * u01(seed, i, 2);
    rr = exp(l10 * (-2.0 + 4.0 * u01(seed, i, 3)));
    pr = exp(l10 * (-2.0 + 4.0 * u01(seed, i, 4)));
    ur = -3.0 + 6.0 * u01(seed, i, 5);
}

// x[i*8 + 0..5] features, x[i*8+6] = jump weight w, y[i] target, ok[i] = 0 for vacuum.
static __global__ void k_gen_samples(unsigned long long seed, long long first, int n, double gamma, double tol,
                                     float* x, float* y, int* ok, double* pstar) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const unsigned long long i = (unsigned long long)(first + k);
    double rl, ul, pl, rr, ur, pr;
    draw_problem(seed, i, rl, ul, pl, rr, ur, pr);
    const exact_euler::Gas G = exact_euler::make_gas(gamma);
    const double cl = sqrt(gamma * pl / rl), cr = sqrt(gamma * pr / rr);
    float f[6];
    double w;
    exact_euler::features(G, rl, ul, pl, rr, ur, pr, f, w);
    for (int j = 0; j < 6; ++j) x[(long long)k * 8 + j] = f[j];
    x[(long long)k * 8 + 6] = (float)w;
    x[(long long)k * 8 + 7] = 0.f;
    if (exact_euler::vacuum(G, ul, cl, ur, cr)) {
        ok[k] = 0;
        y[k] = 0.f;
        if (pstar) pstar[k] = 0.0;
        return;
    }
    double ps, us;
    int it;
    exact_euler::star(G, rl, ul, pl, cl, rr, ur, pr, cr, 0.0, tol, 200, ps, us, it);
    const double p0 = exact_euler::guess_pvrs(G, rl, ul, pl, cl, rr, ur, pr, cr);
    const bool good = ps > 0.0 && p0 > 0.0 && w > 1e-12;
    ok[k] = good ? 1 : 0;
    y[k] = good ? (float)(log(ps / p0) / w) : 0.f;
    if (pstar) pstar[k] = ps;
}

// ---- training ----------------------------------------------------------------
// Gradient of 0.5 * mean squared error over samples [first, first + count), in
// FP32 throughout.
//
// A minibatch of 16384 is 61 M multiply-adds, 2 us of the chip's FP32 rate, so
// the work is in not spending more than that on moving numbers.  One CTA takes
// tiles of TRAIN_TS = 64 samples with 256 threads: warp w holds samples
// 32 (w / 4) + lane and units 8 (w % 4) .. + 7 of each layer, so every weight it
// reads is the same for the whole warp (broadcast, four at a time) and a
// sample's activations pass between its four threads through shared memory.
// The weight gradients are products over the tile's samples, done as a small
// matrix product from shared memory (rows of TRAIN_LD = 68 floats: 16-byte
// aligned, eight rows on distinct banks): 2 x 2 entries of dW2 per thread, the
// other 290 sums one or two per thread.  They stay in registers over all tiles
// of the CTA and go out once, as one row of `part`; train_update adds the rows
// in a fixed order, so the result does not depend on scheduling.
// Measured per minibatch of 16384, with the update: 222 us with one sample per thread
// and a warp shuffle sum per parameter (five shuffles and an atomic on each of 1313
// numbers), 19.7 us in two launches of these tiles, 14.5 us in k_train_epoch.
constexpr int TRAIN_TS = 64, TRAIN_LD = 68, TRAIN_ROW = MLP_NPARAM + 1;  // (a row: the gradient, then the loss)
constexpr int TRAIN_EXTRA = OFF_W2 + (MLP_NPARAM - OFF_B2) + 1;          // sums other than dW2: 290

struct TrainSmem {
    float P[(MLP_NPARAM + 3) / 4 * 4];
    float h1[MLP_H][TRAIN_LD], h2[MLP_H][TRAIN_LD];  // activations [unit][sample]
    float z1[MLP_H][TRAIN_LD], z2[MLP_H][TRAIN_LD];  // loss derivatives at the pre-activations
    float x[MLP_IN][TRAIN_LD];
    float one[TRAIN_LD], dy[TRAIN_LD], loss[TRAIN_LD];
    float out[4][TRAIN_TS];  // output, by unit group
};

// What a thread of a training CTA reads of a tile: two numbers of one sample's features
// (for the CTA), and its own sample's target.
struct TrainIn {
    float2 x;
    float y;
    bool act;
};

__device__ __forceinline__ TrainIn train_load(const float* __restrict__ x, const float* __restrict__ y,
                                              const int* __restrict__ ok, long long first, int count, int t0) {
    const int tid = threadIdx.x, s = 32 * (tid >> 7) + (tid & 31);
    const int k = t0 + (tid >> 2), c = 2 * (tid & 3);
    TrainIn in;
    in.x = make_float2(0.f, 0.f);
    if (c < MLP_IN && k < count) in.x = *reinterpret_cast<const float2*>(x + (first + k) * 8 + c);
    in.act = t0 + s < count && ok[first + t0 + s];
    in.y = in.act ? y[first + t0 + s] : 0.f;
    return in;
}

// A thread's gradient sums: entries of dW2 (rows tj, tj + 16, columns ti, ti + 16), and
// one or two of the others, each the product of two rows over the samples.
struct TrainSums {
    int tj, ti;
    const float *ea[2], *eb[2];
    float g2[2][2], ge[2];

    __device__ __forceinline__ void rows_of(TrainSmem& S) {
        const int tid = threadIdx.x;
        tj = tid >> 4;
        ti = tid & 15;
        if (tid < TRAIN_LD) S.one[tid] = 1.f;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int o = tid + 256 * e;
            ea[e] = S.one;
            eb[e] = S.one;
            if (o < OFF_B1) { ea[e] = S.z1[o / MLP_IN]; eb[e] = S.x[o % MLP_IN]; }
            else if (o < OFF_W2) ea[e] = S.z1[o - OFF_B1];
            else if (o < OFF_W2 + 32) ea[e] = S.z2[o - OFF_W2];
            else if (o < OFF_W2 + 64) { ea[e] = S.h2[o - OFF_W2 - 32]; eb[e] = S.dy; }
            else if (o == OFF_W2 + 64) ea[e] = S.dy;
            else if (o == OFF_W2 + 65) ea[e] = S.loss;
        }
    }
    __device__ __forceinline__ void clear() {
        g2[0][0] = g2[0][1] = g2[1][0] = g2[1][1] = 0.f;
        ge[0] = ge[1] = 0.f;
    }
    __device__ __forceinline__ void store(float* row) const {
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) row[OFF_W2 + (tj + 16 * a) * MLP_H + ti + 16 * b] = g2[a][b];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int o = threadIdx.x + 256 * e;
            if (o < TRAIN_EXTRA) row[o < OFF_W2 ? o : OFF_B2 + (o - OFF_W2)] = ge[e];
        }
    }
};

// Forward and backward of one tile, its sums added to R.
__device__ __forceinline__ void train_tile(TrainSmem& S, const TrainIn& in, float inv_n, TrainSums& R) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int s = 32 * (warp >> 2) + lane;  // this thread's sample of the tile
    const int u0 = 8 * (warp & 3);          // and its units
    __syncthreads();  // parameters in place; the last tile's sums done
    if (2 * (tid & 3) < MLP_IN) {
        S.x[2 * (tid & 3)][tid >> 2] = in.x.x;
        S.x[2 * (tid & 3) + 1][tid >> 2] = in.x.y;
    }
    __syncthreads();
    float h1[8], h2[8];
    {
        float xi[MLP_IN];
#pragma unroll
        for (int i = 0; i < MLP_IN; ++i) xi[i] = S.x[i][s];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float z = S.P[OFF_B1 + u0 + j];
#pragma unroll
            for (int i = 0; i < MLP_IN; ++i) z = fmaf(S.P[OFF_W1 + (u0 + j) * MLP_IN + i], xi[i], z);
            h1[j] = tanhf(z);
            S.h1[u0 + j][s] = h1[j];
        }
    }
    __syncthreads();
    {
        float z[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) z[j] = S.P[OFF_B2 + u0 + j];
#pragma unroll 4
        for (int i = 0; i < MLP_H; i += 4) {
            const float a0 = S.h1[i][s], a1 = S.h1[i + 1][s], a2 = S.h1[i + 2][s], a3 = S.h1[i + 3][s];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float4 w = *reinterpret_cast<const float4*>(&S.P[OFF_W2 + (u0 + j) * MLP_H + i]);
                z[j] = fmaf(w.w, a3, fmaf(w.z, a2, fmaf(w.y, a1, fmaf(w.x, a0, z[j]))));
            }
        }
        float o = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            h2[j] = tanhf(z[j]);
            S.h2[u0 + j][s] = h2[j];
            o = fmaf(S.P[OFF_W3 + u0 + j], h2[j], o);
        }
        S.out[warp & 3][s] = o;
    }
    __syncthreads();
    {
        const float o = S.P[OFF_B3] + ((S.out[0][s] + S.out[1][s]) + (S.out[2][s] + S.out[3][s]));
        const float e = in.act ? o - in.y : 0.f, dy = e * inv_n;
        if ((warp & 3) == 0) {
            S.dy[s] = dy;
            S.loss[s] = 0.5f * e * e * inv_n;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) S.z2[u0 + j][s] = dy * S.P[OFF_W3 + u0 + j] * (1.f - h2[j] * h2[j]);
    }
    __syncthreads();
    {
        float d[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) d[i] = 0.f;
#pragma unroll 8
        for (int j = 0; j < MLP_H; ++j) {
            const float z = S.z2[j][s];
            const float4 wa = *reinterpret_cast<const float4*>(&S.P[OFF_W2 + j * MLP_H + u0]);
            const float4 wb = *reinterpret_cast<const float4*>(&S.P[OFF_W2 + j * MLP_H + u0 + 4]);
            d[0] = fmaf(wa.x, z, d[0]); d[1] = fmaf(wa.y, z, d[1]);
            d[2] = fmaf(wa.z, z, d[2]); d[3] = fmaf(wa.w, z, d[3]);
            d[4] = fmaf(wb.x, z, d[4]); d[5] = fmaf(wb.y, z, d[5]);
            d[6] = fmaf(wb.z, z, d[6]); d[7] = fmaf(wb.w, z, d[7]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) S.z1[u0 + i][s] = d[i] * (1.f - h1[i] * h1[i]);
    }
    __syncthreads();
    auto dot4 = [](const float4& a, const float4& b, float c) {
        return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, c))));
    };
#pragma unroll 4
    for (int k = 0; k < TRAIN_TS; k += 4) {
        const float4 a0 = *reinterpret_cast<const float4*>(&S.z2[R.tj][k]);
        const float4 a1 = *reinterpret_cast<const float4*>(&S.z2[R.tj + 16][k]);
        const float4 b0 = *reinterpret_cast<const float4*>(&S.h1[R.ti][k]);
        const float4 b1 = *reinterpret_cast<const float4*>(&S.h1[R.ti + 16][k]);
        R.g2[0][0] = dot4(a0, b0, R.g2[0][0]);
        R.g2[0][1] = dot4(a0, b1, R.g2[0][1]);
        R.g2[1][0] = dot4(a1, b0, R.g2[1][0]);
        R.g2[1][1] = dot4(a1, b1, R.g2[1][1]);
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        if (tid + 256 * e >= TRAIN_EXTRA) break;
#pragma unroll 4
        for (int k = 0; k < TRAIN_TS; k += 4)
            R.ge[e] = dot4(*reinterpret_cast<const float4*>(R.ea[e] + k),
                           *reinterpret_cast<const float4*>(R.eb[e] + k), R.ge[e]);
    }
}

static __global__ void __launch_bounds__(256) k_train_grad(const float* __restrict__ P, const float* __restrict__ x,
                                                           const float* __restrict__ y, const int* __restrict__ ok,
                                                           long long first, int count, float inv_n,
                                                           float* __restrict__ part) {
    __shared__ __align__(16) TrainSmem S;
    TrainSums R;
    R.rows_of(S);
    R.clear();
    for (int k = threadIdx.x; k < MLP_NPARAM; k += 256) S.P[k] = P[k];
    for (int t0 = blockIdx.x * TRAIN_TS; t0 < count; t0 += gridDim.x * TRAIN_TS)
        train_tile(S, train_load(x, y, ok, first, count, t0), inv_n, R);
    R.store(part + (long long)blockIdx.x * TRAIN_ROW);
}

// Sum of the rows of `part` (in a fixed order) over TRAIN_COLS of the columns and, per
// parameter, Adam (Kingma & Ba 2015) or, with grad non-null, the gradient itself; the
// loss is added to *loss.  32 row groups side by side: the 256 rows of a 16384
// minibatch are eight independent loads per thread.
constexpr int TRAIN_COLS = 8, TRAIN_GROUPS = (TRAIN_ROW + TRAIN_COLS - 1) / TRAIN_COLS;

struct TrainSumSmem {
    float sum[256 / TRAIN_COLS][TRAIN_COLS + 1];
};

__device__ __forceinline__ void train_update(TrainSumSmem& S, int group, const float* part, int rows, float* P,
                                             float* grad, float* m, float* v, float* loss, float lr, float b1, float b2,
                                             float eps, int step) {
    const int tx = threadIdx.x % TRAIN_COLS, ty = threadIdx.x / TRAIN_COLS;
    const int k = group * TRAIN_COLS + tx;
    float a = 0.f;
    if (k < TRAIN_ROW) {
#pragma unroll 8
        for (int r = ty; r < rows; r += 256 / TRAIN_COLS) a += __ldcg(part + (long long)r * TRAIN_ROW + k);
    }
    S.sum[ty][tx] = a;
    __syncthreads();
    if (ty == 0 && k < TRAIN_ROW) {
        float g = 0.f;
#pragma unroll
        for (int r = 0; r < 256 / TRAIN_COLS; ++r) g += S.sum[r][tx];
        if (k == MLP_NPARAM) {
            *loss += g;
        } else if (grad) {
            grad[k] = g;
        } else {
            const float mk = b1 * m[k] + (1.f - b1) * g;
            const float vk = b2 * v[k] + (1.f - b2) * g * g;
            m[k] = mk;
            v[k] = vk;
            const float mh = mk / (1.f - powf(b1, (float)step));
            const float vh = vk / (1.f - powf(b2, (float)step));
            P[k] = __ldcg(P + k) - lr * mh / (sqrtf(vh) + eps);
        }
    }
}

static __global__ void __launch_bounds__(256) k_train_update(const float* part, int rows, float* P, float* grad,
                                                             float* m, float* v, float* loss, float lr, float b1,
                                                             float b2, float eps, int step) {
    __shared__ TrainSumSmem S;
    train_update(S, blockIdx.x, part, rows, P, grad, m, v, loss, lr, b1, b2, eps, step);
}

// An epoch's minibatches [b0, b0 + nb) of `total` in one cooperative launch: what a
// minibatch's two launches cost beyond their work is their start, the parameters' way
// through memory and the first loads of the samples (19.7 us for 16384 samples, 1.26 ms
// for 2^20; here 14.5 us and 0.93 ms): the CTAs stay, two barriers
// per minibatch keep the halves apart (the rows before their sums, the parameters
// before the next forward pass), and the next samples are loaded while the sums are
// made.  What bounds it now is the chain of short phases of a tile and the barriers.
struct TrainCtl {
    unsigned int arrived;  // barrier arrivals so far (modulo 2^32: a wait compares the difference)
    int fault;             // a barrier wait was given up
};

struct TrainArgs {
    float* P;
    const float *x, *y;
    const int* ok;
    float *part, *m, *v, *loss;
    TrainCtl* ctl;
    long long done, total;  // minibatches before this launch, and of the whole run (step size)
    long long b0;           // first minibatch of the epoch's samples
    int batch, nb, step0;   // samples per minibatch, minibatches, Adam steps before
    float lr;
};

// All CTAs of the grid have arrived; false after GRID_SPIN_LIMIT polls.
__device__ __forceinline__ bool train_barrier(TrainCtl* ctl, unsigned int target) {
    __syncthreads();
    bool ok = true;
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&ctl->arrived, 1u);
        int spins = 0;
        while ((int)(ld_acquire(&ctl->arrived) - target) < 0 && ++spins < GRID_SPIN_LIMIT) {}
        ok = spins < GRID_SPIN_LIMIT;
        if (!ok) ctl->fault = 1;
    }
    return __syncthreads_and(ok) != 0;
}

static __global__ void __launch_bounds__(256) k_train_epoch(const TrainArgs a) {
    __shared__ __align__(16) TrainSmem S;
    __shared__ TrainSumSmem U;
    const int tiles = (a.batch + TRAIN_TS - 1) / TRAIN_TS, rows = min(tiles, (int)gridDim.x);
    const bool mine = (int)blockIdx.x < rows;
    const float inv_n = 1.f / a.batch;
    TrainSums R;
    R.rows_of(S);
    long long first = a.b0 * a.batch;
    unsigned int target = 0;
    TrainIn in = train_load(a.x, a.y, a.ok, first, a.batch, blockIdx.x * TRAIN_TS);
    for (int b = 0; b < a.nb; ++b) {
        if (mine) {
            for (int k = threadIdx.x; k < MLP_NPARAM; k += 256) S.P[k] = __ldcg(a.P + k);
            R.clear();
            train_tile(S, in, inv_n, R);
            for (int t = blockIdx.x + gridDim.x; t < tiles; t += gridDim.x)
                train_tile(S, train_load(a.x, a.y, a.ok, first, a.batch, t * TRAIN_TS), inv_n, R);
            R.store(a.part + (long long)blockIdx.x * TRAIN_ROW);
        }
        if (!train_barrier(a.ctl, target += gridDim.x)) return;
        first += a.batch;
        if (b + 1 < a.nb) in = train_load(a.x, a.y, a.ok, first, a.batch, blockIdx.x * TRAIN_TS);
        // step size: linear to a tenth over the run
        const float frac = (float)(a.done + b) / (float)a.total;
        const float lr = a.lr * (1.f - 0.9f * frac);
        for (int g = blockIdx.x; g < TRAIN_GROUPS; g += gridDim.x) {
            train_update(U, g, a.part, rows, a.P, nullptr, a.m, a.v, a.loss, lr, 0.9f, 0.999f, 1e-8f, a.step0 + b + 1);
            __syncthreads();
        }
        if (b + 1 < a.nb && !train_barrier(a.ctl, target += gridDim.x)) return;
    }
}

// ---- BF16 tensor-core inference ---------------------------------------------
// Inference weights: B fragments of each layer in the mma.sync layout, made
// from the FP32 parameters on the host side of this file (mlp_pack).
struct MlpPacked {
    unsigned int w1[4][32][2];     // layer 1: 4 n-tiles (K = 16: 6 inputs + zeros)
    unsigned int w2[4][2][32][2];  // layer 2: 4 n-tiles x 2 k-tiles
    unsigned int w3[2][32][2];     // layer 3: 1 n-tile (column 0) x 2 k-tiles
    float b1[MLP_H], b2[MLP_H], b3;
};

__host__ __device__ __forceinline__ unsigned short bf16_bits(float f) {
    // round-to-nearest-even conversion of an FP32 value to BF16 bits
    unsigned int u;
    memcpy(&u, &f, 4);
    if ((u & 0x7f800000u) == 0x7f800000u) return (unsigned short)((u >> 16) | ((u & 0xffff) ? 0x40 : 0));
    u += 0x7fffu + ((u >> 16) & 1u);
    return (unsigned short)(u >> 16);
}
__host__ __device__ __forceinline__ unsigned int pack2(float lo, float hi) {
    return (unsigned int)bf16_bits(lo) | ((unsigned int)bf16_bits(hi) << 16);
}

// Fill the fragments (host): B[k][n] = W[n][k]; lane = 4g + t holds
// (k = 2t, 2t+1; n = g) in register 0 and (k = 2t+8, 2t+9; n = g) in register 1.
inline void mlp_pack(const float* P, MlpPacked& M) {
    auto w1 = [&](int n, int k) { return k < 6 ? P[OFF_W1 + n * 6 + k] : 0.f; };
    auto w2 = [&](int n, int k) { return P[OFF_W2 + n * MLP_H + k]; };
    auto w3 = [&](int n, int k) { return n == 0 ? P[OFF_W3 + k] : 0.f; };
    for (int lane = 0; lane < 32; ++lane) {
        const int g = lane >> 2, t = lane & 3;
        for (int j = 0; j < 4; ++j) {
            const int n = 8 * j + g;
            M.w1[j][lane][0] = pack2(w1(n, 2 * t), w1(n, 2 * t + 1));
            M.w1[j][lane][1] = pack2(w1(n, 2 * t + 8), w1(n, 2 * t + 9));
            for (int kk = 0; kk < 2; ++kk) {
                M.w2[j][kk][lane][0] = pack2(w2(n, 16 * kk + 2 * t), w2(n, 16 * kk + 2 * t + 1));
                M.w2[j][kk][lane][1] = pack2(w2(n, 16 * kk + 2 * t + 8), w2(n, 16 * kk + 2 * t + 9));
            }
        }
        for (int kk = 0; kk < 2; ++kk) {
            M.w3[kk][lane][0] = pack2(w3(g, 16 * kk + 2 * t), w3(g, 16 * kk + 2 * t + 1));
            M.w3[kk][lane][1] = pack2(w3(g, 16 * kk + 2 * t + 8), w3(g, 16 * kk + 2 * t + 9));
        }
    }
    for (int j = 0; j < MLP_H; ++j) {
        M.b1[j] = P[OFF_B1 + j];
        M.b2[j] = P[OFF_B2 + j];
    }
    M.b3 = P[OFF_B3];
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], const unsigned int (&a)[4], unsigned int b0, unsigned int b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ float tanh_fast(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// MLP outputs for the 16 rows of one M-tile whose layer-1 A fragment is `a1`.
// Returns, in lanes with t == 0, out[0] = row g and out[1] = row g + 8.
__device__ __forceinline__ void mlp_tile(const MlpPacked& M, const unsigned int (&a1)[4], float (&out)[2]) {
    const int lane = threadIdx.x & 31, t = lane & 3;
    unsigned int a2[2][4];
    {
        float d[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float bl = M.b1[8 * j + 2 * t], bh = M.b1[8 * j + 2 * t + 1];
            d[j][0] = bl; d[j][1] = bh; d[j][2] = bl; d[j][3] = bh;
            mma_bf16(d[j], a1, M.w1[j][lane][0], M.w1[j][lane][1]);
        }
        // tanh, then the accumulators of n-tiles (2kk, 2kk+1) are layer 2's A fragment kk
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
            a2[kk][0] = pack2(tanh_fast(d[2 * kk][0]), tanh_fast(d[2 * kk][1]));
            a2[kk][1] = pack2(tanh_fast(d[2 * kk][2]), tanh_fast(d[2 * kk][3]));
            a2[kk][2] = pack2(tanh_fast(d[2 * kk + 1][0]), tanh_fast(d[2 * kk + 1][1]));
            a2[kk][3] = pack2(tanh_fast(d[2 * kk + 1][2]), tanh_fast(d[2 * kk + 1][3]));
        }
    }
    unsigned int a3[2][4];
    {
        float d[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float bl = M.b2[8 * j + 2 * t], bh = M.b2[8 * j + 2 * t + 1];
            d[j][0] = bl; d[j][1] = bh; d[j][2] = bl; d[j][3] = bh;
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) mma_bf16(d[j], a2[kk], M.w2[j][kk][lane][0], M.w2[j][kk][lane][1]);
        }
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
            a3[kk][0] = pack2(tanh_fast(d[2 * kk][0]), tanh_fast(d[2 * kk][1]));
            a3[kk][1] = pack2(tanh_fast(d[2 * kk][2]), tanh_fast(d[2 * kk][3]));
            a3[kk][2] = pack2(tanh_fast(d[2 * kk + 1][0]), tanh_fast(d[2 * kk + 1][1]));
            a3[kk][3] = pack2(tanh_fast(d[2 * kk + 1][2]), tanh_fast(d[2 * kk + 1][3]));
        }
    }
    float d[4] = {M.b3, 0.f, M.b3, 0.f};
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) mma_bf16(d, a3[kk], M.w3[kk][lane][0], M.w3[kk][lane][1]);
    out[0] = d[0];
    out[1] = d[2];
}

// Evaluate the network for 64 feature rows held in shared memory
// (rows[64][8] floats, 6 features used) by one warp; results to res[64].
__device__ __forceinline__ void mlp_warp64(const MlpPacked& M, const float (*rows)[8], float* res) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int mt = 0; mt < 4; ++mt) {
        const int r0 = 16 * mt + g, r1 = r0 + 8;
        auto feat = [&](int r, int c) { return c < 6 ? rows[r][c] : 0.f; };
        unsigned int a[4];
        a[0] = pack2(feat(r0, 2 * t), feat(r0, 2 * t + 1));
        a[1] = pack2(feat(r1, 2 * t), feat(r1, 2 * t + 1));
        a[2] = pack2(feat(r0, 2 * t + 8), feat(r0, 2 * t + 9));
        a[3] = pack2(feat(r1, 2 * t + 8), feat(r1, 2 * t + 9));
        float out[2];
        mlp_tile(M, a, out);
        if (t == 0) {
            res[r0] = out[0];
            res[r1] = out[1];
        }
    }
    __syncwarp();
}

// Network outputs for n feature rows (x[i*8 + 0..5]) -- the raw evaluator
// behind claw2_mlp_infer; one warp per 64 rows.
static __global__ void k_mlp_eval(const MlpPacked* __restrict__ Mg, const float* __restrict__ x, int n, float* y) {
    __shared__ MlpPacked M;
    __shared__ float rows[4][64][8];
    __shared__ float res[4][64];
    for (int k = threadIdx.x; k < (int)(sizeof(MlpPacked) / 4); k += blockDim.x)
        reinterpret_cast<unsigned int*>(&M)[k] = reinterpret_cast<const unsigned int*>(Mg)[k];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long base = ((long long)blockIdx.x * 4 + w) * 64;
    for (int r = lane; r < 64; r += 32)
        for (int c = 0; c < 8; ++c) rows[w][r][c] = (base + r < n) ? x[(base + r) * 8 + c] : 0.f;
    __syncthreads();
    mlp_warp64(M, rows[w], res[w]);
    for (int r = lane; r < 64; r += 32)
        if (base + r < n) y[base + r] = res[w][r];
}

// Learned guesses for every interface of a grid: thread (cp, R) computes the
// x-interface (cp-1 | cp) on row R and the y-interface (R-1 | R) on column cp.
// guess planes: [0] x-interfaces, [1] y-interfaces, q's layout.
static __global__ void __launch_bounds__(128) k_mlp_guess(const MlpPacked* __restrict__ Mg,
                                                          const double* q, Layout L, double gamma, double* guess,
                                                          const EvolveDev* evo, const double* q2) {
    if (evo) {  // the device time loop's record: nothing to do, or the other buffer
        if (evo->done) return;
        if (evo->cur) q = q2;
    }
    __shared__ MlpPacked M;
    __shared__ float rows[4][64][8];
    __shared__ float res[4][64];
    for (int k = threadIdx.x; k < (int)(sizeof(MlpPacked) / 4); k += blockDim.x)
        reinterpret_cast<unsigned int*>(&M)[k] = reinterpret_cast<const unsigned int*>(Mg)[k];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cp = blockIdx.x * 32 + lane;
    const int R = blockIdx.y * 4 + w;
    const int c = min(cp, L.mx + 3), r = min(R, L.my + 3);
    const exact_euler::Gas G = exact_euler::make_gas(gamma);
    const double g1 = gamma - 1.0;
    auto prim = [&](int cc, int rr, double& rho, double& u, double& v, double& p) {
        const long long o = (long long)rr * L.pitch + cc;
        rho = q[o];
        u = q[L.plane + o] / rho;
        v = q[2 * L.plane + o] / rho;
        p = g1 * (q[3 * L.plane + o] - 0.5 * rho * (u * u + v * v));
    };
    double r0, u0, v0, p0, rl, ul, vl, pl, rb, ub, vb, pb;
    prim(c, r, r0, u0, v0, p0);
    prim(max(c - 1, 0), r, rl, ul, vl, pl);
    prim(c, max(r - 1, 0), rb, ub, vb, pb);
    double wx, wy;
    float fx[6], fy[6];
    exact_euler::features(G, rl, ul, pl, r0, u0, p0, fx, wx);
    exact_euler::features(G, rb, vb, pb, r0, v0, p0, fy, wy);
    for (int k = 0; k < 6; ++k) {
        rows[w][lane][k] = isfinite(fx[k]) ? fx[k] : 0.f;
        rows[w][32 + lane][k] = isfinite(fy[k]) ? fy[k] : 0.f;
    }
    __syncthreads();
    // PVRS decides: a weak jump (w below MLP_WMIN) keeps the PVRS guess,
    // which is accurate there and where the network has seen no training data;
    // a warp with only weak jumps skips the network altogether.
    const bool strong = (wx >= MLP_WMIN) || (wy >= MLP_WMIN);
    if (__any_sync(0xffffffffu, strong)) {
        mlp_warp64(M, rows[w], res[w]);
    } else {
        res[w][lane] = 0.f;
        res[w][32 + lane] = 0.f;
    }
    if (wx < MLP_WMIN) wx = 0.0;
    if (wy < MLP_WMIN) wy = 0.0;
    if (cp > L.mx + 3 || R > L.my + 3) return;
    const double cl = sqrt(gamma * pl / rl), c0 = sqrt(gamma * p0 / r0), cb = sqrt(gamma * pb / rb);
    const double gx0 = exact_euler::guess_pvrs(G, rl, ul, pl, cl, r0, u0, p0, c0);
    const double gy0 = exact_euler::guess_pvrs(G, rb, vb, pb, cb, r0, v0, p0, c0);
    const long long o = (long long)R * L.pitch + cp;
    guess[o] = gx0 * exp(wx * (double)res[w][lane]);
    guess[L.plane + o] = gy0 * exp(wy * (double)res[w][32 + lane]);
}

// ---- BF16 inference on the 5th-generation tensor cores (tcgen05 + TMEM) -----
// One CTA of 128 threads evaluates the network for two M = 128 row tiles at a
// time (the x- and the y-interfaces of 128 grid sites, or 256 rows of
// features): thread t owns row t of both tiles, which is TMEM lane t of the
// accumulators, so warp w reads back exactly the lanes 32w..32w+31 it may
// access.  Per tile pair: layer 1 is one tcgen05.mma (M 128, N 32, K 16) per
// tile, the 32 FP32 accumulators of a row come back with one tcgen05.ld,
// tanh and the BF16 rounding run in registers and the row goes back to
// shared memory as layer 2's A operand; layer 2 is two K = 16 MMAs per tile
// into the same TMEM columns; layer 3 (32 -> 1) is a 32-term FP32 dot product
// of the BF16-rounded activations in each thread.  Operands are BF16 in the
// no-swizzle K-major layout of the tcgen05 shared-memory descriptors: element
// (r, k) of an R x K matrix at byte (r/8)*16K + (k/8)*128 + (r%8)*16 + (k%8)*2
// (8 x 16-byte core matrices; the leading, K, offset 128 bytes; the stride
// between 8-row groups 16K bytes).  One elected thread issues the MMAs and
// commits them to an mbarrier; every wait on it is bounded (status bit 1).
struct MlpTcImage {                  // device image of the weights, copied into shared memory
    unsigned short w1[MLP_H * 16];   // layer 1 B operand: N = 32 x K = 16 (6 inputs + zeros)
    unsigned short w2[MLP_H * MLP_H];  // layer 2 B operand: N = 32 x K = 32
    float b1[MLP_H], b2[MLP_H];
    float w3[MLP_H];                 // BF16-rounded, as FP32
    float b3;
    float pad[3];
};
static_assert(sizeof(MlpTcImage) % 16 == 0, "weight image is copied in 16-byte words");

// byte offset of element (r, k) in the no-swizzle K-major image of an R x K matrix
__host__ __device__ constexpr int umma_kmajor_off(int r, int k, int K) {
    return (r >> 3) * (K * 16) + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2;
}

inline float bf16_round(float f) {
    const unsigned int u = (unsigned int)bf16_bits(f) << 16;
    float r;
    memcpy(&r, &u, 4);
    return r;
}

// Fill the weight image (host) from the FP32 parameters: B[n][k] = W[n][k]
// (the MMA computes D = A B^T with both operands K-major).
inline void mlp_pack_tc(const float* P, MlpTcImage& M) {
    memset(&M, 0, sizeof M);
    for (int n = 0; n < MLP_H; ++n) {
        for (int k = 0; k < 16; ++k)
            M.w1[umma_kmajor_off(n, k, 16) / 2] = bf16_bits(k < MLP_IN ? P[OFF_W1 + n * MLP_IN + k] : 0.f);
        for (int k = 0; k < MLP_H; ++k)
            M.w2[umma_kmajor_off(n, k, MLP_H) / 2] = bf16_bits(P[OFF_W2 + n * MLP_H + k]);
        M.b1[n] = P[OFF_B1 + n];
        M.b2[n] = P[OFF_B2 + n];
        M.w3[n] = bf16_round(P[OFF_W3 + n]);
    }
    M.b3 = P[OFF_B3];
}

struct MlpTcSmem {
    alignas(128) unsigned short a1[2][128 * 16];  // layer 1 A operands (features), tiles 0 and 1
    alignas(128) unsigned short a2[2][128 * MLP_H];  // layer 2 A operands (tanh of layer 1)
    alignas(128) MlpTcImage W;
    unsigned long long bar;  // MMA completion
    unsigned int tmem;       // TMEM base address from tcgen05.alloc
};
constexpr int MLP_TC_COLS = 64;  // TMEM columns: tile 0 accumulators 0..31, tile 1 32..63
// With this footprint at most 8 CTAs fit on an SM (228 KB of shared memory,
// 1 KB reserved per CTA), so their 64-column TMEM allocations (8 x 64 = 512
// columns) never wait for one another.
static_assert(9 * (sizeof(MlpTcSmem) + 1024) > 228 * 1024, "TMEM columns would be oversubscribed");

// Shared-memory matrix descriptor: start address, leading (K) byte offset,
// stride (8-row group) byte offset, descriptor version 1, no swizzle.
__device__ __forceinline__ unsigned long long umma_desc(const void* p, unsigned lbo, unsigned sbo) {
    return (unsigned long long)((smem_u32(p) & 0x3FFFFu) >> 4) | ((unsigned long long)(lbo >> 4) << 16) |
           ((unsigned long long)(sbo >> 4) << 32) | (1ull << 46);
}
// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, N = 32, M = 128.
constexpr unsigned MLP_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(MLP_H >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ void umma_bf16(unsigned tmem_d, unsigned long long da, unsigned long long db, int acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem_d),
        "l"(da), "l"(db), "r"(MLP_IDESC), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void umma_commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }

// 16 consecutive FP32 columns of this thread's TMEM lane (warp-collective)
__device__ __forceinline__ void tmem_ld16(unsigned taddr, float (&v)[16]) {
    unsigned r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = __uint_as_float(r[k]);
}

// two FP32 values to packed BF16 (round to nearest even), lo in the low half
__device__ __forceinline__ unsigned int pack2_rn(float lo, float hi) {
    unsigned int r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// CTA set-up: weights into shared memory, the MMA barrier, and the TMEM
// columns (allocated by warp 0, which also frees them in mlp_tc_teardown).
__device__ __forceinline__ void mlp_tc_setup(MlpTcSmem& S, const MlpTcImage* __restrict__ Mg) {
    const uint4* src = reinterpret_cast<const uint4*>(Mg);
    uint4* dst = reinterpret_cast<uint4*>(&S.W);
    for (int k = threadIdx.x; k < (int)(sizeof(MlpTcImage) / 16); k += blockDim.x) dst[k] = src[k];
    if (threadIdx.x == 0) mbar_init(&S.bar);
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem)),
                     "r"(MLP_TC_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
}

__device__ __forceinline__ void mlp_tc_teardown(MlpTcSmem& S) {
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x < 32) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(S.tmem), "r"(MLP_TC_COLS)
                     : "memory");
    }
}

// Write this thread's 6 features as row t of layer 1's A operand of tile j.
__device__ __forceinline__ void mlp_tc_put_features(MlpTcSmem& S, int j, const float (&f)[MLP_IN]) {
    const int t = threadIdx.x;
    uint4 lo, hi;
    lo.x = pack2_rn(f[0], f[1]);
    lo.y = pack2_rn(f[2], f[3]);
    lo.z = pack2_rn(f[4], f[5]);
    lo.w = 0u;
    hi.x = hi.y = hi.z = hi.w = 0u;
    unsigned char* base = reinterpret_cast<unsigned char*>(S.a1[j]);
    *reinterpret_cast<uint4*>(base + umma_kmajor_off(t, 0, 16)) = lo;
    *reinterpret_cast<uint4*>(base + umma_kmajor_off(t, 8, 16)) = hi;
}

// Wait for the phase `phase` of the MMA barrier (bounded); then TMEM reads may start.
__device__ __forceinline__ void mlp_tc_wait(MlpTcSmem& S, unsigned& phase, int* status) {
    if (!mbar_wait(&S.bar, phase & 1u) && status) atomicOr(status, 2);
    ++phase;
    tc_fence_after();
}

// The network for row t of both tiles (features already written with
// mlp_tc_put_features by every thread).  All 128 threads call this together;
// need0 / need1: this thread's row of tile 0 / 1 wants the output.  Rows are
// independent in the products, so a warp none of whose rows of a tile want
// it skips that tile's read-back and activations (its rows of the next
// operand keep stale values, whose results nobody reads); its output is 0.
__device__ __forceinline__ void mlp_tc_pair(MlpTcSmem& S, unsigned& phase, int* status, bool need0, bool need1,
                                            float& out0, float& out1) {
    const int t = threadIdx.x, w = t >> 5;
    const unsigned tm = S.tmem;
    const unsigned lane_base = (unsigned)(32 * w) << 16;
    const bool wj[2] = {__any_sync(0xffffffffu, need0) != 0, __any_sync(0xffffffffu, need1) != 0};
    // layer 1: D_j = A1_j W1^T
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    if (t == 0) {
        tc_fence_after();
        const unsigned long long db = umma_desc(S.W.w1, 128, 16 * 16);
#pragma unroll
        for (int j = 0; j < 2; ++j) umma_bf16(tm + 32 * j, umma_desc(S.a1[j], 128, 16 * 16), db, 0);
        umma_commit(&S.bar);
    }
    mlp_tc_wait(S, phase, status);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        if (!wj[j]) continue;
        unsigned char* base = reinterpret_cast<unsigned char*>(S.a2[j]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float d[16];
            tmem_ld16(tm + lane_base + 32 * j + 16 * h, d);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int k0 = 16 * h + 8 * c;
                uint4 v;
                v.x = pack2_rn(tanh_fast(d[8 * c + 0] + S.W.b1[k0 + 0]), tanh_fast(d[8 * c + 1] + S.W.b1[k0 + 1]));
                v.y = pack2_rn(tanh_fast(d[8 * c + 2] + S.W.b1[k0 + 2]), tanh_fast(d[8 * c + 3] + S.W.b1[k0 + 3]));
                v.z = pack2_rn(tanh_fast(d[8 * c + 4] + S.W.b1[k0 + 4]), tanh_fast(d[8 * c + 5] + S.W.b1[k0 + 5]));
                v.w = pack2_rn(tanh_fast(d[8 * c + 6] + S.W.b1[k0 + 6]), tanh_fast(d[8 * c + 7] + S.W.b1[k0 + 7]));
                *reinterpret_cast<uint4*>(base + umma_kmajor_off(t, k0, MLP_H)) = v;
            }
        }
    }
    // layer 2: D_j = A2_j W2^T, two K = 16 steps (the K offset is two core matrices, 256 bytes)
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    if (t == 0) {
        tc_fence_after();
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int kk = 0; kk < 2; ++kk)
                umma_bf16(tm + 32 * j, umma_desc(reinterpret_cast<const unsigned char*>(S.a2[j]) + 256 * kk, 128, 16 * MLP_H),
                          umma_desc(reinterpret_cast<const unsigned char*>(S.W.w2) + 256 * kk, 128, 16 * MLP_H), kk);
        umma_commit(&S.bar);
    }
    mlp_tc_wait(S, phase, status);
    float o[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        if (!wj[j]) continue;
        float acc = S.W.b3;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float d[16];
            tmem_ld16(tm + lane_base + 32 * j + 16 * h, d);
#pragma unroll
            for (int k = 0; k < 16; k += 2) {
                const unsigned int u =
                    pack2_rn(tanh_fast(d[k] + S.W.b2[16 * h + k]), tanh_fast(d[k + 1] + S.W.b2[16 * h + k + 1]));
                acc = fmaf(__uint_as_float(u << 16), S.W.w3[16 * h + k], acc);
                acc = fmaf(__uint_as_float(u & 0xffff0000u), S.W.w3[16 * h + k + 1], acc);
            }
        }
        o[j] = acc;
    }
    out0 = o[0];
    out1 = o[1];
    // the next pair's MMAs overwrite the accumulators and operands: every
    // thread's reads are done before any thread passes the next barrier
    tc_fence_before();
}

// Network outputs for n feature rows (x[i*8 + 0..5]) -- the raw evaluator
// behind claw2_mlp_infer: 256 rows per tile pair, CTAs loop over the pairs.
static __global__ void __launch_bounds__(128) k_mlp_eval_tc(const MlpTcImage* __restrict__ Mg,
                                                            const float* __restrict__ x, int n, float* y,
                                                            int* status) {
    __shared__ MlpTcSmem S;
    mlp_tc_setup(S, Mg);
    unsigned phase = 0;
    const int t = threadIdx.x;
    const int npairs = (n + 255) / 256;
    for (int pr = blockIdx.x; pr < npairs; pr += gridDim.x) {
        const long long r0 = (long long)pr * 256 + t, r1 = r0 + 128;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const long long r = j ? r1 : r0;
            float f[MLP_IN];
#pragma unroll
            for (int c = 0; c < MLP_IN; ++c) f[c] = (r < n) ? x[r * 8 + c] : 0.f;
            mlp_tc_put_features(S, j, f);
        }
        float o0, o1;
        mlp_tc_pair(S, phase, status, r0 < n, r1 < n, o0, o1);
        if (r0 < n) y[r0] = o0;
        if (r1 < n) y[r1] = o1;
    }
    mlp_tc_teardown(S);
}

// exact_euler::features in FP32 for the inference pass (the features enter
// the network as BF16, so FP32 arithmetic loses nothing that counts): a and
// b are the (rho, u, v, p, c) of the cells left/below and right/above, dir 1
// or 2 picks the normal velocity.  Non-finite features become 0; a
// non-finite jump weight leaves the interface to the PVRS guess.
__device__ __forceinline__ void features_f32(float g, const double (&a)[5], const double (&b)[5], int dir,
                                             float (&x)[MLP_IN], float& w) {
    const float rl = (float)a[0], ul = (float)a[dir], pl = (float)a[3];
    const float rr = (float)b[0], ur = (float)b[dir], pr = (float)b[3];
    const float rb = sqrtf(rl * rr), pb = sqrtf(pl * pr);
    const float cb = sqrtf(__fdividef(g * pb, rb));
    const float icb = __fdividef(1.f, cb);
    const float lr = 0.5f * __logf(__fdividef(rl, rr)), lp = 0.5f * __logf(__fdividef(pl, pr));
    x[0] = lr;
    x[1] = -lr;
    x[2] = ul * icb;
    x[3] = ur * icb;
    x[4] = lp;
    x[5] = -lp;
#pragma unroll
    for (int k = 0; k < MLP_IN; ++k) x[k] = isfinite(x[k]) ? x[k] : 0.f;
    const float dr = __fdividef(rr - rl, rb), dp = __fdividef(pr - pl, pb), du = (ur - ul) * icb;
    const float j2 = dr * dr + dp * dp + du * du;
    w = __fdividef(j2, 1.f + j2);
}

// Learned guesses for every interface of a grid (as k_mlp_guess, with the
// network on tcgen05): thread (cp, R) of a 32 x 4 site tile computes the
// x-interface (cp-1 | cp) on row R (tile 0, row t) and the y-interface
// (R-1 | R) on column cp (tile 1, row t).  CTAs loop over the site tiles.
static __global__ void __launch_bounds__(128, 5) k_mlp_guess_tc(const MlpTcImage* __restrict__ Mg,
                                                             const double* q, Layout L, double gamma, double* guess,
                                                             int* status, const EvolveDev* evo, const double* q2) {
    if (evo) {  // the device time loop's record: nothing to do, or the other buffer
        if (evo->done) return;
        if (evo->cur) q = q2;
    }
    __shared__ MlpTcSmem S;
    __shared__ double sprim[4][5][32];  // each warp's cells (rho, u, v, p, c): the row above's lower neighbours
    mlp_tc_setup(S, Mg);
    unsigned phase = 0;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tx = (L.mx + 4 + 31) / 32, ty = (L.my + 4 + 3) / 4;
    const long long ntiles = (long long)tx * ty;
    const exact_euler::Gas G = exact_euler::make_gas(gamma);
    const double g1 = gamma - 1.0;
    // primitive values and sound speed of one cell
    auto prim = [&](int cc, int rr, double (&v)[5]) {
        const long long o = (long long)rr * L.pitch + cc;
        const double rho = q[o], irho = rcp_nr(rho);
        v[0] = rho;
        v[1] = q[L.plane + o] * irho;
        v[2] = q[2 * L.plane + o] * irho;
        v[3] = g1 * (q[3 * L.plane + o] - 0.5 * rho * (v[1] * v[1] + v[2] * v[2]));
        v[4] = sqrt_nr(gamma * v[3] * irho);
    };
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int cp = (int)(tile % tx) * 32 + lane;
        const int R = (int)(tile / tx) * 4 + w;
        const int c = min(cp, L.mx + 3), r = min(R, L.my + 3);
        // this thread's cell; its left neighbour is the previous lane's cell
        // and its lower neighbour the previous warp's (each computed once),
        // except on the tile's first column and row
        double me[5], lf[5], lo[5];
        prim(c, r, me);
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            lf[k] = __shfl_up_sync(0xffffffffu, me[k], 1);
            sprim[w][k][lane] = me[k];
        }
        if (lane == 0) prim(max(c - 1, 0), r, lf);
        __syncthreads();
        if (w > 0) {
#pragma unroll
            for (int k = 0; k < 5; ++k) lo[k] = sprim[w - 1][k][lane];
        } else {
            prim(c, max(r - 1, 0), lo);
        }
        // features in FP32 (they enter the network as BF16)
        float wxf, wyf;
        float fx[MLP_IN], fy[MLP_IN];
        features_f32((float)gamma, lf, me, 1, fx, wxf);
        features_f32((float)gamma, lo, me, 2, fy, wyf);
        // PVRS decides: a weak jump (w below MLP_WMIN) keeps the PVRS guess;
        // a tile pair with only weak jumps skips the network
        const bool sx = wxf >= (float)MLP_WMIN, sy = wyf >= (float)MLP_WMIN;
        float ox = 0.f, oy = 0.f;
        if (__syncthreads_or(sx || sy)) {
            mlp_tc_put_features(S, 0, fx);
            mlp_tc_put_features(S, 1, fy);
            mlp_tc_pair(S, phase, status, sx, sy, ox, oy);
        }
        if (cp > L.mx + 3 || R > L.my + 3) continue;
        const double gx0 = exact_euler::guess_pvrs(G, lf[0], lf[1], lf[3], lf[4], me[0], me[1], me[3], me[4]);
        const double gy0 = exact_euler::guess_pvrs(G, lo[0], lo[2], lo[3], lo[4], me[0], me[2], me[3], me[4]);
        const long long o = (long long)R * L.pitch + cp;
        guess[o] = sx ? gx0 * (double)__expf(wxf * ox) : gx0;
        guess[L.plane + o] = sy ? gy0 * (double)__expf(wyf * oy) : gy0;
    }
    mlp_tc_teardown(S);
}

// The converged pressures as guesses (a measurement aid, no network): thread
// (cp, R) solves the x-interface (cp-1 | cp) and the y-interface (R-1 | R)
// exactly as the step kernel's Newton iteration would from the adaptive
// guess, to the same tolerance, and writes p* into the guess planes.  A step
// that starts from these needs no Newton update beyond the one that confirms
// convergence, so its time bounds from below what any guess can achieve.
// A deterministic number in [-1, 1) per interface (splitmix64 finaliser of
// its index): the sign and size of the error put on a converged guess.
__device__ __forceinline__ double guess_noise(unsigned long long k) {
    k += 0x9e3779b97f4a7c15ull;
    k = (k ^ (k >> 30)) * 0xbf58476d1ce4e5b9ull;
    k = (k ^ (k >> 27)) * 0x94d049bb133111ebull;
    k ^= k >> 31;
    return (double)(k >> 11) * (2.0 / 9007199254740992.0) - 1.0;
}

// rel > 0: where the adaptive guess needs Newton steps, the converged p* is
// multiplied by 1 + rel * noise, noise in [-1, 1) -- a guess of that
// relative precision -- and elsewhere the step keeps the adaptive guess
// (guess 0): the most a guess of that precision can save with the adaptive
// guess as its fallback, used only where it would help.
static __global__ void __launch_bounds__(128) k_exact_pstar_guess(const double* __restrict__ q, Layout L,
                                                                  double gamma, double tol, double rel,
                                                                  double* guess) {
    const int cp = blockIdx.x * 32 + (threadIdx.x & 31);
    const int R = blockIdx.y * 4 + (threadIdx.x >> 5);
    if (cp > L.mx + 3 || R > L.my + 3) return;
    const exact_euler::Gas G = exact_euler::make_gas(gamma);
    const double g1 = gamma - 1.0;
    // the primitive values and sound speed exactly as RPEulerExact::prepare
    // forms them for the step, so the step's Newton starts at its own root
    auto prim = [&](int cc, int rr, double& rho, double& u, double& v, double& p, double& c) {
        const long long o = (long long)rr * L.pitch + cc;
        rho = q[o];
        const double irho = rcp_nr(rho);
        u = q[L.plane + o] * irho;
        v = q[2 * L.plane + o] * irho;
        p = g1 * (q[3 * L.plane + o] - 0.5 * (q[L.plane + o] * u + q[2 * L.plane + o] * v));
        c = sqrt_nr(gamma * p * irho);
    };
    double r0, u0, v0, p0, c0, rl, ul, vl, pl, cl, rb, ub, vb, pb, cb;
    prim(cp, R, r0, u0, v0, p0, c0);
    prim(max(cp - 1, 0), R, rl, ul, vl, pl, cl);
    prim(cp, max(R - 1, 0), rb, ub, vb, pb, cb);
    double ps, us;
    int it;
    const long long o = (long long)R * L.pitch + cp;
    guess[o] = 0.0;  // vacuum or a failed solve: the step falls back to the adaptive guess
    guess[L.plane + o] = 0.0;
    if (!exact_euler::vacuum(G, ul, cl, u0, c0)) {
        exact_euler::star(G, rl, ul, pl, cl, r0, u0, p0, c0, 0.0, tol, 50, ps, us, it);
        if (rel > 0.0) ps = it > 0 ? ps * (1.0 + rel * guess_noise(2ull * (unsigned long long)o)) : 0.0;
        guess[o] = ps;
    }
    if (!exact_euler::vacuum(G, vb, cb, v0, c0)) {
        exact_euler::star(G, rb, vb, pb, cb, r0, v0, p0, c0, 0.0, tol, 50, ps, us, it);
        if (rel > 0.0) ps = it > 0 ? ps * (1.0 + rel * guess_noise(2ull * (unsigned long long)o + 1ull)) : 0.0;
        guess[L.plane + o] = ps;
    }
}

}  // namespace claw2
