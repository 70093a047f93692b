// Learned warm start: model object, training kernels (forward / backward /
// AdamW, hand-written, FP32) and the C ABI around them.
//
// Training pairs are what the plain routing solves: for every segment solve
// (qup, quc, qdp, ql, dx, s0, n, bw) and the depth the secant converged to
// (recorded by the routing kernel, see troute_record_pairs). The network maps
// standardised logarithms of the eight inputs to the standardised logarithm of
// the depth; the loss is the mean squared error in those units.
#include <cuda_runtime.h>

#include <cmath>
#include <cstddef>
#include <cstring>
#include <vector>

#include "train_buffers.h"
#include "warm.cuh"

namespace tr {

// Flat parameter vector: W1 [64][8] (out x in), b1 [64], W2 [64][64], b2 [64],
// w3 [64], b3.
constexpr int kP_W1 = 0, kP_B1 = kP_W1 + kWHid * kWIn, kP_W2 = kP_B1 + kWHid, kP_B2 = kP_W2 + kWHid * kWHid,
              kP_W3 = kP_B2 + kWHid, kP_B3 = kP_W3 + kWHid, kNParams = kP_B3 + 1;
constexpr int kPairW = 9;  // qup quc qdp ql dx s0 n bw depth

struct Norm {
    float mu[kWIn], sd[kWIn], mu_y, sd_y;
};

__device__ __forceinline__ bool pair_features(const float* pr, const Norm& nm, float (&x)[kWIn], float* y)
{
    const float h = pr[8];
    if (!(h > 0.0f) || !isfinite(h)) return false;
    for (int k = 0; k < kWIn; ++k) {
        const float v = (k < 4) ? pr[k] + kFlowFloor : pr[k];
        if (!(v > 0.0f) || !isfinite(v)) return false;
        x[k] = (logf(v) - nm.mu[k]) / nm.sd[k];
    }
    *y = (logf(h) - nm.mu_y) / nm.sd_y;
    return true;
}

// Per-block sums of the log features and log depth (and their squares) over
// the valid pairs, for the standardisation. Fixed-order reductions: the
// result does not depend on scheduling.
constexpr int kMomThreads = 256;
constexpr int kMomBlocks = 1024;
constexpr int kMomW = 2 * kPairW + 1;

__global__ void __launch_bounds__(kMomThreads) warm_moments_kernel(const float* __restrict__ pairs, long long n,
                                                                   long long stride, double* __restrict__ part)
{
    __shared__ double red[kMomThreads];
    double acc[kMomW] = {};
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i * stride < n;
         i += (long long)gridDim.x * blockDim.x) {
        const float* pr = pairs + (i * stride) * kPairW;
        bool ok = true;
        double v[kPairW];
        for (int k = 0; k < kPairW; ++k) {
            const float raw = (k < 4) ? pr[k] + kFlowFloor : pr[k];
            if (!(raw > 0.0f) || !isfinite(raw)) ok = false;
            v[k] = ok ? log((double)raw) : 0.0;
        }
        if (!ok) continue;
        for (int k = 0; k < kPairW; ++k) {
            acc[k] += v[k];
            acc[kPairW + k] += v[k] * v[k];
        }
        acc[2 * kPairW] += 1.0;
    }
    for (int k = 0; k < kMomW; ++k) {
        red[threadIdx.x] = acc[k];
        __syncthreads();
        for (int w = kMomThreads / 2; w > 0; w >>= 1) {
            if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
            __syncthreads();
        }
        if (threadIdx.x == 0) part[(size_t)blockIdx.x * kMomW + k] = red[0];
        __syncthreads();
    }
}

// Training steps in one cooperative launch. A step: the blocks take the
// mini-batch's tiles of kTrainRows samples, forward and backward, and write each
// tile's gradient (part[tile][kPartLd]) and its samples' (err^2)/2; after a grid
// barrier each block sums its share of the parameters over the tiles in order and
// takes the AdamW step for them; after a second one the next step begins. Sample i
// of the epoch is pair (perm_a * i + perm_b) mod n, a permutation of the pairs when
// gcd(perm_a, n) = 1. Every sum runs in a fixed order, so a training run is
// reproducible bit for bit. (As two launches per step, overlapped by programmatic
// dependent launch, 13 of a step's 30 us lay between the kernels.)
//
// FP32 multiply and add rates and shared-memory bandwidth bound it (both 64 cycles
// of an SM per inner index): three 64 x 64 x 64 products per block (layer 2
// forward, its weight gradient, its input gradient). kGemmThreads threads hold
// 4 x 4 tiles of each product in registers, every sum over its inner index in order
// (one thread per sample with scalar shared-memory reads took 94 us a batch of
// 8,192). A thread's units are 16 apart where they are rows of the shared arrays,
// so that reads of four consecutive inner values are free of bank conflicts and no
// array is needed in both orders. Activations whose derivative is needed later
// stay in the registers of the thread that will use them; the other kChoreThreads
// form the bias and last-layer sums beside the products. (Packed f32x2
// instructions on 2 x 4 tiles of 512 threads were no faster.)
constexpr int kGemmThreads = 256, kChoreThreads = 128;
constexpr int kTLd = 68;         // row of a 64-wide tile: 16-byte aligned, banks shifted by 4
static_assert(kTrainRows == 64 && kWHid == 64 && kPartLd >= kNParams && kPartLd % 4 == 0 && kP_W2 % 4 == 0, "tile shapes");

// The update: kUpdateRows threads per parameter fetch the partials of kUpdateTiles
// tiles at once into shared memory; one adds them up.
constexpr int kUpdateParams = 48, kUpdateRows = (kGemmThreads + kChoreThreads) / kUpdateParams, kUpdateTiles = 128;

struct __align__(16) FbSmem {
    float w1[kWHid][kWIn], b1[kWHid], b2[kWHid], w3[kWHid];
    float x[kTrainRows][kWIn], y[kTrainRows], g[kTrainRows];
    float sums[kUpdateTiles][kUpdateParams];
    float w2[kWHid][kTLd];                              // [out][in]
    float a1[kTrainRows][kTLd], dz2[kTrainRows][kTLd];  // [sample][unit]
    float a2[kTrainRows][kWHid + 1], dz1[kTrainRows][kWHid + 1];
    int valid[kTrainRows], stop;
};
// the arrays read and written as float4
static_assert(offsetof(FbSmem, w1) % 16 == 0 && offsetof(FbSmem, b1) % 16 == 0 && offsetof(FbSmem, b2) % 16 == 0 &&
                  offsetof(FbSmem, w3) % 16 == 0 && offsetof(FbSmem, x) % 16 == 0 && offsetof(FbSmem, w2) % 16 == 0 &&
                  offsetof(FbSmem, a1) % 16 == 0 && offsetof(FbSmem, dz2) % 16 == 0,
              "16-byte aligned");

// SiLU z / (1 + e^-z) and its derivative from one exponential.
__device__ __forceinline__ void silu_both(float z, float* a, float* d)
{
    const float t = 1.0f + expf(-z);
    *a = z / t;
    const float s = 1.0f / t;
    *d = s * (1.0f + z * (1.0f - s));
}

__device__ __forceinline__ void load4(const float* p, float (&v)[4])
{
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
}

// acc[i][j] += u[i] v[j], a product and a sum each.
__device__ __forceinline__ void tile_step(float (&acc)[4][4], const float (&u)[4], const float (&v)[4])
{
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += u[i] * v[j];
}

struct TrainArgs {
    const float* pairs;
    long long n, offset;          // pairs; first sample of the first step
    int batch, steps;             // samples per step (the last may be shorter)
    long long end;                // samples of the epoch
    unsigned long long perm_a, perm_b;
    Norm nm;
    const AdamStep* step;         // [steps], null: gradient only
    float b1, b2, eps, wd;
    float *prm, *grad, *m, *v, *part, *sq_err;   // sq_err [steps][batch]
    unsigned* barrier;            // arrivals; [1] set when a wait ran out
};

// Grid barrier in two halves; the k-th wait ends when k * gridDim.x blocks have
// arrived, or (false, for every block soon after) when it takes too long.
constexpr long long kBarrierCycles = 4000000000LL;   // ~2 s
__device__ __forceinline__ void grid_arrive(unsigned* bar)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(bar, 1u);
    }
}
__device__ __forceinline__ bool grid_wait(unsigned* bar, unsigned k, int* stop)
{
    if (threadIdx.x == 0) {
        const volatile unsigned* p = bar;
        const unsigned want = k * gridDim.x;
        const long long t0 = clock64();
        *stop = 0;
        while ((int)(*p - want) < 0) {
            if (clock64() - t0 > kBarrierCycles) atomicExch(bar + 1, 1u);
            if (p[1]) {
                *stop = 1;
                break;
            }
        }
        __threadfence();
    }
    __syncthreads();
    return *stop == 0;
}

// Features of the tile's samples, by the first kTrainRows threads.
__device__ __forceinline__ void load_samples(const TrainArgs& a, FbSmem& S, long long first, long long end)
{
    const int tid = threadIdx.x;
    if (tid < kTrainRows) {
        float x[kWIn] = {};
        float y = 0.0f;
        bool valid = false;
        if (first + tid < end) {
            const unsigned long long p = (a.perm_a * (unsigned long long)(first + tid) + a.perm_b) % (unsigned long long)a.n;
            valid = pair_features(a.pairs + p * kPairW, a.nm, x, &y);
            if (!valid)
                for (int k = 0; k < kWIn; ++k) x[k] = 0.0f;
        }
        for (int k = 0; k < kWIn; ++k) S.x[tid][k] = x[k];
        S.y[tid] = y;
        S.valid[tid] = valid;
    }
}

// The weights, past L1 (other blocks wrote them). Returns b3.
__device__ __forceinline__ float load_weights(const float* prm, FbSmem& S)
{
    static_assert(kP_B1 % 4 == 0 && kP_W2 % 4 == 0 && kP_B2 % 4 == 0 && kP_W3 % 4 == 0 && kP_B3 % 4 == 0, "float4 groups");
    constexpr int kThreads = kGemmThreads + kChoreThreads, kGroups = kP_B3 / 4, kEach = (kGroups + kThreads - 1) / kThreads;
    float4 v[kEach];
#pragma unroll
    for (int q = 0; q < kEach; ++q) {
        const int i = threadIdx.x + q * kThreads;
        if (i < kGroups) v[q] = __ldcg(reinterpret_cast<const float4*>(prm) + i);
    }
    const float b3 = __ldcg(prm + kP_B3);
#pragma unroll
    for (int q = 0; q < kEach; ++q) {
        const int i = 4 * (threadIdx.x + q * kThreads);
        if (i >= kP_B3) break;
        float* dst = i < kP_B1   ? &S.w1[0][0] + i
                     : i < kP_W2 ? S.b1 + (i - kP_B1)
                     : i < kP_B2 ? &S.w2[(i - kP_W2) / kWHid][(i - kP_W2) % kWHid]
                     : i < kP_W3 ? S.b2 + (i - kP_B2)
                                 : S.w3 + (i - kP_W3);
        *reinterpret_cast<float4*>(dst) = v[q];
    }
    return b3;
}

// One tile: forward and backward; gradient to gp, losses to sq_err (the samples,
// the weights and b3 are in place; ends without a barrier).
__device__ __forceinline__ void train_tile(FbSmem& S, float b3, float inv_batch, float* gp, float* sq_err)
{
    const int tid = threadIdx.x;
    __syncthreads();
    const bool gemm = tid < kGemmThreads;
    const int u0 = (tid / 16) * 4, tx = tid % 16;   // this thread's samples u0 .. u0 + 3, units tx, tx + 16, ...
    float d1[4][4], d2[4][4];                       // SiLU' of layer 1 and 2 (sample, unit)
    if (gemm) {
        // layer 1
        float x[4][kWIn];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int k = 0; k < kWIn; k += 4) load4(&S.x[u0 + i][k], *reinterpret_cast<float(*)[4]>(&x[i][k]));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int unit = tx + 16 * j;
            float w[kWIn];
#pragma unroll
            for (int k = 0; k < kWIn; k += 4) load4(&S.w1[unit][k], *reinterpret_cast<float(*)[4]>(&w[k]));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float z = S.b1[unit], a;
#pragma unroll
                for (int k = 0; k < kWIn; ++k) z += w[k] * x[i][k];
                silu_both(z, &a, &d1[i][j]);
                S.a1[u0 + i][unit] = a;
            }
        }
    }
    __syncthreads();
    if (gemm) {
        // layer 2: z2[s][j] = b2[j] + sum_k W2[j][k] a1[s][k]
        float acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = S.b2[tx + 16 * j];
#pragma unroll 4
        for (int k = 0; k < kWHid; k += 4) {
            float u[4][4], v[4][4];   // [row][k]
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                load4(&S.a1[u0 + i][k], u[i]);
                load4(&S.w2[tx + 16 * i][k], v[i]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float uq[4] = {u[0][q], u[1][q], u[2][q], u[3][q]}, vq[4] = {v[0][q], v[1][q], v[2][q], v[3][q]};
                tile_step(acc, uq, vq);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float a;
                silu_both(acc[i][j], &a, &d2[i][j]);
                S.a2[u0 + i][tx + 16 * j] = a;
            }
    }
    __syncthreads();
    if (tid < kTrainRows) {
        float out = b3;
#pragma unroll 16
        for (int j = 0; j < kWHid; ++j) out += S.w3[j] * S.a2[tid][j];
        const float err = S.valid[tid] ? (out - S.y[tid]) : 0.0f;
        S.g[tid] = err * inv_batch;  // loss = sum(err^2) / (2 batch)
        sq_err[tid] = 0.5f * err * err;
    }
    __syncthreads();
    if (gemm) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) S.dz2[u0 + i][tx + 16 * j] = S.g[u0 + i] * S.w3[tx + 16 * j] * d2[i][j];
    }
    __syncthreads();
    if (gemm) {
        // dA1[s][k] = sum_j W2[j][k] dZ2[s][j]
        float acc[4][4] = {};
#pragma unroll 4
        for (int j = 0; j < kWHid; j += 4) {
            float u[4][4];   // [sample][j]
#pragma unroll
            for (int i = 0; i < 4; ++i) load4(&S.dz2[u0 + i][j], u[i]);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float uq[4] = {u[0][q], u[1][q], u[2][q], u[3][q]};
                const float vq[4] = {S.w2[j + q][tx], S.w2[j + q][tx + 16], S.w2[j + q][tx + 32], S.w2[j + q][tx + 48]};
                tile_step(acc, uq, vq);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) S.dz1[u0 + i][tx + 16 * j] = acc[i][j] * d1[i][j];
        // dW2[j][k] = sum_s dZ2[s][j] a1[s][k]; units j = u0 .. u0 + 3, k = 4 tx .. 4 tx + 3
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
#pragma unroll 8
        for (int s = 0; s < kTrainRows; ++s) {
            float u[4], v[4];
            load4(&S.dz2[s][u0], u);
            load4(&S.a1[s][4 * tx], v);
            tile_step(acc, u, v);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            *reinterpret_cast<float4*>(gp + kP_W2 + (u0 + i) * kWHid + 4 * tx) =
                make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    } else {
        const int c = tid - kGemmThreads;
        if (c < kWHid) {
            float acc = 0.0f;   // dw3[j] = sum_s G[s] a2[s][j]
#pragma unroll 16
            for (int s = 0; s < kTrainRows; ++s) acc += S.g[s] * S.a2[s][c];
            gp[kP_W3 + c] = acc;
        } else {
            const int j = c - kWHid;
            float db = 0.0f;
#pragma unroll 16
            for (int s = 0; s < kTrainRows; ++s) db += S.dz2[s][j];
            gp[kP_B2 + j] = db;
        }
        if (c == 0) {
            float gb = 0.0f;
#pragma unroll 16
            for (int s = 0; s < kTrainRows; ++s) gb += S.g[s];
            gp[kP_B3] = gb;
        }
    }
    __syncthreads();
    if (gemm) {
        const int j = tid / 4, k = (tid % 4) * 2;   // dW1[j][k], dW1[j][k + 1]
        float a = 0.0f, b = 0.0f;
#pragma unroll 16
        for (int s = 0; s < kTrainRows; ++s) {
            const float d = S.dz1[s][j];
            a += d * S.x[s][k];
            b += d * S.x[s][k + 1];
        }
        gp[kP_W1 + j * kWIn + k] = a;
        gp[kP_W1 + j * kWIn + k + 1] = b;
    } else if (tid - kGemmThreads < kWHid) {
        const int j = tid - kGemmThreads;
        float db = 0.0f;
#pragma unroll 16
        for (int s = 0; s < kTrainRows; ++s) db += S.dz1[s][j];
        gp[kP_B1 + j] = db;
    }
}

// The block's share of the parameters: gradient over the tiles in order, AdamW.
__device__ __forceinline__ void update_share(const TrainArgs& a, FbSmem& S, int tiles, int step)
{
    const int c = threadIdx.x % kUpdateParams, row = threadIdx.x / kUpdateParams;
    const int share = (kNParams + gridDim.x - 1) / gridDim.x;
    const int end = min(kNParams, (int)(blockIdx.x + 1) * share);
    for (int p0 = blockIdx.x * share; p0 < end; p0 += kUpdateParams) {
        const int i = p0 + c;
        float g = 0.0f;
        for (int b0 = 0; b0 < tiles; b0 += kUpdateTiles) {
            const int n = min(kUpdateTiles, tiles - b0);
            __syncthreads();
            if (i < end) {
#pragma unroll
                for (int b = row; b < kUpdateTiles; b += kUpdateRows)
                    if (b < n) S.sums[b][c] = __ldcg(a.part + (size_t)(b0 + b) * kPartLd + i);
            }
            __syncthreads();
            if (row == 0 && i < end) {
                if (n == kUpdateTiles) {
#pragma unroll 32
                    for (int b = 0; b < kUpdateTiles; ++b) g += S.sums[b][c];
                } else {
                    for (int b = 0; b < n; ++b) g += S.sums[b][c];
                }
            }
        }
        if (row == 0 && i < end) {
            a.grad[i] = g;
            if (a.step) {
                const AdamStep o = a.step[step];
                const float mi = a.b1 * __ldcg(a.m + i) + (1.0f - a.b1) * g;
                const float vi = a.b2 * __ldcg(a.v + i) + (1.0f - a.b2) * g * g;
                __stcg(a.m + i, mi);
                __stcg(a.v + i, vi);
                const bool is_weight = (i < kP_B1) || (i >= kP_W2 && i < kP_B2) || (i >= kP_W3 && i < kP_B3);
                float p = __ldcg(a.prm + i);
                if (is_weight) p -= o.lr * a.wd * p;
                p -= o.lr * (mi / o.c1) / (sqrtf(vi / o.c2) + a.eps);
                __stcg(a.prm + i, p);
            }
        }
    }
}

__global__ void __launch_bounds__(kGemmThreads + kChoreThreads, 1) warm_train_kernel(const TrainArgs a)
{
    extern __shared__ __align__(16) unsigned char fb_smem[];
    FbSmem& S = *reinterpret_cast<FbSmem*>(fb_smem);
    unsigned arrivals = 0;
    for (int s = 0; s < a.steps; ++s) {
        const long long off = a.offset + (long long)s * a.batch;
        const long long end = min(off + a.batch, a.end);
        const int tiles = (int)((end - off + kTrainRows - 1) / kTrainRows);
        const float inv_batch = 1.0f / (float)(end - off);
        // (the first tile's samples were fetched while the last update ran)
        if (s == 0) load_samples(a, S, off + (long long)blockIdx.x * kTrainRows, end);
        const float b3 = load_weights(a.prm, S);
        for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
            if (t != (int)blockIdx.x) {
                __syncthreads();
                load_samples(a, S, off + (long long)t * kTrainRows, end);
            }
            train_tile(S, b3, inv_batch, a.part + (size_t)t * kPartLd, a.sq_err + (size_t)s * a.batch + (size_t)t * kTrainRows);
        }
        grid_arrive(a.barrier);
        if (s + 1 < a.steps)
            load_samples(a, S, off + a.batch + (long long)blockIdx.x * kTrainRows, min(off + 2ll * a.batch, a.end));
        if (!grid_wait(a.barrier, ++arrivals, &S.stop)) return;
        update_share(a, S, tiles, s);
        if (s + 1 < a.steps) {
            grid_arrive(a.barrier);
            if (!grid_wait(a.barrier, ++arrivals, &S.stop)) return;
        }
    }
}

// Sums of (err^2)/2 in double, in a fixed order: per block of 64 samples, per step
// over its blocks, then *loss_acc += the steps in order.
__global__ void __launch_bounds__(128) warm_block_loss_kernel(const float* __restrict__ sq_err, long long blocks,
                                                              double* __restrict__ block_loss)
{
    const long long b = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (b >= blocks) return;
    double l = 0.0;
    for (int s = 0; s < kTrainRows; ++s) l += (double)sq_err[b * kTrainRows + s];
    block_loss[b] = l;
}

__global__ void __launch_bounds__(256) warm_loss_kernel(const double* __restrict__ block_loss, int nblocks, int steps,
                                                        double* __restrict__ step_loss, double* __restrict__ loss_acc)
{
    for (int s = threadIdx.x; s < steps; s += blockDim.x) {
        double l = 0.0;
        for (int b = 0; b < nblocks; ++b) l += block_loss[(size_t)s * nblocks + b];
        step_loss[s] = l;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = *loss_acc;
        for (int s = 0; s < steps; ++s) a += step_loss[s];
        *loss_acc = a;
    }
}

// Pair compaction: valid rows (depth > 0) per 1024-row block, then their
// scatter to the block's offset in row order.
constexpr int kCompactRows = 1024;

__global__ void __launch_bounds__(kCompactRows) pair_count_kernel(const float* __restrict__ dense, long long n,
                                                                  int* __restrict__ counts)
{
    const long long i = (long long)blockIdx.x * kCompactRows + threadIdx.x;
    const bool ok = i < n && dense[i * kPairW + 8] > 0.0f;
    const int c = __syncthreads_count(ok);
    if (threadIdx.x == 0) counts[blockIdx.x] = c;
}

__global__ void __launch_bounds__(kCompactRows) pair_scatter_kernel(const float* __restrict__ dense, long long n,
                                                                    const long long* __restrict__ offsets,
                                                                    float* __restrict__ out, long long capacity)
{
    __shared__ int warp_cnt[kCompactRows / 32];
    const long long i = (long long)blockIdx.x * kCompactRows + threadIdx.x;
    const bool ok = i < n && dense[i * kPairW + 8] > 0.0f;
    const unsigned b = __ballot_sync(0xffffffffu, ok);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) warp_cnt[w] = __popc(b);
    __syncthreads();
    int before = 0;
    for (int k = 0; k < w; ++k) before += warp_cnt[k];
    before += __popc(b & ((1u << lane) - 1u));
    const long long dst = offsets[blockIdx.x] + before;
    if (ok && dst < capacity)
        for (int k = 0; k < kPairW; ++k) out[dst * kPairW + k] = dense[i * kPairW + k];
}

int compact_pairs(const float* dense, long long n_rows, float* out, long long capacity, long long* n_valid,
                  void* stream)
{
    *n_valid = 0;
    if (n_rows <= 0) return TROUTE_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const long long nb = (n_rows + kCompactRows - 1) / kCompactRows;
    if (nb > 0x7fffffffLL) return set_error(TROUTE_EINVAL, "too many pair rows");
    int* d_counts = nullptr;
    long long* d_off = nullptr;
    cudaError_t e = cudaMalloc(&d_counts, nb * sizeof(int));
    if (e == cudaSuccess) e = cudaMalloc(&d_off, nb * sizeof(long long));
    std::vector<int> counts(nb);
    std::vector<long long> off(nb);
    if (e == cudaSuccess) {
        pair_count_kernel<<<(unsigned)nb, kCompactRows, 0, st>>>(dense, n_rows, d_counts);
        e = cudaMemcpyAsync(counts.data(), d_counts, nb * sizeof(int), cudaMemcpyDeviceToHost, st);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    long long tot = 0;
    for (long long b = 0; b < nb; ++b) {
        off[b] = tot;
        tot += counts[b];
    }
    if (e == cudaSuccess && out && capacity > 0) {
        e = cudaMemcpyAsync(d_off, off.data(), nb * sizeof(long long), cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) {
            pair_scatter_kernel<<<(unsigned)nb, kCompactRows, 0, st>>>(dense, n_rows, d_off, out, capacity);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    }
    cudaFree(d_counts);
    cudaFree(d_off);
    if (e != cudaSuccess) return set_error(TROUTE_ECUDA, "pair compaction: %s", cudaGetErrorString(e));
    *n_valid = tot;
    return TROUTE_OK;
}

}  // namespace tr

using namespace tr;

struct troute_warm {
    float prm[kNParams];
    Norm nm;
    bool trained = false;
    // device: fp32 master copy, AdamW moments, gradient; bf16 inference layout;
    // epoch loss, per-block moments, grid barrier and buffers of the training launches
    float *d_prm = nullptr, *d_m = nullptr, *d_v = nullptr, *d_g = nullptr;
    __nv_bfloat16 *d_w1t = nullptr, *d_w2t = nullptr, *d_w3t = nullptr;
    float *d_b1 = nullptr, *d_b2 = nullptr;
    double *d_loss = nullptr, *d_mom = nullptr;
    unsigned* d_bar = nullptr;
    TrainBuffers buf;

    ~troute_warm()
    {
        for (void* p : {(void*)d_prm, (void*)d_m, (void*)d_v, (void*)d_g, (void*)d_w1t, (void*)d_w2t, (void*)d_w3t,
                        (void*)d_b1, (void*)d_b2, (void*)d_loss, (void*)d_mom, (void*)d_bar})
            if (p) cudaFree(p);
    }
};

static int warm_cuda(cudaError_t e, const char* what)
{
    if (e == cudaSuccess) return TROUTE_OK;
    return set_error(e == cudaErrorMemoryAllocation ? TROUTE_ENOMEM : TROUTE_ECUDA, "%s: %s", what,
                     cudaGetErrorString(e));
}

static int warm_alloc(troute_warm* w)
{
    if (w->d_prm) return TROUTE_OK;
    int rc;
    if ((rc = warm_cuda(cudaMalloc(&w->d_prm, kNParams * sizeof(float)), "cudaMalloc")) ||
        (rc = warm_cuda(cudaMalloc(&w->d_m, kNParams * sizeof(float)), "cudaMalloc")) ||
        (rc = warm_cuda(cudaMalloc(&w->d_v, kNParams * sizeof(float)), "cudaMalloc")) ||
        (rc = warm_cuda(cudaMalloc(&w->d_g, kNParams * sizeof(float)), "cudaMalloc")) ||
        (rc = warm_cuda(cudaMalloc(&w->d_w1t, kWHid * kWK1 * sizeof(__nv_bfloat16)), "cudaMalloc")) ||
        (rc = warm_cuda(cudaMalloc(&w->d_w2t, kWHid * kWHid * sizeof(__nv_bfloat16)), "cudaMalloc")) ||
        (rc = warm_cuda(cudaMalloc(&w->d_w3t, kWOut * kWHid * sizeof(__nv_bfloat16)), "cudaMalloc")) ||
        (rc = warm_cuda(cudaMalloc(&w->d_b1, kWHid * sizeof(float)), "cudaMalloc")) ||
        (rc = warm_cuda(cudaMalloc(&w->d_b2, kWHid * sizeof(float)), "cudaMalloc")) ||
        (rc = warm_cuda(cudaMalloc(&w->d_loss, sizeof(double)), "cudaMalloc")) ||
        (rc = warm_cuda(cudaMalloc(&w->d_bar, 2 * sizeof(unsigned)), "cudaMalloc")) ||
        (rc = warm_cuda(cudaMalloc(&w->d_mom, (size_t)kMomBlocks * kMomW * sizeof(double)), "cudaMalloc")))
        return rc;
    return TROUTE_OK;
}

// Adds the losses of `steps` steps of `tiles` tiles each (their samples from
// sq_err on) to *d_loss.
static int warm_add_losses(troute_warm* w, const float* sq_err, int tiles, int steps)
{
    const long long blocks = (long long)tiles * steps;
    warm_block_loss_kernel<<<(unsigned)((blocks + 127) / 128), 128>>>(sq_err, blocks, w->buf.loss.p);
    warm_loss_kernel<<<1, 256>>>(w->buf.loss.p, tiles, steps, w->buf.loss.p + blocks, w->d_loss);
    return warm_cuda(cudaGetLastError(), "loss launch");
}

// The steps of a (a.steps of them, a.batch samples each but the last) and their
// losses. The tiles of a batch are shared out over as many blocks as fit the GPU.
static int warm_train(troute_warm* w, TrainArgs& a)
{
    int rc, dev = 0, sms = 0, bps = 0;
    const int tiles = (a.batch + kTrainRows - 1) / kTrainRows;
    if ((rc = warm_cuda(cudaGetDevice(&dev), "cudaGetDevice")) ||
        (rc = warm_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "attr")) ||
        (rc = warm_cuda(cudaFuncSetAttribute(warm_train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FbSmem)),
                        "smem attribute")) ||
        (rc = warm_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, warm_train_kernel, kGemmThreads + kChoreThreads,
                                                                      sizeof(FbSmem)),
                        "occupancy")))
        return rc;
    a.nm = w->nm;
    a.prm = w->d_prm;
    a.grad = w->d_g;
    a.m = w->d_m;
    a.v = w->d_v;
    a.part = w->buf.part.p;
    a.sq_err = w->buf.err.p;
    a.barrier = w->d_bar;
    if ((rc = warm_cuda(cudaMemsetAsync(w->d_bar, 0, 2 * sizeof(unsigned), nullptr), "memset"))) return rc;
    void* args[] = {&a};
    if ((rc = warm_cuda(cudaLaunchCooperativeKernel((const void*)warm_train_kernel, dim3(std::min(tiles, sms * std::max(1, bps))),
                                                    dim3(kGemmThreads + kChoreThreads), args, sizeof(FbSmem), nullptr),
                        "training launch")))
        return rc;
    // a last, shorter batch is summed on its own
    const long long last = std::min<long long>(a.batch, a.end - a.offset - (long long)(a.steps - 1) * a.batch);
    const int last_tiles = (int)((last + kTrainRows - 1) / kTrainRows);
    const int full = last_tiles == tiles ? a.steps : a.steps - 1;
    if (full && (rc = warm_add_losses(w, w->buf.err.p, tiles, full))) return rc;
    if (full < a.steps && (rc = warm_add_losses(w, w->buf.err.p + (size_t)full * a.batch, last_tiles, 1))) return rc;
    return TROUTE_OK;
}

// Whether a barrier of the training launches ran out.
static int warm_train_status(troute_warm* w)
{
    unsigned b[2] = {0, 0};
    const int rc = warm_cuda(cudaMemcpy(b, w->d_bar, sizeof b, cudaMemcpyDeviceToHost), "training");
    if (rc) return rc;
    return b[1] ? set_error(TROUTE_ETIMEOUT, "training: a grid barrier ran out") : TROUTE_OK;
}

// Rounds the fp32 weights to the bf16, transposed, padded layout of the MMA path.
static int warm_publish(troute_warm* w)
{
    std::vector<__nv_bfloat16> w1t(kWHid * kWK1), w2t(kWHid * kWHid), w3t(kWOut * kWHid);
    for (int n = 0; n < kWHid; ++n)
        for (int k = 0; k < kWK1; ++k)
            w1t[n * kWK1 + k] = __float2bfloat16_rn(k < kWIn ? w->prm[kP_W1 + n * kWIn + k] : 0.0f);
    for (int n = 0; n < kWHid; ++n)
        for (int k = 0; k < kWHid; ++k) w2t[n * kWHid + k] = __float2bfloat16_rn(w->prm[kP_W2 + n * kWHid + k]);
    for (int n = 0; n < kWOut; ++n)
        for (int k = 0; k < kWHid; ++k) w3t[n * kWHid + k] = __float2bfloat16_rn(n == 0 ? w->prm[kP_W3 + k] : 0.0f);
    int rc;
    if ((rc = warm_cuda(cudaMemcpy(w->d_w1t, w1t.data(), w1t.size() * 2, cudaMemcpyHostToDevice), "H2D")) ||
        (rc = warm_cuda(cudaMemcpy(w->d_w2t, w2t.data(), w2t.size() * 2, cudaMemcpyHostToDevice), "H2D")) ||
        (rc = warm_cuda(cudaMemcpy(w->d_w3t, w3t.data(), w3t.size() * 2, cudaMemcpyHostToDevice), "H2D")) ||
        (rc = warm_cuda(cudaMemcpy(w->d_b1, w->prm + kP_B1, kWHid * 4, cudaMemcpyHostToDevice), "H2D")) ||
        (rc = warm_cuda(cudaMemcpy(w->d_b2, w->prm + kP_B2, kWHid * 4, cudaMemcpyHostToDevice), "H2D")))
        return rc;
    // the routing streams that read them do not wait for this one
    return warm_cuda(cudaStreamSynchronize(nullptr), "H2D");
}

namespace tr {
WarmDev warm_device_view(const troute_warm* w, double delta, int k)
{
    WarmDev m;
    m.w1t = w->d_w1t;
    m.w2t = w->d_w2t;
    m.w3t = w->d_w3t;
    m.b1 = w->d_b1;
    m.b2 = w->d_b2;
    m.b3 = w->prm[kP_B3];
    for (int i = 0; i < kWIn; ++i) {
        m.mu[i] = w->nm.mu[i];
        m.sd[i] = w->nm.sd[i];
        m.inv_sd[i] = 1.0f / w->nm.sd[i];
    }
    m.mu_y = w->nm.mu_y;
    m.sd_y = w->nm.sd_y;
    m.delta = delta;
    m.k = k;
    return m;
}
bool warm_ready(const troute_warm* w) { return w && w->d_w1t && w->trained; }
}  // namespace tr

extern "C" int troute_warm_create(troute_warm** out, uint64_t seed)
{
    if (!out) return set_error(TROUTE_EINVAL, "null pointer");
    auto* w = new (std::nothrow) troute_warm();
    if (!w) return set_error(TROUTE_ENOMEM, "model allocation");
    // He-style initialisation from the seed (counter-based, platform independent)
    for (int i = 0; i < kNParams; ++i) {
        const double u = u01(hash3(seed, 777, (uint64_t)i)) * 2.0 - 1.0;
        double scale = 0.0;
        if (i < kP_B1) scale = std::sqrt(6.0 / kWIn);
        else if (i >= kP_W2 && i < kP_B2) scale = std::sqrt(6.0 / kWHid);
        else if (i >= kP_W3 && i < kP_B3) scale = std::sqrt(6.0 / kWHid);
        w->prm[i] = (float)(u * scale * 0.5);
    }
    for (int k = 0; k < kWIn; ++k) {
        w->nm.mu[k] = 0.0f;
        w->nm.sd[k] = 1.0f;
    }
    w->nm.mu_y = 0.0f;
    w->nm.sd_y = 1.0f;
    *out = w;
    return TROUTE_OK;
}

extern "C" int troute_warm_destroy(troute_warm* w)
{
    delete w;
    return TROUTE_OK;
}

// params: [kNParams] then mu[8], sd[8], mu_y, sd_y
extern "C" int troute_warm_get(const troute_warm* w, float* params, int n)
{
    if (!w || !params || n < kNParams + 2 * kWIn + 2) return set_error(TROUTE_EINVAL, "need %d floats", kNParams + 2 * kWIn + 2);
    std::memcpy(params, w->prm, sizeof w->prm);
    std::memcpy(params + kNParams, w->nm.mu, sizeof w->nm.mu);
    std::memcpy(params + kNParams + kWIn, w->nm.sd, sizeof w->nm.sd);
    params[kNParams + 2 * kWIn] = w->nm.mu_y;
    params[kNParams + 2 * kWIn + 1] = w->nm.sd_y;
    return TROUTE_OK;
}

extern "C" int troute_warm_set(troute_warm* w, const float* params, int n)
{
    if (!w || !params || n < kNParams + 2 * kWIn + 2) return set_error(TROUTE_EINVAL, "need %d floats", kNParams + 2 * kWIn + 2);
    std::memcpy(w->prm, params, sizeof w->prm);
    std::memcpy(w->nm.mu, params + kNParams, sizeof w->nm.mu);
    std::memcpy(w->nm.sd, params + kNParams + kWIn, sizeof w->nm.sd);
    w->nm.mu_y = params[kNParams + 2 * kWIn];
    w->nm.sd_y = params[kNParams + 2 * kWIn + 1];
    int rc = warm_alloc(w);
    if (rc) return rc;
    if ((rc = warm_publish(w))) return rc;
    w->trained = true;
    return TROUTE_OK;
}

// Standardisation constants from the pairs (every stride-th pair).
static int warm_normalise(troute_warm* w, const float* pairs_dev, long long n, long long stride)
{
    int rc;
    warm_moments_kernel<<<kMomBlocks, kMomThreads>>>(pairs_dev, n, stride, w->d_mom);
    std::vector<double> part((size_t)kMomBlocks * kMomW);
    if ((rc = warm_cuda(cudaMemcpy(part.data(), w->d_mom, part.size() * sizeof(double), cudaMemcpyDeviceToHost),
                        "moments")))
        return rc;
    double acc[kMomW] = {};
    for (int b = 0; b < kMomBlocks; ++b)
        for (int k = 0; k < kMomW; ++k) acc[k] += part[(size_t)b * kMomW + k];
    const double cnt = acc[2 * kPairW];
    if (cnt < 2) return set_error(TROUTE_EINVAL, "no valid training pairs");
    float mu[kPairW], sd[kPairW];
    for (int k = 0; k < kPairW; ++k) {
        const double m = acc[k] / cnt;
        const double var = acc[kPairW + k] / cnt - m * m;
        mu[k] = (float)m;
        sd[k] = (float)std::sqrt(var > 1e-12 ? var : 1e-12);
    }
    for (int k = 0; k < kWIn; ++k) {
        w->nm.mu[k] = mu[k];
        w->nm.sd[k] = sd[k];
    }
    w->nm.mu_y = mu[8];
    w->nm.sd_y = sd[8];
    return TROUTE_OK;
}

static unsigned long long coprime_near(unsigned long long n, unsigned long long want)
{
    auto gcd = [](unsigned long long a, unsigned long long b) {
        while (b) { const unsigned long long t = a % b; a = b; b = t; }
        return a;
    };
    unsigned long long a = want % n;
    if (a == 0) a = 1;
    while (gcd(a, n) != 1) a = (a + 1) % n ? (a + 1) % n : 1;
    return a;
}

extern "C" int troute_warm_fit(troute_warm* w, const float* pairs_dev, long long n_pairs, int epochs, int batch,
                               float lr, float weight_decay, uint64_t seed, float* loss_per_epoch)
{
    if (!w || !pairs_dev || n_pairs < 2 || epochs < 1 || batch < kTrainRows || lr <= 0.0f)
        return set_error(TROUTE_EINVAL, "bad training arguments");
    int rc = warm_alloc(w);
    if (rc) return rc;
    if ((rc = warm_normalise(w, pairs_dev, n_pairs, n_pairs > 4000000 ? n_pairs / 4000000 : 1))) return rc;
    batch = (batch / kTrainRows) * kTrainRows;
    if ((rc = warm_cuda(cudaMemcpy(w->d_prm, w->prm, sizeof w->prm, cudaMemcpyHostToDevice), "H2D")) ||
        (rc = warm_cuda(cudaMemset(w->d_m, 0, kNParams * sizeof(float)), "memset")) ||
        (rc = warm_cuda(cudaMemset(w->d_v, 0, kNParams * sizeof(float)), "memset")))
        return rc;
    const long long steps_per_epoch = (n_pairs + batch - 1) / batch;
    const long long total = steps_per_epoch * epochs;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const int tiles = batch / kTrainRows;
    const int keep = train_steps_kept(steps_per_epoch, tiles);
    if ((rc = warm_cuda(w->buf.reserve(tiles, keep), "cudaMalloc"))) return rc;
    std::vector<AdamStep> consts((size_t)keep);
    long long step = 0;
    for (int ep = 0; ep < epochs; ++ep) {
        TrainArgs a = {};
        a.pairs = pairs_dev;
        a.n = n_pairs;
        a.end = n_pairs;
        a.batch = batch;
        a.perm_a = coprime_near((unsigned long long)n_pairs, hash3(seed, 31, ep) | 1ull);
        a.perm_b = hash3(seed, 37, ep) % (unsigned long long)n_pairs;
        a.step = w->buf.step.p;
        a.b1 = b1;
        a.b2 = b2;
        a.eps = eps;
        a.wd = weight_decay;
        if ((rc = warm_cuda(cudaMemset(w->d_loss, 0, sizeof(double)), "memset"))) return rc;
        for (long long s = 0; s < steps_per_epoch; s += keep) {
            a.offset = s * batch;
            a.steps = (int)std::min<long long>(keep, steps_per_epoch - s);
            for (int k = 0; k < a.steps; ++k, ++step) {
                // cosine decay of the step size
                const float frac = (float)step / (float)std::max<long long>(1, total - 1);
                consts[k].lr = lr * 0.5f * (1.0f + std::cos(3.14159265f * frac));
                consts[k].c1 = 1.0f - std::pow(b1, (float)(step + 1));
                consts[k].c2 = 1.0f - std::pow(b2, (float)(step + 1));
            }
            // (a pageable copy: ordered after the launch before, and done when it returns)
            if ((rc = warm_cuda(cudaMemcpy(w->buf.step.p, consts.data(), (size_t)a.steps * sizeof(AdamStep), cudaMemcpyHostToDevice),
                                "step constants")) ||
                (rc = warm_train(w, a)) || (rc = warm_train_status(w)))
                return rc;
        }
        double loss = 0.0;
        if ((rc = warm_cuda(cudaMemcpy(&loss, w->d_loss, sizeof(double), cudaMemcpyDeviceToHost), "loss"))) return rc;
        // each step's loss is sum(err^2)/2 over its batch: the epoch mean per pair
        if (loss_per_epoch) loss_per_epoch[ep] = (float)(loss / (double)n_pairs);
    }
    if ((rc = warm_cuda(cudaMemcpy(w->prm, w->d_prm, sizeof w->prm, cudaMemcpyDeviceToHost), "D2H"))) return rc;
    if ((rc = warm_publish(w))) return rc;
    w->trained = true;
    return warm_cuda(cudaGetLastError(), "training");
}

extern "C" int troute_warm_grad(troute_warm* w, const float* pairs_host, int n, float* grad_out, double* loss_out)
{
    if (!w || !pairs_host || n < 1 || !grad_out) return set_error(TROUTE_EINVAL, "bad arguments");
    int rc = warm_alloc(w);
    if (rc) return rc;
    float* d_pairs = nullptr;
    if ((rc = warm_cuda(cudaMalloc(&d_pairs, (size_t)n * kPairW * sizeof(float)), "cudaMalloc"))) return rc;
    rc = warm_cuda(cudaMemcpy(d_pairs, pairs_host, (size_t)n * kPairW * sizeof(float), cudaMemcpyHostToDevice), "H2D");
    if (!rc) rc = warm_cuda(cudaMemcpy(w->d_prm, w->prm, sizeof w->prm, cudaMemcpyHostToDevice), "H2D");
    if (!rc) rc = warm_cuda(cudaMemset(w->d_loss, 0, sizeof(double)), "memset");
    if (!rc) rc = warm_cuda(w->buf.reserve((n + kTrainRows - 1) / kTrainRows, 1), "cudaMalloc");
    TrainArgs a = {};
    a.pairs = d_pairs;
    a.n = n;
    a.end = n;
    a.batch = n;
    a.steps = 1;
    a.perm_a = 1;
    if (!rc) rc = warm_train(w, a);
    if (!rc) rc = warm_train_status(w);
    if (!rc) rc = warm_cuda(cudaMemcpy(grad_out, w->d_g, kNParams * sizeof(float), cudaMemcpyDeviceToHost), "D2H");
    double loss = 0.0;
    if (!rc) rc = warm_cuda(cudaMemcpy(&loss, w->d_loss, sizeof(double), cudaMemcpyDeviceToHost), "D2H");
    cudaFree(d_pairs);
    if (loss_out) *loss_out = loss / n;
    return rc;
}

extern "C" int troute_warm_predict(troute_warm* w, const float* raw_host, int n, double* depth_out)
{
    if (!w || !raw_host || n < 1 || !depth_out) return set_error(TROUTE_EINVAL, "bad arguments");
    if (!w->trained) return set_error(TROUTE_ESTATE, "model has no weights (train or set them first)");
    float* d_raw = nullptr;
    double* d_out = nullptr;
    int* d_err = nullptr;
    int rc = warm_cuda(cudaMalloc(&d_raw, (size_t)n * kWIn * sizeof(float)), "cudaMalloc");
    if (!rc) rc = warm_cuda(cudaMalloc(&d_out, (size_t)n * sizeof(double)), "cudaMalloc");
    if (!rc) rc = warm_cuda(cudaMalloc(&d_err, sizeof(int)), "cudaMalloc");
    if (!rc) rc = warm_cuda(cudaMemset(d_err, 0, sizeof(int)), "memset");
    if (!rc) rc = warm_cuda(cudaMemcpy(d_raw, raw_host, (size_t)n * kWIn * sizeof(float), cudaMemcpyHostToDevice), "H2D");
    if (!rc) rc = launch_warm_gemm_raw(w, d_raw, n, d_out, d_err, nullptr);
    int err = 0;
    if (!rc) rc = warm_cuda(cudaMemcpy(depth_out, d_out, (size_t)n * sizeof(double), cudaMemcpyDeviceToHost), "D2H");
    if (!rc) rc = warm_cuda(cudaMemcpy(&err, d_err, sizeof(int), cudaMemcpyDeviceToHost), "D2H");
    cudaFree(d_raw);
    cudaFree(d_out);
    cudaFree(d_err);
    if (!rc && err) rc = set_error(err, "warm GEMM: a tensor-core completion wait ran out");
    return rc;
}
