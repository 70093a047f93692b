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
#include <cstring>
#include <vector>

#include "warm.cuh"

namespace tr {

// Flat parameter vector: W1 [64][8] (out x in), b1 [64], W2 [64][64], b2 [64],
// w3 [64], b3.
constexpr int kP_W1 = 0, kP_B1 = kP_W1 + kWHid * kWIn, kP_W2 = kP_B1 + kWHid, kP_B2 = kP_W2 + kWHid * kWHid,
              kP_W3 = kP_B2 + kWHid, kP_B3 = kP_W3 + kWHid, kNParams = kP_B3 + 1;
constexpr int kPairW = 9;  // qup quc qdp ql dx s0 n bw depth
constexpr int kTrainRows = 64;

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

// One mini-batch block of kTrainRows samples: forward, backward, and the
// block's gradient (part[block][kPartLd]) and loss sum (loss_part[block]).
// Sample i of the batch is pair (perm_a * i + perm_b) mod n, a permutation of
// the pairs when gcd(perm_a, n) = 1. Every sum runs in a fixed order, so a
// training run is reproducible bit for bit.
//
// FP32 multiply and add rates bound it: three 64 x 64 x 64 products per block
// (layer 2 forward, its weight gradient, its input gradient), 12.3 k cycles of an
// SM's FP32 lanes. kGemmThreads threads hold 4 x 4 tiles of each product in
// registers, every sum over its inner index in order (what one thread per sample
// did with 64 threads and scalar shared-memory reads in 94 us, batch 8,192);
// activations whose derivative is needed later stay in the registers of the
// thread that will use them. The other kChoreThreads form the bias and last-layer
// sums beside the products.
constexpr int kGemmThreads = 256, kChoreThreads = 128;
constexpr int kTLd = 68;         // row of a 64-wide tile: 16-byte aligned, banks shifted by 4
constexpr int kPartLd = 4804;    // row of the partial gradients, 16-byte aligned
static_assert(kTrainRows == 64 && kWHid == 64 && kPartLd >= kNParams && kPartLd % 4 == 0 && kP_W2 % 4 == 0, "tile shapes");

struct FbSmem {
    float w1[kWHid][kWIn], b1[kWHid], b2[kWHid], w3[kWHid];
    float x[kTrainRows][kWIn], y[kTrainRows], g[kTrainRows], e[kTrainRows];
    int valid[kTrainRows];
    float w2[kWHid][kTLd], w2t[kWHid][kTLd];        // [out][in], [in][out]
    float a1[kTrainRows][kTLd], a1t[kWHid][kTLd];   // [sample][unit], [unit][sample]
    float dz2[kTrainRows][kTLd], dz2t[kWHid][kTLd];
    float a2[kTrainRows][kWHid + 1], dz1[kTrainRows][kWHid + 1];
};

// SiLU z / (1 + e^-z) and its derivative from one exponential.
__device__ __forceinline__ void silu_both(float z, float* a, float* d)
{
    const float t = 1.0f + expf(-z);
    *a = z / t;
    const float s = 1.0f / t;
    *d = s * (1.0f + z * (1.0f - s));
}

// acc[i][j] += u[i] * v[j] over a row of each operand.
__device__ __forceinline__ void tile_step(float (&acc)[4][4], const float* u, const float* v)
{
    const float4 a = *reinterpret_cast<const float4*>(u), b = *reinterpret_cast<const float4*>(v);
    const float ai[4] = {a.x, a.y, a.z, a.w}, bj[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += ai[i] * bj[j];
}

// Programmatic dependent launch: what follows waits for the kernel before.
__device__ __forceinline__ void wait_previous_kernel() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_kernel_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__global__ void __launch_bounds__(kGemmThreads + kChoreThreads, 1)
    warm_fb_kernel(const float* __restrict__ pairs, long long n, long long offset, int batch, unsigned long long perm_a,
                   unsigned long long perm_b, const float* prm, Norm nm, float* __restrict__ part,
                   double* __restrict__ loss_part, float inv_batch)
{
    extern __shared__ __align__(16) unsigned char fb_smem[];
    FbSmem& S = *reinterpret_cast<FbSmem*>(fb_smem);
    const int tid = threadIdx.x;
    let_next_kernel_start();
    // the samples do not depend on the weights: fetched while the last update runs
    if (tid < kTrainRows) {
        const long long i = offset + (long long)blockIdx.x * kTrainRows + tid;
        float x[kWIn] = {};
        float y = 0.0f;
        bool valid = false;
        if (i < offset + batch) {
            const unsigned long long p = (perm_a * (unsigned long long)i + perm_b) % (unsigned long long)n;
            valid = pair_features(pairs + p * kPairW, nm, x, &y);
            if (!valid)
                for (int k = 0; k < kWIn; ++k) x[k] = 0.0f;
        }
        for (int k = 0; k < kWIn; ++k) S.x[tid][k] = x[k];
        S.y[tid] = y;
        S.valid[tid] = valid;
    }
    wait_previous_kernel();
    // (the weights change between launches that overlap: plain loads past L1)
    for (int i = tid; i < kP_B3; i += blockDim.x) {
        const float v = __ldcg(prm + i);
        if (i < kP_B1) S.w1[i / kWIn][i % kWIn] = v;
        else if (i < kP_W2) S.b1[i - kP_B1] = v;
        else if (i < kP_B2) {
            const int j = (i - kP_W2) / kWHid, k = (i - kP_W2) % kWHid;
            S.w2[j][k] = v;
            S.w2t[k][j] = v;
        } else if (i < kP_W3) S.b2[i - kP_B2] = v;
        else S.w3[i - kP_W3] = v;
    }
    const float b3 = __ldcg(prm + kP_B3);
    __syncthreads();
    float* gp = part + (size_t)blockIdx.x * kPartLd;
    const bool gemm = tid < kGemmThreads;
    const int u0 = (tid / 16) * 4, v0 = (tid % 16) * 4;   // this thread's tile
    float d1[4][4], d2[4][4];                             // SiLU' of layer 1 and 2 (sample, unit)
    if (gemm) {
        // layer 1
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float a[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float z = S.b1[v0 + j];
#pragma unroll
                for (int k = 0; k < kWIn; ++k) z += S.w1[v0 + j][k] * S.x[u0 + i][k];
                silu_both(z, &a[i], &d1[i][j]);
                S.a1[u0 + i][v0 + j] = a[i];
            }
            *reinterpret_cast<float4*>(&S.a1t[v0 + j][u0]) = make_float4(a[0], a[1], a[2], a[3]);
        }
    }
    __syncthreads();
    if (gemm) {
        // layer 2: z2[s][j] = b2[j] + sum_k W2[j][k] a1[s][k]
        float acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = S.b2[v0 + j];
#pragma unroll 8
        for (int k = 0; k < kWHid; ++k) tile_step(acc, &S.a1t[k][u0], &S.w2t[k][v0]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float a;
                silu_both(acc[i][j], &a, &d2[i][j]);
                S.a2[u0 + i][v0 + j] = a;
            }
    }
    __syncthreads();
    if (tid < kTrainRows) {
        float out = b3;
#pragma unroll 16
        for (int j = 0; j < kWHid; ++j) out += S.w3[j] * S.a2[tid][j];
        const float err = S.valid[tid] ? (out - S.y[tid]) : 0.0f;
        S.g[tid] = err * inv_batch;  // loss = sum(err^2) / (2 batch)
        S.e[tid] = 0.5f * err * err;
    }
    __syncthreads();
    if (gemm) {
        float t[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int j = 0; j < 4; ++j) t[i][j] = S.g[u0 + i] * S.w3[v0 + j] * d2[i][j];
            *reinterpret_cast<float4*>(&S.dz2[u0 + i][v0]) = make_float4(t[i][0], t[i][1], t[i][2], t[i][3]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            *reinterpret_cast<float4*>(&S.dz2t[v0 + j][u0]) = make_float4(t[0][j], t[1][j], t[2][j], t[3][j]);
    }
    __syncthreads();
    if (gemm) {
        // dW2[j][k] = sum_s dZ2[s][j] a1[s][k]
        float acc[4][4] = {};
#pragma unroll 8
        for (int s = 0; s < kTrainRows; ++s) tile_step(acc, &S.dz2[s][u0], &S.a1[s][v0]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            *reinterpret_cast<float4*>(gp + kP_W2 + (u0 + i) * kWHid + v0) =
                make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        // dA1[s][k] = sum_j W2[j][k] dZ2[s][j]
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
#pragma unroll 8
        for (int j = 0; j < kWHid; ++j) tile_step(acc, &S.dz2t[j][u0], &S.w2[j][v0]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) S.dz1[u0 + i][v0 + j] = acc[i][j] * d1[i][j];
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
            for (int s = 0; s < kTrainRows; ++s) gb += S.g[s];
            gp[kP_B3] = gb;
        }
        if (c == kWHid) {
            double ls = 0.0;
            for (int s = 0; s < kTrainRows; ++s) ls += (double)S.e[s];
            loss_part[blockIdx.x] = ls;
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

// One AdamW step's constants; apply = 0: only the gradient is formed.
struct AdamW {
    float lr, b1, b2, eps, wd, c1, c2;
    int apply;
};

// grad[i] = sum over blocks of part[b][i], blocks in order (their loads in flight
// together), and the AdamW step of parameter i.
constexpr int kUpdateThreads = 64, kUpdateBatch = 32;
__global__ void __launch_bounds__(kUpdateThreads) warm_update_kernel(const float* part, int nblocks, float* __restrict__ grad,
                                                                     float* prm, float* m, float* v, AdamW o)
{
    let_next_kernel_start();
    wait_previous_kernel();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kNParams) return;
    float g = 0.0f;
    for (int b0 = 0; b0 < nblocks; b0 += kUpdateBatch) {
        float t[kUpdateBatch];
#pragma unroll
        for (int b = 0; b < kUpdateBatch; ++b) t[b] = b0 + b < nblocks ? __ldcg(part + (size_t)(b0 + b) * kPartLd + i) : 0.0f;
#pragma unroll
        for (int b = 0; b < kUpdateBatch; ++b)
            if (b0 + b < nblocks) g += t[b];
    }
    grad[i] = g;
    if (!o.apply) return;
    // (launches overlap: what the one before wrote is read past L1)
    const float mi = o.b1 * __ldcg(m + i) + (1.0f - o.b1) * g;
    const float vi = o.b2 * __ldcg(v + i) + (1.0f - o.b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    const bool is_weight = (i < kP_B1) || (i >= kP_W2 && i < kP_B2) || (i >= kP_W3 && i < kP_B3);
    float p = __ldcg(prm + i);
    if (is_weight) p -= o.lr * o.wd * p;
    p -= o.lr * (mi / o.c1) / (sqrtf(vi / o.c2) + o.eps);
    prm[i] = p;
}

// Loss of each step (its blocks in order), then *loss_acc += the steps in order.
__global__ void __launch_bounds__(256) warm_loss_kernel(const double* __restrict__ loss_part, int nblocks, int steps,
                                                        double* __restrict__ step_loss, double* __restrict__ loss_acc)
{
    for (int s = threadIdx.x; s < steps; s += blockDim.x) {
        double l = 0.0;
        for (int b = 0; b < nblocks; ++b) l += loss_part[(size_t)s * nblocks + b];
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
    // per-block partial gradients / losses / moments of the training kernels
    float *d_prm = nullptr, *d_m = nullptr, *d_v = nullptr, *d_g = nullptr;
    __nv_bfloat16 *d_w1t = nullptr, *d_w2t = nullptr, *d_w3t = nullptr;
    float *d_b1 = nullptr, *d_b2 = nullptr;
    double *d_loss = nullptr, *d_mom = nullptr;
    float* d_part = nullptr;
    double* d_lpart = nullptr;
    int part_blocks = 0;
    size_t lpart_n = 0;

    ~troute_warm()
    {
        for (void* p : {(void*)d_prm, (void*)d_m, (void*)d_v, (void*)d_g, (void*)d_w1t, (void*)d_w2t, (void*)d_w3t,
                        (void*)d_b1, (void*)d_b2, (void*)d_loss, (void*)d_mom, (void*)d_part, (void*)d_lpart})
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
        (rc = warm_cuda(cudaMalloc(&w->d_mom, (size_t)kMomBlocks * kMomW * sizeof(double)), "cudaMalloc")))
        return rc;
    return TROUTE_OK;
}

// Room for the partial gradients of a mini-batch of nblocks blocks, and for the
// block losses of `steps` of them with a sum each.
static int warm_parts(troute_warm* w, int nblocks, int steps)
{
    int rc;
    if (nblocks > w->part_blocks) {
        if (w->d_part) cudaFree(w->d_part);
        w->d_part = nullptr;
        w->part_blocks = 0;
        if ((rc = warm_cuda(cudaMalloc(&w->d_part, (size_t)nblocks * kPartLd * sizeof(float)), "cudaMalloc"))) return rc;
        w->part_blocks = nblocks;
    }
    const size_t need = (size_t)steps * ((size_t)nblocks + 1);
    if (need > w->lpart_n) {
        if (w->d_lpart) cudaFree(w->d_lpart);
        w->d_lpart = nullptr;
        w->lpart_n = 0;
        if ((rc = warm_cuda(cudaMalloc(&w->d_lpart, need * sizeof(double)), "cudaMalloc"))) return rc;
        w->lpart_n = need;
    }
    return TROUTE_OK;
}

// Launches kernel so that it may start (up to its wait) while the one before it on
// the stream still runs.
template <class... P, class... A>
static cudaError_t launch_overlapped(void (*kernel)(P...), int blocks, int threads, size_t smem, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

static int warm_fb_attr()
{
    return warm_cuda(cudaFuncSetAttribute(warm_fb_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FbSmem)),
                     "smem attribute");
}

// One mini-batch: gradient into d_g, AdamW step o, block losses into lpart.
static int warm_step(troute_warm* w, const float* pairs, long long n, long long off, int b, unsigned long long pa,
                     unsigned long long pb, float inv_batch, const AdamW& o, double* lpart)
{
    const int nblocks = (b + kTrainRows - 1) / kTrainRows;
    const int rc = warm_cuda(launch_overlapped(warm_fb_kernel, nblocks, kGemmThreads + kChoreThreads, sizeof(FbSmem), pairs, n,
                                               off, b, pa, pb, w->d_prm, w->nm, w->d_part, lpart, inv_batch),
                             "training launch");
    if (rc) return rc;
    return warm_cuda(launch_overlapped(warm_update_kernel, (kNParams + kUpdateThreads - 1) / kUpdateThreads, kUpdateThreads, 0,
                                       w->d_part, nblocks, w->d_g, w->d_prm, w->d_m, w->d_v, o),
                     "update launch");
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
    return TROUTE_OK;
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
    if ((rc = warm_fb_attr())) return rc;
    const long long steps_per_epoch = (n_pairs + batch - 1) / batch;
    const long long total = steps_per_epoch * epochs;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    // block losses are kept for a run of steps and summed together: one thread's
    // sum of 128 doubles takes longer than a whole update
    const int full_blocks = batch / kTrainRows;
    const int keep = (int)std::min<long long>(steps_per_epoch, std::max(1, (1 << 22) / (full_blocks + 1)));
    if ((rc = warm_parts(w, full_blocks, keep))) return rc;
    double* const step_loss = w->d_lpart + (size_t)keep * full_blocks;
    long long step = 0;
    for (int ep = 0; ep < epochs; ++ep) {
        const unsigned long long pa = coprime_near((unsigned long long)n_pairs, hash3(seed, 31, ep) | 1ull);
        const unsigned long long pb = hash3(seed, 37, ep) % (unsigned long long)n_pairs;
        if ((rc = warm_cuda(cudaMemset(w->d_loss, 0, sizeof(double)), "memset"))) return rc;
        int kept = 0;
        for (long long s = 0; s < steps_per_epoch; ++s, ++step) {
            const long long off = s * batch;
            const int b = (int)std::min<long long>(batch, n_pairs - off);
            // cosine decay of the step size
            const float frac = (float)step / (float)std::max<long long>(1, total - 1);
            AdamW o;
            o.lr = lr * 0.5f * (1.0f + std::cos(3.14159265f * frac));
            o.c1 = 1.0f - std::pow(b1, (float)(step + 1));
            o.c2 = 1.0f - std::pow(b2, (float)(step + 1));
            o.b1 = b1;
            o.b2 = b2;
            o.eps = eps;
            o.wd = weight_decay;
            o.apply = 1;
            const int nblocks = (b + kTrainRows - 1) / kTrainRows;
            // (a last, smaller batch is summed on its own: its rows are shorter)
            if (kept == keep || (kept && nblocks != full_blocks)) {
                warm_loss_kernel<<<1, 256>>>(w->d_lpart, full_blocks, kept, step_loss, w->d_loss);
                kept = 0;
            }
            if ((rc = warm_step(w, pairs_dev, n_pairs, off, b, pa, pb, 1.0f / (float)b, o,
                                w->d_lpart + (size_t)kept * full_blocks)))
                return rc;
            ++kept;
            if (nblocks != full_blocks) {
                warm_loss_kernel<<<1, 256>>>(w->d_lpart, nblocks, 1, step_loss, w->d_loss);
                kept = 0;
            }
        }
        if (kept) warm_loss_kernel<<<1, 256>>>(w->d_lpart, full_blocks, kept, step_loss, w->d_loss);
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
    if (!rc) rc = warm_fb_attr();
    const int nblocks = (n + kTrainRows - 1) / kTrainRows;
    if (!rc) rc = warm_parts(w, nblocks, 1);
    if (!rc) rc = warm_step(w, d_pairs, n, 0, n, 1, 0, 1.0f / (float)n, AdamW{}, w->d_lpart);
    if (!rc) {
        warm_loss_kernel<<<1, 256>>>(w->d_lpart, nblocks, 1, w->d_lpart + nblocks, w->d_loss);
        rc = warm_cuda(cudaGetLastError(), "loss launch");
    }
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
