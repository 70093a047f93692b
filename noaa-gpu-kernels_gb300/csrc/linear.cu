// Linearised Muskingum-Cunge: the reference's fast approximate mode
// (water-prediction/t-route/wavefront/linear_mc.cu), with the secant path as
// the yardstick of its error.
//
// Per segment, once: C1..C3 and C4/ql from the channel at a reference depth
// of half bankfull (at least 0.1 m) with X from the Cunge formula at zero
// residual (linear_mc.cu:57-100), FP32. Per step, in topological order:
//   Q_new[i] = C1 Q_up_new + C2 Q_up_old + C3 Q_old[i] + (C4/ql) qlat[i]
// where Q_up is the sum of the upstream reaches' last segments for a reach's
// first segment and the previous segment otherwise (linear_mc.cu:129-165,
// cpu_linear_mc :177-232), FP32 like the reference.
//
// On the GPU: the network is cut into paths, each running from a headwater
// downstream, at every confluence with the deepest upstream reach; the other
// ("light") reaches end paths of their own there. A path's outflow is all that
// other paths read. A warp routes a path for many time steps in one sweep down its
// segments: lane c holds the steps c K .. c K + K - 1 and works on segment i - c in
// round i, so that the segment's discharge after lane c's steps reaches lane c + 1
// by a shuffle for the next round, and the inflow of the segment below stays in
// the lane's registers. Coefficients are read once per sweep, every load is issued
// rounds before its use, and nothing is synchronised within a path.
// Paths are ordered by depth (their deepest chain of reaches): one is only fed by
// shallower ones, so handing them out in that order can wait but not deadlock. The
// outflows are their own flags: the array is filled with a NaN that no operation
// produces, and a reader looks until it finds another value, or until a whole wait
// budget has passed in which no sweep anywhere came to its end or 64 rounds on (14 us
// of a deep path at 48 steps; a count every eight rounds costs 0.1 ms of 2.6).
// What bounds it: the longest path's rounds (the 2.7 M-segment network: 7,400
// segments), so deep paths get a block each and the fewest steps per lane; the many
// short ones share warps and take 8 steps per lane, their bound being the loads.
// (Before: a ready queue of (reach, step) items, one lane each, whose atomics set
// the pace: 2.7 M segments, 48 steps 112 ms.)
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "troute_internal.h"

namespace tr {
namespace {

constexpr unsigned kFull = 0xffffffffu;

// Coefficients of one segment (linear_mc.cu:57-100), FP32 with the reference's
// operation order; powf / sqrtf are CUDA's.
__device__ __forceinline__ float4 lin_coeffs(const troute_chparams_f32& p, float dt)
{
    const float z = (p.cs == 0.0f) ? 1.0f : 1.0f / p.cs;
    float bfd;
    if (p.bw > p.tw) bfd = p.bw / 0.00001f;
    else if (p.bw == p.tw) bfd = p.bw / (2.0f * z);
    else bfd = (p.tw - p.bw) / (2.0f * z);
    const float h = fmaxf(0.5f * bfd, 0.1f);
    const float twl = p.bw + 2.0f * z * h;
    const float A = (p.bw + h * z) * h;
    const float WP = p.bw + 2.0f * h * sqrtf(1.0f + z * z);
    const float R = (WP > 0.0f) ? A / WP : 0.0f;
    const float r23 = powf(R, 2.0f / 3.0f);
    const float r53 = powf(R, 5.0f / 3.0f);
    const float Ck = fmaxf(1e-6f, (sqrtf(p.s0) / p.n_ch) *
                                      ((5.0f / 3.0f) * r23 -
                                       (2.0f / 3.0f) * r53 * (2.0f * sqrtf(1.0f + z * z) / (p.bw + 2.0f * h * z))));
    const float Km = fmaxf(dt, p.dx / Ck);
    const float tw_use = (h > bfd && p.twcc > 0.0f) ? p.twcc : twl;
    float X = 0.25f;
    if (Ck > 0.0f && tw_use * p.s0 * Ck * p.dx > 0.0f)
        X = fminf(0.5f, fmaxf(0.0f, 0.5f * (1.0f - 0.0f / (2.0f * tw_use * p.s0 * Ck * p.dx))));
    float D = Km * (1.0f - X) + dt / 2.0f;
    if (D == 0.0f) D = 1.0f;
    return make_float4((Km * X + dt / 2.0f) / D, (dt / 2.0f - Km * X) / D, (Km * (1.0f - X) - dt / 2.0f) / D, dt / D);
}

__global__ void lin_coeff_kernel(const troute_chparams_f32* __restrict__ p, int n, float dt, float4* __restrict__ c)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) c[i] = lin_coeffs(p[i], dt);
}

// One segment of a path, in path order.
struct __align__(16) LinSeg {
    float c1, c2, c3, c4;
    int idx;    // the caller's segment
    int kind;   // how its inflow is formed (below)
    int up;     // kind 3: path of the light upstream reach; kind 4: row start in `ups`
    int n_up;   // kind 4: upstream reaches
};
enum : int {
    kInner = 0,   // the segment above
    kHead = 1,    // a headwater's first segment: none (it is its path's first)
    kOne = 2,     // a reach's first segment, one upstream reach
    kTwo = 3,     // ... two: the path's own and `up`
    kMany = 4     // ... any list in `ups`: paths, -1 for the path's own
};

constexpr unsigned kUnset = 0xffffffffu;   // outflow not yet written

struct LinRun {
    long long S;
    int T, Tp;                      // steps of this launch; row length of `out`
    const int* path_ptr;            // [paths + 1] into seg
    const LinSeg* seg;
    const int* ups;
    const float* out0;              // [paths] outflow before the launch
    unsigned* out;                  // [paths][Tp] outflow (float bits)
    float* Q;                       // [S] discharge, updated in place
    const float* qlat;              // [T][S]
    const int2* items;              // {first path, paths} of a warp's sweep, shallow first
    int n_items;
    int* ticket;                    // sweeps taken; a warp or block asks again at the end of one
    int* progress;                  // counts 64 rounds of a sweep
    int* error;                     // 0 ok, TROUTE_ETIMEOUT
    long long wait_cycles;
};

// A wait's budget starts again with whatever has been done anywhere since it began.
struct LinBudget {
    const int *ticket, *progress;
    int* error;
    long long wait_cycles, t0;
    int seen;
    __device__ __forceinline__ explicit LinBudget(const LinRun& d)
        : ticket(d.ticket), progress(d.progress), error(d.error), wait_cycles(d.wait_cycles)
    {
        t0 = clock64();
        seen = done();
    }
    __device__ __forceinline__ int done() const
    {
        return *reinterpret_cast<const volatile int*>(ticket) + *reinterpret_cast<const volatile int*>(progress);
    }
    // whether the wait goes on; it does not once a wait anywhere has run out
    __device__ __forceinline__ bool left()
    {
        if (clock64() - t0 > wait_cycles) {
            const int now = done();
            if (now == seen) atomicCAS(error, 0, TROUTE_ETIMEOUT);
            seen = now;
            t0 = clock64();
        }
        return *reinterpret_cast<volatile int*>(error) == 0;
    }
};

__device__ __forceinline__ unsigned ld_out(const unsigned* p) { return *reinterpret_cast<const volatile unsigned*>(p); }

// The outflow at p, waited for. In line for the shallow sweeps, which a call costs
// registers (2.7 M segments, 48 steps 2.60 -> 2.79 ms), and for deep paths of one or two
// steps a lane; a call where the deep paths' loading warps have many places to wait
// (144 steps: 55.0 -> 62.8 G segment-steps/s).
__device__ __noinline__ unsigned wait_on(LinBudget budget, const unsigned* p)
{
    unsigned v;
    do {
        __nanosleep(100);
        v = ld_out(p);
        if (v == kUnset && !budget.left()) v = 0;
    } while (v == kUnset);
    return v;
}

template <bool kCall>
__device__ __forceinline__ float wait_out(const LinRun& d, const unsigned* p)
{
    unsigned v = ld_out(p);
    if (v == kUnset) {
        LinBudget budget(d);
        if (kCall) {
            v = wait_on(budget, p);
        } else {
            do {
                __nanosleep(100);
                v = ld_out(p);
                if (v == kUnset && !budget.left()) v = 0;
            } while (v == kUnset);
        }
    }
    return __uint_as_float(v);
}

// What a lane has asked for of a segment.
template <int K>
struct LinData {
    float4 c;
    int idx, kind, up, n_up;
    float ql[K], q;
    unsigned un[K], up_prev;   // kind 3: the light path's outflow at the lane's steps and the one before
};

// Inflow of a reach with more than two upstream reaches: their outflows and the
// path's own (`own`), added in the network's order from 0.
template <bool kCall>
__device__ __forceinline__ float sum_many(const LinRun& d, int up, int n_up, int t, float own)
{
    float sum = 0.0f;
    for (int m = 0; m < n_up; ++m) {
        const int u = __ldg(d.ups + up + m);
        sum += u < 0 ? own : t < 0 ? __ldg(d.out0 + u) : wait_out<kCall>(d, d.out + (size_t)u * (size_t)d.Tp + t);
    }
    return sum;
}

__device__ __forceinline__ void store_out(unsigned* p, float v)
{
    const unsigned b = __float_as_uint(v);
    *reinterpret_cast<volatile unsigned*>(p) = b == kUnset ? 0x7fffffffu : b;
}

// Shallow paths: K steps per lane, C = 2^lc lanes per path, 32 / C paths per warp,
// a segment's loads issued one round before its use; many warps hide the rest.
template <int K>
__global__ void __launch_bounds__(128) lin_shallow_kernel(const LinRun d, int lc)
{
    const int lane = threadIdx.x & 31;
    const int C = 1 << lc, c = lane & (C - 1);
    while (true) {
        int w = 0;
        if (lane == 0) w = *reinterpret_cast<volatile int*>(d.error) ? d.n_items : atomicAdd(d.ticket, 1);
        w = __shfl_sync(kFull, w, 0);
        if (w >= d.n_items) return;
        const int2 item = __ldg(d.items + w);
        const int path = item.x + (lane >> lc);
        const bool has = (lane >> lc) < item.y;
        const int beg = has ? __ldg(d.path_ptr + path) : 0;
        const int n = has ? __ldg(d.path_ptr + path + 1) - beg : 0;
        const int n_max = __reduce_max_sync(kFull, n);
        for (int tb = 0; tb < d.T; tb += C * K) {
            const int lanes = min(C, (d.T - tb + K - 1) / K);   // that have steps
            const int t0 = tb + c * K, nk = min(K, d.T - t0);
            const bool live = has && c < lanes;
            LinData<K> x;
            int4 r0, r1;
            auto load_rec = [&](int k) {
                if (live && k >= 0 && k < n) {
                    const int4* r = reinterpret_cast<const int4*>(d.seg + beg + k);
                    r0 = __ldg(r);
                    r1 = __ldg(r + 1);
                }
            };
            auto load_data = [&](int k) {
                if (live && k >= 0 && k < n) {
                    x.c = make_float4(__int_as_float(r0.x), __int_as_float(r0.y), __int_as_float(r0.z), __int_as_float(r0.w));
                    x.idx = r1.x;
                    x.kind = r1.y;
                    x.up = r1.z;
                    x.n_up = r1.w;
                    const float* ql = d.qlat + (size_t)t0 * (size_t)d.S + r1.x;
#pragma unroll
                    for (int j = 0; j < K; ++j) x.ql[j] = j < nk ? __ldg(ql + (size_t)j * (size_t)d.S) : 0.0f;
                    if (c == 0) x.q = __ldcg(d.Q + r1.x);
                    if (r1.y == kTwo) {
                        const unsigned* u = d.out + (size_t)r1.z * (size_t)d.Tp + t0;
                        x.up_prev = t0 ? ld_out(u - 1) : __float_as_uint(__ldg(d.out0 + r1.z));
#pragma unroll
                        for (int j = 0; j < K; ++j) x.un[j] = j < nk ? ld_out(u + j) : 0u;
                    }
                }
            };
            load_rec(-c);
            load_data(-c);
            load_rec(1 - c);
            float o[K];              // the segment above: its discharge after each step
            float above_q = 0.0f;    // ... and before the lane's first
            float q_end = 0.0f;
#pragma unroll
            for (int j = 0; j < K; ++j) o[j] = 0.0f;
            const int rounds = n_max + lanes - 1;
            for (int i = 0; i < rounds; ++i) {
                if ((i & 63) == 63 && lane == 0) atomicAdd(d.progress, 1);
                const int k = i - c;
                float q = __shfl_up_sync(kFull, q_end, 1, C);
                if (live && k >= 0 && k < n) {
                    if (c == 0) q = x.q;
                    float po = above_q;
                    // (a headwater's first segment is the path's first: o and po are 0)
                    if (x.kind == kMany) {
                        po = sum_many<false>(d, x.up, x.n_up, t0 - 1, po);
#pragma unroll
                        for (int j = 0; j < K; ++j)
                            if (j < nk) o[j] = sum_many<false>(d, x.up, x.n_up, t0 + j, o[j]);
                    } else if (x.kind != kInner) {
                        // sums from +0, as written: 0 + own (+ light)
                        po = 0.0f + po;
#pragma unroll
                        for (int j = 0; j < K; ++j) o[j] = 0.0f + o[j];
                        if (x.kind == kTwo) {
                            const unsigned* u = d.out + (size_t)x.up * (size_t)d.Tp + t0;
                            po += t0 && x.up_prev == kUnset ? wait_out<false>(d, u - 1) : __uint_as_float(x.up_prev);
#pragma unroll
                            for (int j = 0; j < K; ++j)
                                if (j < nk) o[j] += x.un[j] == kUnset ? wait_out<false>(d, u + j) : __uint_as_float(x.un[j]);
                        }
                    }
                    above_q = q;
#pragma unroll
                    for (int j = 0; j < K; ++j) {
                        const float pn = o[j];
                        if (j < nk) {
                            q = x.c.x * pn + x.c.y * po + x.c.z * q + x.c.w * x.ql[j];
                            o[j] = q;
                        }
                        po = pn;
                    }
                    q_end = q;
                    if (c == lanes - 1) __stcg(d.Q + x.idx, q);
                    if (k == n - 1) {
                        unsigned* row = d.out + (size_t)path * (size_t)d.Tp + t0;
#pragma unroll
                        for (int j = 0; j < K; ++j)
                            if (j < nk) store_out(row + j, o[j]);
                    }
                }
                load_data(k + 1);
                load_rec(k + 2);
            }
            __syncwarp();   // the last lane's discharges, read by the first in the next block of steps
        }
    }
}

// Deep paths, one per block: a lone warp pays ~5 cycles for every instruction and
// over a thousand for a load, and the longest path is the run's critical path, so
// its rounds are stripped to the arithmetic. Warp 0 computes (K steps per lane,
// 32 lanes); the other warps keep a ring of W segments in shared memory filled
// with what a round needs: coefficients, inflow, and the light upstream outflow
// that is added to the segment's inflow: (own + z) + light, where z is -0 inside a
// reach (which changes nothing) and +0 at its head, and light is -0 where there is
// none. They also do the waiting for other paths.
template <int K, int W>
struct DeepRing {
    float ql[W][K][32], light[W][K][32], light_prev[W][32];
    float4 c[W];
    float z[W], q0[W];
    int idx[W], kind[W], up[W], n_up[W];
    volatile int full[W / 8];       // batch of 8 segments last written to each eighth, plus 1
    volatile int rounds;            // rounds computed (in eights)
    int item;
};

// The warp waits until *p >= want; false (for all its lanes) when the budget runs
// out or another warp failed. What was done before the flag was raised (behind a
// fence) is then done for the warp.
__device__ __forceinline__ bool wait_smem(const LinRun& d, const volatile int* p, int want)
{
    bool ok = true;
    if (*p < want) {
        LinBudget budget(d);
        while (ok && *p < want) {
            __nanosleep(20);
            ok = budget.left();
        }
    }
    __threadfence_block();
    return __all_sync(kFull, ok);
}

template <int K, int W, int NP>
__global__ void __launch_bounds__(32 * (NP + 1), 1) lin_deep_kernel(const LinRun d)
{
    constexpr bool kCall = K > 2;   // waiting for other paths
    static_assert(W % 8 == 0 && W >= 40 + 8, "a batch's slots are free 40 rounds after its segments were first used");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    DeepRing<K, W>& R = *reinterpret_cast<DeepRing<K, W>*>(smem_raw);
    const int c = threadIdx.x & 31, warp = threadIdx.x >> 5;
    while (true) {
        if (threadIdx.x == 0)
            R.item = *reinterpret_cast<volatile int*>(d.error) ? d.n_items : atomicAdd(d.ticket, 1);
        __syncthreads();
        const int w = R.item;
        if (w >= d.n_items) return;
        const int path = __ldg(&d.items[w].x), beg = __ldg(d.path_ptr + path), n = __ldg(d.path_ptr + path + 1) - beg;
        for (int tb = 0; tb < d.T; tb += 32 * K) {
            const int lanes = min(32, (d.T - tb + K - 1) / K);
            const int t0 = tb + c * K, nk = min(K, d.T - t0);   // (nk <= 0 from `lanes` on)
            __syncthreads();
            if (threadIdx.x < W / 8) R.full[threadIdx.x] = 0;
            if (threadIdx.x == 0) R.rounds = 0;
            __syncthreads();
            if (warp == 0) {
                float o[K], above_q = 0.0f, q_end = 0.0f;
#pragma unroll
                for (int j = 0; j < K; ++j) o[j] = 0.0f;
                const int rounds = n + lanes - 1;
                for (int i = 0; i < rounds; ++i) {
                    if ((i & 7) == 0) {
                        __syncwarp();
                        __threadfence_block();   // the rounds' reads, before their slots are filled again
                        if (c == 0) R.rounds = i;
                        if (i < n && !wait_smem(d, &R.full[(i >> 3) % (W / 8)], (i >> 3) + 1)) break;
                        if (c == 0 && (i & 63) == 0) atomicAdd(d.progress, 1);   // (arrives before the next fence)
                        __syncwarp();
                    }
                    const int k = i - c;
                    float q = __shfl_up_sync(kFull, q_end, 1);
                    if (k >= 0 && k < n && c < lanes) {
                        const int s = k % W;
                        const float4 cc = R.c[s];
                        const float z = R.z[s];
                        float ql[K];
#pragma unroll
                        for (int j = 0; j < K; ++j) ql[j] = R.ql[s][j][c];
                        if (c == 0) q = R.q0[s];
                        float po;
                        if (R.kind[s] == kMany) {
                            po = sum_many<kCall>(d, R.up[s], R.n_up[s], t0 - 1, above_q);
#pragma unroll
                            for (int j = 0; j < K; ++j)
                                if (j < nk) o[j] = sum_many<kCall>(d, R.up[s], R.n_up[s], t0 + j, o[j]);
                        } else {
                            po = (above_q + z) + R.light_prev[s][c];
#pragma unroll
                            for (int j = 0; j < K; ++j) o[j] = (o[j] + z) + R.light[s][j][c];
                        }
                        above_q = q;
#pragma unroll
                        for (int j = 0; j < K; ++j) {
                            const float pn = o[j];
                            if (j < nk) {
                                q = cc.x * pn + cc.y * po + cc.z * q + cc.w * ql[j];
                                o[j] = q;
                            }
                            po = pn;
                        }
                        q_end = q;
                        if (c == lanes - 1) __stcg(d.Q + R.idx[s], q);
                        if (k == n - 1) {
                            unsigned* row = d.out + (size_t)path * (size_t)d.Tp + t0;
#pragma unroll
                            for (int j = 0; j < K; ++j)
                                if (j < nk) store_out(row + j, o[j]);
                        }
                    }
                }
            } else {
                constexpr int U = K <= 2 ? 8 : K == 4 ? 4 : 2;   // segments whose loads are in flight together
                for (int b = warp - 1; b * 8 < n; b += NP) {
                    const int k0 = b * 8;
                    // the slots' last users: segments k0 - W .. k0 - W + 7, by lane 31 in round k0 - W + 38
                    if (k0 >= W && !wait_smem(d, &R.rounds, k0 - W + 39)) break;
                    int idx = 0, kind = kInner, up = 0;
                    if (c < 8 && k0 + c < n) {
                        const int s = (k0 + c) % W;
                        const int4* r = reinterpret_cast<const int4*>(d.seg + beg + k0 + c);
                        const int4 a = __ldg(r), e = __ldg(r + 1);
                        idx = e.x;
                        kind = e.y;
                        up = e.z;
                        R.q0[s] = __ldcg(d.Q + idx);
                        R.c[s] = make_float4(__int_as_float(a.x), __int_as_float(a.y), __int_as_float(a.z), __int_as_float(a.w));
                        R.z[s] = kind == kInner ? -0.0f : 0.0f;
                        R.idx[s] = idx;
                        R.kind[s] = kind;
                        R.up[s] = up;
                        R.n_up[s] = e.w;
                    }
#pragma unroll
                    for (int u0 = 0; u0 < 8; u0 += U) {
                        float ql[U][K];
                        unsigned un[U][K], prev[U];
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            const int si = __shfl_sync(kFull, idx, u0 + u), sk = __shfl_sync(kFull, kind, u0 + u);
                            const int su = __shfl_sync(kFull, up, u0 + u);
                            const bool in = k0 + u0 + u < n && c < lanes;
                            const unsigned* row = d.out + (size_t)su * (size_t)d.Tp + t0;
                            const bool light = in && sk == kTwo;
                            prev[u] = !light ? 0x80000000u : t0 ? ld_out(row - 1) : __float_as_uint(__ldg(d.out0 + su));
#pragma unroll
                            for (int j = 0; j < K; ++j) {
                                ql[u][j] = in && j < nk ? __ldg(d.qlat + (size_t)(t0 + j) * (size_t)d.S + si) : 0.0f;
                                un[u][j] = light && j < nk ? ld_out(row + j) : 0x80000000u;
                            }
                        }
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            const int su = __shfl_sync(kFull, up, u0 + u);
                            const int s = (k0 + u0 + u) % W;
                            if (k0 + u0 + u < n && c < lanes) {
                                // (only a light outflow can be unset: a value is never waited for elsewhere)
                                const unsigned* row = d.out + (size_t)su * (size_t)d.Tp + t0;
                                R.light_prev[s][c] = t0 && prev[u] == kUnset ? wait_out<kCall>(d, row - 1) : __uint_as_float(prev[u]);
#pragma unroll
                                for (int j = 0; j < K; ++j) {
                                    R.ql[s][j][c] = ql[u][j];
                                    R.light[s][j][c] = un[u][j] == kUnset ? wait_out<kCall>(d, row + j) : __uint_as_float(un[u][j]);
                                }
                            }
                        }
                    }
                    __syncwarp();
                    __threadfence_block();
                    if (c == 0) R.full[b % (W / 8)] = b + 1;
                }
            }
        }
    }
}

// out0 = discharge of each path's last segment before the launch.
__global__ void lin_init_kernel(LinRun d, int n_paths, float* out0)
{
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n_paths; p += gridDim.x * blockDim.x)
        out0[p] = d.Q[d.seg[d.path_ptr[p + 1] - 1].idx];
    if (blockIdx.x == 0 && threadIdx.x < 2) d.ticket[threadIdx.x] = 0;
    if (blockIdx.x == 0 && threadIdx.x == 2) *d.error = *d.progress = 0;
}

// Segment records in path order, one thread per reach: reach r's segments start at
// path_ptr[path[r]] + off[r]; ups: path of every upstream entry, -1 for the main one.
struct LinBuild {
    int R;
    const int *seg_start, *seg_len, *up_ptr, *up_idx, *main_up, *path, *off, *path_ptr;
    const float *c1, *c2, *c3, *c4;
    LinSeg* seg;
    int* ups;
};

__global__ void lin_build_kernel(LinBuild b)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < b.R; r += gridDim.x * blockDim.x) {
        const int u0 = b.up_ptr[r], nu = b.up_ptr[r + 1] - u0, m = b.main_up[r];
        int up = 0;
        for (int k = u0; k < u0 + nu; ++k) {
            const int u = b.up_idx[k], v = u == m ? -1 : b.path[u];
            b.ups[k] = v;
            if (v >= 0) up = v;
        }
        const int s0 = b.seg_start[r], n = b.seg_len[r];
        LinSeg* x = b.seg + b.path_ptr[b.path[r]] + b.off[r];
        for (int i = 0; i < n; ++i) {
            const int s = s0 + i;
            LinSeg y{b.c1[s], b.c2[s], b.c3[s], b.c4[s], s, kInner, 0, 0};
            if (i == 0) {
                y.kind = nu == 0 ? kHead : nu == 1 ? kOne : nu == 2 ? kTwo : kMany;
                y.up = nu > 2 ? u0 : up;
                y.n_up = nu;
            }
            x[i] = y;
        }
    }
}

template <typename T>
struct DArr {
    T* p = nullptr;
    size_t n = 0;
    int alloc(size_t count)
    {
        if (count <= n && p) return TROUTE_OK;
        release();
        const cudaError_t e = cudaMalloc(&p, std::max<size_t>(count, 1) * sizeof(T));
        if (e != cudaSuccess) return set_error(TROUTE_ENOMEM, "cudaMalloc: %s", cudaGetErrorString(e));
        n = count;
        return TROUTE_OK;
    }
    void release()
    {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
    ~DArr() { release(); }
};

int lin_cuda(cudaError_t e, const char* what)
{
    if (e == cudaSuccess) return TROUTE_OK;
    return set_error(e == cudaErrorMemoryAllocation ? TROUTE_ENOMEM : TROUTE_ECUDA, "%s: %s", what,
                     cudaGetErrorString(e));
}

}  // namespace
}  // namespace tr

using namespace tr;

struct troute_linear {
    int R = 0, n_paths = 0;
    long long S = 0;
    std::vector<int> depth_ptr;      // paths of each depth (shallow first)
    int deep_from = 0;               // first path that gets a warp of its own
    DArr<int> path_ptr, ups, ctr;    // ctr: two tickets, error, progress
    DArr<LinSeg> seg;
    DArr<float> out0;
    DArr<unsigned> out;
    DArr<int2> items[6];             // sweeps of 2^k shallow paths
    int n_items[6] = {};
    DArr<int2> deep;                 // sweeps of the deep paths
    int sms = 1;
    cudaStream_t stream = nullptr;
    ~troute_linear()
    {
        if (stream) cudaStreamDestroy(stream);
    }
};

// Paths at least this deep (reaches) get a block each: below it a path's rounds
// are few next to the lanes' skew.
#ifndef TROUTE_LIN_DEEP
#define TROUTE_LIN_DEEP 32
#endif
constexpr int kDeepPath = TROUTE_LIN_DEEP;

extern "C" int troute_linear_coeffs(const troute_chparams_f32* params, int n_segments, double dt, float* c1,
                                    float* c2, float* c3, float* c4oq)
{
    if (n_segments < 0 || !(dt > 0.0)) return set_error(TROUTE_EINVAL, "bad arguments");
    if (n_segments == 0) return TROUTE_OK;
    if (!params || !c1 || !c2 || !c3 || !c4oq) return set_error(TROUTE_EINVAL, "null array");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return set_error(TROUTE_ENODEV, "no CUDA device");
    DArr<troute_chparams_f32> p;
    DArr<float4> c;
    int rc;
    if ((rc = p.alloc(n_segments)) || (rc = c.alloc(n_segments))) return rc;
    if ((rc = lin_cuda(cudaMemcpy(p.p, params, (size_t)n_segments * sizeof *params, cudaMemcpyHostToDevice), "H2D")))
        return rc;
    lin_coeff_kernel<<<std::min(4096, (n_segments + 255) / 256), 256>>>(p.p, n_segments, (float)dt, c.p);
    std::vector<float4> h(n_segments);
    if ((rc = lin_cuda(cudaMemcpy(h.data(), c.p, (size_t)n_segments * sizeof(float4), cudaMemcpyDeviceToHost), "D2H")))
        return rc;
    for (int i = 0; i < n_segments; ++i) {
        c1[i] = h[i].x;
        c2[i] = h[i].y;
        c3[i] = h[i].z;
        c4oq[i] = h[i].w;
    }
    return TROUTE_OK;
}

// Paths and the segments in path order of a validated network.
static int lin_build(troute_linear* L, const troute_topo* topo, const float* c1, const float* c2, const float* c3,
                     const float* c4oq)
{
    const int R = L->R;
    const int* up = topo->reach_up_ptr;
    const int* ui = topo->reach_up_idx;
    // upstream-first order; per reach its depth, its deepest ("main") upstream
    // reach and the segments above it on its path
    std::vector<int> down(R, -1), left(R), order, depth(R, 1), main_up(R, -1), off(R, 0);
    order.reserve(R);
    for (int r = 0; r < R; ++r) {
        left[r] = up[r + 1] - up[r];
        for (int k = up[r]; k < up[r + 1]; ++k) down[ui[k]] = r;
        if (!left[r]) order.push_back(r);
    }
    for (size_t i = 0; i < order.size(); ++i) {
        const int r = order[i], d = down[r];
        for (int k = up[r]; k < up[r + 1]; ++k)
            if (main_up[r] < 0 || depth[ui[k]] + 1 > depth[r]) {
                depth[r] = depth[ui[k]] + 1;
                main_up[r] = ui[k];
            }
        if (main_up[r] >= 0) off[r] = off[main_up[r]] + topo->reach_seg_len[main_up[r]];
        if (d >= 0 && --left[d] == 0) order.push_back(d);
    }
    // a path ends at a reach that is not its downstream reach's main one; paths by
    // depth, within a depth in the caller's order
    auto ends = [&](int r) { return down[r] < 0 || main_up[down[r]] != r; };
    int deepest = 0;
    for (int r = 0; r < R; ++r) deepest = std::max(deepest, depth[r]);
    std::vector<int>& dp = L->depth_ptr;
    dp.assign(deepest + 2, 0);
    for (int r = 0; r < R; ++r)
        if (ends(r)) ++dp[depth[r] + 1];
    for (int k = 1; k <= deepest + 1; ++k) dp[k] += dp[k - 1];   // dp[k]: first path of depth k
    const int P = dp[deepest + 1];
    L->n_paths = P;
    std::vector<int> path(R), pos(dp.begin(), dp.end()), ptr(P + 1, 0);
    for (int r = 0; r < R; ++r)
        if (ends(r)) {
            path[r] = pos[depth[r]]++;
            ptr[path[r] + 1] = off[r] + topo->reach_seg_len[r];
        }
    for (int p = 0; p < P; ++p) ptr[p + 1] += ptr[p];
    for (size_t i = order.size(); i-- > 0;) {   // downstream first
        const int r = order[i];
        if (!ends(r)) path[r] = path[down[r]];
    }
    L->deep_from = deepest >= kDeepPath ? dp[kDeepPath] : P;
    std::vector<int2> deep;
    for (int p = L->deep_from; p < P; ++p) deep.push_back(int2{p, 1});
    const int nnz = R ? up[R] : 0;
    const long long S = L->S;
    DArr<int> d_start, d_len, d_up, d_ui, d_main, d_path, d_off;
    DArr<float> d_c[4];
    const float* cs[4] = {c1, c2, c3, c4oq};
    auto put = [](auto& arr, const auto* src, size_t n) {
        const int rc = arr.alloc(n);
        return rc || !n ? rc : lin_cuda(cudaMemcpy(arr.p, src, n * sizeof *src, cudaMemcpyHostToDevice), "upload");
    };
    int rc;
    if ((rc = put(d_start, topo->reach_seg_start, R)) || (rc = put(d_len, topo->reach_seg_len, R)) ||
        (rc = put(d_up, up, (size_t)R + 1)) || (rc = put(d_ui, ui, nnz)) || (rc = put(d_main, main_up.data(), R)) ||
        (rc = put(d_path, path.data(), R)) || (rc = put(d_off, off.data(), R)) ||
        (rc = put(L->path_ptr, ptr.data(), (size_t)P + 1)) || (rc = put(L->deep, deep.data(), deep.size())) ||
        (rc = L->seg.alloc((size_t)ptr[P])) || (rc = L->ups.alloc(nnz)) || (rc = L->out0.alloc(P)) || (rc = L->ctr.alloc(4)))
        return rc;
    for (int k = 0; k < 4; ++k)
        if ((rc = put(d_c[k], cs[k], (size_t)S))) return rc;
    if (R == 0) return TROUTE_OK;
    const LinBuild b{R, d_start.p, d_len.p, d_up.p, d_ui.p, d_main.p, d_path.p, d_off.p, L->path_ptr.p,
                     d_c[0].p, d_c[1].p, d_c[2].p, d_c[3].p, L->seg.p, L->ups.p};
    lin_build_kernel<<<std::min(4096, (R + 255) / 256), 256>>>(b);
    if ((rc = lin_cuda(cudaGetLastError(), "linear build launch"))) return rc;
    return lin_cuda(cudaStreamSynchronize(nullptr), "linear build");   // the inputs go out of scope
}

// The sweeps of 2^k shallow paths each, of one depth (a path may wait for a
// shallower one, never for one in its own warp). Copied on the stream of the kernel
// that reads them: a copy on the legacy stream may still be on its way then.
static int lin_items(troute_linear* L, int k, cudaStream_t st)
{
    if (L->items[k].p) return TROUTE_OK;
    std::vector<int2> v;
    const int w = 1 << k;
    try {
        for (size_t d = 0; d + 1 < L->depth_ptr.size(); ++d)
            for (int p = L->depth_ptr[d]; p < std::min(L->depth_ptr[d + 1], L->deep_from); p += w)
                v.push_back(int2{p, std::min(w, std::min(L->depth_ptr[d + 1], L->deep_from) - p)});
    } catch (const std::bad_alloc&) {
        return set_error(TROUTE_ENOMEM, "linear sweeps: host memory");
    }
    int rc = L->items[k].alloc(v.size());
    if (!rc && !v.empty())
        rc = lin_cuda(cudaMemcpyAsync(L->items[k].p, v.data(), v.size() * sizeof(int2), cudaMemcpyHostToDevice, st), "upload");
    if (rc) L->items[k].release();
    else L->n_items[k] = (int)v.size();
    return rc;
}

extern "C" int troute_linear_create(troute_linear** out, const troute_topo* topo, const float* c1, const float* c2,
                                    const float* c3, const float* c4oq)
{
    if (!out || !topo) return set_error(TROUTE_EINVAL, "null argument");
    *out = nullptr;
    int rc = troute_validate(topo);
    if (rc) return rc;
    const int R = topo->n_reaches;
    const long long S = topo->n_segments;
    for (int r = 0; r < R; ++r)
        if (topo->reach_seg_len[r] < 1)
            return set_error(TROUTE_ETOPO, "reach %d has no segments (the linear form needs at least one)", r);
    if (S > 0 && (!c1 || !c2 || !c3 || !c4oq)) return set_error(TROUTE_EINVAL, "null coefficient array");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return set_error(TROUTE_ENODEV, "no CUDA device");
    auto* L = new (std::nothrow) troute_linear();
    if (!L) return set_error(TROUTE_ENOMEM, "handle");
    L->R = R;
    L->S = S;
    try {
        rc = lin_build(L, topo, c1, c2, c3, c4oq);
    } catch (const std::bad_alloc&) {
        rc = set_error(TROUTE_ENOMEM, "linear network: host memory");
    }
    if (!rc) rc = lin_cuda(cudaStreamCreateWithFlags(&L->stream, cudaStreamNonBlocking), "stream");
    if (rc) {
        delete L;
        return rc;
    }
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&L->sms, cudaDevAttrMultiProcessorCount, dev);
    *out = L;
    return TROUTE_OK;
}

extern "C" int troute_linear_destroy(troute_linear* L)
{
    delete L;
    return TROUTE_OK;
}

// Steps per launch: the paths' outflows (4 B per path and step) within a quarter
// of the free memory, at most 1024.
static int lin_chunk(const troute_linear* L, int n_ts)
{
    const int most = std::min(n_ts, 1024);
    if ((size_t)L->n_paths * (size_t)((most + 7) / 8 * 8) <= L->out.n) return most;
    size_t fr = 0, tot = 0;
    if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) fr = (size_t)4 << 30;
    const long long fit = (long long)((double)(fr / 4) / (4.0 * std::max(1, L->n_paths))) / 8 * 8;
    return (int)std::max<long long>(1, std::min<long long>(most, std::max<long long>(fit, 8)));
}

template <int K, int W, int NP>
static int lin_launch_deep(const LinRun& d, int sms, cudaStream_t st)
{
    if (d.n_items == 0) return TROUTE_OK;
    const auto kernel = lin_deep_kernel<K, W, NP>;
    const size_t smem = sizeof(DeepRing<K, W>);
    int bps = 0, rc;
    if ((rc = lin_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "smem attribute")) ||
        (rc = lin_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kernel, 32 * (NP + 1), smem), "occupancy")))
        return rc;
    kernel<<<std::min(sms * std::max(1, bps), d.n_items), 32 * (NP + 1), smem, st>>>(d);
    return lin_cuda(cudaGetLastError(), "linear launch");
}

extern "C" int troute_linear_run_device(troute_linear* L, const float* qlat_dev, int n_ts, float* q_dev,
                                        long long wait_cycles, void* stream)
{
    if (!L) return set_error(TROUTE_EINVAL, "null handle");
    if (n_ts < 0) return set_error(TROUTE_EINVAL, "n_ts < 0");
    if (n_ts == 0 || L->R == 0) return TROUTE_OK;
    if (!qlat_dev || !q_dev) return set_error(TROUTE_EINVAL, "null device array");
    const cudaStream_t st = stream ? (cudaStream_t)stream : L->stream;
    const int chunk = lin_chunk(L, n_ts);
    int rc;
    if ((rc = L->out.alloc((size_t)L->n_paths * (size_t)((chunk + 7) / 8 * 8)))) return rc;
    int err = 0;
    for (int t0 = 0; t0 < n_ts && !err; t0 += chunk) {
        LinRun d;
        d.S = L->S;
        d.T = std::min(chunk, n_ts - t0);
        d.Tp = (d.T + 7) / 8 * 8;
        d.path_ptr = L->path_ptr.p;
        d.seg = L->seg.p;
        d.ups = L->ups.p;
        d.out0 = L->out0.p;
        d.out = L->out.p;
        d.Q = q_dev;
        d.qlat = qlat_dev + (size_t)t0 * (size_t)L->S;
        d.error = L->ctr.p + 2;
        d.progress = L->ctr.p + 3;
        d.wait_cycles = wait_cycles > 0 ? wait_cycles : 8000000000LL;
        d.ticket = L->ctr.p;
        // shallow paths: 8 steps per lane, up to 8 lanes each
        int lc = 0;
        while (lc < 3 && (8 << lc) < d.T) ++lc;
        if ((rc = lin_items(L, 5 - lc, st))) return rc;
        d.items = L->items[5 - lc].p;
        d.n_items = L->n_items[5 - lc];
        if ((rc = lin_cuda(cudaMemsetAsync(L->out.p, 0xff, (size_t)L->n_paths * (size_t)d.Tp * sizeof(unsigned), st),
                           "linear set-up")))
            return rc;
        lin_init_kernel<<<std::min<int>(4096, (L->n_paths + 255) / 256), 256, 0, st>>>(d, L->n_paths, L->out0.p);
        if (d.n_items > 0) {
            int bps = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, lin_shallow_kernel<8>, 128, 0);
            lin_shallow_kernel<8><<<std::min(L->sms * std::max(1, bps), (d.n_items + 3) / 4), 128, 0, st>>>(d, lc);
        }
        // deep paths: a block each, the fewest steps per lane that 32 lanes cover
        d.items = L->deep.p;
        d.n_items = L->n_paths - L->deep_from;
        d.ticket = L->ctr.p + 1;
        rc = d.T <= 32 ? lin_launch_deep<1, 128, 7>(d, L->sms, st)
             : d.T <= 64 ? lin_launch_deep<2, 128, 7>(d, L->sms, st)
             : d.T <= 128 ? lin_launch_deep<4, 64, 3>(d, L->sms, st)
                          : lin_launch_deep<8, 64, 3>(d, L->sms, st);
        if (rc) return rc;
        if ((rc = lin_cuda(cudaGetLastError(), "linear launch")) ||
            (rc = lin_cuda(cudaMemcpyAsync(&err, d.error, sizeof err, cudaMemcpyDeviceToHost, st), "status")) ||
            (rc = lin_cuda(cudaStreamSynchronize(st), "linear run")))
            return rc;
    }
    if (err == TROUTE_ETIMEOUT) return set_error(TROUTE_ETIMEOUT, "linear routing: a device wait ran out");
    if (err) return set_error(err, "linear routing: device reported error %d", err);
    return TROUTE_OK;
}

extern "C" int troute_linear_route(const troute_topo* topo, const float* c1, const float* c2, const float* c3,
                                   const float* c4oq, const float* qlat_ts, const float* q0, int n_ts, float* q_out)
{
    if (!topo || n_ts < 0) return set_error(TROUTE_EINVAL, "bad arguments");
    const long long S = topo->n_segments;
    if (S > 0 && (!q0 || !q_out || (n_ts > 0 && !qlat_ts))) return set_error(TROUTE_EINVAL, "null array");
    troute_linear* L = nullptr;
    int rc = troute_linear_create(&L, topo, c1, c2, c3, c4oq);
    if (rc) return rc;
    DArr<float> q, ql;
    if ((rc = q.alloc(S)) || (rc = ql.alloc((size_t)n_ts * S)) ||
        (rc = lin_cuda(cudaMemcpyAsync(q.p, q0, S * sizeof(float), cudaMemcpyHostToDevice, L->stream), "H2D")) ||
        (rc = lin_cuda(cudaMemcpyAsync(ql.p, qlat_ts, (size_t)n_ts * S * sizeof(float), cudaMemcpyHostToDevice, L->stream), "H2D")) ||
        (rc = troute_linear_run_device(L, ql.p, n_ts, q.p, 0, nullptr)) ||
        (rc = lin_cuda(cudaMemcpyAsync(q_out, q.p, S * sizeof(float), cudaMemcpyDeviceToHost, L->stream), "D2H")) ||
        (rc = lin_cuda(cudaStreamSynchronize(L->stream), "D2H"))) {
        troute_linear_destroy(L);
        return rc;
    }
    troute_linear_destroy(L);
    return TROUTE_OK;
}
