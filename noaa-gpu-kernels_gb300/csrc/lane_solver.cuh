// Per-lane secant solver shared by the persistent routing kernels that give
// every lane its own (reach, step): the lane state, the start of a segment
// solve and one "pass" (one depth evaluation plus its secant bookkeeping).
//
// A pass does, for every lane in SOLVE or VEL mode, exactly one evaluation of
// R^fl(2/3) and R^fl(5/3) (pow23_53), so the expensive part of the pass runs
// for all busy lanes of a warp together.
// The evaluation is at h_0 when a solve starts or restarts (need0), otherwise
// at h followed by the secant update and the stop test.
// When a solve stops, the segment's discharge and depth are stored and the next
// segment starts in the same pass; after the reach's last segment the lane goes
// to DONE and the kernel publishes the reach. The velocity, an output that no
// later solve reads, is computed once per run from the final depth
// (velocity_kernel), with the reference's formula (troute_mc_final.cu:132-136).
// The arithmetic is mc_solve's (mc_solve.cuh, the reference's
// troute_mc_final.cu:42-139) split at its evaluations, operation for
// operation.
#pragma once

#include "device_common.cuh"

namespace tr {

// L_BEGIN: the lane's next segment (L.i) starts at the kernel's one
// begin_segment call site before the next evaluation pass; L_START: the lane
// holds an item (L.ri, L.tau) whose inputs are final, started at the kernel's
// one start_item call site. Modes from L_SOLVE up count as busy.
enum : int { L_IDLE = 0, L_WAIT = 1, L_SOLVE = 2, L_BEGIN = 3, L_DONE = 4, L_START = 5 };

// A lane's current segment parameters live in shared memory for the whole
// solve, read by every pass. (Re-reading them from global memory every pass
// misses L2 once a network's parameters outgrow it -- c1's are 260 MB -- and
// costs a DRAM round trip per pass.) Each lane has two buffers: while segment
// i is solved, segment i + 1's parameters, inflow column and scale, discharge,
// depth and (warm start) learned starting depth are copied into the other one by
// cp.async, and one pass later, with the column at hand, its inflow -- all static
// during the launch or final since the reach's previous step completed -- so the
// next solve starts without a global load. Buffer of segment i: i & 1. Its planes,
// in double2: parameters; {inflow scale, inflow column | flags}; the aligned pairs
// of discharge and depth that hold the slot's; {inflow, learned depth}.
// Layout [warp][buffer][plane][lane]: a warp's reads of one plane are 512
// contiguous bytes, free of bank conflicts, whatever the block size.
constexpr int kSegSmemStride = 32;
constexpr int kTailPlane = kParamPlanes, kQPlane = kParamPlanes + 1, kDPlane = kParamPlanes + 2, kInPlane = kParamPlanes + 3;
constexpr int kSegBufPlanes = kParamPlanes + 4;
constexpr int kSegBufStride = kSegBufPlanes * kSegSmemStride;   // double2 from buffer 0 to 1
// double2 of a block's staging array per thread
constexpr int kSegSmemPerThread = 2 * kSegBufPlanes;

// This thread's buffer 0 in a block's array of kSegSmemPerThread x blockDim
// double2.
__device__ __forceinline__ double2* seg_slot_of(double2* seg_sm)
{
    return seg_sm + (threadIdx.x >> 5) * (2 * kSegBufStride) + (threadIdx.x & 31);
}

// The buffer of the lane's segment i.
__device__ __forceinline__ double2* seg_buf(double2* slot, int i) { return slot + (i & 1) * kSegBufStride; }

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// Asynchronous global -> shared copies of this thread; a thread waits only for
// its own (cp.async.wait_all).
__device__ __forceinline__ void cp_async16(void* dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Starts the copies of tile slot s's record, discharge and depth (and learned
// depth for step tau) into buffer buf. The discharge and depth, which other steps
// of the launch write, are copied past L1 (cp.async.cg, whose 16 bytes are the
// pair around the slot: the neighbour's value may be in flux and is not used).
__device__ __forceinline__ void stage_seg_async(const NetDev& net, const RunDev& run, int tau, long long s,
                                                double2* buf)
{
    const SegRec* r = net.seg + s;
#pragma unroll
    for (int k = 0; k < kParamPlanes; ++k) cp_async16(buf + k * kSegSmemStride, r->p + k);
    cp_async16(buf + kTailPlane * kSegSmemStride, &r->qscale);
    cp_async16(buf + kQPlane * kSegSmemStride, net.q + (s & ~1ll));
    cp_async16(buf + kDPlane * kSegSmemStride, net.d + (s & ~1ll));
    if (run.warm) cp_async4(&buf[kInPlane * kSegSmemStride].y, run.start_pred + (size_t)tau * (size_t)net.n_seg_int + s);
}

// Starts the copy of the inflow of column col at step tau into buffer buf.
__device__ __forceinline__ void stage_inflow_async(const RunDev& run, int tau, int col, double2* buf)
{
    cp_async8(&buf[kInPlane * kSegSmemStride].x, run.qlat + (size_t)tau * (size_t)run.qlat_ld + col);
}

__device__ __forceinline__ SegP staged_seg(const double2* slot)
{
    const double2 a = slot[0], b = slot[kSegSmemStride], c = slot[2 * kSegSmemStride];
    const double2 e = slot[3 * kSegSmemStride], f = slot[4 * kSegSmemStride], g = slot[5 * kSegSmemStride];
    SegP p;
    p.dx = a.x; p.bw = a.y; p.twcc = b.x; p.n_ch = b.y; p.ncc = c.x; p.s0 = c.y;
    p.z = e.x; p.bfd = e.y; p.sq_s0 = f.x; p.sq2 = f.y; p.ck_fac = g.x; p.z2 = g.y;
    return p;
}
// Warm-start phase of a solve: the plain bracket, or bracketing the learned
// depth (read from the launch's prediction plane when the solve begins).
enum : int { W_PLAIN = 0, W_ACTIVE = 2 };

// Inflow of the segment to begin next: its column not yet known to have arrived,
// or the copy under way (or done).
enum : int { kInflowLater = 0, kInflowStaged = 1 };

// Everything a lane carries for one (reach, step) and the segment it solves.
struct Lane {
    int mode;
    int ri, tau, g, ns, i, ub, ue, dn;
    int n_up, dn_n_up;     // upstream reaches of this reach and of the one downstream
    int inflow;            // of the next segment (of this one when it begins): kInflow*
    long long base;        // tile slot of segment 0
    long long wait_t0;
    unsigned long long wait_tail;  // queue tail seen when the current wait budget began
    double qup_head, quc_head, q_up_old, q_up_new, q_last;
    // current segment
    long long s;
    double qup, quc, qdp, qldt;   // qldt = ql dt
    double h, h_0, Qj_0, qdc;
    double dpp;            // previous depth (clamped at 0): the plain bracket's centre
    DepthEval e0;
    int need0, iter, attempt, maxiter, total, retried, warm;
    bool irregular;        // outside the ranges of the short arithmetic (mc_solve.cuh)
    bool ahead;            // qmc0_n and Qj0_n hold the next pass's lower discharge and residual (narrow_pass.cuh)
    double qmc0_n, Qj0_n;
};

// A solve's first attempt from the bracket [h_0, h].
__device__ __forceinline__ void restart_bracket(Lane& L, const Tol& tol, double h, double h_0)
{
    L.h = h;
    L.h_0 = h_0;
    L.Qj_0 = 0.0;
    L.qdc = 0.0;
    L.maxiter = tol.maxiter;
    L.attempt = 0;
    L.iter = 0;
    L.need0 = 1;
    L.ahead = false;
}

// The plain starting bracket from the previous depth (troute_mc_final.cu:193).
__device__ __forceinline__ void plain_bracket(Lane& L, const Tol& tol)
{
    restart_bracket(L, tol, L.dpp * 1.33 + kMinDepth, L.dpp * 0.67);
}

// Starts the copy of the next segment's inflow once its column has arrived (a
// pass after the segment's other values were asked for).
__device__ __forceinline__ void stage_next_inflow(Lane& L, const RunDev& run, double2* slot)
{
    if (L.inflow == kInflowLater && L.i + 1 < L.ns) {
        cp_async_wait_all();
        double2* const buf = seg_buf(slot, L.i + 1);
        stage_inflow_async(run, L.tau, __double2loint(buf[kTailPlane * kSegSmemStride].y), buf);
        L.inflow = kInflowStaged;
    }
}

// Starts segment L.i of the lane's reach, staged by the caller (segment 0) or while
// the previous one was solved; consecutive segments that exit early (invalid
// parameters or no flow at all, troute_mc_final.cu:54-63) are stored right away.
// Returns true when a secant solve is pending, false when the reach is complete.
__device__ __forceinline__ bool begin_segment(Lane& L, const NetDev& net, const RunDev& run,
                                              LocalStats& ls, unsigned int* hist_s, double2* slot)
{
    while (L.i < L.ns) {
        L.s = L.base + (long long)L.i * kLanes;
        double2* const buf = seg_buf(slot, L.i);
        cp_async_wait_all();
        if (L.i + 1 < L.ns) stage_seg_async(net, run, L.tau, L.s + kLanes, seg_buf(slot, L.i + 1));
        const double2 tail = buf[kTailPlane * kSegSmemStride], in = buf[kInPlane * kSegSmemStride];
        const double2 q2 = buf[kQPlane * kSegSmemStride], d2 = buf[kDPlane * kSegSmemStride];
        L.qdp = (L.s & 1) ? q2.y : q2.x;
        const double dpp = (L.s & 1) ? d2.y : d2.x;
        double ql = L.inflow == kInflowStaged
                        ? in.x
                        : __ldg(run.qlat + (size_t)L.tau * (size_t)run.qlat_ld + __double2loint(tail.y));
        if (dbits(tail.x) != 0x3ff0000000000000ll) ql = ql * tail.x;   // a scale of 1 changes nothing
        L.inflow = kInflowLater;
        L.qup = (L.i == 0) ? L.qup_head : L.q_up_old;
        L.quc = (L.i == 0) ? L.quc_head : L.q_up_new;
        if (exits_early(staged_seg(buf), ql, L.qup, L.quc, L.qdp)) {
            __stcg(net.q + L.s, 0.0);
            __stcg(net.d + L.s, 0.0);
            __stcg(net.v + L.s, 0.0);
            if (run.q_hist) __stcg(run.q_hist + (size_t)L.tau * (size_t)net.n_seg_int + L.s, 0.0);
            L.q_up_old = L.qdp;
            L.q_up_new = 0.0;
            L.q_last = 0.0;
            SolveOut o;
            o.iters = 0;
            o.retried = 0;
            o.early = 1;
            count_solve(ls, hist_s, o);
            ++L.i;
            continue;
        }
        L.qldt = ql * run.dt;
        L.irregular = !((__double2hiint(tail.y) & 1) && run.dt_regular && flow_regular(L.qup) && flow_regular(L.quc) &&
                        flow_regular(L.qdp) && flow_regular(L.qldt));
        L.dpp = fp_max0(dpp);
        L.total = 0;
        L.retried = 0;
        // the learned starting depth of this solve, predicted before the launch: the
        // bracket [p (1 - delta), p (1 + delta)] around a positive normal float p
        // below 1e4 m (0x461c4000), else the plain bracket
        const unsigned pb = run.warm ? (unsigned)__double2loint(in.y) : 0u;
        if (pb >= 0x00800000u && pb < 0x461c4000u) {
            const double pr = __longlong_as_double(((long long)((pb >> 23) + 896) << 52) |
                                                   ((long long)(pb & 0x7fffff) << 29));  // exact widening
            restart_bracket(L, run.tol, pr * run.warm_hi, pr * run.warm_lo);
            L.warm = W_ACTIVE;
            ls.warm_used++;
            if (run.start_hist) __stcg(run.start_hist + (size_t)L.tau * (size_t)net.n_seg_int + L.s, pr);
        } else {
            plain_bracket(L, run.tol);
            L.warm = W_PLAIN;
        }
        return true;
    }
    return false;
}

// Books one secant iteration of a lane whose pass produced o and (already in
// L.e0) the upper depth's evaluation: the bracket and the stop test. Returns true
// when the solve is done (L.qdc, L.h).
__device__ __forceinline__ bool lane_book(Lane& L, const PassOut& o, const RunDev& run, LocalStats& ls)
{
    const Tol& tol = run.tol;
    L.Qj_0 = o.Qj_0;
    L.qdc = o.qdc;
    const double h = L.h;
    const bool more = secant_more(h, o.h_1, tol);
    L.h_0 = fp_max0(h);
    L.h = fp_max0(o.h_1);
    ++L.iter;
    ++L.total;
    bool stop;
    if (L.warm == W_ACTIVE) {
        // warm phase: accepted once the stop test passes at a depth of at
        // least kMinDepth; otherwise, after warm_k passes (or below
        // kMinDepth), the plain solve restarts from the previous depth
        const bool below_min = fp_lt_pos(L.h, kMinDepth);
        stop = !more && !below_min;
        if (!stop && (below_min || L.iter >= run.warm_k)) {
            L.warm = W_PLAIN;
            ls.warm_fallback++;
            plain_bracket(L, tol);
        }
    } else {
        stop = fp_lt_pos(L.h, kMinDepth) || !(more && L.iter <= L.maxiter);
    }
    if (!stop) return false;
    if (L.warm == W_PLAIN && L.iter >= L.maxiter) {
        // widen the bracket (also after the last attempt, as the reference does)
        L.h *= 1.33;
        L.h_0 *= 0.67;
        L.maxiter += 25;
        L.retried = 1;
        if (++L.attempt < tol.attempts) {
            L.iter = 0;
            L.need0 = 1;
            L.ahead = false;
            return false;
        }
    }
    return true;
}

// Books an iteration; at a stop stores the segment (its velocity is derived from
// the final depth once the run is over, see velocity_kernel) and moves on to the
// next one.
__device__ __forceinline__ void lane_finish(Lane& L, const PassOut& o, const NetDev& net, const RunDev& run,
                                            LocalStats& ls, unsigned int* hist_s, double2* slot)
{
    if (!lane_book(L, o, run, ls)) return;
    __stcg(net.q + L.s, L.qdc);
    __stcg(net.d + L.s, L.h);
    if (run.q_hist) __stcg(run.q_hist + (size_t)L.tau * (size_t)net.n_seg_int + L.s, L.qdc);
    if (run.pairs) {
        float* pr = run.pairs + ((size_t)L.tau * (size_t)net.n_seg_int + L.s) * 9;
        pr[0] = (float)L.qup;
        pr[1] = (float)L.quc;
        pr[2] = (float)L.qdp;
        const SegP p = staged_seg(seg_buf(slot, L.i));
        const double2 tail = seg_buf(slot, L.i)[kTailPlane * kSegSmemStride];
        pr[3] = (float)(__ldg(run.qlat + (size_t)L.tau * (size_t)run.qlat_ld + __double2loint(tail.y)) * tail.x);
        pr[4] = (float)p.dx;
        pr[5] = (float)p.s0;
        pr[6] = (float)p.n_ch;
        pr[7] = (float)p.bw;
        pr[8] = (float)L.h;
    }
    L.q_up_old = L.qdp;
    L.q_up_new = L.qdc;
    L.q_last = L.qdc;
    SolveOut so;
    so.iters = L.total;
    so.retried = L.retried;
    so.early = 0;
    count_solve(ls, hist_s, so);
    ++L.i;
    L.mode = L.i < L.ns ? L_BEGIN : L_DONE;
}

// One evaluation pass of a lane in SOLVE mode (no-op otherwise).
__device__ __forceinline__ bool lane_eval(Lane& L, const RunDev& run, double2* slot, PassOut& o)
{
    const SegP p = staged_seg(seg_buf(slot, L.i));
    const PassFlow f = {L.qup, L.quc, L.qdp, L.qldt, run.dt, run.dt_half};
    DepthEval e;
    secant_pass(p, f, L.need0 ? L.h_0 : L.h, L.need0, L.h, L.h_0, L.Qj_0, L.e0, L.irregular, e, o);
    L.e0 = e;
    L.ahead = false;
    const bool iterated = !L.need0;
    L.need0 = 0;
    return iterated;
}

__device__ __forceinline__ void lane_pass(Lane& L, const NetDev& net, const RunDev& run, LocalStats& ls,
                                          unsigned int* hist_s, double2* slot)
{
    if (L.mode == L_SOLVE) {
        PassOut o;
        if (lane_eval(L, run, slot, o)) lane_finish(L, o, net, run, ls, hist_s, slot);
    }
}

}  // namespace tr
