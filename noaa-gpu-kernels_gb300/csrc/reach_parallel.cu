// Reach-parallel single step: the drop-in for kernel_mc_gpu / cpu_mc
// (troute_mc_final.cu:141-164, :167-252). Independent reaches, a reach's segments
// in sequence, the first segment's current inflow seeded by uq; parameters in the
// caller's AoS layout.
//
// The FP64 pipe bounds it, so the work is arranged to keep a warp's FP64
// instructions full of lanes. Each lane routes a reach of its own and takes the
// next one of its block's share when it is done (one thread per reach left a warp
// running until its longest reach and slowest solve had ended: 2.7 M segments in
// 1.1 M reaches at rtol 1e-8 took 82.1 ms). All lanes share one pass per loop
// (mc_solve.cuh; narrow_pass.cuh where a warp holds at most four).
// A segment's derived values (divisions and square roots, ~55 FP64 instructions)
// and the velocity of the one before it (~65) are not formed when the lane gets
// there -- about four of 32 lanes do in every pass, and each would make the whole
// warp pay -- but for many lanes together: a lane has two buffers in shared
// memory, and once 16 lanes lack their next segment (or one has nothing left to
// solve) the warp forms the velocity of the segment that used each free buffer
// and prepares the next segment in it. All a segment needs beforehand is known
// but its current inflow.
#include "narrow_pass.cuh"

namespace tr {

namespace {
constexpr unsigned kAll = 0xffffffffu;
constexpr int kReachThreads = 128;
constexpr int kBatchLanes = 16;   // lanes lacking a next segment that start a preparation
constexpr int kRunLen = 16;       // consecutive reaches of a share of many

// Planes after the parameters (lane_solver.cuh's buffer layout): {previous
// discharge, upstream previous discharge}, {ql dt, previous depth}, {depth found,
// segment | flags}.
constexpr int kFlowPlane = kParamPlanes, kStartPlane = kParamPlanes + 1, kSegPlane = kParamPlanes + 2;
enum : int { kFirst = 1, kInvalid = 2, kNoFlow = 4, kRegular = 8 };

struct ReachArgs {
    const troute_chparams* p;
    const double *ql, *qu, *qd, *dp;
    const int *rs, *rl;
    double *qo, *vo, *dpo;
    double uq;
    int nr, n_segments, lanes;   // lanes: per warp that take reaches
    int run_len;                 // consecutive reaches of a block's share
    RunDev run;                  // dt, dt_half, tol, stats
};

// Derived values of segment s and its known flows into buffer buf.
__device__ __forceinline__ void prepare_segment(const ReachArgs& a, int s, bool first, double2* buf)
{
    const double* c = reinterpret_cast<const double*>(a.p + s);   // 8-byte loads: the caller's alignment
    const troute_chparams raw = {__ldg(c), __ldg(c + 1), __ldg(c + 2), __ldg(c + 3),
                                 __ldg(c + 4), __ldg(c + 5), __ldg(c + 6), __ldg(c + 7)};
    const double ql = __ldg(a.ql + s), qu = __ldg(a.qu + s), qd = __ldg(a.qd + s), dp = __ldg(a.dp + s);
    const SegP p = derive_seg(raw);
    const double qldt = ql * a.run.dt;
    int flags = first ? kFirst : 0;
    if (fp_le0(p.n_ch) || fp_le0(p.s0) || fp_le0(p.z) || fp_le0(p.bw)) flags |= kInvalid;
    if (fp_le0(ql) && fp_le0(qu) && fp_le0(qd)) flags |= kNoFlow;
    if (seg_regular(p) && value_regular(a.run.dt) && flow_regular(qu) && flow_regular(qd) && flow_regular(qldt))
        flags |= kRegular;
    buf[0] = make_double2(p.dx, p.bw);
    buf[kSegSmemStride] = make_double2(p.twcc, p.n_ch);
    buf[2 * kSegSmemStride] = make_double2(p.ncc, p.s0);
    buf[3 * kSegSmemStride] = make_double2(p.z, p.bfd);
    buf[4 * kSegSmemStride] = make_double2(p.sq_s0, p.sq2);
    buf[5 * kSegSmemStride] = make_double2(p.ck_fac, p.z2);
    buf[kFlowPlane * kSegSmemStride] = make_double2(qd, qu);
    buf[kStartPlane * kSegSmemStride] = make_double2(qldt, fp_max0(dp));
    buf[kSegPlane * kSegSmemStride].y = __hiloint2double(flags, s);
}
}  // namespace

__global__ void __launch_bounds__(kReachThreads, 3) reach_parallel_kernel(const ReachArgs a)
{
    __shared__ unsigned int hist_s[16];
    __shared__ int taken;   // reaches of the block's share handed out
    __shared__ double2 seg_sm[kSegSmemPerThread * kReachThreads];
    double2* const slot = seg_slot_of(seg_sm);
    const int lane = threadIdx.x & 31;
    double2* const warp_seg = slot - lane;
    if (threadIdx.x < 16) hist_s[threadIdx.x] = 0;
    if (threadIdx.x == 0) taken = 0;
    __syncthreads();
    LocalStats ls = {0, 0, 0, 0, 0, 0};
    Lane L;
    L.mode = L_IDLE;
    L.i = 0;                     // the buffer of the segment being solved
    L.warm = W_PLAIN;
    int next = 0, left = 0;      // segments of the lane's reach that are not prepared yet
    bool first = false;          // `next` is its reach's first
    bool more = lane < a.lanes;  // there may be another reach to take
    bool ready = false;          // buffer 1 - L.i holds the next segment
    int owed = 0;                // bit b: buffer b holds a solved segment without its velocity
    double quc = 0.0;            // discharge of the segment before

    while (true) {
        // ---- prepare next segments (and the velocities their buffers owe) ----
        const bool lacks = !ready && (left > 0 || more || owed);
        const unsigned lacking = __ballot_sync(kAll, lacks);
        if (__popc(lacking) >= kBatchLanes || __any_sync(kAll, lacks && L.mode == L_IDLE)) {
            const int spare = 1 - L.i;
            // the buffer whose velocity is formed: the spare one, or at the end the other
            const int b = (owed >> spare) & 1 ? spare : L.i;
            if (lacks && ((owed >> b) & 1) && (b == spare || (L.mode == L_IDLE && left == 0 && !more))) {
                double2* const buf = seg_buf(slot, b);
                const double2 t = buf[kSegPlane * kSegSmemStride];
                a.vo[__double2loint(t.y)] = seg_velocity(staged_seg(buf), t.x);
                owed &= ~(1 << b);
            }
            const bool take = lacks && left == 0 && more;
            const unsigned taking = __ballot_sync(kAll, take);
            if (taking) {
                int k = 0;
                if (lane == 0) k = atomicAdd(&taken, __popc(taking));
                k = __shfl_sync(kAll, k, 0) + __popc(taking & ((1u << lane) - 1u));
                if (take) {
                    const int run = k / a.run_len;
                    const long long at = ((long long)run * gridDim.x + blockIdx.x) * a.run_len + (k - run * a.run_len);
                    more = at < a.nr;
                    if (more) {
                        const int r = (int)at, start = a.rs[r], ns = a.rl[r];
                        if (start < 0 || ns < 0 || (long long)start + ns > (long long)a.n_segments) {
                            record_error(a.run.stats, TROUTE_EINVAL, r, 0, 4);
                        } else {
                            next = start;
                            left = ns;
                            first = true;
                        }
                    }
                }
            }
            if (lacks && left > 0) {
                prepare_segment(a, next, first, seg_buf(slot, spare));
                ++next;
                --left;
                first = false;
                ready = true;
            }
        }

        // ---- idle lanes begin their next segment ----
        if (L.mode == L_IDLE && ready) {
            L.i = 1 - L.i;
            ready = false;
            const double2* const buf = seg_buf(slot, L.i);
            const double2 fl = buf[kFlowPlane * kSegSmemStride], st = buf[kStartPlane * kSegSmemStride];
            const int flags = __double2hiint(buf[kSegPlane * kSegSmemStride].y);
            L.s = __double2loint(buf[kSegPlane * kSegSmemStride].y);
            if (flags & kFirst) quc = a.uq;
            if ((flags & kInvalid) || ((flags & kNoFlow) && fp_le0(quc))) {
                a.qo[L.s] = 0.0;
                a.vo[L.s] = 0.0;
                a.dpo[L.s] = 0.0;
                quc = 0.0;
                SolveOut o;
                o.iters = 0;
                o.retried = 0;
                o.early = 1;
                count_solve(ls, hist_s, o);
            } else {
                L.qup = fl.y;
                L.quc = quc;
                L.qdp = fl.x;
                L.qldt = st.x;
                L.dpp = st.y;
                L.irregular = !((flags & kRegular) && flow_regular(quc));
                L.total = 0;
                L.retried = 0;
                plain_bracket(L, a.run.tol);
                L.mode = L_SOLVE;
            }
        }

        // ---- one pass ----
        const unsigned smask = __ballot_sync(kAll, L.mode == L_SOLVE);
        if (smask) {
            PassOut o;
            bool iterated = false;
            if (__popc(smask) <= kNarrow && !__any_sync(kAll, L.mode == L_SOLVE && L.irregular)) {
                const bool waits = L.mode == L_IDLE && (ready || left > 0 || more);
                int extra;
                iterated = narrow_passes(L, smask, a.run, warp_seg, o, extra, [&](int) { return waits; });
            } else if (L.mode == L_SOLVE) {
                iterated = lane_eval(L, a.run, slot, o);
            }
            if (iterated && lane_book(L, o, a.run, ls)) {
                a.qo[L.s] = L.qdc;
                a.dpo[L.s] = L.h;
                quc = L.qdc;
                seg_buf(slot, L.i)[kSegPlane * kSegSmemStride].x = L.h;
                owed |= 1 << L.i;
                L.mode = L_IDLE;
                SolveOut so;
                so.iters = L.total;
                so.retried = L.retried;
                so.early = 0;
                count_solve(ls, hist_s, so);
            }
        } else if (!__any_sync(kAll, ready || left > 0 || more || owed)) {
            break;
        }
    }
    flush_stats(ls, hist_s, a.run.stats);
}

// Lanes per warp, blocks and their shares. A block's share is known from the start
// and handed out by a counter of its own: one in device memory would be shared by
// calls that overlap, on several streams or in captured graphs, each then missing
// the reaches the other has taken. Runs of 16 reaches keep neighbours, which share
// sectors, in a block; 2,400 reaches a block even out. (2.7 M segments in 1.1 M
// reaches, rtol 1e-8: 14.5 ms, runs within 0.4 %; one counter for the GPU 16-21 ms.)
// One warp per scheduler while four reaches each are enough (narrow passes cost the
// same for one to four); then full passes on one warp per scheduler; from 32 reaches
// a warp on, three warps per scheduler.
int launch_reach_parallel(const troute_chparams* p, const double* ql, const int* rs,
                          const int* rl, const double* qu, const double* qd, const double* dp,
                          double* qo, double* vo, double* dpo, double uq, double dt, int nr,
                          int n_segments, const Tol& tol, DevStats* stats, void* stream)
{
    if (nr <= 0) return TROUTE_OK;
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    constexpr int warps = kReachThreads / 32;
    ReachArgs a = {};
    a.p = p;
    a.ql = ql;
    a.qu = qu;
    a.qd = qd;
    a.dp = dp;
    a.rs = rs;
    a.rl = rl;
    a.qo = qo;
    a.vo = vo;
    a.dpo = dpo;
    a.uq = uq;
    a.nr = nr;
    a.n_segments = n_segments;
    a.run.dt = dt;
    a.run.dt_half = dt / 2.0;
    a.run.tol = tol;
    a.run.stats = stats;
    const long long per_warp = ((long long)nr + warps * sms - 1) / (warps * sms);
    a.lanes = (int)(per_warp < 32 ? per_warp : 32);
    a.run_len = per_warp <= 32 ? warps * a.lanes : kRunLen;
    const int blocks = per_warp <= 32 ? (int)((nr + (long long)warps * a.lanes - 1) / (warps * a.lanes)) : 3 * sms;
    reach_parallel_kernel<<<blocks, kReachThreads, 0, (cudaStream_t)stream>>>(a);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return set_error(TROUTE_ECUDA, "reach_parallel_kernel launch: %s", cudaGetErrorString(e));
    return TROUTE_OK;
}

}  // namespace tr
