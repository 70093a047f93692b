// Persistent tree routing driven by a ready queue (reach-to-warp mapping 3).
//
// The (item, step) pairs of a run form a DAG, an item r being a reach or a piece of
// one (item_segments in network.cpp): (r, t) needs (u, t) for every upstream item u
// (its current-step outflow, the item head's quc) and (r, t-1) (its own previous
// state). Instead of handing items out in a fixed
// order and letting lanes wait on them, each item carries a counter of
// completed dependencies; the lane that completes the last dependency of an
// item appends the item to a global ready queue, and idle lanes pop only from
// that queue. Lanes therefore only ever hold items whose inputs are final, so
// the warps' FP64 work goes to lanes that are actually solving (a warp issues
// every FP64 instruction at full cost however few of its lanes are busy).
//
//   cnt[t][r]   dependencies of (r, t) completed so far; (r, t) is ready at
//               n_up(r) + (t > 0)
//   heads       items without upstream ones at step 0, by level (the farthest from
//               an outlet first); idle lanes claim them (atomic counter) when
//               nothing else is ready
//   rq[i]       the other items in the order they became ready (atomic tail);
//               idle lanes claim slots (atomic head); -1 = not yet written
//   rh[t+1][r]  outflow of item r at step t of this run, rh[0][r] the
//               outflow of the step before the run (from the 4-slot ring of
//               the handle's state, within a reach from the discharge); a whole
//               run is kept, so upstream reaches
//               never wait for downstream ones to consume a value.
// In a warp of few items (and with continue_items in every warp) the lane that
// makes an item ready continues with it itself (the downstream item when two
// became ready), so the longest chain does not pass through the queue. A warp claims only
// slots that are already written (or that a racing warp is about to see
// written); the run ends when the count of completed items reaches n_items.
// Ready items come before heads, so that what has been started is carried on to its
// last step and the long paths, whose heads come first, advance while there is other
// work to fill the GPU; with all heads at the front of one queue they waited for
// every one of them (2.7 M segments, 24 steps, rtol 1e-8: 490 -> 452 ms; 64 members
// of 20,000 segments, warm start: 92.1 -> 86.2 ms; 200,000 segments: the same).
// The head sums at a reach use the upstream order of the reference
// (wavefront_mc.cu:525-531), and the solve is lane_solver.cuh's, i.e. the
// reference's arithmetic.
#include "narrow_pass.cuh"

namespace tr {

namespace {
constexpr unsigned kFullMask = 0xffffffffu;
constexpr int L_FETCH = L_WAIT;  // claimed a queue slot, waiting for it to be written
#ifndef TROUTE_WIDE_ITEMS
#define TROUTE_WIDE_ITEMS 1216
#endif
// Queued items from which on warps fill all their lanes instead of kNarrow.
constexpr int kWideItems = TROUTE_WIDE_ITEMS;
constexpr int kTopUpItems = 64;
constexpr unsigned long long kHeadSlot = 1ull << 63;   // a claimed head, not a queue slot
#ifndef TROUTE_SLEEP_MAX_NS
#define TROUTE_SLEEP_MAX_NS 3200
#endif
constexpr unsigned kSleepMinNs = 200, kSleepMaxNs = TROUTE_SLEEP_MAX_NS;  // idle-warp polling back-off
constexpr unsigned kPrimaryMaxNs = 800;

__device__ __forceinline__ unsigned lanemask_lt_df()
{
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ long long ld_acquire_ll(const long long* p)
{
    long long v;
    asm volatile("ld.acquire.gpu.global.s64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ int2 ld_volatile_int2(const int2* p)
{
    const long long v = *reinterpret_cast<const volatile long long*>(p);
    return make_int2((int)v, (int)(v >> 32));
}

__device__ __forceinline__ unsigned long long ld_volatile_ull(const unsigned long long* p)
{
    return *reinterpret_cast<const volatile unsigned long long*>(p);
}
}  // namespace

// How many more items a warp that holds `held` takes while `avail` are to be had. (A
// narrow warp with work leaves small backlogs to idle ones three passes out of
// four: its atomics would mostly find nothing left.)
__device__ __forceinline__ int claim_room(int2 avail, int held, bool primary, unsigned n_pass)
{
    const int all = max(avail.x, 0) + max(avail.y, 0);
    if (all >= kWideItems) return 32 - held;
    const bool top_up = held == 0 || all >= kTopUpItems || (n_pass & 3) == 0;
    return primary && top_up ? min(all, kNarrow - held) : 0;
}

// Takes up to `want` items from one of the two lists.
__device__ __forceinline__ int claim(int* avail, unsigned long long* head, int want, unsigned long long& base)
{
    const int had = atomicSub(avail, want);
    const int n = max(0, min(want, had));
    if (n < want) atomicAdd(avail, want - n);
    if (n) base = atomicAdd(head, (unsigned long long)n);
    return n;
}

// Loads the reach head inflows of (ri, tau) (all its dependencies are
// complete) and starts its first segment.
__device__ __forceinline__ void start_item(Lane& L, int ri, int tau, int t_base, const NetDev& net,
                                           const RunDev& run, const DataflowDev& df, double2* slot)
{
    const int R = df.n_item;
    const int4* rec = reinterpret_cast<const int4*>(df.item + ri);
    const int4 a = __ldg(rec), b = __ldg(rec + 1);
    const int2 c = __ldg(reinterpret_cast<const int2*>(rec + 2));   // row start in up_idx, inflow column
#ifdef TROUTE_CHECK
    // self-check build (the outflow history is NaN-filled before the run):
    // every value (ri, tau) reads must already be written, and its own output
    // slot must not be
    {
        bool ok = !isnan(__ldcg(df.rh + (size_t)tau * R + ri)) && isnan(__ldcg(df.rh + (size_t)(tau + 1) * R + ri));
        for (int j = 0; j < a.y; ++j) {
            const int u = j == 0 ? b.z : j == 1 ? b.w : __ldg(df.up_idx + c.x + j);
            ok = ok && !isnan(__ldcg(df.rh + (size_t)tau * R + u)) && !isnan(__ldcg(df.rh + (size_t)(tau + 1) * R + u));
        }
        if (!ok) record_error(run.stats, TROUTE_EINVAL, ri, t_base + tau, 7);
    }
#endif
    L.ri = ri;
    L.tau = tau;
    L.g = t_base + tau;
    L.ns = a.x;
    L.n_up = a.y;
    L.dn = a.z;
    L.dn_n_up = a.w;
    L.base = ((long long)b.y << 32) | (unsigned)b.x;
    if (L.ns > 0) {
        stage_seg_async(net, run, tau, L.base, slot);
        stage_inflow_async(run, tau, c.y, slot);
    }
    L.inflow = kInflowStaged;
    // sums over the upstream reaches in their order, from +0 (a first addend of -0
    // becomes +0, as in 0.0 + -0.0); within a reach the value itself
    const double* rprev = df.rh + (size_t)tau * R;
    const double* rcur = df.rh + (size_t)(tau + 1) * R;
    double p = 0.0, q = 0.0;
    if (L.n_up > 0) {
        const double p0 = __ldcg(rprev + b.z), q0 = __ldcg(rcur + b.z);
        double p1 = 0.0, q1 = 0.0;
        if (L.n_up > 1) {
            p1 = __ldcg(rprev + b.w);
            q1 = __ldcg(rcur + b.w);
        }
        p = c.x >= 0 && fp_eq0(p0) ? 0.0 : p0;
        q = c.x >= 0 && fp_eq0(q0) ? 0.0 : q0;
        if (L.n_up > 1) {
            p += p1;
            q += q1;
        }
        for (int j = 2; j < L.n_up; ++j) {
            const int u = __ldg(df.up_idx + c.x + j);
            p += __ldcg(rprev + u);
            q += __ldcg(rcur + u);
        }
    }
    L.qup_head = p;
    L.quc_head = q;
    L.q_up_old = 0.0;
    L.q_up_new = 0.0;
    L.q_last = 0.0;
    L.i = 0;
    L.mode = L_BEGIN;
}

// Threads per block, and the register budget: resident blocks per SM the
// allocation is sized for, or (TROUTE_DF_MAXNREG) a register cap. Two / three / four
// blocks of 128 take 226 / 168 / 128 registers and spill none / 196 B of stores and
// 208 of loads / 646 and 708. Three is the best where all lanes are full, which is
// where the work is largest: 64 members of a 2.7 M-segment network, warm start, 8
// steps 4,640 / 4,198 ms. A single network waits for its longest path, which the
// spills lengthen: 1,000 segments, 288 steps 10.0 / 11.1 / 13.9 ms; 200,000, 24 steps,
// rtol 1e-8 111 / 116 / 132; 64 members of 20,000, warm start, 16 steps 85 / 91 / 105;
// 2.7 M, 24 steps, rtol 1e-8 485 / 502 / 540.
#ifndef TROUTE_DF_THREADS
#define TROUTE_DF_THREADS 128
#endif
#ifndef TROUTE_DF_MINB
#define TROUTE_DF_MINB 3
#endif
#ifdef TROUTE_DF_MAXNREG
#define TROUTE_DF_BOUNDS __maxnreg__(TROUTE_DF_MAXNREG)
#else
#define TROUTE_DF_BOUNDS __launch_bounds__(TROUTE_DF_THREADS, TROUTE_DF_MINB)
#endif
constexpr int kDfThreads = TROUTE_DF_THREADS;
static_assert(kDfThreads % 32 == 0 && kDfThreads >= 32 && kDfThreads <= 1024, "whole warps per block");

// Warm-started runs read each solve's learned starting depth from the
// prediction plane the launch's GEMM filled (warm_gemm.cu) when the solve
// begins (lane_solver.cuh, begin_segment): the same kernel serves plain and
// warm-started runs.
__global__ void TROUTE_DF_BOUNDS route_dataflow_kernel(NetDev net, RunDev run, DataflowDev df)
{
    __shared__ unsigned int hist_s[16];
    __shared__ double2 seg_sm[kSegSmemPerThread * kDfThreads];
    double2* const seg_slot = seg_slot_of(seg_sm);
    double2* const warp_seg = seg_slot - (threadIdx.x & 31);
    if (threadIdx.x < 16) hist_s[threadIdx.x] = 0;
    __syncthreads();
    LocalStats ls = {0, 0, 0, 0, 0, 0};
    const int lane = threadIdx.x & 31;
    const unsigned lt = lanemask_lt_df();
    const int t_base = __ldg(run.step_base);
    const int T = run.n_ts;
    const int R = df.n_item;
    bool failed = false;
    unsigned long long slot = 0;
    const bool primary = blockIdx.x < (unsigned)df.n_primary;
    Lane L;
    L.mode = L_IDLE;
    unsigned long long n_pass = 0, n_busy = 0, n_wait = 0, n_idle = 0, n_solve = 0;
    unsigned idle_ns = kSleepMinNs;  // warp-uniform
    unsigned long long idle_seen = ~0ull;  // warp-uniform: n_done when this warp last saw progress
    long long idle_t0 = clock64();
    // lane 0: unclaimed items and error flag, read before each pass and used after
    // it, so that a solving warp does not wait for them
    int2 seen_avail = make_int2(0, 0);
    int seen_err = 0;

    while (true) {
        // ---- idle lanes claim queue slots (one atomic per warp) ----
        // A warp claims only as many slots as there are queued items that no
        // other warp has claimed (n_avail, taken down before the slots are;
        // claims that outran it would tie later items to whichever lanes raced,
        // however full their warps). While little is queued, the
        // primary warps -- one block per SM, one warp per scheduler -- and warps
        // that have work hold at most kNarrow items, which they solve by
        // narrow passes; once kWideItems are queued (more than the primary
        // warps can take up) every warp fills all its lanes, so that the work
        // lands on full warps: a warp pays for every FP64 instruction whatever
        // the number of its busy lanes.
        const unsigned idle = __ballot_sync(kFullMask, L.mode == L_IDLE);
        if (idle) {
            // ready items before heads: a subtree that has been started is carried on
            int n = 0, nh = 0, err = 0;
            unsigned long long base = 0, base_h = 0;
            if (lane == 0) {
                err = seen_err;
                const int want = claim_room(seen_avail, 32 - __popc(idle), primary, (unsigned)n_pass);
                const int wq = min(want, seen_avail.y);
                if (wq > 0) n = claim(&df.n_avail->y, df.rq_head, wq, base);
                const int wh = min(want - max(wq, 0), seen_avail.x);
                if (wh > 0) nh = claim(&df.n_avail->x, df.head_head, wh, base_h);
            }
            n = __shfl_sync(kFullMask, n, 0);
            nh = __shfl_sync(kFullMask, nh, 0);
            err = __shfl_sync(kFullMask, err, 0);
            if (err) break;
            if (n | nh) {
                base = __shfl_sync(kFullMask, base, 0);
                base_h = __shfl_sync(kFullMask, base_h, 0);
                const int rank = __popc(idle & lt);
                if (L.mode == L_IDLE && rank < n + nh) {
                    slot = rank < n ? base + rank : (base_h + (rank - n)) | kHeadSlot;
                    if ((slot & ~kHeadSlot) < (rank < n ? df.n_items : (unsigned long long)df.n_heads)) {
                        L.mode = L_FETCH;
                        L.wait_t0 = clock64();
                        L.wait_tail = 0;
                    }
                }
            }
        }
        // the run is over once every (reach, step) item has completed; lanes
        // still holding a claimed slot then leave it (it will not be written)
        if (__ballot_sync(kFullMask, L.mode >= L_SOLVE) == 0) {
            unsigned long long nd = 0;
            if (lane == 0) nd = ld_volatile_ull(df.n_done);
            nd = __shfl_sync(kFullMask, nd, 0);
            if (nd >= df.n_items) break;
            // a warp without work that sees no item complete anywhere for a
            // whole wait budget reports a timeout instead of polling forever
            if (nd != idle_seen) {
                idle_seen = nd;
                idle_t0 = clock64();
            } else if (clock64() - idle_t0 > run.wait_cycles) {
                if (lane == 0) record_error(run.stats, TROUTE_ETIMEOUT, -1, -1, 10);
                break;
            }
        } else {
            idle_t0 = clock64();
        }
        {
            const unsigned wmask = __ballot_sync(kFullMask, L.mode == L_FETCH);
            const unsigned bmask = __ballot_sync(kFullMask, L.mode >= L_SOLVE);
            n_pass++;
            n_wait += __popc(wmask);
            n_busy += __popc(bmask);
            n_idle += 32 - __popc(wmask | bmask);
        }

        // ---- lanes with a claimed slot: start the item once it is written ----
        if (L.mode == L_FETCH) {
            // (acquire: the item's inputs were published before it was queued)
            const int2* const at = slot & kHeadSlot ? df.heads + (slot & ~kHeadSlot) : df.rq + slot;
            const long long raw = ld_acquire_ll(reinterpret_cast<const long long*>(at));
            const int ri = (int)(raw & 0xffffffffll);
            const int tau = (int)(raw >> 32);
            if (ri >= 0 && (ri >= R || tau < 0 || tau >= T)) {
                // an entry that names no item of this run: report, never index with it
                record_error(run.stats, TROUTE_EINVAL, ri, tau, 8);
                failed = true;
            } else if (ri >= 0) {
                L.ri = ri;
                L.tau = tau;
                L.mode = L_START;
            } else if (clock64() - L.wait_t0 > run.wait_cycles) {
                // a slot can legitimately stay empty for long while the run
                // advances; give up only if no item completed during a whole
                // wait budget
                const unsigned long long nd = ld_volatile_ull(df.n_done);
                if (nd != L.wait_tail) {
                    L.wait_tail = nd;
                    L.wait_t0 = clock64();
                } else {
                    record_error(run.stats, TROUTE_ETIMEOUT, -1, (int)(slot & 0x7fffffff), 6);
                    failed = true;
                }
            }
        }

        // ---- the inflow of segments asked for before the last pass ----
        if (L.mode == L_SOLVE) stage_next_inflow(L, run, seg_slot);

        // ---- lanes starting an item, then a segment (the one inlined
        // start_item and begin_segment) ----
        if (L.mode == L_START) start_item(L, L.ri, L.tau, t_base, net, run, df, seg_slot);
        if (L.mode == L_BEGIN) L.mode = begin_segment(L, net, run, ls, hist_s, seg_slot) ? L_SOLVE : L_DONE;

        // ---- one pass of the solving lanes ----
        const unsigned smask = __ballot_sync(kFullMask, L.mode == L_SOLVE);
        if (smask && lane == 0) {
            seen_avail = ld_volatile_int2(df.n_avail);
            seen_err = ld_volatile_int(&run.stats->error);
        }
        if (smask) {
            n_solve++;
            PassOut o;
            bool iterated = false;
            if (__popc(smask) <= kNarrow && !__any_sync(kFullMask, L.mode == L_SOLVE && L.irregular)) {
                const unsigned held = __ballot_sync(kFullMask, L.mode != L_IDLE);
                const bool fetching = L.mode == L_FETCH;
                int extra;
                iterated = narrow_passes(L, smask, run, warp_seg, o, extra, [&](int k) {
                    bool out = fetching;
                    if (lane == 0) {
                        out |= seen_err != 0 || claim_room(seen_avail, __popc(held), primary, (unsigned)n_pass + k + 1) > 0;
                        seen_avail = ld_volatile_int2(df.n_avail);
                        seen_err = ld_volatile_int(&run.stats->error);
                    }
                    if (k == 0 && L.mode == L_SOLVE) stage_next_inflow(L, run, seg_slot);
                    return out;
                });
                n_pass += extra;
                n_solve += extra;
                n_busy += (unsigned long long)extra * __popc(smask);
                n_idle += (unsigned long long)extra * (32 - __popc(held));
            } else if (L.mode == L_SOLVE) {
                iterated = lane_eval(L, run, seg_slot, o);
            }
            if (iterated) lane_finish(L, o, net, run, ls, hist_s, seg_slot);
        }

        // ---- completed reaches: publish, count dependencies, queue ready items ----
        int npush = 0;
        int2 push0 = make_int2(-1, -1), push1 = make_int2(-1, -1);
        const unsigned dmask = __ballot_sync(kFullMask, L.mode == L_DONE);
        const bool narrow = primary && __popc(__ballot_sync(kFullMask, L.mode != L_IDLE)) <= kNarrow;
        if (dmask && lane == 0) atomicAdd(df.n_done, (unsigned long long)__popc(dmask));
        if (L.mode == L_DONE) {
            __stcg(df.rh + (size_t)(L.tau + 1) * R + L.ri, L.q_last);
            // what later launches start from
            if (L.tau + kRing >= T) {
                const int reach = __ldg(&df.item[L.ri].reach);
                if (reach >= 0) {
                    __stcg(net.ring + (size_t)(L.g % kRing) * net.n_reach_int + reach, L.q_last);
                    if (L.tau + 1 == T) net.done[reach] = L.g + 1;
                }
            }
            __threadfence();
            // the reach's own next step (needs its upstream reaches too) and the reach
            // downstream: both counters in flight together
            const bool own = L.tau + 1 < T, down = L.dn >= 0;
            int own_old = 0, down_old = 0;
            if (own) own_old = atomicAdd(df.cnt + (size_t)(L.tau + 1) * R + L.ri, 1);
            if (down) down_old = atomicAdd(df.cnt + (size_t)L.tau * R + L.dn, 1);
            if (own && own_old == L.n_up) push0 = make_int2(L.ri, L.tau + 1), npush = 1;
            if (down && down_old + 1 == L.dn_n_up + (L.tau > 0 ? 1 : 0)) {
                if (npush == 0) push0 = make_int2(L.dn, L.tau);
                else push1 = make_int2(L.dn, L.tau);
                ++npush;
            }
            L.mode = L_IDLE;
            if (npush && (df.continue_items || narrow)) {
                // continue with one newly ready item here (the downstream one when
                // there are two: it lies toward the outlet); queue the other
                __threadfence();  // other dependencies' writes, seen through the counters
                const int2 mine = (npush == 2) ? push1 : push0;
                if (npush == 2) push1 = make_int2(-1, -1);
                --npush;
                // started in the next pass, before its evaluation
                L.ri = mine.x;
                L.tau = mine.y;
                L.mode = L_START;
            }
        }
        // warp-aggregated append to the ready queue
        const unsigned push_any = __ballot_sync(kFullMask, npush >= 1), push_two = __ballot_sync(kFullMask, npush == 2);
        if (push_any) {
            const unsigned total = __popc(push_any) + __popc(push_two);
            const unsigned before = __popc(push_any & lt) + __popc(push_two & lt);
            unsigned long long base = 0;
            if (lane == 31) {
                base = atomicAdd(df.rq_tail, (unsigned long long)total);
                atomicAdd(&df.n_avail->y, (int)total);   // a claimer waits for a slot that is about to be written
            }
            base = __shfl_sync(kFullMask, base, 31);
            const unsigned long long pos = base + before;
            if (npush) __threadfence();  // every dependency's writes before the item is visible
            if (npush && pos + npush > df.n_items) {
                // more items than the run has: an accounting error, never write past the queue
                record_error(run.stats, TROUTE_EINVAL, push0.x, push0.y, 9);
                failed = true;
                npush = 0;
            }
            if (npush >= 1) {
                const long long v = ((long long)push0.y << 32) | (unsigned)push0.x;
                *reinterpret_cast<volatile long long*>(df.rq + pos) = v;
            }
            if (npush >= 2) {
                const long long v = ((long long)push1.y << 32) | (unsigned)push1.x;
                *reinterpret_cast<volatile long long*>(df.rq + pos + 1) = v;
            }
        }
        if (__any_sync(kFullMask, failed)) break;
        // a warp without solving lanes sleeps before polling again: briefly when
        // it holds claimed slots (their items are about to be written), with a
        // doubling back-off while it finds nothing at all, so that idle warps
        // do not crowd the queue counters' L2 lines while others solve
        if (__ballot_sync(kFullMask, L.mode >= L_SOLVE) == 0) {
            if (__any_sync(kFullMask, L.mode == L_FETCH)) {
                __nanosleep(kSleepMinNs);
            } else {
                __nanosleep(idle_ns);
                const unsigned most = primary ? kPrimaryMaxNs : kSleepMaxNs;
                idle_ns = idle_ns < most ? 2 * idle_ns : most;
            }
            if (lane == 0) {
                seen_avail = ld_volatile_int2(df.n_avail);
                seen_err = ld_volatile_int(&run.stats->error);
            }
        } else {
            idle_ns = kSleepMinNs;
        }
    }
    if (lane == 0) {
        atomicAdd(&run.stats->warp_passes, n_pass);
        atomicAdd(&run.stats->lane_busy, n_busy);
        atomicAdd(&run.stats->lane_wait, n_wait);
        atomicAdd(&run.stats->lane_idle, n_idle);
        atomicAdd(&run.stats->solve_passes, n_solve);
    }
    cp_async_wait_all();   // a lane that left an item early may still have its next segment in flight
    flush_stats(ls, hist_s, run.stats);
}

// Run set-up on the device: the queue starts empty, the heads are a list of their own
// with n_avail.x of them to be claimed; rh[0] = outflow of the step before the run.
__global__ void dataflow_init_kernel(NetDev net, RunDev run, DataflowDev df)
{
    const int t_base = *run.step_base;
    const int slot = ((t_base - 1) % kRing + kRing) % kRing;
    const double* src = net.ring + (size_t)slot * net.n_reach_int;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < df.n_item; r += gridDim.x * blockDim.x) {
        const ItemRec& c = df.item[r];
        df.rh[r] = c.reach >= 0 ? src[c.reach] : net.q[c.base + (long long)(c.nseg - 1) * kLanes];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *df.rq_head = 0;
        *df.rq_tail = 0;
        *df.head_head = 0;
        *df.n_avail = make_int2(df.n_heads, 0);
        *df.n_done = 0;
    }
}

int launch_route_dataflow(const NetDev& net, const RunDev& run, const DataflowDev& df, int grid, void* stream)
{
    if (run.warm && !run.start_pred) return set_error(TROUTE_ESTATE, "warm start requested without a prediction plane");
    if (df.n_items == 0) return TROUTE_OK;
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t e;
#ifdef TROUTE_CHECK
    if ((e = cudaMemsetAsync(df.rh, 0xff, (size_t)(run.n_ts + 1) * df.n_item * sizeof(double), st)) != cudaSuccess)
        return set_error(TROUTE_ECUDA, "dataflow set-up: %s", cudaGetErrorString(e));
#endif
    if ((e = cudaMemsetAsync(df.cnt, 0, (size_t)run.n_ts * df.n_item * sizeof(int), st)) != cudaSuccess ||
        (e = cudaMemsetAsync(df.rq, 0xff, (size_t)df.n_items * sizeof(int2), st)) != cudaSuccess)
        return set_error(TROUTE_ECUDA, "dataflow set-up: %s", cudaGetErrorString(e));
    int ig = (df.n_item + 255) / 256;
    if (ig > 4096) ig = 4096;
    if (ig < 1) ig = 1;
    dataflow_init_kernel<<<ig, 256, 0, st>>>(net, run, df);
    route_dataflow_kernel<<<grid, kDfThreads, 0, st>>>(net, run, df);
    e = cudaGetLastError();
    if (e != cudaSuccess) return set_error(TROUTE_ECUDA, "route_dataflow_kernel launch: %s", cudaGetErrorString(e));
    return TROUTE_OK;
}

int route_dataflow_threads() { return kDfThreads; }

int route_dataflow_occupancy(int* blocks_per_sm, bool)
{
    const cudaError_t e =
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, route_dataflow_kernel, kDfThreads, 0);
    if (e != cudaSuccess) return set_error(TROUTE_ECUDA, "occupancy query: %s", cudaGetErrorString(e));
    return TROUTE_OK;
}

}  // namespace tr
