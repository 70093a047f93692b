// A pass of at most four solves by the whole warp, eight lanes each.
//
// A narrow river network keeps few lanes of a warp busy, and one FP64 warp
// instruction costs 64-66 cycles whatever the number of its active lanes
// (measured, dependent or not, with one to four warps per SM): the time of a
// run is then the longest chain of passes times the FP64 instructions of a
// pass. Here the idle lanes take part, so that a pass issues 67 FP64 warp
// instructions instead of 141 (a lone warp: 6.4 k cycles a pass against 12.0 k; three
// warps per scheduler share its FP64 pipe, so that from five solves on the full pass
// is the better one):
//  - the eight lanes of a solve form two quads. Within a quad the lanes evaluate
//    at the same time what one lane evaluates in turn: the geometry's linear
//    forms, the reciprocals (wetted perimeter, top width; celerity, conveyance),
//    the quotients by them, the two powers, the four coefficients;
//  - the next pass's lower point has this pass's upper evaluation and this
//    pass's residual, both known before the secant step. Quad A forms the
//    upper coefficients of this pass while quad B forms the lower ones of the
//    next with the same instructions (X differs in its numerator and clamp);
//  - a solve's first pass evaluates h_0 (quad B) and h (quad A) together and so
//    saves the evaluation-only pass.
// Each value is formed by the operations of secant_pass (mc_solve.cuh) in their
// order, so the results are the same bit for bit; products that share an
// instruction with another lane's FMA are FMAs with -0.0 (exact), sums FMAs
// with 1.0. A lane's doubt about a rounding sends its solve's pass to exact_pass.
#pragma once

#include "lane_solver.cuh"

namespace tr {

constexpr int kNarrow = 4;   // solves of a narrow pass

__device__ __forceinline__ double lane_get(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }

// One of two constants with a zero low word, by a lane's role, which the compiler
// does not see through: a select between constants would otherwise be turned into
// two FP64 instructions, one for each side, where the point is to share one.
__device__ __forceinline__ double role_const(bool a, double if_a, double if_not)
{
    int hi = a ? __double2hiint(if_a) : __double2hiint(if_not);
    asm("" : "+r"(hi));
    return __hiloint2double(hi, 0);
}

// What differs between the four lanes of a quad, for a solve.
struct Role {
    int r;              // lane of the quad
    bool xl;            // lanes 1 and 2: X's quotient; 0 and 3: the Manning discharge
    double one_two;     // odd lanes -2, others 1 (the powers' correction)
    double one, neg_zero;
    double rcp_c;       // lane 2 -0, others 1
    double quot_c;      // lane 2 1, others -0
    double om_x, om_c;  // X or 1 - X = om_x X + om_c
    double neg_one;
    double flow;        // qup, quc, qdp, 1
    double dt2;         // lane 2 -dt/2, others dt/2
    double qldt;
};

// v or -v, on the integer pipe
__device__ __forceinline__ double neg_if(bool neg, double v)
{
    return __hiloint2double(__double2hiint(v) ^ (neg ? (int)0x80000000 : 0), __double2loint(v));
}

// One of x^fl(2/3) (odd = false) and x^fl(5/3) (odd = true) as pow23_53_near forms
// them: the same instructions for both, y or 1 as the outer factor.
__device__ __forceinline__ double pow_near_one(double x, bool odd, const Role& kc, bool& doubt)
{
    const int hi = __double2hiint(x);
    const int u = (hi >> 20) - (1023 - 36);
    doubt |= (unsigned)u >= 54u;
    const int k3 = (u * 43) >> 7;
    const int k = k3 - 12;
    const double y = __hiloint2double((hi & 0xfffff) | ((1023 + u - 3 * k3) << 20), __double2loint(x));
    float l;
    double r;
    crpow_seed(y, &l, &r);
    const double c = crpow_widen((float)kFl23Minus23 * ((l + 3.0f * (float)k) * 0.6931472f));
    const double wh = y * r;
    const double wl = __fma_rn(y, r, -wh);
    const double r2 = r * r;
    const double g = __fma_rn(-wl, r2, __fma_rn(-wh, r2, 1.0));
    const double s = g * __fma_rn(g, __fma_rn(g, 14.0 / 81.0, 2.0 / 9.0), 1.0 / 3.0);
    const double m = odd ? y : kc.one;
    const double w0 = m * wh;
    const double we = __fma_rn(m, wl, __fma_rn(m, wh, -w0));
    const double a = __fma_rn(w0, __fma_rn(kc.one_two, c, s), we);
    const double z = w0 + a;
    const double e = a - (z - w0);
    const int h = __double2hiint(z);
    doubt |= ((__double2hiint(e) & 0x7fffffff) >= (((h & 0x7ff00000) - (54 << 20)) | 0x000fffc0)) | ((h & 0xfffff) == 0);
    return __hiloint2double(h + (((odd ? 5 : 2) * k) << 20), __double2loint(z));
}

// Coefficients and discharge of one quad's evaluation: X from num / G clamped to
// [lo, 1/2] (lo2 as in clamped_half), C1..C4 on the quad's four lanes, their sum with the flows; beside X's
// quotient (lanes 1, 2) lanes 0 and 3 form the Manning discharge. W and V hold -G
// and 1/G on lanes 1 and 2 (1/G = 0: none), R^(2/3) and the area on 0 and 3.
struct QuadFlow {
    double q, Qmn;   // on all lanes of the quad
};

__device__ __forceinline__ QuadFlow quad_flow(const Role& k, int quad, double num, int lo2, double Km, double W, double V,
                                              double it, double sq_s0, bool& doubt)
{
    const bool valid = dbits(V) != 0;
    const double q0 = (k.xl ? num : it) * V;
    const double rr = __fma_rn(W, q0, k.xl ? num : k.neg_zero);
    const double qq = __fma_rn(rr, k.xl ? V : sq_s0, k.xl ? q0 : k.neg_zero);
    doubt |= k.xl & valid & quot_doubt(W, q0, rr);
    double X = clamped_half(1.0 - qq, lo2);
    if (!valid) X = 0.5;
    X = lane_get(X, quad | 1);
    QuadFlow o;
    o.Qmn = lane_get(qq, quad);
    // Km X on lanes 0, 1; Km (1 - X) on 2, 3
    const double t = Km * __fma_rn(X, k.om_x, k.om_c);
    // numerators Km X + dt/2, dt/2 - Km X, Km (1 - X) - dt/2; lane 3: the denominator
    const double n = neg_if(k.r == 1, t) + k.dt2;
    const NearRcp rd = near_rcp(lane_get(n, quad | 3));
    const double c = near_quot(k.r == 3 ? k.qldt : n, rd, doubt);
    const double m = c * k.flow;
    const double S3 = lane_get(m, quad) + lane_get(m, quad | 1) + lane_get(m, quad | 2);
    double C4 = lane_get(m, quad | 3);
    if (__any_sync(0xffffffffu, __double2hiint(C4) < 0))
        if (lo2 && fp_lt0(C4) && fp_abs_gt(C4, S3)) C4 = -S3;
    o.q = S3 + C4;
    return o;
}

// secant_more(h, h_1) from h_1 = h - step without FP64 instructions, where it is
// clearly true: the step is at least 2^-30 h, four times rtol h and four times
// atol by the exponents (the roundings of h_1 and of h_1 - h change it by a part in
// 2^21 at most).
__device__ __forceinline__ bool surely_more(double h, double step, const Tol& tol)
{
    const int eh = (__double2hiint(h) >> 20) & 0x7ff, es = (__double2hiint(step) >> 20) & 0x7ff;
    const int er = (__double2hiint(tol.rtol) >> 20) - 1023, ea = __double2hiint(tol.atol) >> 20;
    return (__double2hiint(h) > 0) & (eh != 0) & (es < 0x7ff) & (es - eh >= max(er + 3, -30)) & (es >= ea + 2);
}

// Passes for the lanes of smask (at most kNarrow, none irregular) until one of the
// solves needs its own lane again: it stops, starts a new attempt or the plain
// bracket, or has a doubtful rounding. The whole warp calls it; `warp_seg` is
// buffer 0 of the warp's lane 0. `leave(k)` is asked by every lane after pass k
// (from 0) when all solves would go on; a lane's true ends the call too. A lane of
// smask gets the last pass's o, its L.e0 (and what the next narrow pass starts from)
// as lane_eval leaves them, and the passes before it booked in L; returns whether
// the last one iterated (not after an exact evaluation at h_0 alone). extra: passes
// before the last.
//
// Between its passes the state of a solve stays on its octet, and the loop around
// (claims, item starts, publishing: 4 k cycles of a lone warp beside the pass's 6.4 k)
// is not run. 200,000 segments, 24 steps: 121 -> 114 ms, when a pass took 7.3 k.
template <typename Leave>
__device__ __forceinline__ bool narrow_passes(Lane& L, unsigned smask, const RunDev& run, double2* warp_seg, PassOut& o,
                                              int& extra, Leave leave)
{
    // The solves' own lanes filled the segment buffers (plain stores, or cp.async they
    // waited for) that the other lanes read here, and may fill them again afterwards;
    // shuffles and votes order no memory, so the barriers here and behind the loop do.
    __syncwarp();
    const int lane = threadIdx.x & 31;
    const int r = lane & 3, quad = lane & ~3;
    const bool B = lane & 4;
    // this octet's solve: the (lane / 8)-th lane of smask (the first again when
    // there are fewer)
    unsigned m = smask;
    const int j = lane >> 3;
    if (j > 0) m &= m - 1;
    if (j > 1) m &= m - 1;
    if (j > 2) m &= m - 1;
    const int home = __ffs(m ? m : smask) - 1;
    // passes after which the solve may go on: the warm phase has warm_k
    const int room = (L.warm == W_ACTIVE ? run.warm_k - 1 : L.maxiter) - L.iter;
    const int flags = __shfl_sync(0xffffffffu, (L.i & 1) | (L.need0 << 1) | ((L.ahead ? 1 : 0) << 2), home);
    const int left = __shfl_sync(0xffffffffu, room, home);
    bool need0 = flags & 2, pre = !(flags & 4);
    double h = lane_get(L.h, home), h_0 = lane_get(L.h_0, home);
    double q0n = lane_get(L.qmc0_n, home), Qj0n = lane_get(L.Qj0_n, home);
    Role kc;
    kc.r = r;
    kc.xl = r == 1 || r == 2;
    kc.one_two = role_const(r & 1, -2.0, 1.0);
    kc.one = role_const(true, 1.0, 1.0);
    kc.neg_zero = role_const(true, -0.0, -0.0);
    kc.rcp_c = role_const(r == 2, -0.0, 1.0);
    kc.quot_c = role_const(r == 2, 1.0, -0.0);
    kc.om_x = role_const(r < 2, 1.0, -1.0);
    kc.om_c = role_const(r < 2, -0.0, 1.0);
    kc.neg_one = role_const(true, -1.0, -1.0);
    {
        const double up = lane_get(L.qup, home), uc = lane_get(L.quc, home), dp = lane_get(L.qdp, home);
        kc.flow = r == 0 ? up : r == 1 ? uc : r == 2 ? dp : kc.one;
        kc.qldt = lane_get(L.qldt, home);
        kc.dt2 = neg_if(r == 2, run.dt_half);
    }
    const double2* const rec = warp_seg + home + (flags & 1) * kSegBufStride;
    // this lane's factors of the geometry: WP, A, top width (twice); n, -, s0, s0
    const double* const c1 = reinterpret_cast<const double*>(rec + (r == 0 ? 4 : r == 1 ? 3 : 5) * kSegSmemStride) + (r != 1);
    const double* const c2 = reinterpret_cast<const double*>(rec + (r == 0 ? 1 : 2) * kSegSmemStride) + 1;
    // on quad A of a solve past its first pass here: what the pass before left
    double Km_before = 0.0, W_before = 0.0, V_before = 0.0, Qmn_before = 0.0, Qj_before = 0.0;
    int k = 0;
    while (true) {
        const SegP p = staged_seg(rec);

        // ---- geometry ----
        const double x = (B && need0) ? h_0 : h;
        const bool wet = (__double2hiint(x) | __double2loint(x)) != 0;
        bool unsure = !depth_regular(x);
        const bool over = dbits(x) > dbits(p.bfd);
        // depth above the bank; lane 3: h_0 - h for the secant step
        const double diff = (r == 3 ? h_0 : x) - (r == 3 ? h : p.bfd);
        // lane 0: WP, WP n; lane 1: A; lanes 2, 3: bw + 2 z x and its product with s0
        const double xb = over & (r < 2) ? p.bfd : x;
        double s1 = p.bw + xb * *c1;
        double w = s1 * (r == 1 ? xb : *c2);
        if (__any_sync(0xffffffffu, over)) {
            const double t1 = __fma_rn(r == 0 ? 2.0 : p.twcc, r >= 2 ? p.s0 : diff, r == 0 ? p.twcc : kc.neg_zero);
            const double t2 = (r == 0 ? s1 : w) + t1;
            const double t3 = w + t1 * p.ncc;
            if (over) {
                if (r == 0) s1 = t2, w = t3;
                else w = r == 1 ? t2 : t1;
            }
        }
        // lane 1: R; lane 2: 2 sqrt(1+z^2) / (bw + 2 z x); lanes 0, 3: (WP n) / P
        const double P = lane_get(s1, r == 2 ? lane : quad), wn = lane_get(w, r == 1 ? lane : quad);
        const double q1 = near_quot(r == 2 ? p.sq2 : wn, near_rcp(P), unsure);
        const double z = pow_near_one(lane_get(q1, quad | 1), r & 1, kc, unsure);
        const double sqt = lane_get(q1, quad | 2);
        const double v = neg_if(r & 1, z * ((r & 1) ? 2.0 / 3.0 : 5.0 / 3.0) * ((r & 1) ? sqt : kc.one));
        const double Ck = p.ck_fac * (v + __shfl_xor_sync(0xffffffffu, v, 1));
        const bool moves = wet && __double2hiint(Ck) > 0;
        // lane 1: dx / Ck; lanes 0, 3: 1 / ((WP n) / P); lane 2: G = 2 tw s0 Ck dx, 1 / G
        double W, V, Km, it;
        {
            const bool g2 = r == 2;
            const double b = r == 1 ? Ck : q1, nd = r == 1 ? p.dx : kc.one;
            const double y0 = rcp_seed(b);
            const double nb = neg_if(!g2, g2 ? w : b);
            const double e1 = __fma_rn(nb, g2 ? Ck : y0, kc.rcp_c);
            const double e2 = __fma_rn(e1, g2 ? p.dx : e1, g2 ? kc.neg_zero : e1);
            const double y = __fma_rn(y0, e2, y0);
            const double G = __hiloint2double(__double2hiint(e2) + (1 << 20), __double2loint(e2));
            const double yg0 = rcp_seed(G);
            const double ya = g2 ? yg0 : y, nG = neg_if(true, G);
            const double q0 = __fma_rn(g2 ? nG : nd, ya, kc.quot_c);
            const double rr = __fma_rn(g2 ? q0 : nb, q0, g2 ? q0 : nd);
            const double qq = __fma_rn(rr, ya, g2 ? yg0 : q0);
            unsure |= !g2 & (moves | (r != 1)) & quot_doubt(b, q0, rr);
            it = qq;
            // (shuffles outside the selects: the quads' moves differ)
            W = lane_get(g2 ? nG : z, quad | (kc.xl ? 2 : 0));
            V = lane_get(r == 1 ? w : qq, quad | (kc.xl ? 2 : 1));
            Km = fp_max_pos(run.dt, lane_get(qq, quad | 1));
            if (!moves) {
                if (kc.xl) W = -1.0, V = 0.0;
                Km = run.dt;
            }
        }
        bool doubt = wet & unsure;

        // ---- the lower point of this pass, unless the last narrow pass formed it ----
        double q0 = q0n, Qj_0 = Qj0n;
        if (__any_sync(0xffffffffu, pre)) {
            const double eK = lane_get(L.e0.Km, home), eG = lane_get(L.e0.G, home), ey = lane_get(L.e0.yG, home);
            const double eQ = lane_get(L.e0.Qmn, home), Qp = lane_get(L.Qj_0, home);
            const bool old = kc.xl & !need0;
            bool d = false;
            const QuadFlow a = quad_flow(kc, quad, Qp, 0, need0 ? Km : eK, old ? neg_if(true, eG) : W, old ? ey : V, it, p.sq_s0, d);
            const double Qmn = need0 ? (wet ? a.Qmn : 0.0) : eQ;
            const double res = lane_get(a.q - Qmn, lane | 4), qa = lane_get(a.q, lane | 4);
            if (pre) {
                q0 = qa;
                Qj_0 = res;
                doubt |= B & d;
            }
            // quad B goes on with the upper evaluation
            Km = lane_get(Km, lane & ~4);
            W = lane_get(W, lane & ~4);
            V = lane_get(V, lane & ~4);
            it = lane_get(it, lane & ~4);
        }

        // ---- quad A: upper coefficients of this pass; quad B: lower ones of the next ----
        const QuadFlow a = quad_flow(kc, quad, B ? Qj_0 : q0, B ? 0 : 0x3fe00000, Km, W, V, it, p.sq_s0, doubt);
        const bool flowing = (__double2hiint(h) | __double2loint(h)) != 0;
        const double Qmn = flowing ? a.Qmn : 0.0;
        const double res = a.q - Qmn;
        doubt |= !B & fp_lt0(a.q);   // the negative-flow fallbacks (troute_mc_final.cu:125-130)

        // ---- secant step, on every lane of the octet ----
        // quad A, whose res is Qj: even lanes Qj (h_0 - h), odd ones Qj_0 - Qj
        const double hd = lane_get(diff, quad | 3);
        const double n = __fma_rn(res, (r & 1) ? kc.neg_one : hd, (r & 1) ? Qj_0 : kc.neg_zero);
        const double dQ = lane_get(n, (lane & ~7) | 1), num = lane_get(n, lane & ~7);
        const bool slope = !fp_eq0(dQ);
        bool d2 = false;
        const double q2 = near_quot(num, near_rcp(dQ), d2);
        double h_1 = slope ? h - q2 : h;
        const bool back = fp_lt0(h_1);
        if (back) h_1 = h;
        doubt |= slope & (d2 | !numerator_regular(num));

        // ---- the next pass here, if every solve goes on ----
        const unsigned bad = __ballot_sync(0xffffffffu, doubt);
        const double nh = fp_max0(h_1);
        bool on = ((bad >> (lane & ~7)) & 0xffu) == 0 && k + 1 <= left && !fp_lt_pos(nh, kMinDepth);
        if (__all_sync(0xffffffffu, on)) {
            const bool sure = slope && !back && surely_more(h, q2, run.tol);
            if (!__all_sync(0xffffffffu, sure)) on = secant_more(h, h_1, run.tol);
        }
        if (__all_sync(0xffffffffu, on) && !__any_sync(0xffffffffu, leave(k))) {
            Km_before = Km;
            W_before = W;
            V_before = V;
            Qmn_before = Qmn;
            Qj_before = Qj_0;
            h_0 = fp_max0(h);
            h = nh;
            q0n = lane_get(a.q, lane | 4);
            Qj0n = lane_get(res, lane | 4);
            need0 = pre = false;
            ++k;
            continue;
        }

        // ---- back to the solve's own lane ----
        __syncwarp();
        const int src = (8 * __popc(smask & ((1u << lane) - 1u))) & 31;
        const bool member = (smask >> lane) & 1u;
        extra = k;
        if (k > 0) {
            const double hh = lane_get(h, src), hh_0 = lane_get(h_0, src);
            if (member) {
                L.h = hh;
                L.h_0 = hh_0;
                L.iter += k;
                L.total += k;
                L.need0 = 0;
            }
            if (bad) {
                DepthEval b;
                b.Km = lane_get(Km_before, src);
                b.G = neg_if(true, lane_get(W_before, src + 1));
                b.yG = lane_get(V_before, src + 1);
                b.Qmn = lane_get(Qmn_before, src);
                const double qb = lane_get(Qj_before, src);
                if (member) {
                    L.e0 = b;
                    L.Qj_0 = qb;
                }
            }
        }
        DepthEval e;
        e.Km = lane_get(Km, src);
        e.G = neg_if(true, lane_get(W, src + 1));
        e.yG = lane_get(V, src + 1);
        e.Qmn = lane_get(Qmn, src);
        PassOut po;
        po.Qj_0 = lane_get(Qj_0, src);
        po.qdc = lane_get(a.q, src);
        po.h_1 = lane_get(h_1, src);
        const double qn = lane_get(a.q, src + 4), rn = lane_get(res, src + 4);
        if (!member) return false;
        if ((bad >> src) & 0xffu) {
            const SegP pl = staged_seg(warp_seg + lane + (L.i & 1) * kSegBufStride);
            const PassFlow fl = {L.qup, L.quc, L.qdp, L.qldt, run.dt, run.dt_half};
            redo_pass(pl, fl, L.need0 ? L.h_0 : L.h, L.need0, L.h, L.h_0, L.Qj_0, L.e0, L.irregular, e, po);
            L.e0 = e;
            L.ahead = false;
            const bool iterated = !L.need0;
            L.need0 = 0;
            o = po;
            return iterated;
        }
        L.e0 = e;
        L.need0 = 0;
        L.ahead = true;
        L.qmc0_n = qn;
        L.Qj0_n = rn;
        o = po;
        return true;
    }
}

}  // namespace tr
