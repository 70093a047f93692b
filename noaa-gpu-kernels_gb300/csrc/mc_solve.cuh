// FP64 Muskingum-Cunge secant solve of one segment for one time step, device side.
//
// Arithmetic follows the reference solver operation for operation
// (water-prediction/t-route/troute_mc_final.cu:42-139, the same algorithm as
// cpu_mc :181-248 and mc_solve_d in wavefront/wavefront_mc.cu:215-337):
//   - channel geometry at a depth: trapezoid + compound channel (:30-40);
//   - celerity Ck from Manning (R^(2/3), R^(5/3)), K = max(dt, dx/Ck), X, C1..C4;
//   - X clamped to [0, 0.5] at the lower point and [0.25, 0.5] at the upper
//     point, the upper X using the lower point's C1..C4 (:86 vs :105);
//   - C4 clamp only at the upper point (:109);
//   - up to `attempts` bracket-widening restarts (:121-122);
//   - outflow with the negative-flow fallbacks and trapezoid-only velocity
//     (:125-138).
// R^(2/3) and R^(5/3) are correctly rounded (crpow.cuh), like the host pow() of
// the reference almost always is; with FMA contraction disabled for this code
// (the library builds it with -fmad=false) every other operation rounds exactly
// as the reference's C does.
// One change of evaluation, not of values: every quantity that depends only on
// the lower depth h_0 (geometry, Ck, K, Manning discharge) is carried over from
// the previous iteration's upper-depth evaluation, because each iteration sets
// h_0 = max(0, h) and h >= 0 always holds, so that evaluation is the same
// function of the same number. Only a restart (h_0 *= 0.67) re-evaluates it.
//
// A pass exists in two forms with the same results bit for bit.
//  - secant_pass: what the solves run. The FP64 pipe bounds every routing
//    kernel (one FP64 warp instruction holds an SMSP's pipe for 64 cycles), so
//    the pass is written to issue few of them: about 141 in bank, against 237
//    before (IEEE divisions, 5-instruction shared quotients, 35-instruction
//    powers, the lower depth's X denominator formed anew). Quotients and powers
//    come from near_quot and pow23_53_near, decisions are taken on the integer
//    pipes. Each of these says when it cannot vouch for its rounding; about one
//    pass in 10^4 is then evaluated again by
//  - exact_pass: the same formulas with IEEE divisions, fmin/fmax and the general
//    powers, for any operands, out of line. Solves whose parameters or flows
//    lie outside the ranges in which the short forms are proven
//    (seg_regular, flow_regular) use it for every pass.
#pragma once

#include "crpow.cuh"
#include "fpbits.cuh"
#include "troute_internal.h"

namespace tr {

__device__ __forceinline__ SegP load_seg(const NetDev& net, long long s)
{
    const SegRec* r = net.seg + s;
    const double2 a = __ldg(r->p + 0), b = __ldg(r->p + 1), c = __ldg(r->p + 2);
    const double2 e = __ldg(r->p + 3), f = __ldg(r->p + 4), g = __ldg(r->p + 5);
    SegP p;
    p.dx = a.x; p.bw = a.y; p.twcc = b.x; p.n_ch = b.y; p.ncc = c.x; p.s0 = c.y;
    p.z = e.x; p.bfd = e.y; p.sq_s0 = f.x; p.sq2 = f.y; p.ck_fac = g.x; p.z2 = g.y;
    return p;
}

// Everything at one depth that does not depend on the iteration's X: Km, the
// Manning discharge, and the denominator 2 tw s0 Ck dx of X's quotient with its
// reciprocal. yG = +0 says that X is 1/2 (no celerity, or a denominator that is
// not positive).
struct DepthEval {
    double Km, Qmn, G, yG;
};

// What a pass reads beside the segment's parameters and the depths.
struct PassFlow {
    double qup, quc, qdp, qldt;   // qldt = ql dt
    double dt, dt2;               // dt2 = dt / 2
};

// What a pass with a lower depth produces.
struct PassOut {
    double Qj_0;   // residual at the lower depth (the next iteration's X reads it)
    double qdc;    // outflow of the upper depth's coefficients
    double h_1;    // secant estimate
};

// Ranges in which the short forms are proven: with regular parameters and time
// step (seg_regular, value_regular), depths of +0 or in [2^-100, 2^480) and flows
// below 2^100 every intermediate but the secant's numerator (checked) is zero or
// inside the normal range with room for its residual. The depths reach that far
// in earnest: where the secant does not converge it doubles its bracket pass
// after pass, to 1e136 and beyond, until maxiter (at rtol 1e-8 one iteration in
// four is spent at depths above 1e18 m). Above the bank the area is bounded by
// linear terms, so R tends to twcc / 2 and the discharge grows like the depth.
// A positive depth in [2^-100, 2^480).
__device__ __forceinline__ bool depth_regular(double x)
{
    return (unsigned)(__double2hiint(x) - (923 << 20)) < (580u << 20);
}

// The secant's numerator is below 2^1000.
__device__ __forceinline__ bool numerator_regular(double v) { return (__double2hiint(v) & 0x7fffffff) < (2023 << 20); }

// +0, or a magnitude in [2^-150, 2^100).
__device__ __forceinline__ bool flow_regular(double q)
{
    const int h = __double2hiint(q);
    return (unsigned)((h & 0x7fffffff) - (873 << 20)) < (250u << 20) || (h | __double2loint(q)) == 0;
}

// X = (1 - q) / 2 clamped to [lo, 1/2] from v = 1 - q, on the high words: below 1
// the half is the exponent lowered by one (v is at least 2^-53 there). lo2 is the
// high word of 2 lo: 0 for lo = 0, 0x3fe00000 for lo = 1/4.
__device__ __forceinline__ double clamped_half(double v, int lo2)
{
    const int h = __double2hiint(v);
    const double x = __hiloint2double(h - (1 << 20), __double2loint(v));
    const double lo = __hiloint2double(lo2 ? lo2 - (1 << 20) : 0, 0);
    return h >= 0x3ff00000 ? 0.5 : h <= 0 || h < lo2 ? lo : x;
}

// Evaluation at x (a regular segment; doubt when x is neither +0 nor regular).
__device__ __forceinline__ void eval_near(double x, const SegP& p, double dt, DepthEval& e, bool& doubt)
{
    const bool wet = (__double2hiint(x) | __double2loint(x)) != 0;
    bool unsure = !depth_regular(x);
    const double twl = p.bw + p.z2 * x;  // bw + 2 z x
    const bool over = dbits(x) > dbits(p.bfd);
    const double below = over ? p.bfd : x;
    double AAC = (p.bw + below * p.z) * below;
    double P = p.bw + below * p.sq2;  // bw + 2 below sqrt(1+z^2)
    double WPn = P * p.n_ch;
    if (over) {
        // the compound-channel terms: area A + AC, wetted perimeter WP + WPC,
        // conveyance weight WP n + WPC ncc (2 above is exact: one FMA)
        const double above = x - p.bfd;
        const double WPC = __fma_rn(2.0, above, p.twcc);
        AAC = AAC + p.twcc * above;
        P = P + WPC;
        WPn = WPn + WPC * p.ncc;
    }
    const NearRcp rP = near_rcp(P);
    const double R = near_quot(AAC, rP, unsure);
    double r23, r53;
    pow23_53_near(R, &r23, &r53, unsure);
    // 2 sqrt(1+z^2) / (bw + 2 x z): the denominator is twl
    const double Ck = p.ck_fac * ((5.0 / 3.0) * r23 - (2.0 / 3.0) * r53 * near_quot(p.sq2, near_rcp(twl), unsure));
    e.Qmn = near_one_over(near_quot(WPn, rP, unsure), unsure) * AAC * r23 * p.sq_s0;
    bool unsure_k = false;
    const double K = near_quot(p.dx, near_rcp(Ck), unsure_k);
    const bool moves = wet && __double2hiint(Ck) > 0;
    e.Km = moves ? fp_max_pos(dt, K) : dt;
    const double g = (over ? p.twcc : twl) * p.s0 * Ck * p.dx;
    // 2.0 * tw * s0 * Ck * dx is exactly twice the undoubled product
    e.G = moves ? __hiloint2double(__double2hiint(g) + (1 << 20), __double2loint(g)) : 1.0;
    e.yG = moves ? near_rcp(e.G).y : 0.0;
    if (!wet) e.Qmn = 0.0;
    doubt |= (wet & unsure) | (moves & unsure_k);
}

// Secant update from the lower depth's evaluation e0 and the upper depth's e.
__device__ __forceinline__ void update_near(const DepthEval& e0, const DepthEval& e, const PassFlow& f, double h,
                                            double h_0, double Qj_0, PassOut& o, bool& doubt)
{
    // X at the lower depth, clamped to [0, 0.5] (troute_mc_final.cu:86)
    bool d0 = false, d1 = false, d2 = false;
    double X0 = clamped_half(1.0 - near_quot(Qj_0, {e0.G, e0.yG}, d0), 0);
    const bool v0 = dbits(e0.yG) != 0, v1 = dbits(e.yG) != 0;
    if (!v0) X0 = 0.5;
    const double KX0 = e0.Km * X0, K10 = e0.Km * (1.0 - X0);
    const NearRcp r0 = near_rcp(K10 + f.dt2);
    const double c1 = near_quot(KX0 + f.dt2, r0, doubt);
    const double c2 = near_quot(f.dt2 - KX0, r0, doubt);
    const double c3 = near_quot(K10 - f.dt2, r0, doubt);
    const double c4 = near_quot(f.qldt, r0, doubt);
    const double qmc0 = c1 * f.qup + c2 * f.quc + c3 * f.qdp + c4;
    o.Qj_0 = qmc0 - e0.Qmn;
    // X at the upper depth, clamped to [0.25, 0.5] (troute_mc_final.cu:105)
    double X = clamped_half(1.0 - near_quot(qmc0, {e.G, e.yG}, d1), 0x3fe00000);
    if (!v1) X = 0.5;
    const double KX = e.Km * X, K1 = e.Km * (1.0 - X);
    const NearRcp r1 = near_rcp(K1 + f.dt2);
    const double C1 = near_quot(KX + f.dt2, r1, doubt);
    const double C2 = near_quot(f.dt2 - KX, r1, doubt);
    const double C3 = near_quot(K1 - f.dt2, r1, doubt);
    double C4 = near_quot(f.qldt, r1, doubt);
    const double S3 = C1 * f.qup + C2 * f.quc + C3 * f.qdp;
    if (fp_lt0(C4) && fp_abs_gt(C4, S3)) C4 = -S3;
    // outflow of these coefficients (troute_mc_final.cu:125-130)
    const double Qmc = S3 + C4;
    const double Qj = Qmc - e.Qmn;
    o.qdc = Qmc;
    if (fp_lt0(Qmc)) {
        if (fp_lt0(C4) && fp_abs_gt(C4, S3))
            o.qdc = 0.0;
        else
            o.qdc = fmax(C1 * f.qup + C2 * f.quc + C4, C1 * f.qup + C3 * f.qdp + C4);
    }
    const double dQ = o.Qj_0 - Qj;
    const bool slope = !fp_eq0(dQ);
    const double num = Qj * (h_0 - h);
    o.h_1 = slope ? h - near_quot(num, near_rcp(dQ), d2) : h;
    d2 |= !numerator_regular(num);
    if (fp_lt0(o.h_1)) o.h_1 = h;
    doubt |= (v0 & d0) | (v1 & d1) | (slope & d2);
}

// The same pass for any operands: IEEE divisions, the general powers.
struct ExactPass {
    SegP p;
    PassFlow f;
    double x, h, h_0, Qj_0;
    DepthEval e0, e;   // e0 in, e out
    PassOut o;         // out, unless need0
    int need0;
};

static __device__ __noinline__ void exact_pass(ExactPass* a)
{
    const SegP& p = a->p;
    const double dt = a->f.dt, dt2 = a->f.dt2, h = a->x;
    {
        const double twl = p.bw + p.z2 * h;  // bw + 2 z h
        double above = fmax(h - p.bfd, 0.0);
        double below = fmin(p.bfd, h);
        if (above > 0.0 && p.twcc <= 0.0) {
            above = 0.0;
            below = h;
        }
        const double A = (p.bw + below * p.z) * below;
        const double WP = p.bw + below * p.sq2;  // bw + 2 below sqrt(1+z^2)
        const double AC = p.twcc * above;
        const double WPC = (above > 0.0) ? (p.twcc + 2.0 * above) : 0.0;
        const double P = WP + WPC;
        const double R = (P > 0.0) ? (A + AC) / P : 0.0;
        double r23, r53;
        pow23_53(R, &r23, &r53);
        DepthEval e;
        double Ck = 0.0;
        if (h > 0.0) Ck = fmax(0.0, p.ck_fac * ((5.0 / 3.0) * r23 - (2.0 / 3.0) * r53 * (p.sq2 / twl)));
        e.Km = (Ck > 0.0) ? fmax(dt, p.dx / Ck) : dt;
        const double twu = (h > p.bfd && p.twcc > 0.0) ? p.twcc : twl;
        e.Qmn = (P > 0.0) ? (1.0 / ((WP * p.n_ch + WPC * p.ncc) / P)) * (A + AC) * r23 * p.sq_s0 : 0.0;
        const bool valid = Ck > 0.0 && twu * p.s0 * Ck * p.dx > 0.0;
        e.G = valid ? 2.0 * twu * p.s0 * Ck * p.dx : 1.0;
        // outside near_rcp's range the value only says "valid": such solves stay
        // with this form, which divides by G
        e.yG = !valid ? 0.0 : fp_within(e.G, 400) ? near_rcp(e.G).y : 1.0;
        a->e = e;
    }
    if (a->need0) return;
    const double qup = a->f.qup, quc = a->f.quc, qdp = a->f.qdp, qldt = a->f.qldt;
    const double hu = a->h;
    const DepthEval e0 = a->e0, e = a->e;
    const double X0 = e0.yG != 0.0 ? fmin(0.5, fmax(0.0, 0.5 * (1.0 - a->Qj_0 / e0.G))) : 0.5;
    double D0 = e0.Km * (1.0 - X0) + dt2;
    if (D0 == 0.0) D0 = 1.0;
    const double c1 = (e0.Km * X0 + dt2) / D0;
    const double c2 = (dt2 - e0.Km * X0) / D0;
    const double c3 = (e0.Km * (1.0 - X0) - dt2) / D0;
    const double c4 = qldt / D0;
    const double qmc0 = c1 * qup + c2 * quc + c3 * qdp + c4;
    const double Qj_0 = qmc0 - e0.Qmn;
    const double X = e.yG != 0.0 ? fmin(0.5, fmax(0.25, 0.5 * (1.0 - qmc0 / e.G))) : 0.5;
    double D1 = e.Km * (1.0 - X) + dt2;
    if (D1 == 0.0) D1 = 1.0;
    const double C1 = (e.Km * X + dt2) / D1;
    const double C2 = (dt2 - e.Km * X) / D1;
    const double C3 = (e.Km * (1.0 - X) - dt2) / D1;
    double C4 = qldt / D1;
    const double S3 = C1 * qup + C2 * quc + C3 * qdp;
    if (C4 < 0.0 && fabs(C4) > S3) C4 = -S3;
    const double Qmc = S3 + C4;
    const double Qj = Qmc - e.Qmn;
    double qdc = Qmc;
    if (Qmc < 0.0) {
        if (C4 < 0.0 && fabs(C4) > S3)
            qdc = 0.0;
        else
            qdc = fmax(C1 * qup + C2 * quc + C4, C1 * qup + C3 * qdp + C4);
    }
    double h_1 = (Qj_0 - Qj != 0.0) ? hu - (Qj * (a->h_0 - hu)) / (Qj_0 - Qj) : hu;
    if (h_1 < 0.0) h_1 = hu;
    a->o.Qj_0 = Qj_0;
    a->o.qdc = qdc;
    a->o.h_1 = h_1;
}

// exact_pass on the values of a pass; irregular is set when a depth or
// denominator has left the ranges of the short forms.
__device__ __forceinline__ void redo_pass(const SegP& p, const PassFlow& f, double x, bool need0, double h, double h_0,
                                          double Qj_0, const DepthEval& e0, bool& irregular, DepthEval& e, PassOut& o)
{
    ExactPass a;
    a.p = p;
    a.f = f;
    a.x = x;
    a.h = h;
    a.h_0 = h_0;
    a.Qj_0 = Qj_0;
    a.e0 = e0;
    a.need0 = need0;
    exact_pass(&a);
    e = a.e;
    if (!need0) o = a.o;
    irregular |= !(x == 0.0 || depth_regular(x)) || !fp_within(e.G, 400);
}

// One pass: the evaluation at x into e; unless need0 also the update from e0
// into o. irregular: the segment or its flows are outside the proven ranges.
__device__ __forceinline__ void secant_pass(const SegP& p, const PassFlow& f, double x, bool need0, double h, double h_0,
                                            double Qj_0, const DepthEval& e0, bool& irregular, DepthEval& e, PassOut& o)
{
    bool doubt = irregular;
    eval_near(x, p, f.dt, e, doubt);
    if (!need0) update_near(e0, e, f, h, h_0, Qj_0, o, doubt);
    if (doubt) redo_pass(p, f, x, need0, h, h_0, Qj_0, e0, irregular, e, o);
}

// The stop test's "go on": rerr > rtol && aerr >= atol with rerr = |(h_1 - h) / h|,
// aerr = |h_1 - h| (rerr = 0, aerr = 0.9 for h <= 0); the relative error's
// quotient is only compared with rtol, which quot_gt_pos does exactly without
// dividing.
__device__ __forceinline__ bool secant_more(double h, double h_1, const Tol& tol)
{
    if (fp_gt0(h)) {
        const double aerr = fp_abs(h_1 - h);
        return fp_ge_nonneg(aerr, tol.atol) && quot_gt_pos(aerr, h, tol.rtol);
    }
    return fp_gt_pos(0.0, tol.rtol) && fp_ge_nonneg(0.9, tol.atol);
}

// Velocity from the final depth (troute_mc_final.cu:132-136).
__device__ __forceinline__ double seg_velocity(const SegP& p, double h)
{
    const double twl = p.bw + p.z2 * h;
    double Rv = (h * (p.bw + twl) / 2.0) /
                (p.bw + 2.0 * sqrt(((twl - p.bw) / 2.0) * ((twl - p.bw) / 2.0) + h * h));
    if (Rv < 0.0) Rv = 0.0;
    return (1.0 / p.n_ch) * pow23(Rv) * p.sq_s0;
}

struct SolveOut {
    double q, depth, vel;
    int iters;
    int retried;
    int early;
};

// No solve: invalid parameters or no flow at all (troute_mc_final.cu:54-63).
__device__ __forceinline__ bool exits_early(const SegP& p, double ql, double qup, double quc, double qdp)
{
    return fp_le0(p.n_ch) || fp_le0(p.s0) || fp_le0(p.z) || fp_le0(p.bw) ||
           (fp_le0(ql) && fp_le0(qup) && fp_le0(quc) && fp_le0(qdp));
}

__device__ __forceinline__ SolveOut mc_solve(double dt, double qup, double quc, double qdp,
                                             double ql, const SegP& p, double depthp,
                                             const Tol& tol)
{
    SolveOut o = {0.0, 0.0, 0.0, 0, 0, 0};
    if (exits_early(p, ql, qup, quc, qdp)) {
        o.early = 1;
        return o;
    }
    const PassFlow f = {qup, quc, qdp, ql * dt, dt, dt / 2.0};
    const double depth = fmax(depthp, 0.0);
    double h = depth * 1.33 + kMinDepth;
    double h_0 = depth * 0.67;
    PassOut po = {0.0, 0.0, 0.0};
    int maxiter = tol.maxiter, attempt = 0, iter = 0;
    bool need0 = true;
    bool irregular = !(seg_regular(p) && value_regular(dt) && flow_regular(qup) && flow_regular(quc) && flow_regular(qdp) && flow_regular(f.qldt));
    DepthEval e0, e;
    while (true) {
        secant_pass(p, f, need0 ? h_0 : h, need0, h, h_0, po.Qj_0, e0, irregular, e, po);
        e0 = e;
        if (need0) {
            need0 = false;
            continue;
        }
        const bool more = secant_more(h, po.h_1, tol);
        h_0 = fp_max0(h);
        h = fp_max0(po.h_1);
        ++iter;
        ++o.iters;
        if (!fp_lt_pos(h, kMinDepth) && more && iter <= maxiter) continue;
        if (iter < maxiter) break;
        // widen the bracket (also after the last attempt, as the reference does)
        h *= 1.33;
        h_0 *= 0.67;
        maxiter += 25;
        o.retried = 1;
        if (++attempt >= tol.attempts) break;
        iter = 0;
        need0 = true;
    }
    o.q = po.qdc;
    o.vel = seg_velocity(p, h);
    o.depth = h;
    return o;
}

}  // namespace tr
