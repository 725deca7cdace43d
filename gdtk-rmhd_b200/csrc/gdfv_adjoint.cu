// gdfv_adjoint.cu -- hand-written vector-Jacobian product of the residual,
// g = (dR/dU)^T w, for the Euler path (2D or 3D) with the ausmdv or hllc flux and for
// MHD with hlle and GLM cleaning (FP64), and the adjoints of the predictor-corrector
// step and of a rollout built on it.
//
// The residual (e4/fvcell.d:824-856) is R_c = (1/V) sum_faces +-A F_f, each face
// flux F_f a function of the four stencil states (e4/onedinterp.d:751-989 and
// e4/fluxcalc.d:477-651 or :653-820), each state a function of U through decode_conserved
// (e4/fvcell.d:586-822) or through a boundary condition (ghost cells).  The VJP
// runs in three kernels:
//   1. per cell: decode U -> primitive state P = (rho, v0, v1, v2, u, a);
//   2. tiles of grid lines in the three directions, a thread per cell: recompute
//      reconstruction and the plus face's flux from P, then the reverse of both; a
//      cell's cotangent, summed over its faces of the direction, is added to its gP
//      (atomics), through the ghost-cell maps (mirror, copy, xOrder-1
//      extrapolation, exchange) for ghosts, and to the fixed inflow states;
//   3. per cell: reverse of decode, gU = (dP/dU)^T gP.
// Non-smooth points (limiter, clipping, fmax, Mach-number and upwind switches,
// the entropy fix, |.|) take the branch the primal values took; |x| has
// derivative +1 at x = 0 as in src/ntypes/complex.d:944-955.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <vector>

#include "../../include/gdfv.h"
#include "gdfv_internal.h"
#include "gdfv_launch.h"

namespace gdfv {

namespace {

constexpr int NP = 6;  // rho, v0, v1, v2, u, a

__device__ __forceinline__ double sgn(double x) { return x < 0.0 ? -1.0 : 1.0; }

// Reciprocals and roots for the adjoint arithmetic: FD: without branches (recip, root,
// gdfv_device.cuh), for operands known to be in their range; else, and where no range is known
// (rcp), 0, subnormal and infinite operands give what 1 / x and sqrt(x) give.
__device__ __noinline__ double rcp_out_of_range(double x) { return 1.0 / x; }
template <bool FD>
__device__ __forceinline__ double rcp_of(double x) {
    if constexpr (FD) return recip(x).r;
    else return rcp_out_of_range(x);
}
template <bool FD>
__device__ __forceinline__ double sqrt_of(double x) {
    if constexpr (FD) return root(x);
    else return sqrt(x);
}
__device__ __forceinline__ double rcp(double x) {
    const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
    if (h - ((1023u - 1000u) << 20) >= 2000u << 20) return rcp_out_of_range(x);
    return recip(x).r;
}

// clip_to_limits(q, A, B) (src/nm/limiters.d:41-50; clip_fast, gdfv_stage.cuh) and its reverse,
// which routes g to q, A or B: to the lower bound, which is A when A <= B and else B, or to the
// upper one, A when A > B and else B.  A slip wall's ghost has v = -0 beside a cell at v = +0:
// A <= B there, whichever the side.
__device__ __forceinline__ double clip_adj(double q, double A, double B) {
    const bool down = A > B;
    const double lower = down ? B : A, upper = down ? A : B;
    const double qc = (q > lower) ? q : lower;
    return (qc <= upper) ? qc : upper;
}
__device__ __forceinline__ double clip_rev(double q, double A, double B, double g, double& gA, double& gB) {
    const bool down = A > B;
    const double lower = down ? B : A, upper = down ? A : B;
    const bool below = !(q > lower), above = !below && !(q <= upper), out = below || above;
    const bool to_a = below ? A <= B : down;
    gA += out && to_a ? g : 0.0;
    gB += out && !to_a ? g : 0.0;
    return out ? 0.0 : g;
}

// The l2r2 weights of one cell along a direction: both interface values of a cell come
// from one limiter evaluation (see recon_cell and, for graded blocks, recon_cell_graded).
struct CellWeights {
    double tol, toc, a, twoL, lenR0, lenL0, twoR;
};
template <bool RARE>
__device__ __forceinline__ CellWeights cell_weights(const BlockDesc& B, int D, int c) {
    if (RARE && B.graded) {
        const double* g = B.gw[D] + (long long)(c + 1) * GW_N;
        return CellWeights{g[GW_TOL], g[GW_TOC], g[GW_A], g[GW_TWOL], g[GW_LENR0], g[GW_LENL0], g[GW_TWOR]};
    }
    const double* w = B.w[D];
    return CellWeights{w[W_TOC], w[W_TOC], w[W_AL0], w[W_TWOL], w[W_LENR0], w[W_LENL0], w[W_TWOR]};
}

// lmr/onedinterp.d:147-151: the epsilon of the face between states l and r (scaled by the
// larger of the two), as the forward kernels form it; from: the side it came from (1 l,
// 2 r, 0 the floor).
__device__ __forceinline__ double lmr_epsilon(const NumParams& P, double toc, double l, double r, int& from) {
    const double tiny = 1e-12, a0 = fabs(l), a1 = fabs(r);
    const double m = fmax(fmax(tiny, a0), fmax(tiny, a1));
    from = m == tiny ? 0 : (a0 >= a1 ? 1 : 2);
    return m * P.eps_van_albada * toc;
}

// Both interface values of one scalar of a cell (q1, q0, q2: the cells before, at and after
// it): qm at its minus face, qp at its plus face (e4/onedinterp.d:357-386, clipping as
// src/nm/limiters.d:41-50).  rd: the reciprocal of the limiter's denominator, for the
// reverse (not with lmr, whose two faces have limiters of their own).  top gathers the high words
// of the denominators; with FD the result holds if denominators_in_range(top).
template <bool RARE, bool FD>
__device__ __forceinline__ void cell_recon(const NumParams& P, const CellWeights& w, double q1, double q0, double q2,
                                           double& qm, double& qp, double& rd, unsigned& top) {
    const double em = q0 - q1, ep = q2 - q0, dm = em * w.tol, dp = ep * w.toc;
    double sp = 1.0, sm = 1.0;
    rd = 0.0;
    if (P.apply_limiter) {
        const double p = dm * dp, n = p + fabs(p), d = dm * dm + dp * dp;
        if (RARE && P.lmr_epsilon) {
            int from;
            const double lp = lmr_epsilon(P, w.toc, q0, q2, from), lm = lmr_epsilon(P, w.toc, q1, q0, from);
            sp = (n + lp) * rcp_of<FD>(d + lp);
            sm = (n + lm) * rcp_of<FD>(d + lm);
            top = max(top, max((unsigned)__double2hiint(d + lp), (unsigned)__double2hiint(d + lm)));
        } else {
            rd = rcp_of<FD>(d + P.eps_van_albada);
            top = max(top, (unsigned)__double2hiint(d + P.eps_van_albada));
            sp = sm = (n + P.eps_van_albada) * rd;
        }
    }
    qp = q0 + sp * w.a * (dp * w.twoL + dm * w.lenR0);
    qm = q0 - sm * w.a * (dp * w.lenL0 + dm * w.twoR);
    if (P.extrema_clipping) {
        qp = clip_adj(qp, q0, q2);
        qm = clip_adj(qm, q1, q0);
    }
}

// Reverse of cell_recon: the cotangents gp of qp and gm of qm onto the three cells (g0 added
// to, g1 and g2 set).  Non-smooth points take the branch the values took.
template <bool RARE>
__device__ __forceinline__ void cell_recon_rev(const NumParams& P, const CellWeights& w, double q1, double q0, double q2,
                                               double rd, double gp, double gm, double& g1, double& g0, double& g2) {
    const double em = q0 - q1, ep = q2 - q0, dm = em * w.tol, dp = ep * w.toc;
    const double p = dm * dp, n = p + fabs(p), d = dm * dm + dp * dp;
    const bool lmr = RARE && P.lmr_epsilon;
    double sp = 1.0, sm = 1.0, rp = rd, rm = rd;
    int fp = 0, fm = 0;
    if (P.apply_limiter) {
        if (lmr) {
            const double lp = lmr_epsilon(P, w.toc, q0, q2, fp), lm = lmr_epsilon(P, w.toc, q1, q0, fm);
            rp = rcp(d + lp);
            rm = rcp(d + lm);
            sp = (n + lp) * rp;
            sm = (n + lm) * rm;
        } else {
            sp = sm = (n + P.eps_van_albada) * rd;
        }
    }
    const double X = dp * w.twoL + dm * w.lenR0, Y = dp * w.lenL0 + dm * w.twoR;
    g1 = g2 = 0.0;
    double gvp = 0.0, gvm = 0.0;
    if (P.extrema_clipping) {
        gvp = clip_rev(q0 + sp * w.a * X, q0, q2, gp, g0, g2);
        gvm = clip_rev(q0 - sm * w.a * Y, q1, q0, gm, g1, g0);
    } else {
        gvp = gp;
        gvm = gm;
    }
    g0 += gvp + gvm;
    const double ap = gvp * w.a, am = gvm * w.a;
    const double gX = ap * sp, gY = -am * sm;
    double gdp = gX * w.twoL + gY * w.lenL0, gdm = gX * w.lenR0 + gY * w.twoR;
    if (P.apply_limiter) {
        // s = (p + |p| + eps) / d, p = dm dp, d = dm^2 + dp^2 + eps
        double gn, gd;
        if (lmr) {
            const double gnp = ap * X * rp, gnm = -am * Y * rm;
            const double gdp_ = -gnp * sp, gdm_ = -gnm * sm;
            gn = gnp + gnm;
            gd = gdp_ + gdm_;
            const double k = P.eps_van_albada * w.toc;   // the faces' epsilons enter n and d
            const double kp = (gnp + gdp_) * k, km = (gnm + gdm_) * k;
            if (fp == 1) g0 += kp * sgn(q0);
            else if (fp == 2) g2 += kp * sgn(q2);
            if (fm == 1) g1 += km * sgn(q1);
            else if (fm == 2) g0 += km * sgn(q0);
        } else {
            gn = (ap * X - am * Y) * rd;
            gd = -gn * sp;
        }
        const double gpp = p < 0.0 ? 0.0 : 2.0 * gn;   // |p| rises at 0
        gdm += gpp * dp + 2.0 * gd * dm;
        gdp += gpp * dm + 2.0 * gd * dp;
    }
    g0 += gdm * w.tol - gdp * w.toc;
    g1 -= gdm * w.tol;
    g2 += gdp * w.toc;
}

// ausmdv (e4/fluxcalc.d:477-651) forward with the quantities the reverse needs,
// then its reverse.  Face-local states: r, p, u (normal), v, w (tangential), e, a.
struct FS { double r, p, u, v, w, e, a; };

template <bool FD>
__device__ void ausmdv_vjp(const NumParams& P, const FS& L, const FS& R, const double* gF, FS& gL, FS& gR) {
    // ---- forward
    const double irL = rcp_of<FD>(L.r), irR = rcp_of<FD>(R.r);
    double pLrL = L.p * irL, pRrR = R.p * irR;
    double keL = 0.5 * (L.u * L.u + L.v * L.v + L.w * L.w);
    double keR = 0.5 * (R.u * R.u + R.v * R.v + R.w * R.w);
    double HL = L.e + pLrL + keL, HR = R.e + pRrR + keR;
    double S = pLrL + pRrR;
    const double iS = rcp_of<FD>(S);
    double alphaL = 2.0 * pLrL * iS, alphaR = 2.0 * pRrR * iS;
    bool amL = L.a >= R.a;
    double am = fmax(L.a, R.a);
    const double iam = rcp_of<FD>(am);
    double ML = L.u * iam, MR = R.u * iam;
    double duL = 0.5 * (L.u + fabs(L.u));
    bool subL = fabs(ML) <= 1.0;
    double QL = (L.u + am) * (L.u + am) * (0.25 * iam);
    // p_half enters F linearly: only the cotangents of pLplus and pRminus are needed
    const double uLplus = subL ? alphaL * (QL - duL) + duL : duL;
    double duR = 0.5 * (R.u - fabs(R.u));
    bool subR = fabs(MR) <= 1.0;
    double QR = -(R.u - am) * (R.u - am) * (0.25 * iam);
    const double uRminus = subR ? alphaR * (QR - duR) + duR : duR;
    double ru_half = uLplus * L.r + uRminus * R.r;
    double dp0 = L.p - R.p;
    bool minL = L.p <= R.p;
    double mp = fmin(L.p, R.p);
    const double imp = rcp_of<FD>(mp);
    double dpa = 10.0 * fabs(dp0) * imp;
    bool sLin = dpa < 1.0;
    double s = 0.5 * fmin(1.0, dpa);
    double ru2V = uLplus * L.r * L.u + uRminus * R.r * R.u;
    double ru2D = 0.5 * (ru_half * (L.u + R.u) - fabs(ru_half) * (R.u - L.u));
    bool upL = ru_half >= 0.0;
    const double C = 0.125;
    bool caseA = ((L.u - L.a) < 0.0) && ((R.u - R.a) > 0.0);
    bool caseB = ((L.u + L.a) < 0.0) && ((R.u + R.a) > 0.0);
    double d_ua = 0.0;
    int efix = 0;
    if (P.apply_entropy_fix) {
        if (caseA && !caseB) { d_ua = C * ((R.u - R.a) - (L.u - L.a)); efix = 1; }
        if (caseB && !caseA) { d_ua = C * ((R.u + R.a) - (L.u + L.a)); efix = 2; }
    }
    // ---- reverse
    double gr_L = 0, gp_L = 0, gu_L = 0, gv_L = 0, gw_L = 0, ge_L = 0, ga_L = 0;
    double gr_R = 0, gp_R = 0, gu_R = 0, gv_R = 0, gw_R = 0, ge_R = 0, ga_R = 0;
    double gHL = 0, gHR = 0;
    if (efix && d_ua != 0.0) {
        double gd = -(gF[MASS] * (R.r - L.r) + gF[XMOM] * (R.r * R.u - L.r * L.u) + gF[YMOM] * (R.r * R.v - L.r * L.v) +
                      gF[ZMOM] * (R.r * R.w - L.r * L.w) + gF[TOTENERGY] * (R.r * HR - L.r * HL));
        gr_R -= gF[MASS] * d_ua; gr_L += gF[MASS] * d_ua;
        gr_R -= gF[XMOM] * d_ua * R.u; gu_R -= gF[XMOM] * d_ua * R.r; gr_L += gF[XMOM] * d_ua * L.u; gu_L += gF[XMOM] * d_ua * L.r;
        gr_R -= gF[YMOM] * d_ua * R.v; gv_R -= gF[YMOM] * d_ua * R.r; gr_L += gF[YMOM] * d_ua * L.v; gv_L += gF[YMOM] * d_ua * L.r;
        gr_R -= gF[ZMOM] * d_ua * R.w; gw_R -= gF[ZMOM] * d_ua * R.r; gr_L += gF[ZMOM] * d_ua * L.w; gw_L += gF[ZMOM] * d_ua * L.r;
        gr_R -= gF[TOTENERGY] * d_ua * HR; gHR -= gF[TOTENERGY] * d_ua * R.r;
        gr_L += gF[TOTENERGY] * d_ua * HL; gHL += gF[TOTENERGY] * d_ua * L.r;
        if (efix == 1) { gu_R += C * gd; ga_R -= C * gd; gu_L -= C * gd; ga_L += C * gd; }
        else { gu_R += C * gd; ga_R += C * gd; gu_L -= C * gd; ga_L -= C * gd; }
    }
    double vup = upL ? L.v : R.v, wup = upL ? L.w : R.w, Hup = upL ? HL : HR;
    double g_ru_half = gF[MASS] + gF[YMOM] * vup + gF[ZMOM] * wup + gF[TOTENERGY] * Hup;
    if (upL) { gv_L += gF[YMOM] * ru_half; gw_L += gF[ZMOM] * ru_half; gHL += gF[TOTENERGY] * ru_half; }
    else { gv_R += gF[YMOM] * ru_half; gw_R += gF[ZMOM] * ru_half; gHR += gF[TOTENERGY] * ru_half; }
    double g_ru2 = gF[XMOM], g_p_half = gF[XMOM];
    // ru2 = (0.5+s) ru2V + (0.5-s) ru2D
    double g_s = g_ru2 * (ru2V - ru2D);
    double g_ru2V = g_ru2 * (0.5 + s), g_ru2D = g_ru2 * (0.5 - s);
    // ru2D = 0.5 (ru_half (uL+uR) - |ru_half| (uR-uL))
    g_ru_half += 0.5 * g_ru2D * ((L.u + R.u) - sgn(ru_half) * (R.u - L.u));
    gu_L += 0.5 * g_ru2D * (ru_half + fabs(ru_half));
    gu_R += 0.5 * g_ru2D * (ru_half - fabs(ru_half));
    // ru2V = uLplus rL uL + uRminus rR uR
    double g_uLplus = g_ru2V * L.r * L.u, g_uRminus = g_ru2V * R.r * R.u;
    gr_L += g_ru2V * uLplus * L.u; gu_L += g_ru2V * uLplus * L.r;
    gr_R += g_ru2V * uRminus * R.u; gu_R += g_ru2V * uRminus * R.r;
    // s = 0.5 min(1, dpa), dpa = 10 |dp0| / min(pL, pR)
    if (sLin) {
        double g_dpa = 0.5 * g_s;
        double g_dp0 = g_dpa * 10.0 * sgn(dp0) * imp;
        double g_mp = -g_dpa * dpa * imp;
        gp_L += g_dp0; gp_R -= g_dp0;
        if (minL) gp_L += g_mp; else gp_R += g_mp;
    }
    double g_pLplus = g_p_half, g_pRminus = g_p_half;
    // ru_half = uLplus rL + uRminus rR
    g_uLplus += g_ru_half * L.r; gr_L += g_ru_half * uLplus;
    g_uRminus += g_ru_half * R.r; gr_R += g_ru_half * uRminus;
    double g_am = 0.0, g_alphaL = 0.0, g_alphaR = 0.0, g_duL = 0.0, g_duR = 0.0, g_ML = 0.0, g_MR = 0.0;
    if (subL) {
        gp_L += g_pLplus * (ML + 1.0) * (ML + 1.0) * (2.0 - ML) * 0.25;
        g_ML += g_pLplus * L.p * 0.25 * (2.0 * (ML + 1.0) * (2.0 - ML) - (ML + 1.0) * (ML + 1.0));
        g_alphaL += g_uLplus * (QL - duL);
        double g_Q = g_uLplus * alphaL;
        g_duL += g_uLplus * (1.0 - alphaL);
        gu_L += g_Q * 2.0 * (L.u + am) * (0.25 * iam);
        g_am += g_Q * ((L.u + am) * (0.5 * iam) - QL * iam);
    } else {
        const double iuL = rcp_of<FD>(L.u);
        gp_L += g_pLplus * duL * iuL;
        g_duL += g_pLplus * L.p * iuL;
        gu_L -= g_pLplus * L.p * duL * iuL * iuL;
        g_duL += g_uLplus;
    }
    gu_L += g_duL * 0.5 * (1.0 + sgn(L.u));
    if (subR) {
        gp_R += g_pRminus * (MR - 1.0) * (MR - 1.0) * (2.0 + MR) * 0.25;
        g_MR += g_pRminus * R.p * 0.25 * (2.0 * (MR - 1.0) * (2.0 + MR) + (MR - 1.0) * (MR - 1.0));
        g_alphaR += g_uRminus * (QR - duR);
        double g_Q = g_uRminus * alphaR;
        g_duR += g_uRminus * (1.0 - alphaR);
        gu_R += g_Q * (-2.0 * (R.u - am) * (0.25 * iam));
        g_am += g_Q * ((R.u - am) * (0.5 * iam) - QR * iam);
    } else {
        const double iuR = rcp_of<FD>(R.u);
        gp_R += g_pRminus * duR * iuR;
        g_duR += g_pRminus * R.p * iuR;
        gu_R -= g_pRminus * R.p * duR * iuR * iuR;
        g_duR += g_uRminus;
    }
    gu_R += g_duR * 0.5 * (1.0 - sgn(R.u));
    // ML = uL/am, MR = uR/am
    gu_L += g_ML * iam; g_am -= g_ML * ML * iam;
    gu_R += g_MR * iam; g_am -= g_MR * MR * iam;
    if (amL) ga_L += g_am; else ga_R += g_am;
    // alpha = 2 p/r / S
    double g_pLrL = g_alphaL * 2.0 * iS, g_pRrR = g_alphaR * 2.0 * iS;
    double g_S = -(g_alphaL * alphaL + g_alphaR * alphaR) * iS;
    g_pLrL += g_S; g_pRrR += g_S;
    // H = e + p/r + ke
    ge_L += gHL; g_pLrL += gHL; gu_L += gHL * L.u; gv_L += gHL * L.v; gw_L += gHL * L.w;
    ge_R += gHR; g_pRrR += gHR; gu_R += gHR * R.u; gv_R += gHR * R.v; gw_R += gHR * R.w;
    gp_L += g_pLrL * irL; gr_L -= g_pLrL * pLrL * irL;
    gp_R += g_pRrR * irR; gr_R -= g_pRrR * pRrR * irR;
    gL = FS{gr_L, gp_L, gu_L, gv_L, gw_L, ge_L, ga_L};
    gR = FS{gr_R, gp_R, gu_R, gv_R, gw_R, ge_R, ga_R};
}

// hllc (e4/fluxcalc.d:653-820, factor 1, one gas) forward with the quantities the reverse
// needs, then its reverse.  The Roe-averaged ratio of specific heats is gamma itself for
// one gas (its derivative vanishes); the wave-speed min/max and the star/side switches
// take the branches the primal values took.
template <bool FD>
__device__ void hllc_vjp(const NumParams& P, const FS& L, const FS& R, const double* gF, FS& gL, FS& gR) {
    // ---- forward
    const double g = P.gas.gamma;
    const double keL = 0.5 * (L.u * L.u + L.v * L.v + L.w * L.w);
    const double keR = 0.5 * (R.u * R.u + R.v * R.v + R.w * R.w);
    const double EL = L.r * L.e + L.r * keL, ER = R.r * R.e + R.r * keR;
    const double srL = sqrt_of<FD>(L.r), srR = sqrt_of<FD>(R.r);
    const double D = srL + srR, iD = rcp_of<FD>(D);
    const double uhat = (srL * L.u + srR * R.u) * iD;
    const double ghat = (srL * g + srR * g) * iD;
    const double N1 = srL * L.a * L.a + srR * R.a * R.a;
    const double sD = sqrt_of<FD>(D), isD = rcp_of<FD>(sD);
    const double T = D * isD;
    const double du = R.u - L.u;
    const double c2 = 0.5 * (ghat - 1.0);
    const double ahat2 = N1 * iD + c2 * T * du * du;
    const double ahat = sqrt_of<FD>(ahat2);
    const bool SLfromL = fmin(L.u - L.a, uhat - ahat) == L.u - L.a;
    const double SL = fmin(L.u - L.a, uhat - ahat);
    const bool SRfromR = fmax(R.u + R.a, uhat + ahat) == R.u + R.a;
    const double SR = fmax(R.u + R.a, uhat + ahat);
    const double num = R.p - L.p + L.r * L.u * (SL - L.u) - R.r * R.u * (SR - R.u);
    const double den = L.r * (SL - L.u) - R.r * (SR - R.u);
    const double iden = rcp_of<FD>(den);
    const double Ss = num * iden;
    const bool left = Ss > 0.0;
    const FS& X = left ? L : R;
    const double E = left ? EL : ER, S = left ? SL : SR;
    const bool star = left ? !(SL > 0.0) : !(SR < 0.0);
    const double dn = S - Ss, idn = star ? rcp(dn) : 0.0;
    const double coeff = star ? X.r * (S - X.u) * idn : 0.0;
    // ---- reverse (cotangents of the chosen side's r, p, u, v, w, E, S; of coeff, S*)
    double gr = 0, gp = 0, gu = 0, gv = 0, gw = 0, gE = 0, gS = 0, gc = 0, gSs = 0;
    // mass: r u (+ S (coeff - r))
    gr += gF[MASS] * X.u; gu += gF[MASS] * X.r;
    // momentum: r u u + p, r u v, r u w (+ S (coeff S* - r u), S (coeff - r) v, S (coeff - r) w)
    gr += gF[XMOM] * X.u * X.u; gu += gF[XMOM] * 2.0 * X.r * X.u; gp += gF[XMOM];
    gr += gF[YMOM] * X.u * X.v; gu += gF[YMOM] * X.r * X.v; gv += gF[YMOM] * X.r * X.u;
    gr += gF[ZMOM] * X.u * X.w; gu += gF[ZMOM] * X.r * X.w; gw += gF[ZMOM] * X.r * X.u;
    // energy: u (E + p) (+ S (U* - E))
    gu += gF[TOTENERGY] * (E + X.p); gE += gF[TOTENERGY] * X.u; gp += gF[TOTENERGY] * X.u;
    if (star) {
        gS += gF[MASS] * (coeff - X.r); gc += gF[MASS] * S; gr -= gF[MASS] * S;
        gS += gF[XMOM] * (coeff * Ss - X.r * X.u); gc += gF[XMOM] * S * Ss; gSs += gF[XMOM] * S * coeff;
        gr -= gF[XMOM] * S * X.u; gu -= gF[XMOM] * S * X.r;
        gS += gF[YMOM] * (coeff - X.r) * X.v; gc += gF[YMOM] * S * X.v; gr -= gF[YMOM] * S * X.v;
        gv += gF[YMOM] * S * (coeff - X.r);
        gS += gF[ZMOM] * (coeff - X.r) * X.w; gc += gF[ZMOM] * S * X.w; gr -= gF[ZMOM] * S * X.w;
        gw += gF[ZMOM] * S * (coeff - X.r);
        // U* = coeff (E/r + (S* - u) (S* + p/(r (S - u))))
        const double ir = rcp_of<FD>(X.r), Su = S - X.u, iSu = rcp_of<FD>(Su);
        const double Z = X.p * ir * iSu;
        const double Bq = Ss - X.u, Cq = Ss + Z;
        const double Xs = E * ir + Bq * Cq;
        const double Ust = coeff * Xs;
        gS += gF[TOTENERGY] * (Ust - E);
        gE -= gF[TOTENERGY] * S;
        const double gU = gF[TOTENERGY] * S;
        gc += gU * Xs;
        const double gX = gU * coeff;
        gE += gX * ir; gr -= gX * E * ir * ir;
        gSs += gX * Cq; gu -= gX * Cq;
        const double gZ = gX * Bq;
        gSs += gZ;
        gp += gZ * ir * iSu; gr -= gZ * Z * ir;
        const double gSu = -gZ * Z * iSu;
        gS += gSu; gu -= gSu;
        // coeff = r (S - u) / (S - S*)
        gr += gc * Su * idn;
        gS += gc * X.r * idn; gu -= gc * X.r * idn;
        const double gdn = -gc * coeff * idn;
        gS += gdn; gSs -= gdn;
    }
    // E = r e + r ke on the chosen side
    const double ke = left ? keL : keR;
    gr += gE * (X.e + ke);
    double ge = gE * X.r;
    gu += gE * X.r * X.u; gv += gE * X.r * X.v; gw += gE * X.r * X.w;
    double gr_L = 0, gp_L = 0, gu_L = 0, gv_L = 0, gw_L = 0, ge_L = 0, ga_L = 0;
    double gr_R = 0, gp_R = 0, gu_R = 0, gv_R = 0, gw_R = 0, ge_R = 0, ga_R = 0;
    double gSL = 0, gSR = 0;
    if (left) { gr_L += gr; gp_L += gp; gu_L += gu; gv_L += gv; gw_L += gw; ge_L += ge; gSL += gS; }
    else { gr_R += gr; gp_R += gp; gu_R += gu; gv_R += gv; gw_R += gw; ge_R += ge; gSR += gS; }
    // S* = num / den
    const double gnum = gSs * iden, gden = -gSs * Ss * iden;
    gp_R += gnum; gp_L -= gnum;
    gr_L += gnum * L.u * (SL - L.u); gu_L += gnum * L.r * (SL - 2.0 * L.u); gSL += gnum * L.r * L.u;
    gr_R -= gnum * R.u * (SR - R.u); gu_R -= gnum * R.r * (SR - 2.0 * R.u); gSR -= gnum * R.r * R.u;
    gr_L += gden * (SL - L.u); gSL += gden * L.r; gu_L -= gden * L.r;
    gr_R -= gden * (SR - R.u); gSR -= gden * R.r; gu_R += gden * R.r;
    // SL = min(uL - aL, uhat - ahat), SR = max(uR + aR, uhat + ahat)
    double guhat = 0.0, gahat = 0.0;
    if (SLfromL) { gu_L += gSL; ga_L -= gSL; } else { guhat += gSL; gahat -= gSL; }
    if (SRfromR) { gu_R += gSR; ga_R += gSR; } else { guhat += gSR; gahat += gSR; }
    // ahat2 = N1 / D + c2 T du^2, T = D / sqrt(D); ahat = sqrt(ahat2)
    const double gah2 = gahat * 0.5 * rcp_of<FD>(ahat);
    const double gN1 = gah2 * iD;
    double gD = -gah2 * N1 * iD * iD;
    double gsrL = gN1 * L.a * L.a, gsrR = gN1 * R.a * R.a;
    ga_L += gN1 * 2.0 * srL * L.a; ga_R += gN1 * 2.0 * srR * R.a;
    gD += gah2 * c2 * du * du * 0.5 * isD;
    const double gdu = gah2 * c2 * T * 2.0 * du;
    gu_R += gdu; gu_L -= gdu;
    // uhat = (srL uL + srR uR) / D
    gsrL += guhat * L.u * iD; gu_L += guhat * srL * iD;
    gsrR += guhat * R.u * iD; gu_R += guhat * srR * iD;
    gD -= guhat * uhat * iD;
    gsrL += gD; gsrR += gD;
    gr_L += gsrL * 0.5 * rcp_of<FD>(srL); gr_R += gsrR * 0.5 * rcp_of<FD>(srR);
    gL = FS{gr_L, gp_L, gu_L, gv_L, gw_L, ge_L, ga_L};
    gR = FS{gr_R, gp_R, gu_R, gv_R, gw_R, ge_R, ga_R};
}

// Reverse of the simple outflow flux of cell state q (rho, v0, v1, v2, u, a) through a
// face of normal +axis D (simple_outflow_flux, boundary_flux_effect.d:504-645): F = the
// cell's convective flux plus p n when the mass flux leaves (outsign m > 0), else p n
// alone; g the cotangent of the global-frame flux, added into gq.
template <int D>
__device__ void simple_flux_vjp(const NumParams& P, const double* q, int outsign, const double* g, double* gq) {
    const double rho = q[0], u = q[4];
    const double v[3] = {q[1], q[2], q[3]};
    const double T = u * P.gas.Cvinv;
    const double p = rho * P.gas.R * T;
    const double vn = v[D];
    const double m = rho * vn;
    double gp = 0.0, gm = 0.0, gvn = 0.0, gu = 0.0;
    double gv[3] = {0.0, 0.0, 0.0};
    if (outsign * m > 0.0) {
        gm += g[MASS];
        for (int d = 0; d < 3; ++d) {
            if (d == 2 && P.dims != 3) continue;   // no z momentum flux in 2D
            const double gd = g[XMOM + d];
            if (d == D) gp += gd;
            gv[d] += gd * m;
            gm += gd * v[d];
        }
        const double utot = u + 0.5 * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
        gm += g[TOTENERGY] * utot;
        gu += g[TOTENERGY] * m;
        for (int d = 0; d < 3; ++d) gv[d] += g[TOTENERGY] * m * v[d];
        gp += g[TOTENERGY] * vn;
        gvn += g[TOTENERGY] * p;
    } else {
        gp += g[XMOM + D];
    }
    gq[0] += gm * vn;                     // m = rho vn
    gvn += gm * rho;
    gv[D] += gvn;
    gq[0] += gp * P.gas.R * T;            // p = rho R (u Cvinv)
    gu += gp * rho * P.gas.R * P.gas.Cvinv;
    gq[1] += gv[0];
    gq[2] += gv[1];
    gq[3] += gv[2];
    gq[4] += gu;
}

// hlle for ideal MHD (e4/fluxcalc.d:1608-1780, mu0 = 1) forward with the quantities the
// reverse needs, then its reverse.  Face-local states: r, p, u (normal), v, w
// (tangential), B (normal, tangential, tangential), e (internal energy).  The
// alpha-weighted Cv and R of one gas are Cv and R themselves (their derivatives vanish);
// the wave-speed min/max and the switches at 0 take the branches the primal values took;
// SAFESQRT's floor (|x| <= 1e-14: 0) has derivative 0.
struct FSm { double r, p, u, v, w, Bx, By, Bz, e; };

struct FastSpeed {   // cf = sqrt(0.5 (alf + sqrt(alf^2 - 4 a2 ca2))) with its pieces
    double a2, ca2, alf, als, cf, ir;   // ir = 1 / rho
    bool live;        // SAFESQRT took the root
};
template <bool FD>
__device__ __forceinline__ FastSpeed fast_speed(double gam, double p, double rho, double Bx, double By, double Bz) {
    FastSpeed f;
    const double BB = Bx * Bx + By * By + Bz * Bz;
    f.ir = rcp_of<FD>(rho);
    f.a2 = gam * p * f.ir;
    f.ca2 = Bx * Bx * f.ir;
    f.alf = f.a2 + BB * f.ir;
    const double X = f.alf * f.alf - 4.0 * f.a2 * f.ca2;
    f.live = fabs(X) > 1.0e-14;
    f.als = f.live ? sqrt_of<FD>(X) : 0.0;
    f.cf = sqrt_of<FD>(0.5 * (f.alf + f.als));
    return f;
}
// reverse of fast_speed: gcf into the cotangents of p, rho and B (added)
template <bool FD>
__device__ __forceinline__ void fast_speed_rev(const FastSpeed& f, double gam, double Bx, double By, double Bz,
                                               double gcf, double& gp, double& grho, double& gBx, double& gBy,
                                               double& gBz) {
    const double gcf2 = gcf * 0.5 * rcp_of<FD>(f.cf);
    double galf = 0.5 * gcf2;
    const double gals = galf;
    double ga2 = 0.0, gca2 = 0.0;
    if (f.live) {
        const double gX = gals * 0.5 * rcp_of<FD>(f.als);
        galf += gX * 2.0 * f.alf;
        ga2 += -4.0 * f.ca2 * gX;
        gca2 += -4.0 * f.a2 * gX;
    }
    // alf = a2 + BB / rho
    ga2 += galf;
    const double gBB = galf * f.ir;
    grho -= gBB * (f.alf - f.a2);
    // ca2 = Bx^2 / rho
    double gBx2 = gca2 * f.ir;
    grho -= gBx2 * f.ca2;
    // a2 = gam p / rho
    gp += ga2 * gam * f.ir;
    grho -= ga2 * f.a2 * f.ir;
    gBx2 += gBB;
    gBx += 2.0 * Bx * gBx2;
    gBy += 2.0 * By * gBB;
    gBz += 2.0 * Bz * gBB;
}

// The one-sided fluxes of hlle_mhd: mass, x, y, z momentum, energy, By, Bz (Bx: 0).
__device__ __forceinline__ void mhd_side_flux(const FSm& S, double* f) {
    const double BB = S.Bx * S.Bx + S.By * S.By + S.Bz * S.Bz;
    const double pt = S.p + 0.5 * BB;
    const double uu = S.u * S.u + S.v * S.v + S.w * S.w;
    f[0] = S.r * S.u;
    f[1] = S.r * S.u * S.u - S.Bx * S.Bx + pt;
    f[2] = S.r * S.u * S.v - S.Bx * S.By;
    f[3] = S.r * S.u * S.w - S.Bx * S.Bz;
    f[4] = (S.r * S.e + 0.5 * (S.r * uu + BB) + pt) * S.u - (S.u * S.Bx + S.v * S.By + S.w * S.Bz) * S.Bx;
    f[5] = S.u * S.By - S.v * S.Bx;
    f[6] = S.u * S.Bz - S.w * S.Bx;
}
// reverse of mhd_side_flux: cotangents gf[7] into gS (added)
__device__ __forceinline__ void mhd_side_flux_rev(const FSm& S, const double* gf, FSm& gS) {
    const double BB = S.Bx * S.Bx + S.By * S.By + S.Bz * S.Bz;
    const double pt = S.p + 0.5 * BB;
    const double uu = S.u * S.u + S.v * S.v + S.w * S.w;
    double gpt = 0.0, guu = 0.0, gBB = 0.0;
    // mass
    gS.r += gf[0] * S.u; gS.u += gf[0] * S.r;
    // x momentum r u^2 - Bx^2 + pt
    gS.r += gf[1] * S.u * S.u; gS.u += gf[1] * 2.0 * S.r * S.u; gS.Bx -= gf[1] * 2.0 * S.Bx; gpt += gf[1];
    // y, z momentum
    gS.r += gf[2] * S.u * S.v; gS.u += gf[2] * S.r * S.v; gS.v += gf[2] * S.r * S.u;
    gS.Bx -= gf[2] * S.By; gS.By -= gf[2] * S.Bx;
    gS.r += gf[3] * S.u * S.w; gS.u += gf[3] * S.r * S.w; gS.w += gf[3] * S.r * S.u;
    gS.Bx -= gf[3] * S.Bz; gS.Bz -= gf[3] * S.Bx;
    // energy (H) u - (u Bx + v By + w Bz) Bx, H = r e + (r uu + BB)/2 + pt
    const double H = S.r * S.e + 0.5 * (S.r * uu + BB) + pt;
    const double Sd = S.u * S.Bx + S.v * S.By + S.w * S.Bz;
    const double gH = gf[4] * S.u;
    gS.u += gf[4] * H;
    const double gSd = -gf[4] * S.Bx;
    gS.Bx -= gf[4] * Sd;
    gS.r += gH * (S.e + 0.5 * uu); gS.e += gH * S.r; guu += 0.5 * gH * S.r; gBB += 0.5 * gH; gpt += gH;
    gS.u += gSd * S.Bx; gS.Bx += gSd * S.u; gS.v += gSd * S.By; gS.By += gSd * S.v;
    gS.w += gSd * S.Bz; gS.Bz += gSd * S.w;
    // By, Bz induction
    gS.u += gf[5] * S.By; gS.By += gf[5] * S.u; gS.v -= gf[5] * S.Bx; gS.Bx -= gf[5] * S.v;
    gS.u += gf[6] * S.Bz; gS.Bz += gf[6] * S.u; gS.w -= gf[6] * S.Bx; gS.Bx -= gf[6] * S.w;
    // pt = p + BB/2, uu, BB
    gS.p += gpt; gBB += 0.5 * gpt;
    gS.u += 2.0 * S.u * guu; gS.v += 2.0 * S.v * guu; gS.w += 2.0 * S.w * guu;
    gS.Bx += 2.0 * S.Bx * gBB; gS.By += 2.0 * S.By * gBB; gS.Bz += 2.0 * S.Bz * gBB;
}

// gF: cotangent of the face-local flux in the order MASS, XMOM, YMOM, ZMOM, TOTENERGY, XB,
// YB, ZB; gL, gR receive the cotangents of the two states (added).
template <bool FD>
__device__ void hlle_mhd_vjp(const NumParams& P, const FSm& L, const FSm& R, const double* gF, FSm& gL, FSm& gR) {
    // ---- forward
    const double gam = (P.gas.Cv + P.gas.R) * P.gas.Cvinv, igm1 = rcp_of<FD>(gam - 1.0);
    const double rho = 0.5 * (L.r + R.r), p = 0.5 * (L.p + R.p), u = 0.5 * (L.u + R.u);
    const double Bx = 0.5 * (L.Bx + R.Bx), By = 0.5 * (L.By + R.By), Bz = 0.5 * (L.Bz + R.Bz);
    const FastSpeed fm = fast_speed<FD>(gam, p, rho, Bx, By, Bz);
    const FastSpeed fL = fast_speed<FD>(gam, L.p, L.r, L.Bx, L.By, L.Bz);
    const FastSpeed fR = fast_speed<FD>(gam, R.p, R.r, R.Bx, R.By, R.Bz);
    const double wp = u + fm.cf, wm = u - fm.cf, wmL = L.u - fL.cf, wpR = R.u + fR.cf;
    const bool blL = wmL <= wm, brR = wpR >= wp;
    const double bl = blL ? wmL : wm, br = brR ? wpR : wp;
    const double blm = fmin(bl, 0.0), brp = fmax(br, 0.0);
    double fl[7], fr[7];
    mhd_side_flux(L, fl);
    mhd_side_flux(R, fr);
    const double uuL = L.u * L.u + L.v * L.v + L.w * L.w, uuR = R.u * R.u + R.v * R.v + R.w * R.w;
    const double BBL = L.Bx * L.Bx + L.By * L.By + L.Bz * L.Bz, BBR = R.Bx * R.Bx + R.By * R.By + R.Bz * R.Bz;
    // one-sided fluxes and jumps in the order of F (the Bx flux of either side is 0)
    const double fLF[8] = {fl[0], fl[1], fl[2], fl[3], fl[4], 0.0, fl[5], fl[6]};
    const double fRF[8] = {fr[0], fr[1], fr[2], fr[3], fr[4], 0.0, fr[5], fr[6]};
    const double d[8] = {R.r - L.r, R.r * R.u - L.r * L.u, R.r * R.v - L.r * L.v, R.r * R.w - L.r * L.w,
                         (R.p - L.p) * igm1 + 0.5 * (R.r * uuR + BBR) - 0.5 * (L.r * uuL + BBL),
                         R.Bx - L.Bx, R.By - L.By, R.Bz - L.Bz};
    const double iden = rcp_of<FD>(brp - blm), fac1 = brp * blm;
    // ---- reverse
    double gbrp = 0.0, gblm = 0.0, gfac1 = 0.0, giden = 0.0;
    double gfLF[8], gfRF[8], gd[8];
    for (int q = 0; q < 8; ++q) {
        const double N = brp * fLF[q] - blm * fRF[q] + fac1 * d[q];
        const double gN = gF[q] * iden;
        giden += gF[q] * N;
        gfLF[q] = gN * brp;
        gfRF[q] = -gN * blm;
        gd[q] = gN * fac1;
        gbrp += gN * fLF[q];
        gblm -= gN * fRF[q];
        gfac1 += gN * d[q];
    }
    gbrp += -giden * iden * iden;
    gblm += giden * iden * iden;
    gbrp += gfac1 * blm;
    gblm += gfac1 * brp;
    // fmin(bl, 0), fmax(br, 0) keep their first argument on a tie (src/ntypes/complex.d)
    const double gbl = bl <= 0.0 ? gblm : 0.0, gbr = br >= 0.0 ? gbrp : 0.0;
    double gwm = 0.0, gwp = 0.0, gcfL = 0.0, gcfR = 0.0;
    if (blL) { gL.u += gbl; gcfL -= gbl; } else gwm += gbl;
    if (brR) { gR.u += gbr; gcfR += gbr; } else gwp += gbr;
    // wp = u + cf, wm = u - cf of the averages
    const double gu = gwp + gwm, gcf = gwp - gwm;
    double gp = 0.0, grho = 0.0, gBx = 0.0, gBy = 0.0, gBz = 0.0;
    fast_speed_rev<FD>(fm, gam, Bx, By, Bz, gcf, gp, grho, gBx, gBy, gBz);
    fast_speed_rev<FD>(fL, gam, L.Bx, L.By, L.Bz, gcfL, gL.p, gL.r, gL.Bx, gL.By, gL.Bz);
    fast_speed_rev<FD>(fR, gam, R.Bx, R.By, R.Bz, gcfR, gR.p, gR.r, gR.Bx, gR.By, gR.Bz);
    gL.r += 0.5 * grho; gR.r += 0.5 * grho;
    gL.p += 0.5 * gp; gR.p += 0.5 * gp;
    gL.u += 0.5 * gu; gR.u += 0.5 * gu;
    gL.Bx += 0.5 * gBx; gR.Bx += 0.5 * gBx;
    gL.By += 0.5 * gBy; gR.By += 0.5 * gBy;
    gL.Bz += 0.5 * gBz; gR.Bz += 0.5 * gBz;
    const double gfl[7] = {gfLF[0], gfLF[1], gfLF[2], gfLF[3], gfLF[4], gfLF[6], gfLF[7]};
    const double gfr[7] = {gfRF[0], gfRF[1], gfRF[2], gfRF[3], gfRF[4], gfRF[6], gfRF[7]};
    mhd_side_flux_rev(L, gfl, gL);
    mhd_side_flux_rev(R, gfr, gR);
    // jumps
    gR.r += gd[0]; gL.r -= gd[0];
    gR.r += gd[1] * R.u; gR.u += gd[1] * R.r; gL.r -= gd[1] * L.u; gL.u -= gd[1] * L.r;
    gR.r += gd[2] * R.v; gR.v += gd[2] * R.r; gL.r -= gd[2] * L.v; gL.v -= gd[2] * L.r;
    gR.r += gd[3] * R.w; gR.w += gd[3] * R.r; gL.r -= gd[3] * L.w; gL.w -= gd[3] * L.r;
    const double ig = gd[4] * igm1;
    gR.p += ig; gL.p -= ig;
    gR.r += 0.5 * gd[4] * uuR; gL.r -= 0.5 * gd[4] * uuL;
    gR.u += gd[4] * R.r * R.u; gR.v += gd[4] * R.r * R.v; gR.w += gd[4] * R.r * R.w;
    gL.u -= gd[4] * L.r * L.u; gL.v -= gd[4] * L.r * L.v; gL.w -= gd[4] * L.r * L.w;
    gR.Bx += gd[4] * R.Bx; gR.By += gd[4] * R.By; gR.Bz += gd[4] * R.Bz;
    gL.Bx -= gd[4] * L.Bx; gL.By -= gd[4] * L.By; gL.Bz -= gd[4] * L.Bz;
    gR.Bx += gd[5]; gL.Bx -= gd[5];
    gR.By += gd[6]; gL.By -= gd[6];
    gR.Bz += gd[7]; gL.Bz -= gd[7];
}

struct AdjArgs {
    const BlockDesc* blocks;
    const InflowState* inflow;
    const double* U;
    const double* W;
    double* Pp;        // [6][total]
    double* gP;        // [6][total]
    double* gU;        // [nq][total]
    double* gInflow;   // [ninflow][6]
    const double* rot; // rotations of exchange faces with an Rmatrix (9 doubles each)
    const long long* tile_off;  // [3][nblocks+1] prefix counts of line tiles per direction
    double* lam;       // [nq][total] adjoint state of a fused step (modes 1, 2)
    double* bbuf;      // [nq][total] b = dt/2 lam + dt mu (mode 1 writes, mode 2 is its W)
    double w_scale;    // W enters scaled by this
    double dt;
    long long total;
    int nblocks;
    int mode;          // 0: gU = result; 1: mu -> bbuf, lam += mu; 2: lam += result
    NumParams P;
    double c_h;        // MHD: the GLM wave speed of the residual (the context's current one)
    // MHD with cleaning in a step adjoint: {c_h, psi damping factor} of the step (device;
    // null: c_h above, no damping); chd_slot is where the step adjoint forms them
    const double* chd;
    double* chd_slot;
};

__device__ __forceinline__ void decode_cell(const AdjArgs& a, long long g) {
    double u[5];
    for (int q = 0; q < 5; ++q) u[q] = a.U[q * a.total + g];
    Prim<double> s;
    double p, T;
    decode(a.P, u, s, p, T);
    double v[NP] = {s.rho, s.v[0], s.v[1], s.v[2], s.u, s.a};
    for (int m = 0; m < NP; ++m) { a.Pp[m * a.total + g] = v[m]; a.gP[m * a.total + g] = 0.0; }
}

__global__ void adj_decode_kernel(AdjArgs a) {
    long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (g < a.total) decode_cell(a, g);
}

// Stencil cell state from P (with the ghost maps) and the reverse map of a cotangent.
struct Src {
    const BlockDesc* blk;
    long long c0, c1;
    int kind, axis, inflow;
};

// RARE: some exchange rotates its ghosts' vectors, some face is an outflow boundary
// with a ghost or flux rule of its own, the limiter is lmr's, or some block is graded
// (the kernels without it carry none of that code)
template <bool RARE>
__device__ Src adj_resolve(const AdjArgs& a, const BlockDesc& B, int i, int j, int k) {
    StageArgs A{};
    A.blocks = a.blocks;
    CellSrc s = resolve<RARE, RARE>(A, B, i, j, k);
    return Src{s.blk, s.c0, s.c1, s.kind, s.axis, s.inflow};
}

template <bool RARE>
__device__ void adj_load(const AdjArgs& a, const Src& s, double* c) {
    if (s.kind == SRC_INFLOW) {
        const InflowState& in = a.inflow[s.inflow];
        c[0] = in.rho; c[1] = in.vel[0]; c[2] = in.vel[1]; c[3] = in.vel[2]; c[4] = in.u; c[5] = in.a;
        return;
    }
    const long long g0 = s.blk->offset + s.c0;
    double e[NP];
    for (int m = 0; m < NP; ++m) e[m] = a.Pp[m * a.total + g0];
    if (s.kind == SRC_EXTRAP1_G0 || s.kind == SRC_EXTRAP1_G1) {
        const long long g1 = s.blk->offset + s.c1;
        double f[NP];
        for (int m = 0; m < NP; ++m) f[m] = a.Pp[m * a.total + g1];
        // ghost0 = 2e - f1, ghost1 = 2 ghost0 - e (rho, v, u); a from the edge cell
        for (int m = 0; m < 5; ++m) {
            double g0v = 2.0 * e[m] - f[m];
            c[m] = (s.kind == SRC_EXTRAP1_G0) ? g0v : 2.0 * g0v - e[m];
        }
        c[5] = e[5];
        return;
    }
    for (int m = 0; m < NP; ++m) c[m] = e[m];
    if (s.kind == SRC_MIRROR) c[1 + s.axis] = -c[1 + s.axis];
    if (RARE && s.kind == SRC_ROTATE) {   // ghost velocity R v (flowstate.d:393-400)
        const double* R = a.rot + 9 * s.inflow;
        for (int r = 0; r < 3; ++r) c[1 + r] = R[3 * r] * e[1] + R[3 * r + 1] * e[2] + R[3 * r + 2] * e[3];
    }
    if (RARE && s.kind == SRC_FIXEDP) {   // fixed_p.d:98-119: rho, u from p_outside at the cell's T
        const double T = e[4] * a.P.gas.Cvinv;
        c[0] = a.inflow[s.inflow].p / (T * a.P.gas.R);
        c[4] = a.P.gas.Cv * T;
    }
    if (RARE && s.kind == SRC_FIXEDPT) {  // fixed_pt.d:105-128: rho, u from p_outside, T_outside
        c[0] = a.inflow[s.inflow].rho;
        c[4] = a.inflow[s.inflow].u;
    }
}

template <bool RARE>
__device__ void adj_scatter(const AdjArgs& a, const Src& s, const double* gc) {
    if (s.kind == SRC_INFLOW) {
        for (int m = 0; m < NP; ++m) atomicAdd(&a.gInflow[s.inflow * NP + m], gc[m]);
        return;
    }
    const long long g0 = s.blk->offset + s.c0;
    if (s.kind == SRC_EXTRAP1_G0 || s.kind == SRC_EXTRAP1_G1) {
        const long long g1 = s.blk->offset + s.c1;
        const double ce = (s.kind == SRC_EXTRAP1_G0) ? 2.0 : 3.0, cf = (s.kind == SRC_EXTRAP1_G0) ? -1.0 : -2.0;
        for (int m = 0; m < 5; ++m) {
            atomicAdd(&a.gP[m * a.total + g0], ce * gc[m]);
            atomicAdd(&a.gP[m * a.total + g1], cf * gc[m]);
        }
        atomicAdd(&a.gP[5 * a.total + g0], gc[5]);
        return;
    }
    if (RARE && (s.kind == SRC_FIXEDP || s.kind == SRC_FIXEDPT)) {
        // velocity and sound speed pass through; rho and u are the outside state's
        // (FixedPT) or, FixedP, rho = p/(T R) and u = Cv T with T = u_cell / Cv
        double gu = 0.0;
        if (s.kind == SRC_FIXEDP) {
            const double u = a.Pp[4 * a.total + g0];
            const double T = u * a.P.gas.Cvinv;
            const double rho = a.inflow[s.inflow].p / (T * a.P.gas.R);
            gu = gc[0] * (-rho / T) * a.P.gas.Cvinv + gc[4] * a.P.gas.Cv * a.P.gas.Cvinv;
        }
        atomicAdd(&a.gP[1 * a.total + g0], gc[1]);
        atomicAdd(&a.gP[2 * a.total + g0], gc[2]);
        atomicAdd(&a.gP[3 * a.total + g0], gc[3]);
        if (gu != 0.0) atomicAdd(&a.gP[4 * a.total + g0], gu);
        atomicAdd(&a.gP[5 * a.total + g0], gc[5]);
        return;
    }
    if (RARE && s.kind == SRC_ROTATE) {   // the transpose of the ghost's rotation R v
        const double* R = a.rot + 9 * s.inflow;
        for (int m = 0; m < NP; ++m) {
            const double v = (m >= 1 && m <= 3)
                                 ? R[m - 1] * gc[1] + R[3 + m - 1] * gc[2] + R[6 + m - 1] * gc[3]
                                 : gc[m];
            atomicAdd(&a.gP[m * a.total + g0], v);
        }
        return;
    }
    for (int m = 0; m < NP; ++m) {
        double v = gc[m];
        if (s.kind == SRC_MIRROR && m == 1 + s.axis) v = -v;
        atomicAdd(&a.gP[m * a.total + g0], v);
    }
}

// ---------------------------------------------------------------- MHD (residual VJP)
// Primitives of an MHD cell: rho, v0, v1, v2, u, a, B0, B1, B2, psi.
constexpr int NPM = 10;

// Stencil state of an MHD source (the ghost rules of finish_cell): (x, y) is the centre
// of the stencil cell, for the slip wall's dipole field (internal_copy_then_reflect.d:
// 140-143: Bx, By of a slip-wall ghost with |x| < 0.4136 are the dipole's, constants).
__device__ void adj_load_mhd(const AdjArgs& a, const Src& s, double x, double y, double* c) {
    if (s.kind == SRC_INFLOW) {
        const InflowState& in = a.inflow[s.inflow];
        c[0] = in.rho; c[1] = in.vel[0]; c[2] = in.vel[1]; c[3] = in.vel[2]; c[4] = in.u; c[5] = in.a;
        c[6] = in.B[0]; c[7] = in.B[1]; c[8] = in.B[2]; c[9] = in.psi;
        return;
    }
    const long long g0 = s.blk->offset + s.c0;
    double e[NPM];
    for (int m = 0; m < NPM; ++m) e[m] = a.Pp[m * a.total + g0];
    for (int m = 0; m < NPM; ++m) c[m] = e[m];
    if (s.kind == SRC_EXTRAP1_G0 || s.kind == SRC_EXTRAP1_G1) {
        // extrapolate_copy.d:171-201: rho, u, v, B extrapolated; a and psi of the edge cell
        const long long g1 = s.blk->offset + s.c1;
        for (int m = 0; m < NPM; ++m) {
            if (m == 5 || m == 9) continue;
            const double f = a.Pp[m * a.total + g1];
            const double g0v = 2.0 * e[m] - f;
            c[m] = (s.kind == SRC_EXTRAP1_G0) ? g0v : 2.0 * g0v - e[m];
        }
    } else if (s.kind == SRC_MIRROR) {
        c[1 + s.axis] = -c[1 + s.axis];   // B is not reflected (ghost_cell.d:56-67)
        if (x > -0.4136 && x < 0.4136) dipole_field(x, y, c[6], c[7]);
    } else if (s.kind == SRC_ROTATE) {
        const double* R = a.rot + 9 * s.inflow;
        for (int r = 0; r < 3; ++r) {
            c[1 + r] = R[3 * r] * e[1] + R[3 * r + 1] * e[2] + R[3 * r + 2] * e[3];
            c[6 + r] = R[3 * r] * e[6] + R[3 * r + 1] * e[7] + R[3 * r + 2] * e[8];
        }
    }
}

__device__ void adj_scatter_mhd(const AdjArgs& a, const Src& s, double x, double y, const double* gc) {
    if (s.kind == SRC_INFLOW) {
        for (int m = 0; m < NPM; ++m) atomicAdd(&a.gInflow[s.inflow * NPM + m], gc[m]);
        return;
    }
    const long long g0 = s.blk->offset + s.c0;
    if (s.kind == SRC_EXTRAP1_G0 || s.kind == SRC_EXTRAP1_G1) {
        const long long g1 = s.blk->offset + s.c1;
        const double ce = (s.kind == SRC_EXTRAP1_G0) ? 2.0 : 3.0, cf = (s.kind == SRC_EXTRAP1_G0) ? -1.0 : -2.0;
        for (int m = 0; m < NPM; ++m) {
            if (m == 5 || m == 9) { atomicAdd(&a.gP[m * a.total + g0], gc[m]); continue; }
            atomicAdd(&a.gP[m * a.total + g0], ce * gc[m]);
            atomicAdd(&a.gP[m * a.total + g1], cf * gc[m]);
        }
        return;
    }
    double g[NPM];
    for (int m = 0; m < NPM; ++m) g[m] = gc[m];
    if (s.kind == SRC_MIRROR) {
        g[1 + s.axis] = -g[1 + s.axis];
        if (x > -0.4136 && x < 0.4136) { g[6] = 0.0; g[7] = 0.0; }   // the dipole's constants
    } else if (s.kind == SRC_ROTATE) {
        const double* R = a.rot + 9 * s.inflow;
        for (int m = 0; m < 3; ++m) {
            g[1 + m] = R[m] * gc[1] + R[3 + m] * gc[2] + R[6 + m] * gc[3];
            g[6 + m] = R[m] * gc[6] + R[3 + m] * gc[7] + R[6 + m] * gc[8];
        }
    }
    for (int m = 0; m < NPM; ++m) atomicAdd(&a.gP[m * a.total + g0], g[m]);
}

// ---------------------------------------------------------------- the face sweep
// The transpose of reconstruction and flux along one direction, as tiles of cells of grid
// lines: one thread per cell, which also takes the face on its plus side.
//
// What bounds it: FP64 latency and issue, not bytes.  A thread per face would
// evaluate the limiter of each of its two cells forward, again in its reverse, and the two
// reverses (20 limiters forward and 10 reverse a face for Euler), hold the four stencil
// cells and their cotangents (168 registers, 12 warps per SM) and scatter all four with
// atomics (measured: 817 us a product's faces at 128x128x64 against 388).  Per cell there is
// one limiter a scalar, forward once and reverse once; the
// faces' states and the cotangents pass between neighbouring threads in shared memory, and
// a cell's own cotangent, summed over its faces in this direction, is added once:
//   1  primitives and W of the tile's cells into shared memory (ghosts by their rules)
//   2  per cell: reconstruction; minus-face states to shared memory, plus-face ones kept
//   3  per face: flux cotangent from W, reverse of the flux; the cotangent of the right
//      state goes to the next cell
//   4  per cell: reverse of the limiter: cotangents of the cells before, at and after it
//   5  per cell: their sum, added to gP (atomically: the three directions and the tiles'
//      ends meet there)
// Along i a tile is 256 (MHD 192) consecutive slots of the block's lines laid end to end, each with
// its two ghosts on either side; along j and k it is 32 lines (lanes, i fastest, so global
// accesses are coalesced) by 8 (MHD 6) cells.  Neighbouring tiles share their end cells: each adds
// the part of the faces it owns (all but the last slot's, or the last cell's).
#ifndef GDFV_ADJ_J
#define GDFV_ADJ_J 8
#endif
// MHD: 6 layers, 2 CTAs of 192 threads at 168 registers (0.4 KB of spills): 272 us a product
// on Orszag-Tang 256x256x4 and 251 us at 64^3.  Without the faces' range tests 269 / 249, against
// 298 / 263 with 8 layers at 128 registers, 292 / 253 with 4 layers at 3 CTAs and 342 / 262
// with 12 at one.  Euler: 8
// layers, 2 CTAs at 128 registers 454 us at 128x128x64; 6 or 5 layers at 96 registers 461 / 446
#ifndef GDFV_ADJ_J_MHD
#define GDFV_ADJ_J_MHD 6
#endif
template <bool MHD>
struct LineGeo {
    static constexpr int J = MHD ? GDFV_ADJ_J_MHD : GDFV_ADJ_J;   // cells along j or k per tile
    static constexpr int CTA = 32 * J;
    static constexpr int NPr = MHD ? NPM : NP;   // primitives of a cell
    static constexpr int NS = MHD ? 9 : 5;       // reconstructed scalars
    static constexpr int NQ = MHD ? 10 : 5;
    static constexpr int PAD = (J + 2) * 32;                  // cells with one halo layer on either side
    static constexpr int O_P = 0;                                  // [NS][PAD] reconstructed primitives
    static constexpr int O_W = O_P + NS * PAD;                     // [NQ][CTA] W (zero outside the block)
    static constexpr int O_M = O_W + NQ * CTA;                // [NS][CTA] minus-face state, then its cotangent, then g1
    static constexpr int O_R = O_M + NS * CTA;                // [NS][CTA] limiter reciprocal, then g2
    static constexpr int O_A = O_R + NS * CTA;                // Euler: [CTA] sound speed, [CTA] its cotangent from the left face
    static constexpr int O_IN = O_A + (MHD ? 0 : 2 * CTA);    // [J][NPr] inflow sums of the warps
    static constexpr int O_END = O_IN + J * NPr;
    static constexpr size_t bytes = sizeof(double) * (size_t)O_END;
    // place of primitive v among the reconstructed ones (MHD never reconstructs the sound speed)
    static __host__ __device__ constexpr int slot(int v) { return MHD && v > 5 ? v - 1 : v; }
    static __host__ __device__ constexpr int prim(int s) { return MHD && s >= 5 ? s + 1 : s; }
};

// The state of cell (i, j, k) of block B, inside it or a ghost beyond one face.
template <bool MHD, bool RARE>
__device__ __noinline__ void line_ghost_load(const AdjArgs& a, const BlockDesc& B, int i, int j, int k, double* c) {
    const Src s = adj_resolve<RARE>(a, B, i, j, k);
    if constexpr (MHD)
        adj_load_mhd(a, s, B.x0 + ((double)i + 0.5) * B.len[0], B.y0 + ((double)j + 0.5) * B.len[1], c);
    else
        adj_load<RARE>(a, s, c);
}
template <bool MHD, bool RARE>
__device__ __noinline__ void line_ghost_scatter(const AdjArgs& a, const BlockDesc& B, int i, int j, int k,
                                                const double* gc) {
    const Src s = adj_resolve<RARE>(a, B, i, j, k);
    if constexpr (MHD)
        adj_scatter_mhd(a, s, B.x0 + ((double)i + 0.5) * B.len[0], B.y0 + ((double)j + 0.5) * B.len[1], gc);
    else
        adj_scatter<RARE>(a, s, gc);
}

// Reverse of the flux of one face for Euler: left and right states in scalar order (normal
// and tangential velocity, rho, u) with the sound speeds, gF in the face's frame; gl, gr
// receive the cotangents in the same order, gaL, gaR those of the sound speeds.
template <int FLUX, bool FD>
__device__ __forceinline__ void euler_face_rev(const NumParams& P, const double* l, double aL, const double* r, double aR,
                                               const double* gF, double* gl, double& gaL, double* gr, double& gaR) {
    const double Rg = P.gas.R, Cvinv = P.gas.Cvinv;
    const FS L{l[3], l[3] * Rg * (l[4] * Cvinv), l[0], l[1], l[2], l[4], aL};
    const FS R{r[3], r[3] * Rg * (r[4] * Cvinv), r[0], r[1], r[2], r[4], aR};
    FS gL, gR;
    if constexpr (FLUX == FLUX_HLLC) hllc_vjp<FD>(P, L, R, gF, gL, gR);
    else ausmdv_vjp<FD>(P, L, R, gF, gL, gR);
    // p = rho R (u Cvinv)
    gl[0] = gL.u; gl[1] = gL.v; gl[2] = gL.w;
    gl[3] = gL.r + gL.p * Rg * (l[4] * Cvinv);
    gl[4] = gL.e + gL.p * l[3] * Rg * Cvinv;
    gaL = gL.a;
    gr[0] = gR.u; gr[1] = gR.v; gr[2] = gR.w;
    gr[3] = gR.r + gR.p * Rg * (r[4] * Cvinv);
    gr[4] = gR.e + gR.p * r[3] * Rg * Cvinv;
    gaR = gR.a;
}

// The same for MHD: scalars with the face-frame B and psi after them; gF in the order of
// the conserved quantities (face frame), psi and divB included.  F[divB] = (BxR - BxL)/2 and
// the GLM terms (fluxcalc.d:139-150, with the reference's third term added to F[xB] under
// glm_reference_indexing) with c_h held fixed, then hlle.
template <bool FD>
__device__ __forceinline__ void mhd_face_rev(const AdjArgs& a, const double* l, const double* r, const double* gF,
                                             double* gl, double* gr) {
    const NumParams& P = a.P;
    const double Rg = P.gas.R, Cvinv = P.gas.Cvinv;
    const FSm L{l[3], l[3] * Rg * (l[4] * Cvinv), l[0], l[1], l[2], l[5], l[6], l[7], l[4]};
    const FSm R{r[3], r[3] * Rg * (r[4] * Cvinv), r[0], r[1], r[2], r[5], r[6], r[7], r[4]};
    FSm gL{}, gR{};
    gl[8] = gr[8] = 0.0;
    gR.Bx += 0.5 * gF[DIVB]; gL.Bx -= 0.5 * gF[DIVB];
    if (P.divergence_cleaning) {
        const double ch = a.chd ? a.chd[0] : a.c_h;
        const double gt3 = P.glm_reference_indexing ? gF[XB] : gF[ZB];
        const double gpa = gF[XB] + gF[YB] + gt3;
        gR.Bx -= 0.5 * ch * gF[XB]; gL.Bx += 0.5 * ch * gF[XB];
        gR.By -= 0.5 * ch * gF[YB]; gL.By += 0.5 * ch * gF[YB];
        gR.Bz -= 0.5 * ch * gt3; gL.Bz += 0.5 * ch * gt3;
        gl[8] += 0.5 * gpa; gr[8] += 0.5 * gpa;
        const double gps = gF[PSI] * ch * ch;
        gL.Bx += 0.5 * gps; gR.Bx += 0.5 * gps;
        gr[8] -= 0.5 * gF[PSI] * ch; gl[8] += 0.5 * gF[PSI] * ch;   // gps / (2 c_h)
    }
    hlle_mhd_vjp<FD>(P, L, R, gF, gL, gR);
    auto back = [&](const FSm& S, const FSm& gS, double* g) {
        g[0] = gS.u; g[1] = gS.v; g[2] = gS.w;
        g[3] = gS.r + gS.p * Rg * (S.e * Cvinv);   // p = rho R (u Cvinv)
        g[4] = gS.e + gS.p * S.r * Rg * Cvinv;
        g[5] = gS.Bx; g[6] = gS.By; g[7] = gS.Bz;
    };
    back(L, gL, gl);
    back(R, gR, gr);
}

// place (prim slot) of scalar s of direction D: face-frame velocity, rho, u, face-frame B, psi
template <int D, bool MHD>
__device__ constexpr int scalar_slot(int s) {
    return s < 3 ? 1 + (D + s) % 3 : s == 3 ? 0 : s == 4 ? 4 : s < 8 ? LineGeo<MHD>::slot(6 + (D + s - 5) % 3) : 8;
}
template <int N>
struct Scalars { double q[N]; };
// Phase 2 of a cell whose limiters are out of the branch-free reciprocals' range (differences of
// 1e45 a cell length and more, infinities, NaN): with divisions.  The plus-face states are
// returned.
template <int D, bool MHD, bool RARE>
__device__ __noinline__ Scalars<LineGeo<MHD>::NS> line_recon_out_of_range(const NumParams& P, CellWeights w,
                                                                          const double* cell, double* minus,
                                                                          double* recips) {
    using G = LineGeo<MHD>;
    constexpr int step = D == 0 ? 1 : 32;
    Scalars<G::NS> plus;
    unsigned top = 0u;
#pragma unroll
    for (int s = 0; s < G::NS; ++s) {
        const double* v = cell + scalar_slot<D, MHD>(s) * G::PAD;
        double qm, rd = 0.0;
        if (s == 8 && MHD && !P.divergence_cleaning) plus.q[s] = qm = v[0];
        else cell_recon<RARE, false>(P, w, v[-step], v[0], v[step], qm, plus.q[s], rd, top);
        minus[s * G::CTA] = qm;
        recips[s * G::CTA] = rd;
    }
    return plus;
}

// Cotangent of a face's flux in its frame, from W of the cells to the left and right (at wl and wr).
template <int D, bool MHD>
__device__ __forceinline__ void face_cotangent(const double* wl, const double* wr, double AVl, double AVr, double* gF) {
    constexpr int T = LineGeo<MHD>::CTA;
#pragma unroll
    for (int q = 0; q < LineGeo<MHD>::NQ; ++q) {
        // momentum and B components in the order normal, tangents
        const int qg = q >= 1 && q <= 3 ? 1 + (D + q - 1) % 3 : (MHD && q >= 5 && q <= 7 ? 5 + (D + q - 5) % 3 : q);
        gF[q] = AVr * wr[qg * T] - AVl * wl[qg * T];
    }
}
// Phase 3 of a face whose states l and r (minus-face state of the cell to the right, replaced by
// its cotangent) are out of the branch-free reciprocals' range: with divisions.  The cotangents of
// l and, after them, of its sound speed are returned; sa: the sound speeds of the cells.  It reads W
// and r again: handed over in registers they cost a product 4 to 5 us (hllc 470 against 465,
// MHD 277 against 272).
template <int D, bool MHD, int FLUX>
__device__ __noinline__ Scalars<LineGeo<MHD>::NS + 1> line_face_out_of_range(const AdjArgs& a, Scalars<LineGeo<MHD>::NS> l,
                                                                             double AVl, double AVr, const double* wl,
                                                                             double* minus, double* sa) {
    using G = LineGeo<MHD>;
    constexpr int step = D == 0 ? 1 : 32;
    Scalars<G::NS + 1> out;
    double gF[G::NQ], r[G::NS], gr[G::NS];
    face_cotangent<D, MHD>(wl, wl + step, AVl, AVr, gF);
#pragma unroll
    for (int s = 0; s < G::NS; ++s) r[s] = minus[s * G::CTA];
    out.q[G::NS] = 0.0;
    if constexpr (MHD)
        mhd_face_rev<false>(a, l.q, r, gF, out.q, gr);
    else
        euler_face_rev<FLUX, false>(a.P, l.q, sa[0], r, sa[step], gF, out.q, out.q[G::NS], gr, sa[G::CTA + step]);
#pragma unroll
    for (int s = 0; s < G::NS; ++s) minus[s * G::CTA] = gr[s];
    return out;
}
// flux_in_range of the states l and r of a face in scalar order
template <int FLUX>
__device__ __forceinline__ bool face_in_range(const GasParams& gas, const double* l, double aL, const double* r, double aR) {
    const double pL = l[3] * gas.R * (l[4] * gas.Cvinv), pR = r[3] * gas.R * (r[4] * gas.Cvinv);
    return flux_in_range<FLUX>(l[3], pL, aL, l, l + 5, r[3], pR, aR, r, r + 5);
}

template <int D, bool MHD, int FLUX, bool RARE>
__device__ __forceinline__ void line_tile(const AdjArgs& a, unsigned tile, double* sm) {
    using G = LineGeo<MHD>;
    constexpr int NS = G::NS, NQ = G::NQ, NPr = G::NPr, T = G::CTA, PAD = G::PAD, LINE_J = G::J;
    constexpr int ax0 = D, ax1 = (D + 1) % 3, ax2 = (D + 2) % 3;
    constexpr int step = D == 0 ? 1 : 32;   // to the next cell along D, in shared memory
    double* SP = sm + G::O_P;
    double* SW = sm + G::O_W;
    double* SM = sm + G::O_M;
    double* SR = sm + G::O_R;
    double* SA = sm + G::O_A;
    double* SIN = sm + G::O_IN;
    const NumParams& P = a.P;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int pv[9] = {scalar_slot<D, MHD>(0), scalar_slot<D, MHD>(1), scalar_slot<D, MHD>(2),
                           scalar_slot<D, MHD>(3), scalar_slot<D, MHD>(4), scalar_slot<D, MHD>(5),
                           scalar_slot<D, MHD>(6), scalar_slot<D, MHD>(7), scalar_slot<D, MHD>(8)};

    const long long* off = a.tile_off + D * (a.nblocks + 1);
    const int b = block_of_tile(off, a.nblocks, tile);
    const BlockDesc& B = a.blocks[b];
    const unsigned lt = (unsigned)((long long)tile - off[b]);
    const int n0 = B.n[0], n1 = B.n[1], nD = B.n[D];
    // this thread's cell: line l, index c along D (-2 .. nD + 1)
    int c, i, j, k;
    bool valid, first, last;   // first, last: the ends of the tile along D
    if (D == 0) {
        const unsigned long long x = (unsigned long long)lt * (T - 1) + (unsigned)tid;
        valid = x < (unsigned long long)(n0 + 4) * ((unsigned long long)n1 * B.n[2]);
        const unsigned xs = valid ? (unsigned)x : 0u, l = xs / (unsigned)(n0 + 4);
        c = (int)(xs - l * (unsigned)(n0 + 4)) - 2;
        i = c;
        k = (int)(l / (unsigned)n1);
        j = (int)(l - (unsigned)k * (unsigned)n1);
        first = tid == 0;
        last = tid == T - 1;
    } else {
        const unsigned lines = (unsigned)n0 * (unsigned)(D == 1 ? B.n[2] : n1), groups = (lines + 31) / 32;
        const unsigned m = lt / groups, l0 = (lt - m * groups) * 32 + lane, l = l0 < lines ? l0 : 0u;
        c = (int)m * (LINE_J - 1) - 1 + warp;
        valid = l0 < lines && c <= nD + 1;
        const int q = (int)(l / (unsigned)n0);
        i = (int)(l - (unsigned)q * (unsigned)n0);
        j = D == 1 ? c : q;
        k = D == 1 ? q : c;
        first = warp == 0;
        last = warp == LINE_J - 1;
    }
    const bool inside = valid && c >= 0 && c < nD;
    const bool active = valid && c >= -1 && c <= nD;          // cells with a face of the block
    const bool has_face = active && c < nD && !last;          // its plus face, when the tile owns it
    const bool has_left = active && c >= 0 && !first;         // its minus face is the tile's too
    const int pi = D == 0 ? tid + 1 : tid + 32;               // own cell in the padded arrays
    const int sD = D == 0 ? 1 : (D == 1 ? n0 : n0 * n1);
    const long long g = B.offset + (long long)(unsigned)(inside ? i + n0 * (j + n1 * k) : 0);
    const bool ends = active && (first || last);              // the tile's end cells also handle the next cell

    // ---------------- 1: primitives (the tile's cells and one beyond either end) and W
    if (inside) {
#pragma unroll
        for (int s = 0; s < NS; ++s) SP[s * PAD + pi] = a.Pp[G::prim(s) * a.total + g];
        if (!MHD) SA[tid] = a.Pp[5 * a.total + g];
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) SW[q * T + tid] = inside ? a.W[q * a.total + g] : 0.0;
    if ((valid && !inside) || ends) {
        const int e = first ? -1 : 1;
#pragma unroll 1
        for (int pass = inside ? 1 : 0; pass < (ends ? 2 : 1); ++pass) {
            const int d = pass ? e : 0;
            const int ce = c + d;
            double cp[NPr];
            if (ce >= 0 && ce < nD) {
                const long long ge = B.offset + (long long)(unsigned)((D == 0 ? ce : i) + n0 * ((D == 1 ? ce : j) + n1 * (D == 2 ? ce : k)));
#pragma unroll
                for (int m = 0; m < NPr; ++m) cp[m] = a.Pp[m * a.total + ge];
            } else {
                line_ghost_load<MHD, RARE>(a, B, D == 0 ? ce : i, D == 1 ? ce : j, D == 2 ? ce : k, cp);
            }
#pragma unroll
            for (int s = 0; s < NS; ++s) SP[s * PAD + pi + d * step] = cp[G::prim(s)];
            if (!MHD && pass == 0) SA[tid] = cp[5];
        }
    }
    __syncthreads();

    // ---------------- 2: reconstruction
    const CellWeights w = cell_weights<RARE>(B, D, active ? c : 0);
    const bool clean = !MHD || P.divergence_cleaning;
    double qp[NS];
    bool bad_p = false, bad_m = false;   // e4/onedinterp.d:44-74: the face takes the cell-centre state
    if (active) {
        double qm_r = 1.0, qm_u = 1.0;
        unsigned top = 0u;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            const double* v = SP + pv[s] * PAD + pi;
            double qm, rd = 0.0;
            if (s == 8 && !clean) qp[s] = qm = v[0];
            else cell_recon<RARE, true>(P, w, v[-step], v[0], v[step], qm, qp[s], rd, top);
            SM[s * T + tid] = qm;
            SR[s * T + tid] = rd;
            if (s == 3) qm_r = qm;
            if (s == 4) qm_u = qm;
        }
        if (!P.eps_in_range || !denominators_in_range(top)) {
            const Scalars<NS> again = line_recon_out_of_range<D, MHD, RARE>(P, w, SP + pi, SM + tid, SR + tid);
#pragma unroll
            for (int s = 0; s < NS; ++s) qp[s] = again.q[s];
            qm_r = SM[3 * T + tid];
            qm_u = SM[4 * T + tid];
        }
        bad_p = qp[4] <= 0.0 || qp[3] <= 0.0;
        bad_m = qm_u <= 0.0 || qm_r <= 0.0;
        if (bad_m) {
#pragma unroll
            for (int s = 0; s < NS; ++s) SM[s * T + tid] = SP[pv[s] * PAD + pi];
        }
        if (bad_p) {
#pragma unroll
            for (int s = 0; s < NS; ++s) qp[s] = SP[pv[s] * PAD + pi];
        }
    }
    __syncthreads();

    // ---------------- 3: flux of the plus face; qp becomes its cotangent
    double ga = 0.0;
    if (has_face) {
        // cotangent of the face flux: F enters R of the right cell with +A/V and of the left with -A/V
        double AVr = B.area[D] * B.vol_inv * a.w_scale, AVl = AVr;
        if (RARE && B.graded) {
            // graded: the face's area from its cells' lengths across it, each side's own volume
            const int ic[3] = {i + (D == 0), j + (D == 1), k + (D == 2)};
            double Lr[3], Ll[3];
            for (int d = 0; d < 3; ++d) {
                Lr[d] = B.glen[d][ic[d] + 2];
                Ll[d] = B.glen[d][ic[d] - (d == D) + 2];
            }
            const bool threeD = P.dims == 3;
            const double Af = threeD ? (D == 0 ? Lr[1] * Lr[2] : (D == 1 ? Lr[2] * Lr[0] : Lr[0] * Lr[1]))
                                     : (D == 0 ? Lr[1] : Lr[0]);
            AVr = Af * rcp(threeD ? Lr[0] * Lr[1] * Lr[2] : Lr[0] * Lr[1]) * a.w_scale;
            AVl = Af * rcp(threeD ? Ll[0] * Ll[1] * Ll[2] : Ll[0] * Ll[1]) * a.w_scale;
        }
        const int nb = tid + step;   // the cell to the right
        const int bface = c == -1 ? 2 * D : (c == nD - 1 ? 2 * D + 1 : -1);
        bool simple = false;
        if constexpr (RARE && !MHD) simple = bface >= 0 && B.bc_type[bface] == BC_SIMPLE_FLUX;
        if constexpr (RARE && !MHD) {
            if (simple) {
                // OutFlowBC_SimpleFlux (boundary_flux_effect.d:504-645): the boundary face's flux is
                // the interior cell's outflow flux, or only its pressure on a closed face
                const int at = pi + ((bface & 1) ? 0 : step);
                double gF[NQ];
                face_cotangent<D, MHD>(SW + tid, SW + nb, AVl, AVr, gF);
                double gg[5] = {gF[MASS], 0.0, 0.0, 0.0, gF[TOTENERGY]}, cs[6], gs[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
                gg[1 + ax0] = gF[1]; gg[1 + ax1] = gF[2]; gg[1 + ax2] = gF[3];
                for (int s = 0; s < 5; ++s) cs[s] = SP[s * PAD + at];
                cs[5] = 0.0;
                simple_flux_vjp<D>(P, cs, (bface & 1) ? 1 : -1, gg, gs);
                const long long gi = B.offset + (long long)(unsigned)(i + n0 * (j + n1 * k) + ((bface & 1) ? 0 : sD));
                for (int m = 0; m < 5; ++m) atomicAdd(&a.gP[m * a.total + gi], gs[m]);
#pragma unroll
                for (int s = 0; s < NS; ++s) { qp[s] = 0.0; SM[s * T + nb] = 0.0; }
                SA[T + nb] = 0.0;
            }
        }
        if (!simple) {
            double r[NS];
#pragma unroll
            for (int s = 0; s < NS; ++s) r[s] = SM[s * T + nb];
            if (face_in_range<FLUX>(P.gas, qp, MHD ? 1.0 : SA[tid], r, MHD ? 1.0 : SA[nb])) {
                double gF[NQ], gl[NS], gr[NS];
                face_cotangent<D, MHD>(SW + tid, SW + nb, AVl, AVr, gF);
                if constexpr (MHD)
                    mhd_face_rev<true>(a, qp, r, gF, gl, gr);
                else
                    euler_face_rev<FLUX, true>(P, qp, SA[tid], r, SA[nb], gF, gl, ga, gr, SA[T + nb]);
#pragma unroll
                for (int s = 0; s < NS; ++s) { qp[s] = gl[s]; SM[s * T + nb] = gr[s]; }
            } else {
                Scalars<NS> l;
#pragma unroll
                for (int s = 0; s < NS; ++s) l.q[s] = qp[s];
                const Scalars<NS + 1> g = line_face_out_of_range<D, MHD, FLUX>(a, l, AVl, AVr, SW + tid, SM + nb, SA + tid);
#pragma unroll
                for (int s = 0; s < NS; ++s) qp[s] = g.q[s];
                ga = g.q[NS];
            }
        }
    } else {
#pragma unroll
        for (int s = 0; s < NS; ++s) qp[s] = 0.0;
    }
    __syncthreads();

    // ---------------- 4: reverse of the limiter; the cotangents of the cells before and after
    // the own one go to shared memory, the own one's stays
    double gc[NPr];
#pragma unroll
    for (int m = 0; m < NPr; ++m) gc[m] = 0.0;
    if (active) {
        if (!MHD) gc[5] = ga + (has_left ? SA[T + tid] : 0.0);
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            const double* v = SP + pv[s] * PAD + pi;
            double gp = qp[s], gm = has_left ? SM[s * T + tid] : 0.0, g0 = 0.0, g1 = 0.0, g2 = 0.0;
            if (bad_p) { g0 += gp; gp = 0.0; }
            if (bad_m) { g0 += gm; gm = 0.0; }
            if (s == 8 && !clean) g0 += gp + gm;
            else cell_recon_rev<RARE>(P, w, v[-step], v[0], v[step], SR[s * T + tid], gp, gm, g1, g0, g2);
            SM[s * T + tid] = g1;
            SR[s * T + tid] = g2;
            gc[G::prim(pv[s])] = g0;
        }
    }
    __syncthreads();

    // ---------------- 5: the cell's sum; ghosts pass it on by their rules
    const bool from_left = valid && !first && c >= 0 && c - 1 <= nD;       // the cells before and after that
    const bool from_right = valid && !last && c + 1 <= nD;                 // were active in this tile
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        const int m = G::prim(pv[s]);
        if (from_left) gc[m] += SR[s * T + tid - step];
        if (from_right) gc[m] += SM[s * T + tid + step];
    }
    if (inside) {
#pragma unroll
        for (int m = 0; m < NPr; ++m)
            if (!MHD || m != 5) atomicAdd(&a.gP[m * a.total + g], gc[m]);
    }
    // the tile's ends and the ghosts; inflow ghosts (one state a face) are summed over the tile first
    double vin[NPr];
    bool in = false;
    int side = 0;
    if ((valid && !inside && (active || from_left || from_right)) || ends) {
        const int e = first ? -1 : 1;
#pragma unroll 1
        for (int pass = inside ? 1 : 0; pass < (ends ? 2 : 1); ++pass) {
            const int ce = c + (pass ? e : 0);
            if (pass) {
                if (!MHD) gc[5] = 0.0;
#pragma unroll
                for (int s = 0; s < NS; ++s) gc[G::prim(pv[s])] = (first ? SM : SR)[s * T + tid];
            }
            if (ce >= 0 && ce < nD) {
                const long long ge = B.offset + (long long)(unsigned)((D == 0 ? ce : i) + n0 * ((D == 1 ? ce : j) + n1 * (D == 2 ? ce : k)));
#pragma unroll
                for (int m = 0; m < NPr; ++m)
                    if (m != 5) atomicAdd(&a.gP[m * a.total + ge], gc[m]);
            } else {
                side = ce < 0 ? 0 : 1;
                if (B.bc_type[2 * D + side] == BC_INFLOW) {
#pragma unroll
                    for (int m = 0; m < NPr; ++m) vin[m] = (in ? vin[m] : 0.0) + gc[m];
                    in = true;
                } else {
                    double t[NPr];   // (a copy, so that gc itself stays in registers)
#pragma unroll
                    for (int m = 0; m < NPr; ++m) t[m] = gc[m];
                    line_ghost_scatter<MHD, RARE>(a, B, D == 0 ? ce : i, D == 1 ? ce : j, D == 2 ? ce : k, t);
                }
            }
        }
    }
    if (B.bc_type[2 * D] == BC_INFLOW || B.bc_type[2 * D + 1] == BC_INFLOW) {
#pragma unroll 1
        for (int sd = 0; sd < 2; ++sd) {
            if (!__syncthreads_or(in && side == sd)) continue;
#pragma unroll
            for (int m = 0; m < NPr; ++m) {
                double v = in && side == sd ? vin[m] : 0.0;
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0) SIN[warp * NPr + m] = v;
            }
            __syncthreads();
            if (tid < NPr) {
                double v = 0.0;
                for (int wv = 0; wv < T / 32; ++wv) v += SIN[wv * NPr + tid];
                atomicAdd(&a.gInflow[B.bc_inflow[2 * D + sd] * NPr + tid], v);
            }
        }
    }
}

// All tiles of the three directions in one launch: CTAs [0, nb0) take the i lines,
// [nb0, nb0 + nb1) the j lines, the rest the k lines.
#ifndef GDFV_ADJ_MINB
#define GDFV_ADJ_MINB 2
#endif
#ifndef GDFV_ADJ_MINB_MHD
#define GDFV_ADJ_MINB_MHD 2
#endif
template <bool MHD, int FLUX, bool RARE>
__global__ void __launch_bounds__(LineGeo<MHD>::CTA, MHD ? GDFV_ADJ_MINB_MHD : GDFV_ADJ_MINB)
    adj_lines_kernel(const __grid_constant__ AdjArgs a, unsigned nb0, unsigned nb1) {
    extern __shared__ double smem_lines[];
    const unsigned bid = blockIdx.x;
    if (bid < nb0) line_tile<0, MHD, FLUX, RARE>(a, bid, smem_lines);
    else if (bid < nb0 + nb1) line_tile<1, MHD, FLUX, RARE>(a, bid - nb0, smem_lines);
    else line_tile<2, MHD, FLUX, RARE>(a, bid - nb0 - nb1, smem_lines);
}

// Tiles of one direction of a block (line_tile's decomposition).
template <bool MHD>
long long line_tiles_of(const int* n, int D) {
    constexpr int J = LineGeo<MHD>::J, T = LineGeo<MHD>::CTA;
    if (D == 0) return ((long long)(n[0] + 4) * n[1] * n[2] - 1 + T - 2) / (T - 1);
    const long long lines = (long long)n[0] * (D == 1 ? n[2] : n[1]);
    return (lines + 31) / 32 * ((n[D] + 1 + J - 2) / (J - 1));
}
long long line_tiles(bool mhd, const int* n, int D) { return mhd ? line_tiles_of<true>(n, D) : line_tiles_of<false>(n, D); }

template <bool MHD, int FLUX, bool RARE>
cudaError_t launch_lines_of(const AdjArgs& a, const unsigned* nb, cudaStream_t s) {
    using G = LineGeo<MHD>;
    auto* kernel = adj_lines_kernel<MHD, FLUX, RARE>;
    // the attribute is the device's: set for every launch (a host-side table look-up)
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::bytes);
    if (e != cudaSuccess) return e;
    kernel<<<nb[0] + nb[1] + nb[2], G::CTA, G::bytes, s>>>(a, nb[0], nb[1]);
    return cudaGetLastError();
}

// The face sweep of the context's flux calculator, with the rare rules when some exchange
// rotates, some face is an outflow boundary of its own, the limiter is lmr's or a block graded.
cudaError_t launch_lines(const AdjArgs& a, int flux, const unsigned* nb, cudaStream_t s) {
    const bool rare = a.P.rotating || a.P.outflow_bcs || a.P.lmr_epsilon || a.P.graded;
    if (a.P.mhd)
        return rare ? launch_lines_of<true, FLUX_HLLE, true>(a, nb, s) : launch_lines_of<true, FLUX_HLLE, false>(a, nb, s);
    if (flux == FLUX_HLLC)
        return rare ? launch_lines_of<false, FLUX_HLLC, true>(a, nb, s) : launch_lines_of<false, FLUX_HLLC, false>(a, nb, s);
    return rare ? launch_lines_of<false, FLUX_AUSMDV, true>(a, nb, s) : launch_lines_of<false, FLUX_AUSMDV, false>(a, nb, s);
}

// MHD decode (e4/fvcell.d:586-822): the ten primitives of each cell, gP cleared.
__device__ __forceinline__ void decode_cell_mhd(const AdjArgs& a, long long g) {
    double u[10];
    for (int q = 0; q < 10; ++q) u[q] = a.U[q * a.total + g];
    if (a.mode == 1 && a.chd) {
        // the corrector's stencils read the predictor state with psi damped, U1' = D U1
        // (D: psi times the step's damping factor), and its cotangent is D lam
        const double damp = a.chd[1];
        u[PSI] *= damp;
        a.lam[PSI * a.total + g] *= damp;
    }
    Prim<double> s;
    double p, T;
    decode(a.P, u, s, p, T);
    const double v[NPM] = {s.rho, s.v[0], s.v[1], s.v[2], s.u, s.a, s.B[0], s.B[1], s.B[2], s.psi};
    for (int m = 0; m < NPM; ++m) { a.Pp[m * a.total + g] = v[m]; a.gP[m * a.total + g] = 0.0; }
}

__global__ void adj_decode_mhd_kernel(AdjArgs a) {
    const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (g < a.total) decode_cell_mhd(a, g);
}

// gU = (dP/dU)^T gP for the MHD decode: u = (E - |B|^2/2)/rho - |v|^2/2, B and psi
// copied, a = sqrt(gamma R u / Cv); divB does not enter the primitives.  The modes
// of back_cell (the predictor-corrector adjoint's lam and b updates) over ten
// conserved quantities.
__device__ __forceinline__ void back_cell_mhd(const AdjArgs& a, long long g) {
    double U[10], gp[NPM];
    for (int q = 0; q < 10; ++q) U[q] = a.U[q * a.total + g];
    for (int m = 0; m < NPM; ++m) gp[m] = a.gP[m * a.total + g];
    const double rho = U[MASS], dinv = 1.0 / rho;
    const double v0 = U[XMOM] * dinv, v1 = U[YMOM] * dinv, v2 = U[ZMOM] * dinv;
    const double rE = U[TOTENERGY] - 0.5 * (U[XB] * U[XB] + U[YB] * U[YB] + U[ZB] * U[ZB]);
    const double u = rE * dinv - 0.5 * (v0 * v0 + v1 * v1 + v2 * v2);
    const double gR = a.P.gas.gamma * a.P.gas.R;
    const double aa = sqrt(gR * u * a.P.gas.Cvinv);
    const double gu = gp[4] + gp[5] * gR * a.P.gas.Cvinv / (2.0 * aa);
    const double gv0 = gp[1] - gu * v0, gv1 = gp[2] - gu * v1, gv2 = gp[3] - gu * v2;
    const double gdinv = gu * rE + gv0 * U[XMOM] + gv1 * U[YMOM] + gv2 * U[ZMOM];
    double r[10];
    r[MASS] = gp[0] - gdinv * dinv * dinv;
    r[XMOM] = gv0 * dinv; r[YMOM] = gv1 * dinv; r[ZMOM] = gv2 * dinv;
    r[TOTENERGY] = gu * dinv;
    r[XB] = gp[6] - gu * dinv * U[XB];
    r[YB] = gp[7] - gu * dinv * U[YB];
    r[ZB] = gp[8] - gu * dinv * U[ZB];
    r[PSI] = gp[9];
    r[DIVB] = 0.0;
    if (a.mode == 0) {
        for (int q = 0; q < 10; ++q) a.gU[q * a.total + g] = r[q];
    } else if (a.mode == 1) {
        if (a.chd) r[PSI] *= a.chd[1];   // mu is the cotangent of U1' = D U1: D mu is U1's
        for (int q = 0; q < 10; ++q) {
            const double l = a.lam[q * a.total + g];
            a.bbuf[q * a.total + g] = 0.5 * a.dt * l + a.dt * r[q];
            a.lam[q * a.total + g] = l + r[q];
        }
    } else {
        for (int q = 0; q < 10; ++q) a.lam[q * a.total + g] += r[q];
    }
}

__global__ void adj_back_mhd_kernel(AdjArgs a) {
    const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (g < a.total) back_cell_mhd(a, g);
}

__global__ void adj_back_decode_mhd_kernel(AdjArgs back, AdjArgs next) {
    const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (g >= back.total) return;
    back_cell_mhd(back, g);
    decode_cell_mhd(next, g);
}

// gU = (dP/dU)^T gP for P = decode(U) (e4/fvcell.d:586-822 with ideal_gas.d:98-139)
__device__ __forceinline__ void back_cell(const AdjArgs& a, long long g) {
    double U[5];
    for (int q = 0; q < 5; ++q) U[q] = a.U[q * a.total + g];
    double gp[NP];
    for (int m = 0; m < NP; ++m) gp[m] = a.gP[m * a.total + g];
    const double rho = U[0], dinv = 1.0 / rho;
    const double v0 = U[1] * dinv, v1 = U[2] * dinv, v2 = U[3] * dinv;
    const double u = U[4] * dinv - 0.5 * (v0 * v0 + v1 * v1 + v2 * v2);
    const double T = u * a.P.gas.Cvinv;
    const double gR = a.P.gas.gamma * a.P.gas.R;
    const double aa = sqrt(gR * T);
    double gu = gp[4] + gp[5] * gR * a.P.gas.Cvinv / (2.0 * aa);
    double gv0 = gp[1] - gu * v0, gv1 = gp[2] - gu * v1, gv2 = gp[3] - gu * v2;
    double gdinv = gu * U[4] + gv0 * U[1] + gv1 * U[2] + gv2 * U[3];
    const double r[5] = {gp[0] - gdinv * dinv * dinv, gv0 * dinv, gv1 * dinv, gv2 * dinv, gu * dinv};
    if (a.mode == 0) {
        for (int q = 0; q < 5; ++q) a.gU[q * a.total + g] = r[q];
    } else if (a.mode == 1) {
        // predictor-corrector adjoint, first product: r = mu = J(U1)^T (dt/2 lam)
        for (int q = 0; q < 5; ++q) {
            const double l = a.lam[q * a.total + g];
            a.bbuf[q * a.total + g] = 0.5 * a.dt * l + a.dt * r[q];
            a.lam[q * a.total + g] = l + r[q];
        }
    } else {
        // second product: r = J(U0)^T b
        for (int q = 0; q < 5; ++q) a.lam[q * a.total + g] += r[q];
    }
}


__global__ void adj_decode_back_kernel(AdjArgs a) {
    long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (g < a.total) back_cell(a, g);
}

// The reverse decode of one product and the decode of the next, in one pass per
// cell (the cell's cotangent gP is read, then cleared for the next product).
__global__ void adj_back_decode_kernel(AdjArgs back, AdjArgs next) {
    long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (g >= back.total) return;
    back_cell(back, g);
    decode_cell(next, g);
}

}  // namespace

}  // namespace gdfv

using namespace gdfv;

namespace {

// The forms the VJP, step and rollout adjoints take.
bool vjp_supported(int ctx, const AdjView& v) {
    if (!v.prepared) { adjoint_set_error(ctx, "call gdfv_prepare first"); return false; }
    if (v.mhd) {
        for (const BlockDesc& B : v.h_blocks)
            for (int f = 0; f < 6; ++f)
                if (B.bc_type[f] == BC_FIXED_P || B.bc_type[f] == BC_FIXED_PT) {
                    adjoint_set_error(ctx, "the MHD residual VJP does not take outflow_fixed_p boundaries");
                    return false;
                }
        return true;
    }
    if (v.flux != FLUX_AUSMDV && v.flux != FLUX_HLLC) {
        adjoint_set_error(ctx, "the adjoint supports flux_calculator=ausmdv or hllc (and hlle with MHD in "
                               "gdfv_residual_vjp)");
        return false;
    }
    return true;
}

// Scratch layout, np = 6 primitives (Euler) or 10 (MHD), nq conserved quantities:
// P [np][total] | gP [np][total] | b [nq][total] | tile offsets [3][nblocks+1] | inflow
// cotangents [ninflow][np].  Tile offsets are uploaded once per allocation.
cudaError_t vjp_setup(const AdjView& v, AdjArgs& a, std::vector<long long>& off) {
    const long long total = v.total;
    const long long np = v.mhd ? NPM : NP, nq = v.mhd ? 10 : 5;
    const long long need = (2 * np + nq) * total + 3 * (v.nblocks + 1) + np * (long long)v.ninflow + 8;
    cudaError_t e = cudaSuccess;
    if (*v.scratch_n < need) {
        if (*v.scratch) cudaFree(*v.scratch);
        *v.scratch = nullptr;
        *v.scratch_n = 0;
        *v.scratch_ready = 0;
        e = context_malloc(v.ctx, (void**)v.scratch, sizeof(double) * need);
        if (e != cudaSuccess) return e;
        *v.scratch_n = need;
    }
    double* base = *v.scratch;
    a = AdjArgs{};
    a.blocks = v.d_blocks;
    a.inflow = v.d_inflow;
    a.rot = v.d_rot;
    a.Pp = base;
    a.gP = base + np * total;
    a.bbuf = base + 2 * np * total;
    a.tile_off = reinterpret_cast<const long long*>(base + (2 * np + nq) * total);
    a.gInflow = base + (2 * np + nq) * total + 3 * (v.nblocks + 1);
    a.chd_slot = a.gInflow + np * v.ninflow;   // two doubles of the tail
    a.c_h = v.c_h;
    a.total = total;
    a.nblocks = v.nblocks;
    a.P = v.P;
    a.w_scale = 1.0;
    off.assign(3 * (v.nblocks + 1), 0);
    for (int d = 0; d < 3; ++d) {
        for (int b = 0; b < v.nblocks; ++b) {
            const BlockDesc& B = v.h_blocks[b];
            // 2D blocks have no k faces (the residual sums four faces)
            const long long nt = (v.dims == 2 && d == 2) ? 0 : line_tiles(v.mhd, B.n, d);
            off[d * (v.nblocks + 1) + b + 1] = off[d * (v.nblocks + 1) + b] + nt;
        }
    }
    if (!*v.scratch_ready) {
        e = cudaMemcpy((void*)a.tile_off, off.data(), sizeof(long long) * off.size(), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) return e;
        *v.scratch_ready = 1;
    }
    return cudaSuccess;
}

// The MHD residual VJP: decode, the line tiles of the three directions, reverse decode.
cudaError_t enqueue_vjp_mhd(const AdjView& v, const AdjArgs& a, const std::vector<long long>& off) {
    const int nt = 256;
    const unsigned nb_cells = (unsigned)((v.total + nt - 1) / nt);
    adj_decode_mhd_kernel<<<nb_cells, nt, 0, v.stream>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    unsigned nb[3];
    for (int d = 0; d < 3; ++d) nb[d] = (unsigned)off[d * (v.nblocks + 1) + v.nblocks];
    if ((e = launch_lines(a, v.flux, nb, v.stream)) != cudaSuccess) return e;
    adj_back_mhd_kernel<<<nb_cells, nt, 0, v.stream>>>(a);
    return cudaGetLastError();
}

// decode, the line tiles of the three directions (cotangents added to gP) and the reverse decode.
cudaError_t enqueue_vjp(const AdjView& v, const AdjArgs& a, const std::vector<long long>& off) {
    const int nt = 256;
    const long long total = v.total;
    adj_decode_kernel<<<(unsigned)((total + nt - 1) / nt), nt, 0, v.stream>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) {
        unsigned nb[3];
        for (int d = 0; d < 3; ++d) nb[d] = (unsigned)off[d * (v.nblocks + 1) + v.nblocks];
        e = launch_lines(a, v.flux, nb, v.stream);
    }
    if (e == cudaSuccess) {
        adj_decode_back_kernel<<<(unsigned)((total + nt - 1) / nt), nt, 0, v.stream>>>(a);
        e = cudaGetLastError();
    }
    return e;
}

}  // namespace

extern "C" int gdfv_residual_vjp(int ctx, const double* U_dev, const double* W_dev, double* G_dev,
                                 double* g_inflow_host) {
    AdjView v;
    if (!adjoint_view(ctx, &v)) return GDFV_ERR_ARG;
    if (!vjp_supported(ctx, v)) return v.prepared ? GDFV_ERR_ARG : GDFV_ERR_STATE;
    if (!U_dev || !W_dev || !G_dev) { adjoint_set_error(ctx, "null pointer"); return GDFV_ERR_ARG; }
    AdjArgs a;
    std::vector<long long> off;
    cudaError_t e = vjp_setup(v, a, off);
    a.U = U_dev;
    a.W = W_dev;
    a.gU = G_dev;
    a.mode = 0;
    const int np = v.mhd ? NPM : NP;
    if (e == cudaSuccess && v.ninflow > 0) e = cudaMemsetAsync(a.gInflow, 0, sizeof(double) * np * v.ninflow, v.stream);
    if (e == cudaSuccess) e = v.mhd ? enqueue_vjp_mhd(v, a, off) : enqueue_vjp(v, a, off);
    if (e == cudaSuccess && g_inflow_host && v.ninflow > 0)
        e = cudaMemcpyAsync(g_inflow_host, a.gInflow, sizeof(double) * np * v.ninflow, cudaMemcpyDeviceToHost, v.stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(v.stream);
    if (e != cudaSuccess) { adjoint_set_error(ctx, cudaGetErrorString(e)); return GDFV_ERR_CUDA; }
    return GDFV_OK;
}

namespace {

// A chain of products: the reverse decode of each product runs fused with the
// decode of the next one (adj_back_decode_kernel, or its MHD form); finish() ends
// the chain.
struct VjpChain {
    bool pending = false;
    AdjArgs back{};
    cudaError_t product(const AdjView& v, const AdjArgs& a, const std::vector<long long>& off) {
        const int nt = 256;
        const unsigned nb_cells = (unsigned)((v.total + nt - 1) / nt);
        if (v.mhd) {
            if (pending) adj_back_decode_mhd_kernel<<<nb_cells, nt, 0, v.stream>>>(back, a);
            else adj_decode_mhd_kernel<<<nb_cells, nt, 0, v.stream>>>(a);
        } else {
            if (pending) adj_back_decode_kernel<<<nb_cells, nt, 0, v.stream>>>(back, a);
            else adj_decode_kernel<<<nb_cells, nt, 0, v.stream>>>(a);
        }
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) {
            unsigned nb[3];
            for (int d = 0; d < 3; ++d) nb[d] = (unsigned)off[d * (v.nblocks + 1) + v.nblocks];
            e = launch_lines(a, v.flux, nb, v.stream);
        }
        back = a;
        pending = true;
        return e;
    }
    cudaError_t finish(const AdjView& v) {
        if (!pending) return cudaSuccess;
        pending = false;
        const int nt = 256;
        const unsigned nb_cells = (unsigned)((v.total + nt - 1) / nt);
        if (v.mhd) adj_back_mhd_kernel<<<nb_cells, nt, 0, v.stream>>>(back);
        else adj_decode_back_kernel<<<nb_cells, nt, 0, v.stream>>>(back);
        return cudaGetLastError();
    }
};

// The adjoint of one predictor-corrector step, enqueued on v.stream:
// mu = J(U1)^T (dt/2 lam); b = dt/2 lam + dt mu; lam += mu; then lam += J(U0)^T b.
// MHD with cleaning: the step's c_h and psi damping factor are formed first from U0
// (as gdfv_run forms them at the step's start); the corrector evaluated R at U1 with
// psi damped, and damped psi again in U2:
//   U2 = D (U0 + dt/2 R(U0) + dt/2 R(D U1)),  U1 = U0 + dt R(U0),
// so lam' = D lam, mu = J(D U1)^T (dt/2 lam'), b = dt/2 lam' + dt D mu,
// lam <- lam' + D mu + J(U0)^T b (the mode-1 decode and reverse decode apply D).
cudaError_t enqueue_step_adjoint(int ctx, const AdjView& v, AdjArgs a, const std::vector<long long>& off,
                                 const double* U0, const double* U1, double dt, double* lam, VjpChain& chain) {
    a.chd = nullptr;
    if (v.mhd && v.P.divergence_cleaning) {
        cudaError_t e = enqueue_step_ch(ctx, v.stream, U0, dt, a.chd_slot);
        if (e != cudaSuccess) return e;
        a.chd = a.chd_slot;
    }
    a.lam = lam;
    a.dt = dt;
    a.U = U1;
    a.W = lam;
    a.w_scale = 0.5 * dt;
    a.mode = 1;
    cudaError_t e = chain.product(v, a, off);
    a.U = U0;
    a.W = a.bbuf;
    a.w_scale = 1.0;
    a.mode = 2;
    if (e == cudaSuccess) e = chain.product(v, a, off);
    return e;
}

}  // namespace

extern "C" int gdfv_step_adjoint(int ctx, const double* U0_dev, const double* U1_dev, double dt, double* lam_dev,
                                 double* g_inflow_dev) {
    AdjView v;
    if (!adjoint_view(ctx, &v)) return GDFV_ERR_ARG;
    if (!vjp_supported(ctx, v)) return v.prepared ? GDFV_ERR_ARG : GDFV_ERR_STATE;
    if (!U0_dev || !U1_dev || !lam_dev || (v.ninflow > 0 && !g_inflow_dev) || !(dt > 0.0)) {
        adjoint_set_error(ctx, "gdfv_step_adjoint needs U0, U1, lam (and g_inflow with inflow faces) and dt > 0");
        return GDFV_ERR_ARG;
    }
    if (v.mhd && v.P.divergence_cleaning) {   // the scan scratch of the step's c_h
        const int st = steps_dt_prepare(ctx);
        if (st) return st;
    }
    AdjArgs a;
    std::vector<long long> off;
    cudaError_t e = vjp_setup(v, a, off);
    if (v.ninflow > 0) a.gInflow = g_inflow_dev;
    VjpChain chain;
    if (e == cudaSuccess) e = enqueue_step_adjoint(ctx, v, a, off, U0_dev, U1_dev, dt, lam_dev, chain);
    if (e == cudaSuccess) e = chain.finish(v);
    if (e != cudaSuccess) { adjoint_set_error(ctx, cudaGetErrorString(e)); return GDFV_ERR_CUDA; }
    return GDFV_OK;
}

extern "C" int gdfv_rollout_adjoint(int ctx, const double* const* ckpt_dev, int n_ckpt, const double* dts, int nsteps,
                                    int checkpoint_every, double* const* work_dev, int last_ready, double* lam_dev,
                                    double* g_inflow_dev) {
    AdjView v;
    if (!adjoint_view(ctx, &v)) return GDFV_ERR_ARG;
    if (!vjp_supported(ctx, v)) return v.prepared ? GDFV_ERR_ARG : GDFV_ERR_STATE;
    const int K = checkpoint_every;
    if (!ckpt_dev || !dts || !work_dev || !lam_dev || (v.ninflow > 0 && !g_inflow_dev) || nsteps < 1 || K < 1 ||
        K > 64 || n_ckpt != (nsteps + K - 1) / K) {
        adjoint_set_error(ctx, "gdfv_rollout_adjoint: needs one checkpoint per segment of checkpoint_every (<= 64) "
                               "steps, 4*checkpoint_every work arrays, lam (and g_inflow with inflow faces)");
        return GDFV_ERR_ARG;
    }
    for (int m = 0; m < 4 * K; ++m)
        if (!work_dev[m]) { adjoint_set_error(ctx, "gdfv_rollout_adjoint: null work array"); return GDFV_ERR_ARG; }
    for (int m = 0; m < nsteps; ++m)
        if (!(dts[m] > 0.0)) { adjoint_set_error(ctx, "gdfv_rollout_adjoint: dt must be > 0"); return GDFV_ERR_ARG; }
    int st = steps_dt_prepare(ctx);
    if (st) return st;
    AdjArgs a;
    std::vector<long long> off;
    cudaError_t e = vjp_setup(v, a, off);
    if (v.ninflow > 0) a.gInflow = g_inflow_dev;
    cudaStream_t aux = context_aux_stream(ctx, 0);     // recomputation, lowest priority
    AdjView vh = v;                                    // adjoint sweep, highest priority
    vh.stream = context_aux_stream(ctx, 1);
    if (e == cudaSuccess && (!aux || !vh.stream)) e = cudaErrorNotReady;
    // Work arrays: two sets of (K states, K predictor states); segment s uses set
    // (nseg-1-s) % 2.  The recomputation of segment s-1 (aux stream) runs while the
    // adjoint of segment s (context stream) runs; events order the reuse of a set.
    cudaEvent_t start = nullptr, rec_done[2] = {nullptr, nullptr}, adj_done[2] = {nullptr, nullptr};
    for (cudaEvent_t* ev : {&start, &rec_done[0], &rec_done[1], &adj_done[0], &adj_done[1]})
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(ev, cudaEventDisableTiming);
    const int nseg = n_ckpt;
    auto seg_len = [&](int s) { return std::min(K, nsteps - s * K); };
    bool first = true;
    auto recompute = [&](int s, int p) -> cudaError_t {
        // the state after a segment's last step is the next checkpoint: not recomputed
        double* outs[64];
        const int len = seg_len(s);
        for (int m = 0; m < len; ++m) outs[m] = m < len - 1 ? work_dev[2 * K * p + m] : nullptr;
        cudaError_t r = enqueue_steps_dt(ctx, aux, ckpt_dev[s], outs, work_dev + 2 * K * p + K,
                                         dts + (size_t)s * K, len, first);
        first = false;
        if (r == cudaSuccess) r = cudaEventRecord(rec_done[p], aux);
        return r;
    };
    if (e == cudaSuccess) e = cudaEventRecord(start, v.stream);   // inputs written on the context stream
    if (e == cudaSuccess) e = cudaStreamWaitEvent(aux, start, 0);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(vh.stream, start, 0);
    VjpChain chain;
    // the last segment's states and predictor states may come from the forward pass
    if (e == cudaSuccess) e = last_ready ? cudaEventRecord(rec_done[0], aux) : recompute(nseg - 1, 0);
    for (int idx = 0; idx < nseg && e == cudaSuccess; ++idx) {
        const int s = nseg - 1 - idx, p = idx % 2, q = 1 - p;
        if (s >= 1) {
            if (idx >= 1) e = cudaStreamWaitEvent(aux, adj_done[q], 0);   // set q free again
            if (e == cudaSuccess) e = recompute(s - 1, q);
        }
        if (e == cudaSuccess) e = cudaStreamWaitEvent(vh.stream, rec_done[p], 0);
        double* const* outs = work_dev + 2 * K * p;
        double* const* preds = work_dev + 2 * K * p + K;
        for (int n = seg_len(s) - 1; n >= 0 && e == cudaSuccess; --n) {
            const double* U0 = n == 0 ? ckpt_dev[s] : outs[n - 1];
            e = enqueue_step_adjoint(ctx, vh, a, off, U0, preds[n], dts[(size_t)s * K + n], lam_dev, chain);
        }
        // each segment ends its chain, so that every reader of the set precedes adj_done
        if (e == cudaSuccess) e = chain.finish(vh);
        if (e == cudaSuccess) e = cudaEventRecord(adj_done[p], vh.stream);
    }
    if (e == cudaSuccess) {
        if (!first) st = steps_dt_status(ctx, aux);   // failure counters of the recomputed segments
        else e = cudaStreamSynchronize(aux);
        if (st == GDFV_OK && e == cudaSuccess) e = cudaStreamSynchronize(vh.stream);
    }
    for (cudaEvent_t ev : {start, rec_done[0], rec_done[1], adj_done[0], adj_done[1]})
        if (ev) cudaEventDestroy(ev);
    if (e != cudaSuccess) { adjoint_set_error(ctx, cudaGetErrorString(e)); return GDFV_ERR_CUDA; }
    return st;
}
