// Rate derivatives of one reaction at one point, from its DRxn record: shared
// by the derivative kernels (derivs.cu) and, for reactions without a
// pre-decoded form, by the quad ones (deriv_quad.cu).
#pragma once

#include <cuda_runtime.h>

#include "cg_math.cuh"
#include "rates_common.cuh"

namespace cg {
namespace {

constexpr double kLn10 = 2.302585092994045684;

struct DState {
    double* C;
    double* E;
    double* D;
    double* A;
    int64_t s;       // stride between species of C and E
    int64_t sd;      // and of D
};

__device__ __forceinline__ double arr_ln(double lnA, double b, double theta, const PointT& pt) {
    return fma(b, pt.lnT, lnA) - theta * pt.invT;
}
__device__ __forceinline__ double arr_dln(double b, double theta, const PointT& pt) {
    return fma(theta, pt.invT, b) * pt.invT;
}

// Forward rate constant of a falloff reaction and its derivatives:
// dlkf = d ln kf/dT at fixed M, gM = d ln kf/dM.
inline __device__ void falloff_d(int kind, int flags, const DRxn& R, const DFall& f, double x2, double M, const PointT& pt,
                          double& kf, double& dlkf, double& gM) {
    const double lkinf = arr_ln(R.lnA, R.b, R.theta, pt);
    const double lr = arr_ln(f.lnA0, f.b0, f.theta0, pt) - lkinf;
    const double Pr = cgm::cg_exp_clamped(lr) * M * (f.sgn0 * R.sgn);
    const double dlkinf = arr_dln(R.b, R.theta, pt);
    const double dlPr = arr_dln(f.b0, f.theta0, pt) - dlkinf;
    const double ipr = cgm::cg_rcp(1.0 + Pr);
    double lnF = 0.0, gpr = ipr, dlF_T = 0.0;
    if (kind == CG_TROE) {
        const double e3 = cgm::cg_exp_clamped(-pt.T * f.p[1]);
        const double e1 = cgm::cg_exp_clamped(-pt.T * f.p[3]);
        double Fc = fma(f.p[0], e3, f.p[2] * e1);
        double dFc = fma(-f.p[0] * f.p[1], e3, -f.p[2] * f.p[3] * e1);
        if (flags & CG_F_TROE_T2) {
            const double e2 = cgm::cg_exp_clamped(-x2 * pt.invT);
            Fc += e2;
            dFc = fma(x2 * pt.invT * pt.invT, e2, dFc);
        }
        const double lFc = cgm::cg_log10(Fc);
        const double u = fma(lr, 1.0 / kLn10, cgm::cg_log10(M)) + fma(-0.67, lFc, -0.4);
        const double nn = fma(-1.27, lFc, 0.75);
        const double den = fma(-0.14, u, nn);
        const double iden = cgm::cg_rcp(den);
        const double f1 = u * iden;
        const double q1 = cgm::cg_rcp(fma(f1, f1, 1.0));
        lnF = kLn10 * lFc * q1;
        const double dF_df1 = -2.0 * lFc * f1 * q1 * q1;
        const double dF_dlpr = dF_df1 * nn * iden * iden;
        const double df1_dlfc = (-0.67 * den + 1.1762 * u) * iden * iden;
        const double dF_dlfc = fma(dF_df1, df1_dlfc, q1);
        gpr = ipr + dF_dlpr;
        dlF_T = dF_dlfc * dFc * cgm::cg_rcp(Fc);
    } else if (kind == CG_SRI) {
        const double lp = fma(lr, 1.0 / kLn10, cgm::cg_log10(M));
        const double X = cgm::cg_rcp(fma(lp, lp, 1.0));
        const double eb = cgm::cg_exp_clamped(-f.p[1] * pt.invT);
        const double ec = cgm::cg_exp_clamped(-pt.T * f.p[2]);
        const double base = fma(f.p[0], eb, ec);
        const double dbase = fma(f.p[0] * f.p[1] * pt.invT * pt.invT, eb, -f.p[2] * ec);
        const double lb = cgm::cg_log(base);
        lnF = cgm::cg_log(f.p[3]) + fma(X, lb, x2 * pt.lnT);
        gpr = ipr - 2.0 * lp * X * X * lb / kLn10;
        dlF_T = fma(X, dbase * cgm::cg_rcp(base), x2 * pt.invT);
    }
    kf = R.sgn * cgm::cg_exp_clamped(lkinf + lnF) * (Pr * ipr);
    dlkf = fma(gpr, dlPr, dlkinf) + dlF_T;
    gM = gpr * cgm::cg_rcp(M);
}

// PLOG forward rate, d ln kf/dT and d ln kf/d ln P (plog.j2:4-38).
inline __device__ void plog_d(const DevMech& m, int row, double P, double lnP, const PointT& pt, double& kf, double& dlkf,
                       double& dlkf_lnP) {
    const int l0 = __ldg(m.plog_ptr + row), l1 = __ldg(m.plog_ptr + row + 1);
    int l = l0;
    while (l < l1 && !(P < __ldg(m.plog_p + l))) ++l;
    int la, lb;
    if (l == l0) la = lb = l0;
    else if (l == l1) la = lb = l1 - 1;
    else {
        la = l - 1;
        lb = l;
    }
    double k[2] = {0.0, 0.0}, d[2] = {0.0, 0.0};
    const int lev[2] = {la, lb};
    for (int s = 0; s < 2; ++s) {
        for (int t = __ldg(m.plog_tptr + lev[s]); t < __ldg(m.plog_tptr + lev[s] + 1); ++t) {
            const double4 c = m.plog_term[t];
            const double x = c.w * cgm::cg_exp_clamped(arr_ln(c.x, c.y, c.z, pt));
            k[s] += x;
            d[s] = fma(x, arr_dln(c.y, c.z, pt), d[s]);
        }
        d[s] *= cgm::cg_rcp(k[s]);
    }
    if (la == lb) {
        kf = k[0];
        dlkf = d[0];
        dlkf_lnP = 0.0;
        return;
    }
    const double a = __ldg(m.plog_lnp + la), b = __ldg(m.plog_lnp + lb);
    const double w = (lnP - a) / (b - a);
    const double kl = cgm::cg_log(k[0]), kh = cgm::cg_log(k[1]);
    kf = cgm::cg_exp_clamped(kl + (kh - kl) * w);
    dlkf = fma(w, d[1] - d[0], d[0]);
    dlkf_lnP = (kh - kl) / (b - a);
}

// One side of a reaction: species, coefficients (compact or general rows).
// NMAX = 3 holds the compact form only; its loops unroll, so the arrays stay
// in registers.
template <int NMAX>
struct SideT {
    int n;
    int sp[NMAX];
    double nu[NMAX];
};
using Side = SideT<16>;

__device__ __forceinline__ void load_sides3(const DRxn& R, SideT<3>& re, SideT<3>& pr) {
    re.n = R.nre;
    pr.n = R.npr;
#pragma unroll
    for (int j = 0; j < kMaxCompact; ++j) {
        re.sp[j] = slot_species(R.sp[j]);
        re.nu[j] = slot_nu(R.sp[j]);
        pr.sp[j] = slot_species(R.sp[3 + j]);
        pr.nu[j] = slot_nu(R.sp[3 + j]);
    }
}

__device__ __forceinline__ void load_sides(const DevMech& m, const DRxn& R, Side& re, Side& pr) {
    if (R.flags & kFCompact) {
        re.n = R.nre;
        pr.n = R.npr;
        for (int j = 0; j < kMaxCompact; ++j) {
            re.sp[j] = slot_species(R.sp[j]);
            re.nu[j] = slot_nu(R.sp[j]);
            pr.sp[j] = slot_species(R.sp[3 + j]);
            pr.nu[j] = slot_nu(R.sp[3 + j]);
        }
        return;
    }
    const int g = R.gen;
    const int r0 = __ldg(m.gen_rptr + g), r1 = __ldg(m.gen_rptr + g + 1);
    const int p0 = __ldg(m.gen_pptr + g), p1 = __ldg(m.gen_pptr + g + 1);
    re.n = min(r1 - r0, 16);
    pr.n = min(p1 - p0, 16);
    for (int j = 0; j < re.n; ++j) {
        re.sp[j] = __ldg(m.gen_sp + r0 + j);
        re.nu[j] = __ldg(m.gen_nu + r0 + j);
    }
    for (int j = 0; j < pr.n; ++j) {
        pr.sp[j] = __ldg(m.gen_sp + p0 + j);
        pr.nu[j] = __ldg(m.gen_nu + p0 + j);
    }
}

__device__ __forceinline__ double powi(double x, double nu) {
    if (nu == 1.0) return x;
    if (nu == 2.0) return x * x;
    if (nu == 3.0) return x * x * x;
    return pow(x, nu);
}

// d(c^nu)/dc
__device__ __forceinline__ double dpowi(double x, double nu) {
    if (nu == 1.0) return 1.0;
    if (nu == 2.0) return 2.0 * x;
    if (nu == 3.0) return 3.0 * x * x;
    return nu * pow(x, nu - 1.0);
}

// Derivative of prod_i c_i^nu_i with respect to factor j (product of the others).
template <int NMAX>
__device__ __forceinline__ double dprod(const SideT<NMAX>& s, const double* c, int j) {
    double p = dpowi(c[j], s.nu[j]);
#pragma unroll(NMAX == 3 ? 3 : 1)
    for (int i = 0; i < NMAX; ++i)
        if (i < s.n && i != j) p *= powi(c[i], s.nu[i]);
    return p;
}

// Rate of progress of reaction r at one point and its derivatives: dqdT at
// fixed C, dqdM (three-body and falloff), and dq/dC_j over the reaction's own
// species (dsp[0..nd)); re/pr are its sides.  State C, EGp and dE are read
// with stride st.s.
template <int NMAX>
struct RxnGradT {
    int kind;
    bool usesM;
    double qnet, dqdT, dqdM, dlkf_lnP;
    int nd;
    int dsp[2 * NMAX];
    double dqc[2 * NMAX];
};
using RxnGrad = RxnGradT<16>;

// The rate constants of reaction r at one point: kf and its d ln kf/dT,
// kb, and for three-body and falloff reactions M and d ln kf/dM (gM).  The
// row-owner Jacobian computes them once per reaction and tile (KC = 5
// values, stride 32 apart, in `kc`); reaction_grad can take them from there.
// per-reaction slots of the row-owner kernel's tile cache: a compact
// reaction's derivatives (dq/dT, dq/dM, dq/dC of its six slots), or another
// reaction's five rate constants (kf, kb, dlkf, gM, M)
constexpr int kDC = 8;

__device__ __forceinline__ void reaction_k(const DevMech& m, int r, const DRxn& R, int kind, const PointT& pt,
                                           double ctot, double Pv, double lnP, const DState& st, double& kf,
                                           double& kb, double& dlkf, double& gM, double& M, double& dlkf_lnP) {
    M = 0.0;
    gM = 0.0;
    dlkf_lnP = 0.0;
    if (kind != CG_STANDARD && kind != CG_PLOG) {
        M = ctot;
        for (int e = __ldg(m.eff_ptr + r); e < __ldg(m.eff_ptr + r + 1); ++e)
            M = fma(__ldg(m.eff_val + e), st.C[__ldg(m.eff_sp + e) * st.s], M);
    }
    if (kind == CG_STANDARD || kind == CG_THIRD_BODY) {
        kf = R.sgn * cgm::cg_exp_clamped(arr_ln(R.lnA, R.b, R.theta, pt));
        dlkf = arr_dln(R.b, R.theta, pt);
    } else if (kind == CG_PLOG) {
        plog_d(m, R.aux, Pv, lnP, pt, kf, dlkf, dlkf_lnP);
    } else {
        const DFall f = load_fall(m.fall + R.aux);
        falloff_d(kind, R.flags, R, f, __ldg(&m.fall2[R.aux].T2), M, pt, kf, dlkf, gM);
    }
    kb = 0.0;
    if (R.flags & CG_F_REVERSIBLE) {
        double num = 1.0, den = 1.0;
        if (R.flags & kFCompact) {
#pragma unroll
            for (int j = 0; j < kMaxCompact; ++j) {
                if (j < R.nre) num *= ipow3(st.E[slot_species(R.sp[j]) * st.s], slot_nu(R.sp[j]));
                if (j < R.npr) den *= ipow3(st.E[slot_species(R.sp[3 + j]) * st.s], slot_nu(R.sp[3 + j]));
            }
        } else {
            const int g = R.gen;
            for (int j = __ldg(m.gen_rptr + g); j < __ldg(m.gen_rptr + g + 1); ++j)
                num *= powi(st.E[__ldg(m.gen_sp + j) * st.s], __ldg(m.gen_nu + j));
            for (int j = __ldg(m.gen_pptr + g); j < __ldg(m.gen_pptr + g + 1); ++j)
                den *= powi(st.E[__ldg(m.gen_sp + j) * st.s], __ldg(m.gen_nu + j));
        }
        kb = kf * num * cgm::cg_rcp(den);
    }
}

// NMAX = 3: compact reactions only (the caller checks kFCompact).  With
// CACHED the rate constants come from kc (reaction_k's values).
template <int NMAX, bool CACHED = false>
__device__ __forceinline__ void reaction_grad(const DevMech& m, int r, const DRxn& R, const PointT& pt, double ctot,
                                              double Pv, double lnP, const DState& st, SideT<NMAX>& re,
                                              SideT<NMAX>& pr, RxnGradT<NMAX>& g, const double* kc = nullptr) {
    int kind = CG_STANDARD;
    while (kind < CG_PLOG && r >= m.seg[kind + 1]) ++kind;
    if constexpr (NMAX == 3) load_sides3(R, re, pr);
    else load_sides(m, R, re, pr);
    double M, kf, kb_c, dlkf, gM, dlkf_lnP = 0.0;
    if constexpr (CACHED) {
        kf = kc[0];
        kb_c = kc[32];
        dlkf = kc[64];
        gM = kc[96];
        M = kc[128];
    } else {
        reaction_k(m, r, R, kind, pt, ctot, Pv, lnP, st, kf, kb_c, dlkf, gM, M, dlkf_lnP);
    }
    double cr[NMAX], cp[NMAX];
    double pf = 1.0;
#pragma unroll(NMAX == 3 ? 3 : 1)
    for (int j = 0; j < NMAX; ++j)
        if (j < re.n) {
            cr[j] = st.C[re.sp[j] * st.s];
            pf *= powi(cr[j], re.nu[j]);
        }
    const double qf = kf * pf;
    double kb = 0.0, qb = 0.0, dlKc = 0.0;
    if (R.flags & CG_F_REVERSIBLE) {
        double pb_ = 1.0;
#pragma unroll(NMAX == 3 ? 3 : 1)
        for (int j = 0; j < NMAX; ++j)
            if (j < re.n) dlKc = fma(re.nu[j], st.D[re.sp[j] * st.sd], dlKc);
#pragma unroll(NMAX == 3 ? 3 : 1)
        for (int j = 0; j < NMAX; ++j)
            if (j < pr.n) {
                cp[j] = st.C[pr.sp[j] * st.s];
                pb_ *= powi(cp[j], pr.nu[j]);
                dlKc = fma(-pr.nu[j], st.D[pr.sp[j] * st.sd], dlKc);
            }
        kb = kb_c;
        qb = kb * pb_;
    }
    const double mfac = (kind == CG_THIRD_BODY) ? M : 1.0;
    g.kind = kind;
    g.qnet = qf - qb;
    g.dlkf_lnP = dlkf_lnP;
    g.dqdT = mfac * fma(qf, dlkf, -qb * (dlkf + dlKc));
    g.dqdM = (kind == CG_THIRD_BODY) ? (qf - qb) : ((kind >= CG_LINDEMANN && kind <= CG_SRI) ? (qf - qb) * gM : 0.0);
    g.usesM = kind >= CG_THIRD_BODY && kind <= CG_SRI;
    const bool rev = (R.flags & CG_F_REVERSIBLE) != 0;
    if constexpr (NMAX == 3) {
        // fixed slots: 0..2 reactants, 3..5 products (unused: zero derivative
        // on species 0), so that every loop over the slots unrolls
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const bool on = j < re.n;
            g.dsp[j] = on ? re.sp[j] : 0;
            g.dqc[j] = on ? mfac * kf * dprod(re, cr, j) : 0.0;
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const bool on = rev && j < pr.n;
            g.dsp[3 + j] = on ? pr.sp[j] : 0;
            g.dqc[3 + j] = on ? -mfac * kb * dprod(pr, cp, j) : 0.0;
        }
        g.nd = 6;
    } else {
        int nd = 0;
        for (int j = 0; j < re.n; ++j) {
            g.dsp[nd] = re.sp[j];
            g.dqc[nd++] = mfac * kf * dprod(re, cr, j);
        }
        if (rev)
            for (int j = 0; j < pr.n; ++j) {
                g.dsp[nd] = pr.sp[j];
                g.dqc[nd++] = -mfac * kb * dprod(pr, cp, j);
            }
        g.nd = nd;
    }
}

}  // namespace
}  // namespace cg
