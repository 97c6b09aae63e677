// Rates of reactions evaluated from their DRxn record: any stoichiometry, kind
// and sign of A.  Shared by the one-thread-per-point kernels and by the quad
// kernels' reactions that have no pre-decoded form.
#pragma once

#include "cg_math.cuh"
#include "rates_common.cuh"

namespace cg {

// kb and the net rate of progress mfac * (qf - qb) of one reaction with
// forward rate kf (reactions/standard.j2:3-19).  mfac is the third-body
// concentration for three-body reactions, 1 otherwise (third_body.j2:30-31).
// C and EGp are read with stride B.
template <int B>
__device__ __forceinline__ double net_rate(const DevMech& m, const DRxn& R, double kf, double mfac, const double* C,
                                          const double* E) {
    if (R.flags & kFCompact) {
        double qf = kf, qb = 0.0;
        if (R.flags & CG_F_REVERSIBLE) {
            double num = 1.0, den = 1.0, cp = 1.0;
#pragma unroll
            for (int j = 0; j < kMaxCompact; ++j)
                if (j < R.nre) num *= ipow3(E[slot_species(R.sp[j]) * B], slot_nu(R.sp[j]));
#pragma unroll
            for (int j = 0; j < kMaxCompact; ++j)
                if (j < R.npr) {
                    const int s = slot_species(R.sp[3 + j]), nu = slot_nu(R.sp[3 + j]);
                    den *= ipow3(E[s * B], nu);
                    cp *= ipow3(C[s * B], nu);
                }
            qb = kf * num * rcp_nr(den) * cp;
        }
#pragma unroll
        for (int j = 0; j < kMaxCompact; ++j)
            if (j < R.nre) qf *= ipow3(C[slot_species(R.sp[j]) * B], slot_nu(R.sp[j]));
        return mfac * (qf - qb);
    }
    const int g = R.gen;
    const int r0 = __ldg(m.gen_rptr + g), r1 = __ldg(m.gen_rptr + g + 1);
    const int p0 = __ldg(m.gen_pptr + g), p1 = __ldg(m.gen_pptr + g + 1);
    double qf = kf, qb = 0.0;
    for (int j = r0; j < r1; ++j) {
        const int s = __ldg(m.gen_sp + j);
        const double nu = __ldg(m.gen_nu + j);
        qf *= (nu == 1.0) ? C[s * B] : pow(C[s * B], nu);
    }
    if (R.flags & CG_F_REVERSIBLE) {
        double ratio = 1.0, cp = 1.0;
        for (int j = r0; j < r1; ++j) {
            const int s = __ldg(m.gen_sp + j);
            const double nu = __ldg(m.gen_nu + j);
            ratio *= (nu == 1.0) ? E[s * B] : pow(E[s * B], nu);
        }
        for (int j = p0; j < p1; ++j) {
            const int s = __ldg(m.gen_sp + j);
            const double nu = __ldg(m.gen_nu + j);
            ratio /= (nu == 1.0) ? E[s * B] : pow(E[s * B], nu);
            cp *= (nu == 1.0) ? C[s * B] : pow(C[s * B], nu);
        }
        qb = kf * ratio * cp;
    }
    return mfac * (qf - qb);
}

__device__ __forceinline__ double arrhenius(double lnA, double b, double theta, double sgn, const PointT& pt) {
    return sgn * cgm::cg_exp_clamped(fma(b, pt.lnT, lnA) - theta * pt.invT);
}

// Falloff forward rate: kinf * Pr/(1+Pr) * F (troe.j2:21-45); Lindemann F = 1,
// SRI F = d [a cgm::cg_exp_clamped(-b/T) + cgm::cg_exp_clamped(-T/c)]^X T^e with X = 1/(1 + cgm::cg_log10(Pr)^2).
__device__ __forceinline__ double falloff_kf(int kind, int flags, const DRxn& R, const DFall& f, double e_sri_or_t2,
                                             double M, const PointT& pt) {
    const double kinf = arrhenius(R.lnA, R.b, R.theta, R.sgn, pt);
    const double k0 = arrhenius(f.lnA0, f.b0, f.theta0, f.sgn0, pt);
    const double Pr = k0 * M / kinf;
    double F = 1.0;
    if (kind == CG_TROE) {
        double Fc = fma(f.p[0], cgm::cg_exp_clamped(-pt.T * f.p[1]), f.p[2] * cgm::cg_exp_clamped(-pt.T * f.p[3]));
        if (flags & CG_F_TROE_T2) Fc += cgm::cg_exp_clamped(-e_sri_or_t2 * pt.invT);
        const double lFc = cgm::cg_log10(Fc);
        const double c1 = fma(-0.67, lFc, -0.4);
        const double n1 = fma(-1.27, lFc, 0.75);
        const double lp = cgm::cg_log10(Pr) + c1;
        const double f1 = lp / fma(-0.14, lp, n1);
        F = cgm::cg_exp_clamped(2.302585092994045684 * lFc / fma(f1, f1, 1.0));
    } else if (kind == CG_SRI) {
        const double lp = cgm::cg_log10(Pr);
        const double X = 1.0 / fma(lp, lp, 1.0);
        const double base = fma(f.p[0], cgm::cg_exp_clamped(-f.p[1] * pt.invT), cgm::cg_exp_clamped(-pt.T * f.p[2]));
        F = f.p[3] * cgm::cg_exp_clamped(fma(X, cgm::cg_log(base), e_sri_or_t2 * pt.lnT));
    }
    return kinf * (Pr / (1.0 + Pr)) * F;
}

// PLOG (plog.j2:4-38): bracket P between tabulated pressures and interpolate
// ln kf linearly in ln P; below the first / above the last level the
// nearest level's rate is used.
__device__ __forceinline__ double plog_kf(const DevMech& m, int row, double P, double lnP, const PointT& pt) {
    const int l0 = __ldg(m.plog_ptr + row), l1 = __ldg(m.plog_ptr + row + 1);
    int l = l0;
    while (l < l1 && !(P < __ldg(m.plog_p + l))) ++l;
    int la, lb;
    if (l == l0) {
        la = lb = l0;
    } else if (l == l1) {
        la = lb = l1 - 1;
    } else {
        la = l - 1;
        lb = l;
    }
    double kfl = 0.0, kfh = 0.0;
    for (int t = __ldg(m.plog_tptr + la); t < __ldg(m.plog_tptr + la + 1); ++t) {
        const double4 c = m.plog_term[t];
        kfl += arrhenius(c.x, c.y, c.z, c.w, pt);
    }
    if (lb == la) return kfl;
    for (int t = __ldg(m.plog_tptr + lb); t < __ldg(m.plog_tptr + lb + 1); ++t) {
        const double4 c = m.plog_term[t];
        kfh += arrhenius(c.x, c.y, c.z, c.w, pt);
    }
    const double a = __ldg(m.plog_lnp + la), b = __ldg(m.plog_lnp + lb);
    const double lkl = cgm::cg_log(kfl);
    return cgm::cg_exp_clamped(lkl + (cgm::cg_log(kfh) - lkl) * (lnP - a) / (b - a));
}

// Net rate of progress of reaction r; C and EGp are read with stride B.
template <int B>
__device__ __noinline__ double generic_rate(const DevMech& m, unsigned r, PointT pt, double P, double lnP,
                                            double ctot, const double* C, const double* E) {
    const DRxn R = load_rxn(m.rxn + r);
    int kind = CG_STANDARD;
    while (kind < CG_PLOG && (int)r >= m.seg[kind + 1]) ++kind;
    double M = ctot;
    if (kind >= CG_THIRD_BODY && kind <= CG_SRI)
        for (int e = __ldg(m.eff_ptr + r); e < __ldg(m.eff_ptr + r + 1); ++e)
            M = fma(__ldg(m.eff_val + e), C[__ldg(m.eff_sp + e) * B], M);
    double kf;
    if (kind <= CG_THIRD_BODY) kf = arrhenius(R.lnA, R.b, R.theta, R.sgn, pt);
    else if (kind == CG_PLOG) kf = plog_kf(m, R.aux, P, lnP, pt);
    else kf = falloff_kf(kind, R.flags, R, load_fall(m.fall + R.aux), __ldg(&m.fall2[R.aux].T2), M, pt);
    return net_rate<B>(m, R, kf, kind == CG_THIRD_BODY ? M : 1.0, C, E);
}

}  // namespace cg
