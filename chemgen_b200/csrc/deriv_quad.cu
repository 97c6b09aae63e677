// Analytic derivatives on eight-point tiles, four reactions to a warp
// (quad.cuh): the dense Jacobian d wdot / d(T, Y) and the adjoint.  The rate
// law and the chain rule are those of derivs.cu's header.
//
// Per reaction the kernels form, in shared memory, one row (eight points) for
// each derivative that something else gathers:
//   dq/dC of each molecule's species (a species on a side twice has two rows);
//   for the Jacobian dq/dT - s/T and ctot dq/dM - s, with s = sum_j dq/dC_j C_j
//   (M's share included); for three-body and falloff reactions dq/dM (for the
//   efficiencies).  For the adjoint every row is already multiplied by the
//   reaction's cotangent gq = sum_k nu_k G_k.
// Then every output has one owner, which sums its row list: no accumulation
// in memory, no atomics, one order of summation.
//   Jacobian: entry (k, j) is (ctot sum_r nu_kr dq_r/dC_j + bk) / (W_j S) with
//     bk = sum_r nu_kr (ctot dq_r/dM - s_r), and column T is
//     sum_r nu_kr (dq_r/dT - s_r / T): the product of a row with C comes from
//     the s's, so an entry needs no other entry and goes straight to J.
//   Adjoint: rho = sum_j dL/dC_j C_j = sum_r gq_r s_r, so dL/dY_j needs no
//     second pass over the species either.
// What bounds them: the load/store unit (60-70 % busy: state, records, rows)
// and the issue rate (47 %), with one CTA per SM for the Jacobian (its 2000
// rows take 130 KB; 24 warps, or 32 for FP32 storage), two of 12 for the
// adjoint.  J itself is written once, in 64-byte pieces.  Measured on B200 at
// 53/325, 65536 points, against the kernels they replaced (32-point tiles; the
// Jacobian's derivatives cached in L2 and gathered row by row, the adjoint added
// into per-warp copies): Jacobian FP64 3.17 -> 1.12 ms, FP32 3.10 -> 1.14 ms,
// adjoint 1.66 -> 0.39 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <utility>
#include <vector>

#include "deriv_common.cuh"
#include "quad.cuh"

namespace cg {

// A short entry (k, column j + 1) of the Jacobian: up to eight signed rows (row |
// sign << 15) and two weighted ones.  Most entries hold a handful of rows, and
// the generic list's padding and decoding cost four times as much as the
// sum itself; an entry of at most four rows is one 16-byte load here.
struct __align__(16) JEnt {
    unsigned at;                       // k (ns + 1) + j + 1
    unsigned short k, j;               // byte offsets of bk and of 1/(W_j S): 64 k, 64 j
    unsigned short row[8];
    unsigned short grow[2];
    unsigned pad;
    double coef[2];
};
static_assert(sizeof(JEnt) == 48, "JEnt must stay 48 bytes");
constexpr int kJRows[] = {1, 2, 3, 4, 6, 8};           // rows of class c / 3; c % 3 weighted ones
// Up to four entries (k, j + 1) of a row that no reaction touches.
struct __align__(16) JZero {
    unsigned at;                       // k (ns + 1) + 1
    unsigned short k, n;               // 64 k
    unsigned short j[4];               // 64 j
};
static_assert(sizeof(JZero) == 16, "JZero must stay 16 bytes");

struct GradPlan {
    int adjoint = 0, other = 0;        // other: PLOG reactions, or some without a pre-decoded form
    int nchunk = 0, rows = 0, warps = 0, nown = 0, nrow = 0, nzero = 0;
    size_t smem = 0;
    int grid = 0;
    const QRec* rec = nullptr;
    const int* qrow = nullptr;         // first row of each quad within its chunk
    const int4* run = nullptr;         // {class, first quad, how many, 0}
    const int* rbeg = nullptr;         // [nchunk W + 1] first run of each warp in each chunk
    const int2* efl = nullptr;
    const QEff* eff = nullptr;
    const QFall* fall = nullptr;
    const double* th = nullptr;
    QLists lists{};                    // Jacobian: [nown] long entries, owner k << 16 | column; adjoint: [nchunk][nown]
    QLists rlists{};                   // Jacobian: [nrow], owner k of the row sums bk
    const JEnt* ent = nullptr;         // Jacobian: short entries, quads of one class
    const int4* erun = nullptr;        // {class, first quad, how many, 0}
    const int* ebeg = nullptr;         // [W + 1] first run of each warp
    const JZero* zero = nullptr;       // [nzero][4] species pairs that no reaction touches
    void* dbuf = nullptr;
};

struct GradView {
    int nchunk, rows, nown, nrow, nzero;
    const QRec* __restrict__ rec;
    const int* __restrict__ qrow;
    const int4* __restrict__ run;
    const int* __restrict__ rbeg;
    const int2* __restrict__ efl;
    const QEff* __restrict__ eff;
    const QFall* __restrict__ fall;
    const double* __restrict__ th;
    QLists lists;
    QLists rlists;
    const JEnt* __restrict__ ent;
    const int4* __restrict__ erun;
    const int* __restrict__ ebeg;
    const JZero* __restrict__ zero;
};

namespace {

struct GradCtx {
    PointT pt;
    double P, lnP, ctot;
    const double2* ce;                 // {C, EGp}
    const double* dg;                  // adjoint: pairs {dE, G}; Jacobian: dE
    const double* tab;
    double* out;                       // this lane's slot of row 0
    int g;
};

// {dE, G} of the species at byte offset `off` of the state.  The Jacobian has
// no G, and its dE rows are half as long.
template <bool ADJ>
__device__ __forceinline__ double2 grad_row(const GradCtx& c, unsigned off) {
    if (ADJ) return quad_row(reinterpret_cast<const double2*>(c.dg), off);
    return make_double2(*reinterpret_cast<const double*>(reinterpret_cast<const char*>(c.dg) + (off >> 1)), 0.0);
}

// Adjoint sums of a lane's reactions.
struct AdjSums {
    double t = 0.0, a = 0.0, rho = 0.0, p = 0.0;
};

// Falloff: forward rate constant kf = kfm M, d ln kf/dT at fixed M, and gpr =
// d ln kf / d ln M (falloff_d's formulas).  kfm and not kf, so that nothing
// divides by M, which is zero where no collider is present.
__device__ __forceinline__ void quad_falloff_d(int kind, const QRec& R, const QFall* fall, double M, const PointT& pt,
                                               const double* tab, double& kfm, double& dlkf, double& gpr) {
    const double2* q = reinterpret_cast<const double2*>(fall + R.aux);
    const double2 f0 = __ldg(q), f1 = __ldg(q + 1), f2 = __ldg(q + 2), f3 = __ldg(q + 3);
    const double lkinf = fma(R.b, pt.lnT, R.lnA) - R.th * pt.invT;
    const double lr = (fma(f0.y, pt.lnT, f0.x) - f1.x * pt.invT) - lkinf;
    const double k0r = q_exp(lr, tab), Pr = k0r * M;   // k0 / kinf
    const double dlkinf = fma(R.th, pt.invT, R.b) * pt.invT;
    const double dlPr = fma(f1.x, pt.invT, f0.y) * pt.invT - dlkinf;
    const double ipr = q_rcp(1.0 + Pr);
    double lnF = 0.0, dlF_T = 0.0;
    gpr = ipr;
    constexpr double kIln10 = 0.43429448190325182765, kLn10c = 2.302585092994045684;
    if (kind == CG_TROE) {
        const double e3 = f1.y * q_exp(fmax(-pt.T * f2.x, kQMinArg), tab);
        const double e1 = f2.y * q_exp(fmax(-pt.T * f3.x, kQMinArg), tab);
        double Fc = e3 + e1;
        double dFc = -fma(f2.x, e3, f3.x * e1);
        if (f3.y != 0.0) {
            const double e2 = q_exp(fmax(-f3.y * pt.invT, kQMinArg), tab);
            Fc += e2;
            dFc = fma(f3.y * pt.invT * pt.invT, e2, dFc);
        }
        const double lFc = cgm::cg_log10(Fc);
        const double u = fma(lr, kIln10, cgm::cg_log10(M)) + fma(-0.67, lFc, -0.4);
        const double nn = fma(-1.27, lFc, 0.75);
        const double den = fma(-0.14, u, nn);
        const double iden = q_rcp(den);
        const double f = u * iden;
        const double q1 = q_rcp(fma(f, f, 1.0));
        lnF = kLn10c * lFc * q1;
        const double dF_df1 = -2.0 * lFc * f * q1 * q1;
        const double df1_dlfc = (-0.67 * den + 1.1762 * u) * iden * iden;
        gpr = fma(dF_df1 * nn, iden * iden, ipr);
        dlF_T = fma(dF_df1, df1_dlfc, q1) * dFc * q_rcp(Fc);
    } else if (kind == CG_SRI) {
        const double lp = fma(lr, kIln10, cgm::cg_log10(M));
        const double X = q_rcp(fma(lp, lp, 1.0));
        const double eb = f1.y * q_exp(fmax(-f2.x * pt.invT, kQMinArg), tab);
        const double ec = q_exp(fmax(-pt.T * f2.y, kQMinArg), tab);
        const double base = eb + ec;
        const double dbase = fma(f2.x * pt.invT * pt.invT, eb, -f2.y * ec);
        const double lb = cgm::cg_log(base);
        lnF = cgm::cg_log(f3.x) + fma(X, lb, f3.y * pt.lnT);
        gpr = ipr - 2.0 * lp * X * X * lb * kIln10;
        dlF_T = fma(X, dbase * q_rcp(base), f3.y * pt.invT);
    }
    kfm = cgm::cg_exp_clamped(lkinf + lnF) * (k0r * ipr);
    dlkf = fma(gpr, dlPr, dlkinf) + dlF_T;
}

// The rows of one reaction with q = mul (qf - qb): mul is M for a three-body or
// falloff reaction (kf then lacks that factor), otherwise 1.  scale: dq/dM =
// scale (qf - qb) (M itself is no divisor: it is zero where a species without
// efficiency stands alone), add: the reaction's share of s = add mul (qf - qb)
// beside the molecules' (ord counts M of a three-body reaction).  plog: kf
// depends on P, dlnp = d ln kf / d ln P.
template <bool ADJ, bool WIDE, bool REV>
__device__ __forceinline__ void grad_rows(const GradCtx& c, const QRec& R, double kf, double dlkf, bool usesM,
                                          double mul, double scale, double add, double* out, AdjSums& sum,
                                          bool plog = false, double dlnp = 0.0) {
    constexpr int N = WIDE ? 3 : 2;
    unsigned so[3] = {R.s[0], R.s[1], R.s2}, po[3] = {R.p[0], R.p[1], R.p2};
    double x[N], d[N];
    double num = 1.0, dlKc = 0.0, gq = 0.0;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const double2 a = quad_row(c.ce, so[j]);
        x[j] = a.x;
        if (REV) num = j ? num * a.y : a.y;
        if (REV || ADJ) {
            const double2 b = grad_row<ADJ>(c, so[j]);
            if (REV) dlKc += b.x;
            if (ADJ) gq -= b.y;
        }
    }
    d[0] = WIDE ? x[1] * x[N - 1] : x[1];
    d[1] = WIDE ? x[0] * x[N - 1] : x[0];
    if (WIDE) d[N - 1] = x[0] * x[1];
    const double qf = kf * (d[0] * x[0]);
    double kb = 0.0, qb = 0.0, e[N];
    if (REV) {
        double den = 1.0, y[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const double2 a = quad_row(c.ce, po[j]);
            const double2 b = grad_row<ADJ>(c, po[j]);
            y[j] = a.x;
            den = j ? den * a.y : a.y;
            dlKc -= b.x;
            if (ADJ) gq += b.y;
        }
        e[0] = WIDE ? y[1] * y[N - 1] : y[1];
        e[1] = WIDE ? y[0] * y[N - 1] : y[0];
        if (WIDE) e[N - 1] = y[0] * y[1];
        kb = kf * num * q_rcp(den);
        qb = kb * (e[0] * y[0]);
    } else if (ADJ) {
#pragma unroll
        for (int j = 0; j < N; ++j) gq += grad_row<ADJ>(c, po[j]).y;
    }
    const double net = qf - qb;
    double dT = net * dlkf - (REV ? qb * dlKc : 0.0);
    double s = fma((double)(R.ord & 0xffu), qf, fma(add, net, -(double)((R.ord >> 8) & 0xffu) * qb));
    const double m = scale * net;
    double f = ADJ ? gq * kf : kf, b = ADJ ? -gq * kb : -kb;
    if (usesM) {
        dT *= mul;
        s *= mul;
        f *= mul;
        b *= mul;
    }
    int o = 0;
#pragma unroll
    for (int j = 0; j < N; ++j) out[32 * o++] = f * d[j];
    if (REV) {
#pragma unroll
        for (int j = 0; j < N; ++j) out[32 * o++] = b * e[j];
    }
    if (ADJ) {
        sum.t = fma(gq, dT, sum.t);
        sum.rho = fma(gq, s, sum.rho);
        if (plog) sum.p = fma(gq, net * dlnp / c.P, sum.p);
        if (usesM) {
            const double gm = gq * m;
            sum.a += gm;
            out[32 * o] = gm;
        }
    } else {
        out[32 * o++] = fma(-s, c.pt.invT, dT);
        out[32 * o++] = fma(c.ctot, m, -s);
        if (usesM) out[32 * o] = m;
    }
}

// grad_rows of the class cls.
template <bool ADJ>
__device__ __forceinline__ void grad_rows_of(int cls, const GradCtx& c, const QRec& R, double kf, double dlkf,
                                             bool usesM, double mul, double scale, double add, double* out,
                                             AdjSums& sum, bool plog = false, double dlnp = 0.0) {
    switch (cls & (kQWide | kQRev)) {
        case 0: grad_rows<ADJ, false, false>(c, R, kf, dlkf, usesM, mul, scale, add, out, sum, plog, dlnp); break;
        case kQRev: grad_rows<ADJ, false, true>(c, R, kf, dlkf, usesM, mul, scale, add, out, sum, plog, dlnp); break;
        case kQWide: grad_rows<ADJ, true, false>(c, R, kf, dlkf, usesM, mul, scale, add, out, sum, plog, dlnp); break;
        default: grad_rows<ADJ, true, true>(c, R, kf, dlkf, usesM, mul, scale, add, out, sum, plog, dlnp); break;
    }
}

// PLOG: {kf, d ln kf/dT, d ln kf/d ln P}.  Evaluated like the reactions below,
// its arrays in local memory, 8 of 40 took a 15-species adjoint to 430 us for
// 100003 points, now 219 (321 with the 32-point tiles before).
__device__ __noinline__ double3 quad_plog_d(const DevMech& m, int row, double P, double lnP, PointT pt) {
    double3 k;
    plog_d(m, row, P, lnP, pt, k.x, k.y, k.z);
    return k;
}

// A reaction evaluated from its DRxn record: its rows in the same order.  With
// PLOG those too, from their pre-decoded records.
template <bool ADJ, bool PLOG>
__device__ __noinline__ AdjSums grad_rows_generic(const DevMech& m, GradCtx c, int cls, const QRec* rec, double* out) {
    AdjSums sum;
    if (PLOG && (cls & 15) == CG_PLOG) {
        const QRec R = load_qrec(rec);
        double kf, dlkf, dlnp;
        plog_d(m, (int)R.aux, c.P, c.lnP, c.pt, kf, dlkf, dlnp);
        grad_rows_of<ADJ>(cls, c, R, kf, dlkf, false, 1.0, 0.0, 0.0, out, sum, true, dlnp);
        return sum;
    }
    const unsigned r = __ldg(&rec->r);
    if (r == kQNone) return sum;
    const double* s0 = reinterpret_cast<const double*>(c.ce);
    const double* d0 = c.dg;
    const DState st{const_cast<double*>(s0), const_cast<double*>(s0 + 1), const_cast<double*>(d0), nullptr, 2 * kQP,
                    ADJ ? 2 * kQP : kQP};
    Side re, pr;
    RxnGrad rg;
    reaction_grad<16>(m, (int)r, load_rxn(m.rxn + r), c.pt, c.ctot, c.P, c.lnP, st, re, pr, rg);
    double gq = 1.0;
    if (ADJ) {
        gq = 0.0;
        for (int j = 0; j < re.n; ++j) gq = fma(-re.nu[j], d0[re.sp[j] * 2 * kQP + 1], gq);
        for (int j = 0; j < pr.n; ++j) gq = fma(pr.nu[j], d0[pr.sp[j] * 2 * kQP + 1], gq);
    }
    double s = 0.0;
    for (int j = 0; j < rg.nd; ++j) {
        s = fma(rg.dqc[j], s0[rg.dsp[j] * 2 * kQP], s);
        out[32 * j] = gq * rg.dqc[j];
    }
    if (rg.usesM) {
        double M = c.ctot;
        for (int e = __ldg(m.eff_ptr + r); e < __ldg(m.eff_ptr + r + 1); ++e)
            M = fma(__ldg(m.eff_val + e), s0[__ldg(m.eff_sp + e) * 2 * kQP], M);
        s = fma(rg.dqdM, M, s);
    }
    int o = rg.nd;
    if (ADJ) {
        sum.t = fma(gq, rg.dqdT, sum.t);
        sum.rho = fma(gq, s, sum.rho);
        if (rg.usesM) {
            sum.a = fma(gq, rg.dqdM, sum.a);
            out[32 * o] = gq * rg.dqdM;
        }
        if (rg.kind == CG_PLOG) sum.p = fma(gq, rg.qnet * rg.dlkf_lnP / c.P, sum.p);
    } else {
        out[32 * o++] = fma(-s, c.pt.invT, rg.dqdT);
        out[32 * o++] = fma(c.ctot, rg.usesM ? rg.dqdM : 0.0, -s);
        if (rg.usesM) out[32 * o] = rg.dqdM;
    }
    return sum;
}

// Elementary reactions: the n quads of a run; the next quad's record and first
// row are loaded while this one is evaluated.
template <int W, bool ADJ, bool WIDE, bool REV>
__device__ __forceinline__ void grad_standard(const GradCtx& c, const QRec* rec, const int* qrow, int n,
                                              AdjSums& sum) {
    QRec N = load_qrec(rec);
    int row = __ldg(qrow);
    for (; n > 0; --n) {
        const QRec R = N;
        double* out = c.out + row * kQP;
        rec += kQG * W;
        qrow += W;
        if (n > 1) {
            N = load_qrec(rec);
            row = __ldg(qrow);
        }
        const double kf = q_exp(fma(R.b, c.pt.lnT, R.lnA) - R.th * c.pt.invT, c.tab);
        grad_rows<ADJ, WIDE, REV>(c, R, kf, fma(R.th, c.pt.invT, R.b) * c.pt.invT, false, 1.0, 0.0, 0.0, out, sum);
    }
}

// OTHER: the mechanism has PLOG reactions or some without a pre-decoded form.
// Instances of their own for those, because what the call needs beside the loops
// spills: without it 53/325 takes 325 instead of 351 us for the rates and adjoint
// of 32768 points, 1118 instead of 1155 for the Jacobian of 65536.  (In 32 warps,
// with 64 registers, PLOG goes out of line as a whole: in line it took 1.5 % more.)
template <int W, bool ADJ, bool OTHER>
__device__ __forceinline__ void grad_run(const DevMech& m, const GradView& v, const GradCtx& c, int cls, int q, int n,
                                         AdjSums& sum) {
    const int kind = cls & 15;
    const QRec* rec = v.rec + kQG * q + c.g;
    if (kind == CG_STANDARD) {
        switch (cls) {
            case 0: grad_standard<W, ADJ, false, false>(c, rec, v.qrow + q, n, sum); break;
            case kQRev: grad_standard<W, ADJ, false, true>(c, rec, v.qrow + q, n, sum); break;
            case kQWide: grad_standard<W, ADJ, true, false>(c, rec, v.qrow + q, n, sum); break;
            default: grad_standard<W, ADJ, true, true>(c, rec, v.qrow + q, n, sum); break;
        }
        return;
    }
    for (; n > 0; --n, q += W, rec += kQG * W) {
        double* out = c.out + __ldg(v.qrow + q) * kQP;
        if (OTHER && (W == 32 ? kind >= CG_PLOG : kind == kQKindGeneric)) {
            const AdjSums x = grad_rows_generic<ADJ, W == 32>(m, c, cls, rec, out);
            if (ADJ) {
                sum.t += x.t;
                sum.a += x.a;
                sum.rho += x.rho;
                sum.p += x.p;
            }
            continue;
        }
        const QRec R = load_qrec(rec);
        if (OTHER && W < 32 && kind == CG_PLOG) {
            const double3 k = quad_plog_d(m, (int)R.aux, c.P, c.lnP, c.pt);
            grad_rows_of<ADJ>(cls, c, R, k.x, k.y, false, 1.0, 0.0, 0.0, out, sum, true, k.z);
            continue;
        }
        const double M = quad_m(v.eff, __ldg(v.efl + q), c.g, c.ctot, c.ce);
        double kf, dlkf, scale = 1.0, add = 0.0;
        if (kind == CG_THIRD_BODY) {
            kf = q_exp(fma(R.b, c.pt.lnT, R.lnA) - R.th * c.pt.invT, c.tab);
            dlkf = fma(R.th, c.pt.invT, R.b) * c.pt.invT;
        } else {
            quad_falloff_d(kind, R, v.fall, M, c.pt, c.tab, kf, dlkf, add);
            scale = add;
        }
        grad_rows_of<ADJ>(cls, c, R, kf, dlkf, true, M, scale, add, out, sum);
    }
}

// The rows of a chunk's reactions.
template <int W, bool ADJ, bool OTHER>
__device__ __forceinline__ void grad_chunk(const DevMech& m, const GradView& v, const GradCtx& c, int chunk, int warp,
                                           AdjSums& sum) {
    const int* rb = v.rbeg + chunk * W + warp;
    const int r1 = __ldg(rb + 1);
    for (int r = __ldg(rb); r < r1; ++r) {
        const int4 rn = __ldg(v.run + r);
        const int cls = __shfl_sync(0xffffffffu, rn.x, 0), n = __shfl_sync(0xffffffffu, rn.z, 0);
        grad_run<W, ADJ, OTHER>(m, v, c, cls, rn.y, n, sum);
    }
}

// The tile's state {C, EGp}, {dE, G} (for the Jacobian dE, and 1/(W S) in rows
// of their own after dE's) from its head, Y and G; leaves ctot, P and the temperature functions in c and
// returns 1/S, S = sum Y/W.
template <int W, bool ADJ>
__device__ __forceinline__ double grad_state(const DevMech& m, const GradView& v, GradCtx& c, bool act, int64_t i,
                                             int64_t ng, const double* h, const double* __restrict__ Y,
                                             const double* __restrict__ G, int warp, int p, double2* sCE, double* sDG,
                                             double* sRed) {
    const int ns = m.ns;
    c.pt.T = h[p];
    c.pt.lnT = h[kQP + p];
    c.pt.invT = h[2 * kQP + p];
    c.P = h[3 * kQP + p];
    c.lnP = m.seg[CG_PLOG] < m.seg[CG_PLOG + 1] ? cgm::cg_log(c.P) : 0.0;
    const double T = c.pt.T, pfac = kPatm / kR0 * c.pt.invT;
    double part = 0.0;
    for (int k = 4 * warp + c.g; k < ns; k += 4 * W) {
        const double w = __ldg(m.inv_mw + k);
        const double x = (act ? __ldcs(Y + (int64_t)k * ng + i) : 1.0) * w;
        double cf[8];
        quad_thermo(v.th, k, T, cf);
        const double smh = smh_poly(cf, T, c.pt.lnT, c.pt.invT);
        // d smh/dT - 1/T
        const double dp = fma(fma(fma(4.0 * cf[5], T, 3.0 * cf[4]), T, 2.0 * cf[3]), T, cf[2]);
        part += x;
        sCE[k * kQP + p] = make_double2(x, q_exp(smh, c.tab) * pfac);
        const double dE = dp + fma(cf[6], c.pt.invT, cf[1]) * c.pt.invT - c.pt.invT;
        if (ADJ)
            reinterpret_cast<double2*>(sDG)[k * kQP + p] =
                make_double2(dE, act ? __ldcs(G + (int64_t)k * ng + i) : 0.0);
        else
            sDG[k * kQP + p] = dE;
    }
    part += __shfl_xor_sync(0xffffffffu, part, 8);
    part += __shfl_xor_sync(0xffffffffu, part, 16);
    if (c.g == 0) sRed[warp * kQP + p] = part;
    __syncthreads();
    const double S = quad_total<W>(sRed, c.g), iS = cgm::cg_rcp(S);
    const double fac = c.P * cgm::cg_rcp(kR0 * S * T);
    c.ctot = S * fac;
    for (int k = 4 * warp + c.g; k < ns; k += 4 * W) {
        sCE[k * kQP + p].x *= fac;
        // (written after the barrier: the last tile's entries read it before)
        if (!ADJ) sDG[(ns + 1 + k) * kQP + p] = __ldg(m.inv_mw + k) * iS;
    }
    __syncthreads();
    return iS;
}

// Runs fn on the owner records of quads first + warp, first + warp + W, ..., the
// next quad's record loaded before fn runs on this one's.
template <int W, typename Fn>
__device__ __forceinline__ void for_owners(const QLists& L, int n, int first, int warp, int g, Fn fn) {
    if (warp >= n) return;
    const QOwn* op = L.own + kQG * (first + warp) + g;
    QOwn N = load_qown(op);
    for (int s = warp; s < n; s += W) {
        const QOwn o = N;
        op += kQG * W;
        if (s + W < n) N = load_qown(op);
        fn(o);
    }
}

// Row `e & 0x7fff` with the sign of bit 15, from the low or the high half of w.
__device__ __forceinline__ double signed_row(const double* rows, unsigned w, bool high) {
    const unsigned off = (high ? w >> 10 : w << 6) & 0x1fffc0u, sg = (high ? w : w << 16) & 0x80000000u;
    const double x = *reinterpret_cast<const double*>(reinterpret_cast<const char*>(rows) + off);
    return __hiloint2double(__double2hiint(x) ^ (int)sg, __double2loint(x));
}

// The short entries of one class: n quads of the warp's run.
__device__ __forceinline__ double at_byte(const void* p, unsigned off) {
    return *reinterpret_cast<const double*>(static_cast<const char*>(p) + off);
}

template <int W, int C, int G, typename JT>
__device__ __forceinline__ void jac_entries(const JEnt* e, int n, const double* rows, const double* bk,
                                            const double* wj, double ctot, JT* Ji, unsigned ng, bool act) {
    const uint4* q = reinterpret_cast<const uint4*>(e);
    uint4 n0 = __ldg(q), n1{};
    double2 nc{};
    if (C > 4 || G > 0) n1 = __ldg(q + 1);
    if (G > 0) nc = __ldg(reinterpret_cast<const double2*>(q + 2));
    for (; n > 0; --n) {
        const uint4 a = n0, b = n1;
        const double2 cf = nc;
        q += 3 * kQG * W;
        if (n > 1) {
            n0 = __ldg(q);
            if (C > 4 || G > 0) n1 = __ldg(q + 1);
            if (G > 0) nc = __ldg(reinterpret_cast<const double2*>(q + 2));
        }
        const unsigned w[4] = {a.z, a.w, b.x, b.y};
        double x = signed_row(rows, w[0], false);
#pragma unroll
        for (int j = 1; j < C; ++j) x += signed_row(rows, w[j >> 1], j & 1);
        if (G > 0) x = fma(cf.x, rows[(b.z & 0xffffu) * kQP], x);
        if (G > 1) x = fma(cf.y, rows[(b.z >> 16) * kQP], x);
        const double y = fma(ctot, x, at_byte(bk, a.y & 0xffffu)) * at_byte(wj, a.y >> 16);
        if (act) __stcs(Ji + (uint64_t)a.x * ng, (JT)y);
    }
}

// ---------------------------------------------------------------- Jacobian
template <int W, int MINB, bool OTHER, typename JT>
__global__ void __launch_bounds__(32 * W, MINB)
    jacobian_quad(const __grid_constant__ DevMech m, const __grid_constant__ GradView v, const double* __restrict__ P,
                  const double* __restrict__ Tg, const double* __restrict__ Y, JT* __restrict__ J, int64_t ng) {
    extern __shared__ __align__(16) double smem[];
    const int ns = m.ns, ncol = ns + 1;
    const int lane = threadIdx.x & 31, p = lane & (kQP - 1), g = lane >> 3;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    double* sTab = smem;                                   // [16]
    double* sH = sTab + 16;                                // [2][4][8] heads of this tile and the next
    double* sRed = sH + 8 * kQP;                           // [W][8]
    double2* sCE = reinterpret_cast<double2*>(sRed + W * kQP);   // [ns + 1][8]
    double* sDG = reinterpret_cast<double*>(sCE + (ns + 1) * kQP);  // [ns + 1][8] dE, [ns][8] 1/(W S)
    double* sB = sDG + (2 * ns + 1) * kQP;                 // [ns][8] bk
    double* sV = sB + ns * kQP;                            // [rows + 1][8]
    if (threadIdx.x < 16) sTab[threadIdx.x] = kQExpTab[threadIdx.x];
    if (warp == W - 1 && g == 0) quad_head(sH, (int64_t)blockIdx.x * kQP + p, ng, P, Tg);
    if (threadIdx.x < kQP) {
        sV[v.rows * kQP + p] = 0.0;
        sCE[ns * kQP + p] = make_double2(1.0, 1.0);
        sDG[ns * kQP + p] = 0.0;
    }
    __syncthreads();
    GradCtx c;
    c.ce = sCE + p;
    c.dg = sDG + p;
    c.tab = sTab;
    c.out = sV + lane;
    c.g = g;
    const int64_t stride = (int64_t)gridDim.x * kQP;
    int buf = 0;
    for (int64_t t0 = (int64_t)blockIdx.x * kQP; t0 < ng; t0 += stride, buf ^= 1) {
        const int64_t i = t0 + p;
        const bool act = i < ng;
        grad_state<W, false>(m, v, c, act, i, ng, sH + buf * 4 * kQP, Y, nullptr, warp, p, sCE, sDG, sRed);
        AdjSums none;
        grad_chunk<W, false, OTHER>(m, v, c, 0, warp, none);
        if (warp == W - 1 && g == 0 && t0 + stride < ng) quad_head(sH + (buf ^ 1) * 4 * kQP, i + stride, ng, P, Tg);
        __syncthreads();
        for_owners<W>(v.rlists, v.nrow, 0, warp, g, [&](const QOwn& o) {
            const double x = list_sum(v.rlists, o, g, sV + p);
            if (o.own >= 0) sB[o.own * kQP + p] = x;
        });
        __syncthreads();
        const double* bk = sB + p;
        const double* wj = sDG + (ns + 1) * kQP + p;
        const unsigned n32 = (unsigned)ng;                 // the launch function keeps ng below 2^32
        JT* Ji = J + i;
        for_owners<W>(v.lists, v.nown, 0, warp, g, [&](const QOwn& o) {
            const double x = list_sum(v.lists, o, g, sV + p);
            if (o.own < 0 || !act) return;
            const int k = o.own >> 16, col = o.own & 0xffff;   // column 0: T
            const double y = col ? fma(c.ctot, x, bk[k * kQP]) * wj[(col - 1) * kQP] : x;
            __stcs(Ji + (uint64_t)(unsigned)(k * ncol + col) * n32, (JT)y);
        });
        const int r1 = __ldg(v.ebeg + warp + 1);
        for (int r = __ldg(v.ebeg + warp); r < r1; ++r) {
            const int4 rn = __ldg(v.erun + r);
            const int cls = __shfl_sync(0xffffffffu, rn.x, 0), n = __shfl_sync(0xffffffffu, rn.z, 0);
            const JEnt* e = v.ent + kQG * rn.y + g;
#define CG_JAC_ENTRIES(K, C)                                                                      \
    case 3 * K: jac_entries<W, C, 0>(e, n, sV + p, bk, wj, c.ctot, Ji, n32, act); break;     \
    case 3 * K + 1: jac_entries<W, C, 1>(e, n, sV + p, bk, wj, c.ctot, Ji, n32, act); break; \
    case 3 * K + 2: jac_entries<W, C, 2>(e, n, sV + p, bk, wj, c.ctot, Ji, n32, act); break
            switch (cls) {
                CG_JAC_ENTRIES(0, 1);
                CG_JAC_ENTRIES(1, 2);
                CG_JAC_ENTRIES(2, 3);
                CG_JAC_ENTRIES(3, 4);
                CG_JAC_ENTRIES(4, 6);
                CG_JAC_ENTRIES(5, 8);
            }
#undef CG_JAC_ENTRIES
        }
        // entries that no reaction touches: four of a row to a record
        for (int q = 4 * warp + g; q < v.nzero; q += 4 * W) {
            const uint4 z = __ldg(reinterpret_cast<const uint4*>(v.zero + q));
            const int n = (int)(z.y >> 16);
            const double b0 = at_byte(bk, z.y & 0xffffu);
            const unsigned j[4] = {z.z & 0xffffu, z.z >> 16, z.w & 0xffffu, z.w >> 16};
            JT* Jk = Ji + (uint64_t)z.x * n32;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const double y = b0 * at_byte(wj, j[u]);
                if (act && u < n) __stcs(Jk + (uint64_t)(j[u] >> 6) * n32, (JT)y);
            }
        }
        // the next tile's rows are written after two more barriers
    }
}

// ----------------------------------------------------------------- adjoint
template <int W, int MINB, bool OTHER>
__global__ void __launch_bounds__(32 * W, MINB)
    vjp_quad(const __grid_constant__ DevMech m, const __grid_constant__ GradView v, const double* __restrict__ P,
             const double* __restrict__ Tg, const double* __restrict__ Y, const double* __restrict__ G,
             double* __restrict__ gT, double* __restrict__ gY, double* __restrict__ gP, int64_t ng) {
    extern __shared__ __align__(16) double smem[];
    const int ns = m.ns;
    const int lane = threadIdx.x & 31, p = lane & (kQP - 1), g = lane >> 3;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    double* sTab = smem;                                   // [16]
    double* sH = sTab + 16;                                // [2][4][8] heads of this tile and the next
    double* sRed = sH + 8 * kQP;                           // [4][W][8]
    double2* sCE = reinterpret_cast<double2*>(sRed + 4 * W * kQP);   // [ns + 1][8]
    double* sDG = reinterpret_cast<double*>(sCE + (ns + 1) * kQP);  // [ns + 1][8] pairs
    double* sV = sDG + 2 * (ns + 1) * kQP;                 // [rows + 1][8]
    double* sW = sV + (v.rows + 1) * kQP;                  // [ns][8], several chunks only
    if (threadIdx.x < 16) sTab[threadIdx.x] = kQExpTab[threadIdx.x];
    if (warp == W - 1 && g == 0) quad_head(sH, (int64_t)blockIdx.x * kQP + p, ng, P, Tg);
    if (threadIdx.x < kQP) {
        sV[v.rows * kQP + p] = 0.0;
        sCE[ns * kQP + p] = make_double2(1.0, 1.0);
        reinterpret_cast<double2*>(sDG)[ns * kQP + p] = make_double2(0.0, 0.0);
    }
    __syncthreads();
    GradCtx c;
    c.ce = sCE + p;
    c.dg = sDG + 2 * p;
    c.tab = sTab;
    c.out = sV + lane;
    c.g = g;
    const int64_t stride = (int64_t)gridDim.x * kQP;
    int buf = 0;
    for (int64_t t0 = (int64_t)blockIdx.x * kQP; t0 < ng; t0 += stride, buf ^= 1) {
        const int64_t i = t0 + p;
        const bool act = i < ng;
        const double iS =
            grad_state<W, true>(m, v, c, act, i, ng, sH + buf * 4 * kQP, Y, G, warp, p, sCE, sDG, sRed);
        AdjSums sum;
        for (int ch = 0; ch < v.nchunk; ++ch) {
            grad_chunk<W, true, OTHER>(m, v, c, ch, warp, sum);
            if (ch == 0 && warp == W - 1 && g == 0 && t0 + stride < ng)
                quad_head(sH + (buf ^ 1) * 4 * kQP, i + stride, ng, P, Tg);
            const bool last = ch == v.nchunk - 1;
            if (last) {
                double x[4] = {sum.t, sum.a, sum.rho, sum.p};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    x[j] += __shfl_xor_sync(0xffffffffu, x[j], 8);
                    x[j] += __shfl_xor_sync(0xffffffffu, x[j], 16);
                    if (g == 0) sRed[(j * W + warp) * kQP + p] = x[j];
                }
            }
            __syncthreads();
            double ab = 0.0, rho = 0.0;
            if (last) {
                ab = quad_total<W>(sRed + W * kQP, g);
                rho = quad_total<W>(sRed + 2 * W * kQP, g);
                if (warp == 0) {
                    const double tb = quad_total<W>(sRed, g), pb = quad_total<W>(sRed + 3 * W * kQP, g);
                    if (g == 0 && act) {
                        __stcs(gT + i, fma(-rho, c.pt.invT, tb));
                        if (gP) __stcs(gP + i, fma(rho, 1.0 / c.P, pb));
                    }
                }
            }
            for_owners<W>(v.lists, v.nown, ch * v.nown, warp, g, [&](const QOwn& o) {
                double x = list_sum(v.lists, o, g, sV + p);
                const int k = o.own;
                if (k < 0) return;
                if (ch > 0) x += sW[k * kQP + p];
                if (!last) sW[k * kQP + p] = x;
                else if (act)
                    __stcs(gY + (int64_t)k * ng + i, fma(c.ctot, x + ab, -rho) * (__ldg(m.inv_mw + k) * iS));
            });
            // before the next chunk's rows, and before sRed is written again
            __syncthreads();
        }
    }
}

template <bool OTHER>
const void* grad_kernel(const GradPlan* p, int precision) {
    if (p->adjoint)
        return p->warps == 8 ? (const void*)vjp_quad<8, 3, OTHER>
                             : p->warps == 12 ? (const void*)vjp_quad<12, 2, OTHER> : (const void*)vjp_quad<24, 1, OTHER>;
    // (64 registers: the instance without the call took 104.5 instead of 102.4 us for
    // GRI30, 5003 points)
    if (p->warps == 32) return (const void*)jacobian_quad<32, 1, true, float>;
    if (precision == 0)
        return p->warps == 8 ? (const void*)jacobian_quad<8, 3, OTHER, double>
                             : p->warps == 12 ? (const void*)jacobian_quad<12, 2, OTHER, double>
                                              : (const void*)jacobian_quad<24, 1, OTHER, double>;
    return p->warps == 8 ? (const void*)jacobian_quad<8, 3, OTHER, float>
                         : p->warps == 12 ? (const void*)jacobian_quad<12, 2, OTHER, float>
                                          : (const void*)jacobian_quad<24, 1, OTHER, float>;
}

const void* grad_kernel(const GradPlan* p, int precision) {
    return p->other ? grad_kernel<true>(p, precision) : grad_kernel<false>(p, precision);
}

}  // namespace

void grad_release(GradPlan* p);

// adjoint: any mechanism whose state fits (the reactions run in chunks).
// Jacobian: the rows of every reaction at once (about 520 reactions).  At most
// 511 species.  cudaErrorNotSupported otherwise.  f32: the Jacobian's plan for FP32 storage
// where it has one of its own (the FP64 plan serves both otherwise, and this
// returns cudaErrorNotSupported).
cudaError_t grad_prepare(const DevMech& m, const cg_mech_view& v, int device, int adjoint, int f32, GradPlan** out) {
    *out = nullptr;
    const int ns = m.ns, nr = m.nr;
    if (nr == 0 || ns >= 0x10000 / kQRow) return cudaErrorNotSupported;
    const int32_t* flags = (const int32_t*)v.a[CG_FLAGS];
    const int32_t* rp = (const int32_t*)v.a[CG_RPTR];
    const int32_t* pp = (const int32_t*)v.a[CG_PPTR];
    const int32_t* rsp = (const int32_t*)v.a[CG_RSP];
    const int32_t* psp = (const int32_t*)v.a[CG_PSP];
    const double* rnu = (const double*)v.a[CG_RNU];
    const double* pnu = (const double*)v.a[CG_PNU];
    const int32_t* ep = (const int32_t*)v.a[CG_EFF_PTR];
    const int32_t* es = (const int32_t*)v.a[CG_EFF_SP];
    const double* ev = (const double*)v.a[CG_EFF_VAL];
    DeviceLimits dev;
    cudaError_t e = device_limits(device, &dev);
    if (e != cudaSuccess) return e;
    const size_t limit = dev.smem_block, per_sm = dev.smem_sm;
    HostQuads h;
    build_quads(v, h, adjoint != 0, true);
    auto uses_m = [&](int r) {
        return r >= m.seg[CG_THIRD_BODY] && r < m.seg[CG_PLOG];
    };
    auto generic = [&](int q) { return h.key[q] == kQKindGeneric; };
    // rows of a quad: per-molecule (per-species for generic reactions)
    // derivatives, then dT and s (Jacobian), then dM
    std::vector<int> order(nr), nval(h.nquad, 0), nslot(nr, 0);
    for (int r = 0; r < nr; ++r) order[r] = r;
    std::sort(order.begin(), order.end(), [&](int a, int b) { return h.at[a] < h.at[b]; });
    for (int r : order) {
        const int q = h.at[r] / kQG;
        const bool rev = (flags[r] & CG_F_REVERSIBLE) != 0;
        if (generic(q)) nslot[r] = (rp[r + 1] - rp[r]) + (rev ? pp[r + 1] - pp[r] : 0);
        else nslot[r] = ((h.key[q] & kQWide) ? 3 : 2) * (rev ? 2 : 1);
        nval[q] = std::max(nval[q], nslot[r] + (adjoint ? 0 : 2) + (uses_m(r) ? 1 : 0));
    }
    GradPlan pl;
    pl.adjoint = adjoint;
    pl.other = h.ngeneric + h.nplog > 0;
    auto bytes = [&](size_t rows, int chunks, int warps) {
        const size_t state = (size_t)8 + 4 * (ns + 1) + rows + 1 + (adjoint ? 4 : 1) * warps +
                             (adjoint ? (chunks > 1 ? ns : 0) : ns);
        return (16 + state * kQP) * sizeof(double);
    };
    // chunks of quads whose rows fit
    size_t total = 0, most = 0;
    for (int q = 0; q < h.nquad; ++q) {
        total += 4 * nval[q];
        most = std::max<size_t>(most, 4 * nval[q]);
    }
    size_t cap = total;
    if (bytes(total, 1, 24) > limit || total >= 0xffff) {
        if (!adjoint) return cudaErrorNotSupported;
        if (bytes(most, 2, 24) > limit) return cudaErrorNotSupported;
        cap = std::min<size_t>((limit - bytes(0, 2, 24)) / (kQP * sizeof(double)), 0xfff0);
        // even chunks
        const size_t n = (total + cap - most) / (cap - most + 1) + 1;
        cap = std::min(cap, total / n + most);
    }
    std::vector<int> chunk(h.nquad), qbeg(1, 0);
    std::vector<int> qrow(h.nquad);
    size_t used = 0;
    for (int q = 0; q < h.nquad; ++q) {
        if (used + 4 * nval[q] > cap) {
            qbeg.push_back(q);
            used = 0;
        }
        chunk[q] = (int)qbeg.size() - 1;
        qrow[q] = (int)used;
        used += 4 * nval[q];
        pl.rows = std::max(pl.rows, (int)used);
    }
    pl.nchunk = (int)qbeg.size();
    qbeg.push_back(h.nquad);
    const int fit = (int)(per_sm / (bytes(pl.rows, pl.nchunk, 24) + 1024));
    pl.warps = fit >= 3 ? 8 : fit == 2 ? 12 : 24;
    if (f32) {
        // one CTA per SM: 32 warps of 64 registers.  FP32 J at 53/325: 106 -> 97 us
        // for 5003 points, 581 -> 540 for 32768; FP64 J, whose stores weigh more,
        // goes from 579 to 599 us there and stays with 24 warps of 80
        if (pl.warps != 24 || bytes(pl.rows, pl.nchunk, 32) > limit) return cudaErrorNotSupported;
        pl.warps = 32;
    }
    pl.smem = bytes(pl.rows, pl.nchunk, pl.warps);
    const int resident = std::max(1, std::min((int)(per_sm / (pl.smem + 1024)), f32 ? 1 : 24 / pl.warps));
    pl.grid = dev.sms * resident;
    std::vector<int4> run;
    std::vector<int> rbeg;
    build_runs(h, qbeg, pl.warps, run, rbeg);
    // row of value j of reaction r within its chunk
    auto row = [&](int r, int j) { return qrow[h.at[r] / kQG] + 4 * j + h.at[r] % kQG; };
    // species of each slot row, as the kernels lay them out
    auto slots = [&](int r, std::vector<int>& sp) {
        sp.assign(nslot[r], -1);
        const bool rev = (flags[r] & CG_F_REVERSIBLE) != 0;
        const int q = h.at[r] / kQG;
        if (generic(q)) {
            int o = 0;
            for (int j = rp[r]; j < rp[r + 1]; ++j) sp[o++] = rsp[j];
            if (rev)
                for (int j = pp[r]; j < pp[r + 1]; ++j) sp[o++] = psp[j];
            return;
        }
        const int n = (h.key[q] & kQWide) ? 3 : 2;
        int o = 0;
        for (int j = rp[r]; j < rp[r + 1]; ++j)
            for (int u = 0; u < (int)rnu[j]; ++u) sp[o++] = rsp[j];
        o = n;
        if (rev)
            for (int j = pp[r]; j < pp[r + 1]; ++j)
                for (int u = 0; u < (int)pnu[j]; ++u) sp[o++] = psp[j];
    };
    using List = ListBuilder::List;
    ListBuilder lb, rb;
    std::vector<int> sp, ebeg;
    std::vector<int4> erun;
    std::vector<JEnt> jent;
    std::vector<JZero> zero;
    if (adjoint) {
        std::vector<std::vector<List>> lists(pl.nchunk, std::vector<List>(ns));
        for (int r : order) {
            std::vector<List>& L = lists[chunk[h.at[r] / kQG]];
            slots(r, sp);
            for (int j = 0; j < (int)sp.size(); ++j)
                if (sp[j] >= 0) L[sp[j]].push_back({row(r, j), 1.0});
            if (uses_m(r))
                for (int x = ep[r]; x < ep[r + 1]; ++x) L[es[x]].push_back({row(r, nslot[r]), ev[x]});
        }
        std::vector<List> all(ns);
        for (const auto& L : lists)
            for (int k = 0; k < ns; ++k) all[k].insert(all[k].end(), L[k].begin(), L[k].end());
        std::vector<const List*> al;
        for (const List& l : all) al.push_back(&l);
        const auto quads = ListBuilder::group(al, pl.warps);
        pl.nown = (int)quads.size();
        for (const auto& L : lists)
            for (const auto& q : quads) {
                std::vector<const List*> o;
                for (int k : q) o.push_back(&L[k]);
                lb.add_quad(o, q, pl.rows);
            }
    } else {
        std::vector<List> sums(ns);
        std::map<int, List> ent;
        std::vector<double> net(ns, 0.0);
        for (int r : order) {
            slots(r, sp);
            const int n = nslot[r];
            for (int j = rp[r]; j < rp[r + 1]; ++j) net[rsp[j]] -= rnu[j];
            for (int j = pp[r]; j < pp[r + 1]; ++j) net[psp[j]] += pnu[j];
            for (int side = 0; side < 2; ++side)
                for (int j = side ? pp[r] : rp[r]; j < (side ? pp[r + 1] : rp[r + 1]); ++j) {
                    const int k = side ? psp[j] : rsp[j];
                    const double nu = net[k];
                    net[k] = 0.0;
                    if (nu == 0.0) continue;
                    for (int x = 0; x < n; ++x)
                        if (sp[x] >= 0) ent[k << 16 | (sp[x] + 1)].push_back({row(r, x), nu});
                    ent[k << 16].push_back({row(r, n), nu});
                    sums[k].push_back({row(r, n + 1), nu});
                    if (uses_m(r))
                        for (int x = ep[r]; x < ep[r + 1]; ++x)
                            ent[k << 16 | (es[x] + 1)].push_back({row(r, n + 2), nu * ev[x]});
                }
        }
        std::vector<const List*> el, sl;
        std::vector<int> code, scode;
        std::vector<std::pair<int, JEnt>> shorts;
        for (int k = 0; k < ns; ++k) {
            ent[k << 16];              // column T exists even if no reaction touches k
            scode.push_back(k);
            sl.push_back(&sums[k]);
        }
        for (const auto& x : ent) {
            // short entries by class; the rest, and column T, as lists
            const int k = x.first >> 16, col = x.first & 0xffff;
            JEnt e;
            std::memset(&e, 0, sizeof(e));
            e.at = (unsigned)(k * (ns + 1) + col);
            e.k = (unsigned short)(k * 8 * kQP);
            e.j = (unsigned short)((col - 1) * 8 * kQP);
            size_t nr_ = 0, ng_ = 0;
            for (const auto& y : x.second) {
                const double a = std::fabs(y.second);
                if (a == 1.0 || a == 2.0 || a == 3.0) {
                    for (int u = 0; u < (int)a; ++u, ++nr_)
                        if (nr_ < 8) e.row[nr_] = (unsigned short)(y.first | (y.second < 0.0 ? 0x8000 : 0));
                } else if (a != 0.0) {
                    if (ng_ < 2) {
                        e.grow[ng_] = (unsigned short)y.first;
                        e.coef[ng_] = y.second;
                    }
                    ++ng_;
                }
            }
            if (col == 0 || nr_ > 8 || ng_ > 2 || pl.rows >= 0x8000) {
                code.push_back(x.first);
                el.push_back(&x.second);
                continue;
            }
            int c = 0;
            while ((size_t)kJRows[c] < nr_) ++c;
            for (size_t u = nr_; u < 8; ++u) e.row[u] = (unsigned short)pl.rows;
            for (size_t u = ng_; u < 2; ++u) e.grow[u] = (unsigned short)pl.rows;
            shorts.push_back({3 * c + (int)ng_, e});
        }
        std::stable_sort(shorts.begin(), shorts.end(),
                         [](const std::pair<int, JEnt>& a, const std::pair<int, JEnt>& b) { return a.first > b.first; });
        HostQuads eq;
        for (size_t x = 0; x < shorts.size();) {
            size_t y = x;
            while (y < shorts.size() && y < x + kQG && shorts[y].first == shorts[x].first) ++y;
            // a quad short of four repeats its last entry (the same value twice)
            for (size_t g = 0; g < (size_t)kQG; ++g) jent.push_back(shorts[std::min(x + g, y - 1)].second);
            eq.key.push_back(shorts[x].first);
            x = y;
        }
        build_runs(eq, {0, (int)eq.key.size()}, pl.warps, erun, ebeg);
        auto build = [&](ListBuilder& b, const std::vector<const List*>& l, const std::vector<int>& what) {
            const auto quads = ListBuilder::group(l, pl.warps);
            for (const auto& q : quads) {
                std::vector<const List*> o;
                std::vector<int> w;
                for (int x : q) {
                    o.push_back(l[x]);
                    w.push_back(what[x]);
                }
                b.add_quad(o, w, pl.rows);
            }
            return (int)quads.size();
        };
        pl.nown = build(lb, el, code);
        pl.nrow = build(rb, sl, scode);
        for (int k = 0; k < ns; ++k) {
            JZero z;
            z.n = 0;
            for (int j = 0; j <= ns; ++j) {
                if (j < ns && !ent.count(k << 16 | (j + 1))) z.j[z.n++] = (unsigned short)(j * 8 * kQP);
                if (z.n == 4 || (j == ns && z.n > 0)) {
                    z.at = (unsigned)(k * (ns + 1) + 1);
                    z.k = (unsigned short)(k * 8 * kQP);
                    for (int u = z.n; u < 4; ++u) z.j[u] = 0;
                    zero.push_back(z);
                    z.n = 0;
                }
            }
        }
        pl.nzero = (int)zero.size();
    }
    if (!lb.fits || !rb.fits) return cudaErrorNotSupported;
    Image im;
    const size_t o_rec = im.put(h.rec), o_qr = im.put(qrow), o_run = im.put(run), o_rb = im.put(rbeg);
    const size_t o_efl = im.put(h.efl), o_eff = im.put(h.eff), o_fall = im.put(h.fall);
    const size_t o_th = im.put(quad_thermo_rows(v)), o_li = im.put(lb.own);
    const size_t o_le = im.put(lb.ent), o_lg = im.put(lb.gen), o_ri = im.put(rb.own);
    const size_t o_re = im.put(rb.ent), o_rg = im.put(rb.gen), o_z = im.put(zero);
    const size_t o_je = im.put(jent), o_er = im.put(erun), o_eb = im.put(ebeg);
    GradPlan* p = new GradPlan(pl);
    e = im.upload(&p->dbuf);
    for (int precision = 0; precision < 2 && e == cudaSuccess; ++precision)
        e = raise_smem_limit(grad_kernel(p, precision), p->smem);
    if (e != cudaSuccess) {
        grad_release(p);
        return e;
    }
    char* d = (char*)p->dbuf;
    p->rec = (const QRec*)(d + o_rec);
    p->qrow = (const int*)(d + o_qr);
    p->run = (const int4*)(d + o_run);
    p->rbeg = (const int*)(d + o_rb);
    p->efl = (const int2*)(d + o_efl);
    p->eff = (const QEff*)(d + o_eff);
    p->fall = (const QFall*)(d + o_fall);
    p->th = (const double*)(d + o_th);
    p->lists = QLists{(const QOwn*)(d + o_li), (const uint4*)(d + o_le), (const QGen*)(d + o_lg)};
    p->rlists = QLists{(const QOwn*)(d + o_ri), (const uint4*)(d + o_re), (const QGen*)(d + o_rg)};
    p->zero = (const JZero*)(d + o_z);
    p->ent = (const JEnt*)(d + o_je);
    p->erun = (const int4*)(d + o_er);
    p->ebeg = (const int*)(d + o_eb);
    *out = p;
    return cudaSuccess;
}

void grad_release(GradPlan* p) {
    if (!p) return;
    if (p->dbuf) cudaFree(p->dbuf);
    delete p;
}

namespace {
GradView grad_view(const GradPlan* p) {
    return GradView{p->nchunk, p->rows, p->nown, p->nrow, p->nzero, p->rec, p->qrow, p->run, p->rbeg,
                    p->efl, p->eff, p->fall, p->th, p->lists, p->rlists, p->ent, p->erun, p->ebeg, p->zero};
}

cudaError_t launch_grad(const GradPlan* p, int precision, int64_t ng, void** args, cudaStream_t s) {
    const int64_t tiles = (ng + kQP - 1) / kQP;
    return cudaLaunchKernel(grad_kernel(p, precision), dim3((unsigned)std::min<int64_t>(tiles, p->grid)),
                            dim3(32u * (unsigned)p->warps), args, p->smem, s);
}
}  // namespace

cudaError_t launch_jacobian_quad(const GradPlan* p, const DevMech& m, int precision, const double* P, const double* T,
                                 const double* Y, void* J, int64_t ng, cudaStream_t s) {
    if (ng <= 0) return cudaSuccess;
    if (ng >= ((int64_t)1 << 32)) return cudaErrorInvalidValue;   // J would be 2^32 ns (ns + 1) values: no GPU holds it
    DevMech dm = m;
    GradView v = grad_view(p);
    void* args[] = {&dm, &v, &P, &T, &Y, &J, &ng};
    return launch_grad(p, precision, ng, args, s);
}

cudaError_t launch_vjp_quad(const GradPlan* p, const DevMech& m, const double* P, const double* T, const double* Y,
                            const double* G, double* gT, double* gY, double* gP, int64_t ng, cudaStream_t s) {
    if (ng <= 0) return cudaSuccess;
    DevMech dm = m;
    GradView v = grad_view(p);
    void* args[] = {&dm, &v, &P, &T, &Y, &G, &gT, &gY, &gP, &ng};
    return launch_grad(p, 0, ng, args, s);
}

}  // namespace cg
