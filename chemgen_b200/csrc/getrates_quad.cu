// getrates on eight-point tiles, four reactions to a warp (quad.cuh), FP64
// and mixed precision.
//
// Computes the same quantities as the reference's generated getrates
// (chemgen/templates/python_header.j2:25-56, ytoc.j2, exp_g.j2,
// reactions/{standard,third_body,troe,plog}.j2), with Lindemann and SRI
// falloff added.  A CTA owns a tile of eight points and keeps its state
// {C, EGp} (FP64) or {log2 Gibbs, C * 2^32} (mixed) in shared memory:
//   1  species quads: C and EGp of the tile;
//   2  reaction quads: the net rates of progress q, into shared memory, all
//      reactions at once when they fit, else chunk by chunk;
//   3  species quads: wdot = sum nu q from per-species row lists
//      (reactions/standard.j2:21-27), each species with one owner, so no
//      atomics and one order of summation.
// What bounds it: the load/store unit's 128 bytes per clock (76 % busy at
// 348 species: the four 16-byte state loads of a reaction, its record, the
// list rows) and the issue rate (59 %).  Measured on B200, FP64: 348/2163,
// 2^17 points, 5.63 -> 3.14 ms against the kernel it replaced (32-point tiles,
// one reaction a warp, 13 chunks with two barriers each); JetSurf 2.0 3.6 ms;
// 53/325 on the table-driven path 191 -> 290 Mpts/s.  A loop per class (build_runs)
// is 18 % faster than a dispatch per quad (3.31 against 4.04 ms at 348/2163, then).
// The mixed form repeats the generated mixed kernel's arithmetic to the last
// bit: FP64 exponents, FP32 2^f, products and falloff blend, the sums over
// species and reactions in the generated code's order.  It runs the batches
// (and the remainders past whole waves) that would leave the generated
// kernel's wave mostly empty: 53/325, 4096 points, FP64 98 -> 21 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <utility>
#include <vector>

#include "quad.cuh"
#include "rates_generic.cuh"

namespace cg {

struct QuadPlan {
    int nquad = 0, nchunk = 0, nsq = 0, rows = 0, warps = 0;
    int mixed = 0, general = 0;        // general: reactions of kQKindGeneric
    size_t smem = 0;
    int grid = 0;
    const QRec* rec = nullptr;
    const int4* run = nullptr;         // {class, first quad, how many, first slot}
    const int2* efl = nullptr;         // [nquad] efficiency lists
    const QEff* eff = nullptr;
    const QFall* fall = nullptr;
    const int* rbeg = nullptr;         // [nchunk W + 1] first run of each warp in each chunk
    const double* th = nullptr;        // quad_thermo's rows
    QLists lists{};                    // owners: species, [nchunk][nsq] quads
    void* dbuf = nullptr;
};

struct QuadView {
    int nchunk, nsq, rows;
    const QRec* __restrict__ rec;
    const int4* __restrict__ run;
    const int2* __restrict__ efl;
    const QEff* __restrict__ eff;
    const QFall* __restrict__ fall;
    const int* __restrict__ rbeg;
    const double* __restrict__ th;
    QLists lists;
};

// qf - qb of this lane's reaction with forward rate constant kf
// (reactions/standard.j2:3-19).
template <bool WIDE, bool REV>
__device__ __forceinline__ double quad_net(const QRec& R, double kf, const double2* ce) {
    const double2 a0 = quad_row(ce, R.s[0]), a1 = quad_row(ce, R.s[1]);
    double cf = a0.x * a1.x, num = a0.y * a1.y;
    if (WIDE) {
        const double2 a2 = quad_row(ce, R.s2);
        cf *= a2.x;
        num *= a2.y;
    }
    if (!REV) return kf * cf;
    const double2 b0 = quad_row(ce, R.p[0]), b1 = quad_row(ce, R.p[1]);
    double cb = b0.x * b1.x, den = b0.y * b1.y;
    if (WIDE) {
        const double2 b2 = quad_row(ce, R.p2);
        cb *= b2.x;
        den *= b2.y;
    }
    return kf * cf - kf * num * q_rcp(den) * cb;
}

__device__ __forceinline__ double quad_net(int cls, const QRec& R, double kf, const double2* ce) {
    switch (cls & (kQWide | kQRev)) {
        case 0: return quad_net<false, false>(R, kf, ce);
        case kQRev: return quad_net<false, true>(R, kf, ce);
        case kQWide: return quad_net<true, false>(R, kf, ce);
        default: return quad_net<true, true>(R, kf, ce);
    }
}

struct QuadCtx {
    PointT pt;
    double P, lnP, ctot;
    const double2* ce;
    const double* tab;
    int g;
};

// Elementary reactions: the n quads of a run.  The record of the next quad is
// loaded while this one is evaluated.
template <int W, bool WIDE, bool REV>
__device__ __forceinline__ void quad_standard(const QuadCtx& c, const QRec* rec, int n, double* out) {
    QRec N = load_qrec<WIDE>(rec);
    for (; n > 0; --n, out += 32 * W) {
        const QRec R = N;
        rec += kQG * W;
        if (n > 1) N = load_qrec<WIDE>(rec);
        *out = quad_net<WIDE, REV>(R, q_exp(fma(R.b, c.pt.lnT, R.lnA) - R.th * c.pt.invT, c.tab), c.ce);
    }
}

template <int W>
__device__ __forceinline__ void quad_run(const DevMech& m, const QuadView& v, const QuadCtx& c, int cls, int q, int n,
                                         double* out) {
    const int kind = cls & 15;
    const QRec* rec = v.rec + kQG * q + c.g;
    if (kind == CG_STANDARD) {
        switch (cls) {
            case 0: quad_standard<W, false, false>(c, rec, n, out); break;
            case kQRev: quad_standard<W, false, true>(c, rec, n, out); break;
            case kQWide: quad_standard<W, true, false>(c, rec, n, out); break;
            default: quad_standard<W, true, true>(c, rec, n, out); break;
        }
        return;
    }
    if (kind == kQKindGeneric) {
        for (; n > 0; --n, rec += kQG * W, out += 32 * W) {
            const unsigned r = __ldg(&rec->r);
            const double* s = reinterpret_cast<const double*>(c.ce);
            *out = r == kQNone ? 0.0 : generic_rate<2 * kQP>(m, r, c.pt, c.P, c.lnP, c.ctot, s, s + 1);
        }
        return;
    }
    for (; n > 0; --n, q += W, rec += kQG * W, out += 32 * W) {
        const QRec R = load_qrec(rec);
        const double M = quad_m(v.eff, __ldg(v.efl + q), c.g, c.ctot, c.ce);
        if (kind == CG_THIRD_BODY)
            *out = M * quad_net(cls, R, q_exp(fma(R.b, c.pt.lnT, R.lnA) - R.th * c.pt.invT, c.tab), c.ce);
        else
            *out = quad_net(cls, R, quad_falloff(kind, R, v.fall, M, c.pt, c.tab), c.ce);
    }
}

struct MixPt {
    double lnT2, invT;
    float ctot32, Tf, invTf, lnT2f;
};

// The state of the mixed form in its 16-byte pair: G in x, C * 2^32 in the
// low word of y.
__device__ __forceinline__ float mix_c(const double2& s) { return __int_as_float(__double2loint(s.y)); }

// Net rate of progress, mixed precision: the generated mixed kernel's
// expressions (emit_cuda.py reaction32, falloff32) with molecules as slots.
// CLS: the class when it is known at compile time, else -1.
template <int CLS>
__device__ __forceinline__ double quad_rate_mixed(const QuadView& v, int rcls, int q, const QRec& R, int g,
                                                  const MixPt& pt, const double2* ce) {
    const int cls = CLS < 0 ? rcls : CLS;
    const int kind = cls & 15;
    float Ms = pt.ctot32;
    if (kind != CG_STANDARD) {
        const int2 list = __ldg(v.efl + q);
        const double2* e = reinterpret_cast<const double2*>(v.eff + list.x + g);
        for (int k = 0; k < list.y; k += 4) {
            double2 x[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) x[u] = __ldg(e + kQG * (k + u));
#pragma unroll
            for (int u = 0; u < 4; ++u)
                Ms = fmaf(__int_as_float(__double2hiint(x[u].y)), mix_c(quad_row(ce, __double2loint(x[u].y))), Ms);
        }
    }
    double akf = fma(-R.th, pt.invT, fma(R.b, pt.lnT2, R.lnA));
    if (kind > CG_THIRD_BODY) {
        const double2* fp = reinterpret_cast<const double2*>(v.fall + R.aux);
        const double2 f0 = __ldg(fp), f1 = __ldg(fp + 1), f2 = __ldg(fp + 2);
        const float c0 = __int_as_float(__double2loint(f1.y)), c1 = __int_as_float(__double2hiint(f1.y));
        const float c2 = __int_as_float(__double2loint(f2.x)), c3 = __int_as_float(__double2hiint(f2.x));
        const float c4 = __int_as_float(__double2loint(f2.y));
        const double ainf = akf;
        const double a0 = fma(-f1.x, pt.invT, fma(f0.y, pt.lnT2, f0.x));
        int npr;
        float fpr;
        cgg::split2(a0 - ainf, npr, fpr);
        float mpr = cgg::ex2f(fpr) * Ms;
        const int ex = ((__float_as_int(mpr) >> 23) & 0xff) - 126;
        npr += ex - 32;
        mpr = __int_as_float((__float_as_int(mpr) & 0x807fffff) | (126 << 23));   // [0.5, 1)
        float l2r;
        int nfix;
        const float l2m = cgg::lg2f(mpr), l2pr = (float)npr + l2m;
        cgg::falloff_blend(mpr, npr, l2m, l2r, nfix);
        constexpr float kL = 0.30102999566398119521f, kIL = (float)(1.0 / 0.30102999566398119521);
        float l2k = l2r;               // log2 of Pr/(1+Pr) F / 2^nfix
        if (kind == CG_TROE) {
            float Fc = fmaf(c0, cgg::ex2f(c1 * pt.Tf), c2 * cgg::ex2f(c3 * pt.Tf));
            if (c4 != 0.0f) Fc = Fc + cgg::ex2f(c4 * pt.invTf);
            const float lFc = kL * cgg::lg2f(Fc);
            const float lp = kL * l2pr + fmaf(-0.67f, lFc, -0.4f);
            const float f = __fdividef(lp, fmaf(-0.14f, lp, fmaf(-1.27f, lFc, 0.75f)));
            l2k = fmaf(kIL, __fdividef(lFc, fmaf(f, f, 1.0f)), l2r);
        } else if (kind == CG_SRI) {
            const float lp = kL * l2pr;
            const float X = __fdividef(1.0f, fmaf(lp, lp, 1.0f));
            const float base = fmaf(c0, cgg::ex2f(c1 * pt.invTf), cgg::ex2f(c2 * pt.Tf));
            l2k = l2r + (c3 + X * cgg::lg2f(base) + c4 * pt.lnT2f);
        }
        akf = ainf + ((double)nfix + (double)l2k);
    }
    // products and Gibbs sums in the generated code's order: a species that
    // is on a side twice adds 2 G in one rounding
    const float mf = kind == CG_THIRD_BODY ? Ms : 1.0f;
    const double2 a0 = quad_row(ce, R.s[0]), a1 = quad_row(ce, R.s[1]);
    float cf = mix_c(a0) * mix_c(a1);
    double gs = a0.x + a1.x;
    if (cls & kQWide) {
        const double2 a2 = quad_row(ce, R.s2);
        cf *= mix_c(a2);
        gs = R.s[1] == R.s2 ? a0.x + (a1.x + a2.x) : gs + a2.x;
    }
    int n;
    float f;
    cgg::split2(akf, n, f);
    const float e2 = kind <= CG_THIRD_BODY && R.aux ? __uint_as_float(R.aux) : cgg::ex2f(f);
    double rr = (double)(e2 * (cf * mf)) * cgg::exp2i(n - 32 * (int)(R.ord & 0xffu));   // rate2

    if (cls & kQRev) {
        const double2 b0 = quad_row(ce, R.p[0]), b1 = quad_row(ce, R.p[1]);
        float cb = mix_c(b0) * mix_c(b1);
        const double g0 = R.p[0] == R.p[1] ? gs - (b0.x + b1.x) : (gs - b0.x) - b1.x;
        if (cls & kQWide) {
            const double2 b2 = quad_row(ce, R.p2);
            cb *= mix_c(b2);
            gs = R.p[1] != R.p2 ? g0 - b2.x : R.p[0] == R.p2 ? fma(-3.0, b0.x, gs) : (gs - b0.x) - (b1.x + b2.x);
        } else {
            gs = g0;
        }
        rr -= cgg::rate2(akf + gs, cb * mf, -32 * (int)((R.ord >> 8) & 0xffu));
    }
    return rr;
}

// The n quads of a run, mixed (see quad_standard).
template <int W, int CLS>
__device__ __forceinline__ void quad_run_mixed(const QuadView& v, int cls, int q, int n, int g, const MixPt& pt,
                                               const double2* ce, double* out) {
    const QRec* rec = v.rec + kQG * q + g;
    QRec N = load_qrec(rec);
    for (; n > 0; --n, q += W, out += 32 * W) {
        const QRec R = N;
        rec += kQG * W;
        if (n > 1) N = load_qrec(rec);
        *out = quad_rate_mixed<CLS>(v, cls, q, R, g, pt, ce);
    }
}

// wdot of this quarter-warp's species, mixed: the reactions' rates added one by
// one in file order as the generated kernel does (its bits: the two serve
// batches of different sizes).  Entries: row | {0, 2, 3 for coefficients
// 1, 2, 3} << 13 | minus << 15.
__device__ __forceinline__ double sequence_sum(const QLists& L, const QOwn& o, int g, const double* rows) {
    double acc = 0.0;
    auto add = [&](unsigned e) {
        // 1.0, 2.0, 3.0 are 0x3ff00000 + 0x80000 {0, 2, 3}: the entry holds {0, 2, 3}
        const int hi = (int)((((e & 0x6000u) << 6) + 0x3ff00000u) | ((e & 0x8000u) << 16));
        acc = fma(__hiloint2double(hi, 0), rows[(e & 0x1fffu) * kQP], acc);
    };
    const uint4* q = L.ent + o.ptr + g;
    const int n = (int)o.cnt;
    uint4 w = o.rows;
    for (int k = 0; k < n; ++k) {
        const uint4 c = w;
        if (k + 1 < n) w = __ldg(q + kQG * k);
        add(c.x & 0xffffu), add(c.x >> 16), add(c.y & 0xffffu), add(c.y >> 16);
        add(c.z & 0xffffu), add(c.z >> 16), add(c.w & 0xffffu), add(c.w >> 16);
    }
    return acc;
}

template <int W, int MINB, bool MIXED>
__global__ void __launch_bounds__(32 * W, MINB)
    getrates_quad(const __grid_constant__ DevMech m, const __grid_constant__ QuadView v, const double* __restrict__ P, const double* __restrict__ Tg,
                  const double* __restrict__ Y, double* __restrict__ wdot, int64_t i0, int64_t ng, int64_t n1,
                  const unsigned long long* __restrict__ count) {
    extern __shared__ __align__(16) double smem[];
    const int ns = m.ns;
    const int lane = threadIdx.x & 31, p = lane & (kQP - 1), g = lane >> 3;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);   // warp-uniform
    double* sTab = smem;                                   // [16] 2^(j/16)
    double* sH = sTab + 16;                                // [2][4][8] this tile's and the next one's T, ln T, 1/T, P
    double* sRed = sH + 8 * kQP;                           // [W][8]
    double2* sCE = reinterpret_cast<double2*>(sRed + W * kQP);   // [ns + 1][8]
    double* sQ = reinterpret_cast<double*>(sCE + (ns + 1) * kQP);   // [rows + 1][8]
    double* sW = sQ + (v.rows + 1) * kQP;                  // [ns][8], several chunks only
    // points [i0, n1) of arrays with stride ng; with a device-side count only
    // those below min(*count, n1)
    const int64_t npts = count ? min(n1, (int64_t)*count) : n1;
    if (threadIdx.x < 16) sTab[threadIdx.x] = kQExpTab[threadIdx.x];
    if (warp == W - 1 && g == 0) quad_head<MIXED>(sH, i0 + (int64_t)blockIdx.x * kQP + p, npts, P, Tg);
    if (threadIdx.x < kQP) {
        sQ[v.rows * kQP + p] = 0.0;                        // the zero row of the lists
        if (MIXED) sCE[ns * kQP + p] = make_double2(0.0, __hiloint2double(0, __float_as_int(1.0f)));
        else sCE[ns * kQP + p] = make_double2(1.0, 1.0);
    }
    __syncthreads();
    const double2* ce = sCE + p;
    const int64_t step = (int64_t)gridDim.x * kQP;
    int buf = 0;
    for (int64_t t0 = i0 + (int64_t)blockIdx.x * kQP; t0 < npts; t0 += step, buf ^= 1) {
        const int64_t i = t0 + p;
        const bool act = i < npts;
        const double* h = sH + buf * 4 * kQP + p;
        PointT pt;
        pt.T = h[0];
        pt.lnT = h[kQP];
        pt.invT = h[2 * kQP];
        const double T = pt.T, Pp = h[3 * kQP];
        MixPt mp;
        mp.lnT2 = pt.lnT * cgg::kLog2e;
        mp.invT = pt.invT;
        // exp_g.j2:2-27 with pfac = Patm/(R0 T) folded in; the sum of Y/W
        const double pfac = kPatm / kR0 * pt.invT;
        const double lpfac2 = -6.35856916300311 - mp.lnT2;   // log2(Patm/R0) - log2 T
        double part = 0.0;
        for (int k = 4 * warp + g; k < ns; k += 4 * W) {
            const double c = (act ? __ldcs(Y + (int64_t)k * ng + i) : 1.0) * __ldg(m.inv_mw + k);
            double cf[8];
            quad_thermo(v.th, k, T, cf);
            const double smh = smh_poly(cf, T, pt.lnT, pt.invT);
            part += c;
            if (MIXED) sCE[k * kQP + p] = make_double2(fma(smh, cgg::kLog2e, lpfac2), c);
            else sCE[k * kQP + p] = make_double2(c, q_exp(smh, sTab) * pfac);
        }
        double fac, ctot;
        if (MIXED) {
            // the generated kernel's order of summation: one warp adds species
            // after species
            __syncthreads();
            if (warp == 0) {
                double csum = 0.0, ct = 0.0;
#pragma unroll 4
                for (int k = 0; k < ns; ++k) csum += sCE[k * kQP + p].y;
                const double facs = Pp * cgm::cg_rcp(kR0 * csum * T) * 4294967296.0;
#pragma unroll 4
                for (int k = 0; k < ns; ++k) ct += sCE[k * kQP + p].y * facs;
                if (g == 0) {
                    sRed[p] = facs;
                    sRed[kQP + p] = ct;
                }
            }
            __syncthreads();
            fac = sRed[p];             // times 2^32
            ctot = sRed[kQP + p];
        } else {
            part += __shfl_xor_sync(0xffffffffu, part, 8);
            part += __shfl_xor_sync(0xffffffffu, part, 16);
            if (g == 0) sRed[warp * kQP + p] = part;
            __syncthreads();
            const double csum = quad_total<W>(sRed, g);
            fac = Pp * cgm::cg_rcp(kR0 * csum * T);            // ytoc.j2:3-18
            ctot = csum * fac;
        }
        for (int k = 4 * warp + g; k < ns; k += 4 * W) {
            if (MIXED) {
                const float c = (float)(sCE[k * kQP + p].y * fac);
                sCE[k * kQP + p].y = __hiloint2double(0, __float_as_int(c));
            } else {
                sCE[k * kQP + p].x *= fac;
            }
        }
        mp.ctot32 = (float)ctot;           // mixed: scaled by 2^32
        mp.Tf = (float)T;
        mp.invTf = (float)pt.invT;
        mp.lnT2f = (float)mp.lnT2;
        const double lnP = (!MIXED && m.seg[CG_PLOG] < m.seg[CG_PLOG + 1]) ? cgm::cg_log(Pp) : 0.0;
        __syncthreads();
        for (int c = 0; c < v.nchunk; ++c) {
            const int* rb = v.rbeg + c * W + warp;
            const int r1 = __ldg(rb + 1);
            for (int r = __ldg(rb); r < r1; ++r) {
                const int4 rn = __ldg(v.run + r);
                const int cls = __shfl_sync(0xffffffffu, rn.x, 0), n = __shfl_sync(0xffffffffu, rn.z, 0);
                double* out = sQ + rn.w + lane;
                if (MIXED) {
                    switch (cls) {
                        case 0: quad_run_mixed<W, 0>(v, cls, rn.y, n, g, mp, ce, out); break;
                        case kQRev: quad_run_mixed<W, kQRev>(v, cls, rn.y, n, g, mp, ce, out); break;
                        case kQWide: quad_run_mixed<W, kQWide>(v, cls, rn.y, n, g, mp, ce, out); break;
                        case kQWide | kQRev: quad_run_mixed<W, (kQWide | kQRev)>(v, cls, rn.y, n, g, mp, ce, out); break;
                        default: quad_run_mixed<W, -1>(v, cls, rn.y, n, g, mp, ce, out); break;
                    }
                } else {
                    const QuadCtx qc{pt, Pp, lnP, ctot, ce, sTab, g};
                    quad_run<W>(m, v, qc, cls, rn.y, n, out);
                }
            }
            if (c == 0 && warp == W - 1 && g == 0 && t0 + step < npts)
                quad_head<MIXED>(sH + (buf ^ 1) * 4 * kQP, t0 + step + p, npts, P, Tg);
            __syncthreads();
            const bool last = c == v.nchunk - 1;
            if (warp < v.nsq) {
                const QOwn* op = v.lists.own + kQG * (c * v.nsq + warp) + g;
                QOwn N = load_qown(op);
                for (int s = warp; s < v.nsq; s += W) {
                    const QOwn o = N;
                    op += kQG * W;
                    if (s + W < v.nsq) N = load_qown(op);
                    double acc = MIXED ? sequence_sum(v.lists, o, g, sQ + p) : list_sum(v.lists, o, g, sQ + p);
                    const int k = o.own;
                    if (k >= 0) {
                        if (c > 0) acc += sW[k * kQP + p];
                        if (!last) sW[k * kQP + p] = acc;
                        else if (act) __stcs(wdot + (int64_t)k * ng + i, acc);
                    }
                }
            }
            if (!last) __syncthreads();
        }
    }
}

using QuadKernel = void (*)(const DevMech, const QuadView, const double*, const double*, const double*, double*, int64_t, int64_t,
                            int64_t, const unsigned long long*);

static QuadKernel quad_kernel(int warps, int mixed) {
    switch (warps) {
        case 8: return mixed ? getrates_quad<8, 4, true> : getrates_quad<8, 4, false>;
        case 16: return mixed ? getrates_quad<16, 2, true> : getrates_quad<16, 2, false>;
        default: return mixed ? getrates_quad<32, 1, true> : getrates_quad<32, 1, false>;
    }
}

// Species up to which the FP64 call has needed no workspace from its caller
// (what 32-point tiles of C and EGp left of shared memory); beyond, the
// global-scratch kernel asks for one, although the tiles would fit to 511.
constexpr int kQuadMaxSpecies = 437;

int quad_tile_points() { return kQP; }
int quad_general(const QuadPlan* p) { return p->general; }

// latency: 32 warps to a tile whatever its size, for batches of few tiles.
cudaError_t quad_prepare(const DevMech& m, const cg_mech_view& v, int device, int mixed, int latency,
                         QuadPlan** out) {
    *out = nullptr;
    const int ns = m.ns, nr = m.nr;
    if (nr == 0 || ns > kQuadMaxSpecies) return cudaErrorNotSupported;
    HostQuads h;
    build_quads(v, h);
    if (mixed && (!h.mixed_ok || 4 * h.nquad >= 0x1fff)) return cudaErrorNotSupported;
    DeviceLimits dev;
    cudaError_t e = device_limits(device, &dev);
    if (e != cudaSuccess) return e;
    const size_t limit = dev.smem_block, per_sm = dev.smem_sm;
    QuadPlan pl;
    pl.mixed = mixed;
    pl.nquad = h.nquad;
    pl.general = h.ngeneric;
    // chunks: every reaction at once when the rates fit beside the state
    auto bytes = [&](int rows, int chunks, int warps) {
        return (16 + ((size_t)8 + 2 * (ns + 1) + rows + 1 + warps + (chunks > 1 ? ns : 0)) * kQP) * sizeof(double);
    };
    int qpc = h.nquad;
    if (bytes(4 * qpc, 1, 32) > limit) {
        qpc = (int)((limit - bytes(0, 2, 32)) / (4 * kQP * sizeof(double)));
        qpc = std::min(qpc, 16000);                        // rows are 16-bit indices
    }
    pl.nchunk = (h.nquad + qpc - 1) / qpc;
    qpc = (h.nquad + pl.nchunk - 1) / pl.nchunk;
    pl.rows = 4 * qpc;
    // warps per CTA and CTAs per SM: 32 resident warps of 64 registers, in as
    // many CTAs as shared memory allows (against 24 of 80 registers: 348/2163 at
    // 2^17 points 3.31 -> 3.14 ms, 53/325 at 4096 points 26.6 -> 20.9 us)
    const int fit = (int)(per_sm / (bytes(pl.rows, pl.nchunk, 32) + 1024));
    if (latency && fit < 2) return cudaErrorNotSupported;   // the plan for throughput is the same
    pl.warps = latency || fit < 2 ? 32 : fit <= 3 ? 16 : 8;
    pl.smem = bytes(pl.rows, pl.nchunk, pl.warps);
    const int resident = std::max(1, std::min((int)(per_sm / (pl.smem + 1024)), 32 / pl.warps));
    pl.grid = dev.sms * resident;
    // per-species lists of (row, net coefficient), in sorted-reaction order
    std::vector<int> qbeg(pl.nchunk + 1);
    for (int c = 0; c <= pl.nchunk; ++c) qbeg[c] = std::min(h.nquad, c * qpc);
    std::vector<int4> run;
    std::vector<int> rbeg;
    build_runs(h, qbeg, pl.warps, run, rbeg);
    for (int c = 0; c < pl.nchunk; ++c)
        for (int r = rbeg[c * pl.warps]; r < rbeg[(c + 1) * pl.warps]; ++r) run[r].w = (run[r].y - qbeg[c]) * 32;
    const int32_t* rp = (const int32_t*)v.a[CG_RPTR];
    const int32_t* pp = (const int32_t*)v.a[CG_PPTR];
    const int32_t* rsp = (const int32_t*)v.a[CG_RSP];
    const int32_t* psp = (const int32_t*)v.a[CG_PSP];
    const double* rnu = (const double*)v.a[CG_RNU];
    const double* pnu = (const double*)v.a[CG_PNU];
    std::vector<int> order(nr);
    for (int r = 0; r < nr; ++r) order[r] = r;
    std::sort(order.begin(), order.end(), [&](int a, int b) { return h.at[a] < h.at[b]; });
    std::vector<std::vector<ListBuilder::List>> lists(pl.nchunk, std::vector<ListBuilder::List>(ns));
    std::vector<double> net(ns, 0.0);
    for (int r : order) {
        const int c = (h.at[r] / 4) / qpc, row = h.at[r] - 4 * qbeg[c];
        for (int j = rp[r]; j < rp[r + 1]; ++j) net[rsp[j]] -= rnu[j];
        for (int j = pp[r]; j < pp[r + 1]; ++j) net[psp[j]] += pnu[j];
        for (int side = 0; side < 2; ++side)
            for (int j = side ? pp[r] : rp[r]; j < (side ? pp[r + 1] : rp[r + 1]); ++j) {
                const int k = side ? psp[j] : rsp[j];
                if (net[k] != 0.0) lists[c][k].push_back({row, net[k]});
                net[k] = 0.0;
            }
    }
    // (with several chunks, grouped by the lists over all of them)
    std::vector<ListBuilder::List> all(ns);
    for (const auto& l : lists)
        for (int k = 0; k < ns; ++k) all[k].insert(all[k].end(), l[k].begin(), l[k].end());
    std::vector<const ListBuilder::List*> al;
    for (const auto& l : all) al.push_back(&l);
    const std::vector<std::vector<int>> quads = ListBuilder::group(al, pl.warps);
    pl.nsq = (int)quads.size();
    ListBuilder lb;
    for (int c = 0; c < pl.nchunk; ++c)
        for (const std::vector<int>& q : quads) {
            std::vector<const ListBuilder::List*> own;
            for (int k : q) own.push_back(&lists[c][k]);
            lb.add_quad(own, q, pl.rows);
        }
    if (!lb.fits) return cudaErrorNotSupported;
    if (mixed) {
        // every coefficient of every side, in file order; one chunk
        if (pl.nchunk > 1) return cudaErrorNotSupported;
        const int32_t* orig = (const int32_t*)v.a[CG_ORIG];
        std::vector<int> file(nr);
        for (int r = 0; r < nr; ++r) file[r] = r;
        std::sort(file.begin(), file.end(), [&](int a, int b) { return orig[a] < orig[b]; });
        std::vector<std::vector<unsigned>> seq(ns);
        for (int r : file)
            for (int side = 0; side < 2; ++side)
                for (int j = side ? pp[r] : rp[r]; j < (side ? pp[r + 1] : rp[r + 1]); ++j) {
                    const double nu = side ? pnu[j] : rnu[j];
                    const unsigned mult = nu == 1.0 ? 0u : nu == 2.0 ? 0x4000u : 0x6000u;   // integers up to 3: a fast form
                    seq[side ? psp[j] : rsp[j]].push_back((unsigned)h.at[r] | mult | (side ? 0u : 0x8000u));
                }
        std::vector<int> sp(ns);
        for (int k = 0; k < ns; ++k) sp[k] = k;
        std::stable_sort(sp.begin(), sp.end(), [&](int a, int b) { return seq[a].size() > seq[b].size(); });
        lb = ListBuilder();
        pl.nsq = (ns + kQG - 1) / kQG;
        for (int s = 0; s < pl.nsq; ++s) {
            const unsigned n8 = std::max<unsigned>((unsigned)(seq[sp[kQG * s]].size() + 7) / 8, 1);
            QOwn own[kQG];
            const int ptr = (int)lb.ent.size();
            for (unsigned k = 0; k < n8; ++k)
                for (int g = 0; g < kQG; ++g) {
                    const int i = kQG * s + g;
                    unsigned e[8];
                    for (unsigned u = 0; u < 8; ++u)
                        e[u] = i < ns && 8 * k + u < seq[sp[i]].size() ? seq[sp[i]][8 * k + u] : (unsigned)pl.rows;
                    const uint4 w =
                        make_uint4(e[0] | e[1] << 16, e[2] | e[3] << 16, e[4] | e[5] << 16, e[6] | e[7] << 16);
                    if (k == 0) own[g] = QOwn{i < ns ? sp[i] : -1, n8, ptr, 0u, w};
                    else lb.ent.push_back(w);
                }
            lb.own.insert(lb.own.end(), own, own + kQG);
        }
    }
    Image im;
    const size_t o_rec = im.put(mixed ? h.rec2 : h.rec), o_run = im.put(run), o_efl = im.put(h.efl), o_eff = im.put(h.eff);
    const size_t o_fall = im.put(mixed ? h.fall2 : h.fall), o_rb = im.put(rbeg), o_th = im.put(quad_thermo_rows(v));
    const size_t o_li = im.put(lb.own), o_le = im.put(lb.ent), o_lg = im.put(lb.gen);
    QuadPlan* q = new QuadPlan(pl);
    e = im.upload(&q->dbuf);
    if (e == cudaSuccess) e = raise_smem_limit((const void*)quad_kernel(q->warps, mixed), q->smem);
    if (e != cudaSuccess) {
        if (q->dbuf) cudaFree(q->dbuf);
        delete q;
        return e;
    }
    char* d = (char*)q->dbuf;
    q->rec = (const QRec*)(d + o_rec);
    q->run = (const int4*)(d + o_run);
    q->efl = (const int2*)(d + o_efl);
    q->eff = (const QEff*)(d + o_eff);
    q->fall = (const QFall*)(d + o_fall);
    q->rbeg = (const int*)(d + o_rb);
    q->th = (const double*)(d + o_th);
    q->lists = QLists{(const QOwn*)(d + o_li), (const uint4*)(d + o_le), (const QGen*)(d + o_lg)};
    *out = q;
    return cudaSuccess;
}

void quad_release(QuadPlan* p) {
    if (!p) return;
    if (p->dbuf) cudaFree(p->dbuf);
    delete p;
}

// Points [i0, n1) of arrays laid out for ng points (all: i0 = 0, n1 = ng).
cudaError_t launch_getrates_quad(const QuadPlan* p, const DevMech& m, const double* P, const double* T,
                                 const double* Y, double* wdot, int64_t i0, int64_t ng, int64_t n1, cudaStream_t s,
                                 const unsigned long long* count) {
    if (n1 <= i0) return cudaSuccess;
    const int64_t tiles = (n1 - i0 + kQP - 1) / kQP;
    const unsigned grid = (unsigned)std::min<int64_t>(tiles, p->grid);
    const QuadView v{p->nchunk, p->nsq, p->rows, p->rec, p->run, p->efl, p->eff, p->fall, p->rbeg, p->th, p->lists};
    const QuadKernel fn = quad_kernel(p->warps, p->mixed);
    fn<<<grid, 32u * (unsigned)p->warps, p->smem, s>>>(m, v, P, T, Y, wdot, i0, ng, n1, count);
    return cudaGetLastError();
}

}  // namespace cg
