// Shared pieces of the quad kernels: table-driven kernels in which a tile is
// eight grid points and a warp works on four reactions at once, lane =
// 8 * (reaction of the quad) + (point of the tile).
//
// Why eight points.  With one point per lane a tile's C and EGp took 16 ns 32
// bytes (178 KB at 348 species), which left room to stage only ~180 rates of
// progress, so a 2163-reaction mechanism went through 13 chunks with two
// block barriers each.  With eight points the state takes a quarter of that
// and the rates of all 2163 reactions fit beside it (45 + 139 KB): one pass
// over the reactions, one over the species.  A 53-species tile takes 28 KB, so
// several independent CTAs share an SM, and a batch of a few thousand points
// still fills the chip.  Reactions are sorted by kind and size on the host,
// so the four reactions of a quad run the same code and no lane diverges.
//
// The state of a species at a point is one 16-byte pair {C, EGp} (FP64) or
// {log2 Gibbs term, C * 2^32} (mixed), so that a molecule costs one 16-byte
// shared load; a quarter-warp (8 lanes, 128 bytes) reads one species row, and
// no access has a bank conflict.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <vector>

#include "cg_math.cuh"
#include "gen_common.cuh"
#include "rates_common.cuh"

namespace cg {

constexpr int kQP = 8;                 // points per tile
constexpr int kQG = 4;                 // reactions (species, entries) per warp
constexpr int kQRow = 16 * kQP;        // bytes of one species' row of the state
constexpr int kQKindGeneric = 6;       // reactions evaluated from their DRxn record

// ------------------------------------------------------------ exponential
// exp(x) = 2^n 2^(j/16) e^r with 16 n + j = round(16 x / ln 2): r <= ln2/32, so
// the series needs degree 7 instead of 12, and 2^(j/16) comes from a 16-entry
// table in shared memory (16 banks pairs: no conflict whatever the lanes'
// j).  ln2/16 is split into a 21-bit head (its product with the integer is
// exact, and its low word is zero, as are those of the coefficients 1/5! ..
// 1/7!, rounded to 21 bits where their rounding stays below 2^-57 of the
// result: such constants are immediates of the FP64 instruction) and a tail.
// Largest error 1.7 ulp over [-700, 700].  The exponent is taken from bits
// 4..35 of the rounded 16 x / ln 2 and saturates to 0 or +inf as cg_exp's does,
// so no x with |x| < 1.4e9 needs a clamp.  For that the FP64 kernels keep 1/T <=
// 700 and evaluate reactions with Ea/Rc > 1e6 K elsewhere: a difference of two
// exponents (falloff's ln k0 - ln kinf) then reaches it too.  Down to T = 1/700
// K nothing is clamped; below, the clamp changes only rates with Ea/Rc < 1 K,
// all others being 0 or +inf already.
struct QExp {
    double l16, lo, c4, c3;
};
static __constant__ QExp kQExp = {23.083120654223414, -2.9683281493947953e-08, 0.041666666666666664,
                                  0.16666666666666666};
static __constant__ double kQExpTab[16] = {
    1.0, 1.0442737824274138, 1.0905077326652577, 1.1387886347566916, 1.189207115002721, 1.241857812073484,
    1.2968395546510096, 1.3542555469368927, 1.4142135623730951, 1.4768261459394993, 1.5422108254079407,
    1.6104903319492543, 1.681792830507429, 1.7562521603732995, 1.8340080864093424, 1.9152065613971474};
constexpr double kQMaxInvT = 700.0, kQMaxTheta = 1e6, kQMinArg = -9e7;

__device__ __forceinline__ double q_exp(double x, const double* tab) {
    const double t = fma(x, kQExp.l16, cgm::kRound);
    const double k = t - cgm::kRound;
    double r = fma(k, -0.04332166910171509, x);
    r = fma(k, kQExp.lo, r);
    const int n = __double2loint(t), k2 = (int)__funnelshift_r(n, __double2hiint(t), 4);   // floor(16 x / ln 2 / 16)
    double p = fma(0.00019841268658638, r, 0.00138888880610466);
    p = fma(p, r, 0.00833333283662796);
    p = fma(p, r, kQExp.c4);
    p = fma(p, r, kQExp.c3);
    p = fma(p, r, 0.5);
    p = fma(p, r, 1.0);
    const double b = tab[n & 15];
    const int e = max(0, min(k2 + 1023, 2047));
    return fma(b, p * r, b) * __hiloint2double(e << 20, 0);
}

// 1/x from the hardware's approximation a (error e < 2^-20): a (1 + e + e^2).
__device__ __forceinline__ double q_rcp(double x) {
    double a;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(a) : "d"(x));
    const double e = fma(-x, a, 1.0);
    return fma(a, fma(e, e, e), a);
}

// One reaction, 48 bytes.  s, p: byte offset (species * kQRow) of each
// reactant and product molecule's row of the state; unused slots name the
// dummy species ns (C = EGp = 1, G = 0).  FP64 tables hold
// ln|A|, b, Ea/Rc; mixed ones log2|A|, b, (Ea/Rc) log2 e.  An elementary
// reaction with at most two molecules a side needs the first 32 bytes only.
struct __align__(16) QRec {
    double lnA, b, th;
    unsigned short s[2], p[2];         // the first two molecules of each side
    unsigned short s2, p2;             // the third ones
    unsigned int r;                    // reaction in kernel order
    unsigned int aux;                  // falloff or PLOG row; mixed: 2^f of a constant rate as FP32 bits, else 0
    unsigned int ord;                  // molecules a side, << 0 / << 8 (M included)
};
static_assert(sizeof(QRec) == 48, "QRec must stay 48 bytes");

// One third-body efficiency: M += val C, sp the byte offset of the species' row.
struct __align__(16) QEff {
    double val;
    unsigned int sp;
    float fval;
};

// Falloff parameters: ln A0, b0, Ea0/Rc and Troe {1-a, 1/T3, a, 1/T1, T2} or
// SRI {a, b, 1/c, d, e}; in the mixed tables log2 A0, b0, (Ea0/Rc) log2 e and
// the FP32 constants of the generated mixed kernel.
struct __align__(16) QFall {
    double lnA0, b0, th0, p[5];
};
static_assert(sizeof(QFall) == 64, "QFall must stay 64 bytes");

// Class of a quad's reactions: kind | kQWide (three molecules on a side that
// counts) | kQRev.
constexpr int kQWide = 16, kQRev = 32;
constexpr unsigned kQNone = 0xffffffffu;   // QRec.r of a repeat that fills a quad

// Weighted entry of a row list (net coefficients other than +-1).
struct __align__(16) QGen {
    double coef;
    unsigned int row, pad;
};

// Row lists.  A quad is either four owners (species, matrix entries), one to a
// quarter-warp, or one owner with a long list split four ways, whose parts
// are added by shuffles.  An owner's list is n4 half-steps of four 16-bit rows
// -- n4neg half-steps of rows to subtract, then rows to add -- two to a step,
// and ngen weighted entries.  The first step is in the owner's record, so
// that a short list costs one load, which the loop over quads makes a quad
// ahead; the others follow at ent[ptr], uint4 per step and quarter-warp.
struct __align__(16) QOwn {
    int own;                           // what the sum is for; < 0: nothing
    unsigned cnt;                      // n4neg | n4 << 16 | kOwnWide
    int ptr;
    unsigned gen;                      // first weighted entry / kQG | ngen << 20
    uint4 rows;
};
static_assert(sizeof(QOwn) == 32, "QOwn must stay 32 bytes");
constexpr unsigned kOwnWide = 1u << 31;
struct QLists {
    const QOwn* own;                   // [4 quads]
    const uint4* ent;
    const QGen* gen;
};

__device__ __forceinline__ QOwn load_qown(const QOwn* p) {
    const uint4* q = reinterpret_cast<const uint4*>(p);
    QOwn o;
    uint4* d = reinterpret_cast<uint4*>(&o);
    d[0] = __ldg(q);
    d[1] = __ldg(q + 1);
    return o;
}

template <bool ALL = true>
__device__ __forceinline__ QRec load_qrec(const QRec* p) {
    const int4* q = reinterpret_cast<const int4*>(p);
    QRec r;
    int4* d = reinterpret_cast<int4*>(&r);
    d[0] = __ldg(q);
    d[1] = __ldg(q + 1);
    if (ALL) d[2] = __ldg(q + 2);
    return r;
}

// Coefficients of smh for this lane's temperature (T < Tmid -> low), from
// rows of eight doubles {c0 .. c6, Tmid}, low then high: a lane loads the one
// range that it needs (64 bytes; both ranges and a select per coefficient
// were a quarter of a large mechanism's load bandwidth).
__device__ __forceinline__ void quad_thermo(const double* th, int k, double T, double (&c)[8]) {
    const double* row = th + 16 * k + (T < __ldg(th + 16 * k + 7) ? 0 : 8);
#pragma unroll
    for (int j = 0; j < 4; ++j)
        reinterpret_cast<double2*>(c)[j] = __ldg(reinterpret_cast<const double2*>(row) + j);
}

// The row of the state at byte offset `off`, this lane's point.
__device__ __forceinline__ double2 quad_row(const double2* ce, unsigned off) {
    return *reinterpret_cast<const double2*>(reinterpret_cast<const char*>(ce) + off);
}

// Sum of the row list of this quarter-warp's owner.  `rows` points at this
// lane's point of row 0 (a row is kQP doubles).  Steps after the first are
// loaded two ahead: with one in flight, a large mechanism's longest list,
// coming from L2, took longer than its reactions.
__device__ __forceinline__ double list_sum(const QLists& L, const QOwn& o, int g, const double* rows) {
    const int neg = (int)(o.cnt & 0xffffu), n4 = (int)((o.cnt >> 16) & 0x7fffu);
    auto row = [&](unsigned r) { return rows[r * kQP]; };
    auto half = [&](unsigned a, unsigned b, bool minus) {
        const double x = (row(a & 0xffffu) + row(a >> 16)) + (row(b & 0xffffu) + row(b >> 16));
        return minus ? -x : x;
    };
    double acc = half(o.rows.x, o.rows.y, neg > 0);
    if (n4 > 1) acc += half(o.rows.z, o.rows.w, neg > 1);
    if (n4 > 2) {
        const int n = (n4 + 1) >> 1;
        auto step = [&](double x, int k, const uint4& c) {
            x += half(c.x, c.y, 2 * k < neg);
            return x + half(c.z, c.w, 2 * k + 1 < neg);    // rows of zeros past n4
        };
        const uint4* e = L.ent + o.ptr + g;
        uint4 w0 = __ldg(e), w1 = n > 2 ? __ldg(e + kQG) : w0;
        for (int k = 1; k < n; k += 2) {
            const uint4 c0 = w0, c1 = w1;
            e += 2 * kQG;
            if (k + 2 < n) w0 = __ldg(e);
            if (k + 3 < n) w1 = __ldg(e + kQG);
            acc = step(acc, k, c0);
            if (k + 1 < n) acc = step(acc, k + 1, c1);
        }
    }
    const int ngen = (int)(o.gen >> 20);
    if (ngen) {
        const double2* ge = reinterpret_cast<const double2*>(L.gen + kQG * (o.gen & 0xfffffu) + g);
        for (int k = 0; k < ngen; k += 2) {                 // padded to pairs
            const double2 v0 = __ldg(ge + kQG * k), v1 = __ldg(ge + kQG * (k + 1));
            acc = fma(v0.x, row((unsigned)__double2loint(v0.y)), acc);
            acc = fma(v1.x, row((unsigned)__double2loint(v1.y)), acc);
        }
    }
    if (o.cnt & kOwnWide) {
        acc += __shfl_xor_sync(0xffffffffu, acc, 8);
        acc += __shfl_xor_sync(0xffffffffu, acc, 16);
    }
    return acc;
}

// M = ctot + sum_e (eff_e - 1) C[sp_e] (third_body.j2:18-31), in the table's order.
__device__ __forceinline__ double quad_m(const QEff* eff, int2 list, int g, double ctot, const double2* ce) {
    double M = ctot;
    const double2* e = reinterpret_cast<const double2*>(eff + list.x + g);
    for (int k = 0; k < list.y; k += 4) {          // lists are padded to fours (dummy species, 0)
        double2 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = __ldg(e + kQG * (k + u));
#pragma unroll
        for (int u = 0; u < 4; ++u) M = fma(v[u].x, quad_row(ce, __double2loint(v[u].y)).x, M);
    }
    return M;
}

// Falloff forward rate constant (troe.j2:21-45; Lindemann F = 1; SRI) with
// Pr = exp(ln k0 - ln kinf) M and ln F folded into the exponent of kinf.
__device__ __forceinline__ double quad_falloff(int kind, const QRec& R, const QFall* fall, double M,
                                               const PointT& pt, const double* tab) {
    const double2* q = reinterpret_cast<const double2*>(fall + R.aux);
    const double2 f0 = __ldg(q), f1 = __ldg(q + 1), f2 = __ldg(q + 2), f3 = __ldg(q + 3);
    const double lkinf = fma(R.b, pt.lnT, R.lnA) - R.th * pt.invT;
    const double lr = (fma(f0.y, pt.lnT, f0.x) - f1.x * pt.invT) - lkinf;
    const double Pr = q_exp(lr, tab) * M;
    double lnF = 0.0;
    if (kind == CG_TROE) {
        double Fc = fma(f1.y, q_exp(fmax(-pt.T * f2.x, kQMinArg), tab), f2.y * q_exp(fmax(-pt.T * f3.x, kQMinArg), tab));
        if (f3.y != 0.0) Fc += q_exp(fmax(-f3.y * pt.invT, kQMinArg), tab);
        const double lFc = cgm::cg_log10(Fc);
        const double lp = fma(lr, 0.43429448190325182765, cgm::cg_log10(M)) + fma(-0.67, lFc, -0.4);
        const double f = lp * q_rcp(fma(-0.14, lp, fma(-1.27, lFc, 0.75)));
        lnF = 2.302585092994045684 * lFc * q_rcp(fma(f, f, 1.0));
    } else if (kind == CG_SRI) {
        const double lp = fma(lr, 0.43429448190325182765, cgm::cg_log10(M));
        const double X = q_rcp(fma(lp, lp, 1.0));
        const double base = fma(f1.y, q_exp(fmax(-f2.x * pt.invT, kQMinArg), tab), q_exp(fmax(-pt.T * f2.y, kQMinArg), tab));
        lnF = cgm::cg_log(f3.x) + fma(X, cgm::cg_log(base), f3.y * pt.lnT);
    }
    return cgm::cg_exp_clamped(lkinf + lnF) * (Pr * q_rcp(1.0 + Pr));
}

// A tile's T, ln T, 1/T and P, [4][8] in shared memory.  One warp forms the
// next tile's while the others evaluate reactions: ln T in every warp was a
// tenth of a 53-species tile's instructions.  The mixed form has no q_exp and
// takes 1/T as it is, like the generated kernel.
template <bool MIXED = false>
__device__ __forceinline__ void quad_head(double* h, int64_t i, int64_t n, const double* P, const double* Tg) {
    const int p = threadIdx.x & (kQP - 1);
    const double T = i < n ? __ldcs(Tg + i) : 1000.0;
    h[p] = T;
    h[kQP + p] = cgm::cg_log(T);
    h[2 * kQP + p] = MIXED ? cgm::cg_rcp(T) : fmin(cgm::cg_rcp(T), kQMaxInvT);
    h[3 * kQP + p] = i < n ? __ldcs(P + i) : kPatm;
}

// Sum over the warps' parts sRed[w][8], each quarter-warp a share of them.
template <int W>
__device__ __forceinline__ double quad_total(const double* red, int g) {
    double x = 0.0;
    const int p = threadIdx.x & (kQP - 1);
#pragma unroll
    for (int w = 0; w < W / kQG; ++w) x += red[(kQG * w + g) * kQP + p];
    x += __shfl_xor_sync(0xffffffffu, x, 8);
    return x + __shfl_xor_sync(0xffffffffu, x, 16);
}

// ------------------------------------------------------------------ host
// The reactions sorted into quads.
struct HostQuads {
    int ns = 0, nr = 0, nquad = 0, ngeneric = 0, nplog = 0;
    std::vector<QRec> rec, rec2;       // [4 nquad] FP64 and log2 (mixed) tables
    std::vector<int> key;              // [nquad] class
    std::vector<int2> efl;             // [nquad]
    std::vector<QEff> eff;
    std::vector<QFall> fall, fall2;
    std::vector<int> at;               // position (4 quad + group) of each reaction
    bool mixed_ok = true;              // every reaction has a pre-decoded form
};

// The rows of quad_thermo.
inline std::vector<double> quad_thermo_rows(const cg_mech_view& v) {
    const int ns = (int)v.s[CG_S_NS];
    const double* tmid = (const double*)v.a[CG_TMID];
    const double* rng[2] = {(const double*)v.a[CG_SMH_LO], (const double*)v.a[CG_SMH_HI]};
    std::vector<double> th((size_t)16 * ns);
    for (int k = 0; k < ns; ++k)
        for (int h = 0; h < 2; ++h) {
            for (int j = 0; j < 7; ++j) th[16 * k + 8 * h + j] = rng[h][7 * k + j];
            th[16 * k + 8 * h + 7] = tmid[k];
        }
    return th;
}

// `products`: a side of three products makes a reaction wide even when it is
// irreversible (the adjoint reads every product).  `plog`: PLOG reactions have a
// class of their own (else they are evaluated from their DRxn records).
inline void build_quads(const cg_mech_view& v, HostQuads& h, bool products = false, bool plog = false) {
    const int ns = h.ns = (int)v.s[CG_S_NS], nr = h.nr = (int)v.s[CG_S_NR];
    const int32_t* flags = (const int32_t*)v.a[CG_FLAGS];
    const int32_t* rp = (const int32_t*)v.a[CG_RPTR];
    const int32_t* pp = (const int32_t*)v.a[CG_PPTR];
    const int32_t* rsp = (const int32_t*)v.a[CG_RSP];
    const int32_t* psp = (const int32_t*)v.a[CG_PSP];
    const double* rnu = (const double*)v.a[CG_RNU];
    const double* pnu = (const double*)v.a[CG_PNU];
    const double* arh = (const double*)v.a[CG_ARH];
    const double* karh = (const double*)v.a[CG_KARH];
    const double* fall = (const double*)v.a[CG_FALL];
    const double* kfall = (const double*)v.a[CG_KFALL];
    const int32_t* ep = (const int32_t*)v.a[CG_EFF_PTR];
    const int32_t* es = (const int32_t*)v.a[CG_EFF_SP];
    const double* ev = (const double*)v.a[CG_EFF_VAL];
    int seg[CG_NKINDS + 1];
    seg[0] = 0;
    for (int k = 0; k < CG_NKINDS; ++k) seg[k + 1] = seg[k] + (int)v.s[CG_S_NSTD + k];
    constexpr double kLog2e = 1.4426950408889634074;
    struct Item {
        int key, neff, r;
        QRec a, b;
    };
    std::vector<Item> items(nr);
    for (int r = 0; r < nr; ++r) {
        Item& it = items[r];
        std::memset(&it.a, 0, sizeof(QRec));
        int kind = CG_STANDARD;
        while (kind < CG_PLOG && r >= seg[kind + 1]) ++kind;
        const bool falloff = kind >= CG_LINDEMANN && kind <= CG_SRI;
        const bool third = kind == CG_THIRD_BODY;
        unsigned short mol[2][3];
        for (int j = 0; j < 6; ++j) mol[j / 3][j % 3] = (unsigned short)(ns * kQRow);
        int n[2] = {0, 0};
        bool ok = (flags[r] & CG_F_INT_NU) && ns < 0x10000 / kQRow;
        if (kind == CG_PLOG) {
            ok = ok && plog;
            it.a.aux = (unsigned)(r - seg[CG_PLOG]);
            ++h.nplog;
        } else {
            ok = ok && arh[3 * r] > 0.0 && std::fabs(karh[4 * r + 2]) < kQMaxTheta;
        }
        if (falloff) {
            const int f = r - seg[CG_LINDEMANN];
            ok = ok && fall[8 * f] > 0.0 && std::fabs(kfall[4 * f + 2]) < kQMaxTheta;
            it.a.aux = (unsigned)f;
        }
        for (int side = 0; ok && side < 2; ++side) {
            const int32_t* ptr = side ? pp : rp;
            const int32_t* sp = side ? psp : rsp;
            const double* nu = side ? pnu : rnu;
            for (int j = ptr[r]; ok && j < ptr[r + 1]; ++j)
                for (int q = 0; q < (int)nu[j]; ++q) {
                    if (n[side] == 3) ok = false;
                    else mol[side][n[side]++] = (unsigned short)(sp[j] * kQRow);
                }
        }
        const bool rev = (flags[r] & CG_F_REVERSIBLE) != 0;
        it.r = r;
        it.neff = (third || falloff) ? ep[r + 1] - ep[r] : 0;
        it.a.r = (unsigned)r;
        it.a.lnA = karh[4 * r];
        it.a.b = karh[4 * r + 1];
        it.a.th = karh[4 * r + 2];
        it.a.ord = (unsigned)(n[0] + (third ? 1 : 0)) | (unsigned)(n[1] + (third ? 1 : 0)) << 8;
        for (int j = 0; j < 2; ++j) {
            it.a.s[j] = mol[0][j];
            it.a.p[j] = mol[1][j];
        }
        it.a.s2 = mol[0][2];
        it.a.p2 = mol[1][2];
        it.b = it.a;
        if (ok) {
            it.b.lnA = std::log2(std::fabs(arh[3 * r]));
            it.b.th = it.a.th * kLog2e;
            if (kind <= CG_THIRD_BODY && it.b.b == 0.0 && it.b.th == 0.0) {
                // a constant rate: in generated code the compiler evaluates its
                // 2^f, to the nearest float and not as the hardware does
                const float f = (float)(it.b.lnA - std::nearbyint(it.b.lnA)), e = (float)std::exp2((double)f);
                std::memcpy(&it.b.aux, &e, sizeof(e));
            }
            const bool wide = n[0] > 2 || ((rev || products) && n[1] > 2);
            it.key = kind | (wide ? kQWide : 0) | (rev ? kQRev : 0);
        } else {
            it.key = kQKindGeneric;
            it.neff = 0;
            h.mixed_ok = false;
            ++h.ngeneric;
        }
    }
    // the costly kinds first (they are dealt out round robin to the warps),
    // then by size; within a class the longest efficiency lists first
    auto cost = [](int key) {
        const int kind = key & 15;
        return (kind == kQKindGeneric ? 4 : kind >= CG_LINDEMANN ? 3 : kind == CG_THIRD_BODY ? 2 : 1) * 1000 + key;
    };
    std::stable_sort(items.begin(), items.end(), [&](const Item& x, const Item& y) {
        const int a = cost(x.key), b = cost(y.key);
        return a != b ? a > b : x.neff > y.neff;
    });
    h.at.assign(nr, 0);
    for (size_t i = 0; i < items.size();) {
        size_t e = i;
        while (e < items.size() && e < i + kQG && items[e].key == items[i].key) ++e;
        const int2 in = make_int2((int)h.eff.size(), (items[i].neff + 3) / 4 * 4);
        for (int k = 0; k < in.y; ++k)
            for (size_t g = 0; g < kQG; ++g) {
                const Item& it = items[std::min(i + g, e - 1)];
                QEff q;
                const bool on = k < it.neff;
                q.sp = (unsigned)((on ? es[ep[it.r] + k] : ns) * kQRow);
                q.val = on ? ev[ep[it.r] + k] : 0.0;
                q.fval = (float)q.val;
                h.eff.push_back(q);
            }
        for (size_t g = 0; g < kQG; ++g) {
            // a quad short of four repeats its last reaction on the dummy
            // species: no list names the repeats, and their adjoint is zero
            const Item& it = items[std::min(i + g, e - 1)];
            QRec a = it.a, b = it.b;
            if (i + g >= e) {
                for (QRec* x : {&a, &b}) {
                    x->s[0] = x->s[1] = x->p[0] = x->p[1] = x->s2 = x->p2 = (unsigned short)(ns * kQRow);
                    x->r = kQNone;
                }
            }
            h.rec.push_back(a);
            h.rec2.push_back(b);
            if (i + g < e) h.at[it.r] = 4 * h.nquad + (int)g;
        }
        h.key.push_back(items[i].key);
        h.efl.push_back(in);
        ++h.nquad;
        i = e;
    }
    const int nfall = (int)(v.s[CG_S_NLIND] + v.s[CG_S_NTROE] + v.s[CG_S_NSRI]);
    for (int f = 0; f < nfall; ++f) {
        const double* row = fall + 8 * f;
        const int r = seg[CG_LINDEMANN] + f;
        QFall a;
        std::memset(&a, 0, sizeof(a));
        a.lnA0 = kfall[4 * f];
        a.b0 = kfall[4 * f + 1];
        a.th0 = kfall[4 * f + 2];
        QFall b = a;
        b.lnA0 = row[0] != 0.0 ? std::log2(std::fabs(row[0])) : 0.0;
        b.th0 = a.th0 * kLog2e;
        float* c = reinterpret_cast<float*>(b.p);
        if (r >= seg[CG_TROE] && r < seg[CG_TROE + 1]) {
            const double T2 = (flags[r] & CG_F_TROE_T2) ? row[6] : 0.0;
            const double p[5] = {row[7], 1.0 / row[4], row[3], 1.0 / row[5], T2};
            std::memcpy(a.p, p, sizeof(p));
            c[0] = (float)row[7];
            c[1] = (float)(-kLog2e / row[4]);
            c[2] = (float)row[3];
            c[3] = (float)(-kLog2e / row[5]);
            c[4] = (float)(-kLog2e * T2);
        } else if (r >= seg[CG_SRI] && r < seg[CG_SRI + 1]) {
            const double p[5] = {row[3], row[4], 1.0 / row[5], row[6], row[7]};
            std::memcpy(a.p, p, sizeof(p));
            c[0] = (float)row[3];
            c[1] = (float)(-kLog2e * row[4]);
            c[2] = (float)(-kLog2e / row[5]);
            c[3] = (float)(row[6] > 0.0 ? std::log2(row[6]) : -200.0);
            c[4] = (float)row[7];
        }
        h.fall.push_back(a);
        h.fall2.push_back(b);
    }
}

// Builder of row lists.  Each owner has (row, coefficient) contributions.
// Owners are grouped four to a quad, the longest lists first; an owner whose
// list is longer than kListSplit takes a quad of its own.  The quads are then
// dealt out to the warps (quad j W + w runs on warp w), longest first, each
// to the warp with the least work, so that the warps finish together.
struct ListBuilder {
    using List = std::vector<std::pair<int, double>>;
    static constexpr size_t kListSplit = 24;

    std::vector<QOwn> own;
    std::vector<uint4> ent;
    std::vector<QGen> gen;
    bool fits = true;                  // every count fits its field

    // steps of one owner's rows and coefficients: +-1, +-2, +-3 as repeated
    // rows, others weighted
    struct Split {
        std::vector<int> pos, neg;
        List ge;
    };
    static void split(const List& l, Split* out, int parts) {
        size_t np = 0, nn = 0, ng = 0;
        for (const auto& x : l) {
            const double a = std::fabs(x.second);
            if (a == 1.0 || a == 2.0 || a == 3.0)
                for (int q = 0; q < (int)a; ++q)
                    if (x.second > 0.0) out[np++ % parts].pos.push_back(x.first);
                    else out[nn++ % parts].neg.push_back(x.first);
            else if (a != 0.0) out[ng++ % parts].ge.push_back(x);
        }
    }
    static size_t length(const List& l) {
        size_t n = 0;
        for (const auto& x : l) {
            const double a = std::fabs(x.second);
            n += (a == 1.0 || a == 2.0 || a == 3.0) ? (size_t)a : 2;
        }
        return n;
    }

    static size_t weighted(const List& l) {
        size_t n = 0;
        for (const auto& x : l) {
            const double a = std::fabs(x.second);
            n += a != 0.0 && a != 1.0 && a != 2.0 && a != 3.0;
        }
        return n;
    }

    // One owner's list, split four ways, or those of two to four owners;
    // `zero` is a row of zeros.
    void add_quad(const std::vector<const List*>& lists, const std::vector<int>& what, int zero) {
        Split q[kQG];
        const bool wide = lists.size() == 1;
        if (wide) split(*lists[0], q, kQG);
        else
            for (size_t g = 0; g < lists.size(); ++g) split(*lists[g], q + g, 1);
        size_t np = 0, nn = 0, ng = 0;
        for (int g = 0; g < kQG; ++g) {
            np = std::max(np, (q[g].pos.size() + 3) / 4);
            nn = std::max(nn, (q[g].neg.size() + 3) / 4);
            ng = std::max(ng, q[g].ge.size());
        }
        ng = (ng + 1) / 2 * 2;
        const size_t n4 = np + nn, n8 = std::max<size_t>((n4 + 1) / 2, 1);
        fits = fits && nn < 0xffff && n4 < 0x7fff && ng < 0xfff && gen.size() / kQG < 0xfffff;
        QOwn o[kQG];
        for (int g = 0; g < kQG; ++g) {
            o[g].own = wide ? what[0] : g < (int)what.size() ? what[g] : -1;
            o[g].cnt = (unsigned)nn | (unsigned)n4 << 16 | (wide ? kOwnWide : 0u);
            o[g].ptr = (int)ent.size();
            o[g].gen = (unsigned)(gen.size() / kQG) | (unsigned)ng << 20;
        }
        for (size_t k = 0; k < n8; ++k)
            for (int g = 0; g < kQG; ++g) {
                unsigned r[8];
                for (size_t u = 0; u < 8; ++u) {
                    const size_t h = 2 * k + u / 4;          // half-step
                    const std::vector<int>& l = h < nn ? q[g].neg : q[g].pos;
                    const size_t j = 4 * (h < nn ? h : h - nn) + u % 4;
                    r[u] = j < l.size() ? (unsigned)l[j] : (unsigned)zero;
                }
                const uint4 w = make_uint4(r[0] | r[1] << 16, r[2] | r[3] << 16, r[4] | r[5] << 16, r[6] | r[7] << 16);
                if (k == 0) o[g].rows = w;
                else ent.push_back(w);
            }
        for (size_t k = 0; k < ng; ++k)
            for (int g = 0; g < kQG; ++g) {
                const List& l = q[g].ge;
                QGen x;
                x.coef = k < l.size() ? l[k].second : 0.0;
                x.row = k < l.size() ? (unsigned)l[k].first : (unsigned)zero;
                x.pad = 0;
                gen.push_back(x);
            }
        own.insert(own.end(), o, o + kQG);
    }

    // Groups the owners of the lists into quads and orders the quads for
    // `warps` warps; each quad names its owners.
    static std::vector<std::vector<int>> group(const std::vector<const List*>& lists, int warps) {
        const size_t no = lists.size();
        std::vector<size_t> len(no), wt(no);
        std::vector<int> own(no);
        for (size_t k = 0; k < no; ++k) {
            own[k] = (int)k;
            len[k] = length(*lists[k]);
            wt[k] = weighted(*lists[k]);
        }
        // long lists first, then lists with weighted entries together
        std::stable_sort(own.begin(), own.end(), [&](int a, int b) {
            const bool la = len[a] > kListSplit, lb = len[b] > kListSplit;
            if (la != lb) return la;
            if (!la && wt[a] != wt[b]) return wt[a] > wt[b];
            return len[a] > len[b];
        });
        std::vector<std::vector<int>> quads;
        std::vector<size_t> cost;
        for (size_t k = 0; k < own.size();) {
            std::vector<int> q{own[k]};
            size_t l = len[own[k++]];
            if (l <= kListSplit)
                while (q.size() < (size_t)kQG && k < own.size()) {
                    l = std::max(l, len[own[k]]);
                    q.push_back(own[k++]);
                }
            cost.push_back(12 + (q.size() == 1 ? l / 4 : l));
            quads.push_back(q);
        }
        std::vector<int> by(quads.size());
        for (size_t k = 0; k < by.size(); ++k) by[k] = (int)k;
        std::stable_sort(by.begin(), by.end(), [&](int a, int b) { return cost[a] > cost[b]; });
        std::vector<std::vector<int>> mine(warps);
        std::vector<size_t> load(warps, 0);
        const int n = (int)quads.size();
        for (int q : by) {
            int best = -1;
            for (int w = 0; w < warps; ++w)
                if ((int)mine[w].size() < (n - w + warps - 1) / warps && (best < 0 || load[w] < load[best])) best = w;
            mine[best].push_back(q);
            load[best] += cost[q];
        }
        std::vector<std::vector<int>> out(n);
        for (int w = 0; w < warps; ++w)
            for (size_t j = 0; j < mine[w].size(); ++j) out[j * warps + w] = quads[mine[w][j]];
        return out;
    }
};

// Runs: the quads of one class that one warp takes, quads first, first + W,
// ....  Quad q of a chunk runs on warp (q - chunk's first) mod W; each warp has
// the list of its runs, so that a loop over one class holds no dispatch and
// no warp looks at classes it has no quad of.
//   run = {class, first quad, how many, 0}; of warp w in chunk c:
//   run[beg[c W + w]] .. run[beg[c W + w + 1] - 1]
inline void build_runs(const HostQuads& h, const std::vector<int>& qbeg, int warps, std::vector<int4>& run,
                       std::vector<int>& beg) {
    beg.assign(1, 0);
    for (size_t c = 0; c + 1 < qbeg.size(); ++c)
        for (int w = 0; w < warps; ++w) {
            const size_t first = run.size();
            for (int q = qbeg[c] + w; q < qbeg[c + 1]; q += warps) {
                if (run.size() == first || run.back().x != h.key[q]) run.push_back(make_int4(h.key[q], q, 0, 0));
                ++run.back().z;
            }
            beg.push_back((int)run.size());
        }
}

// Raises a kernel's limit of dynamic shared memory to `bytes` on the current
// device.  Every plan of one kernel instance (one per handle) has its own size:
// the limit is never lowered, so a launch needs no call and no lock for it
// (0.5 us of a small batch's 12).
inline cudaError_t raise_smem_limit(const void* fn, size_t bytes) {
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    cudaFuncAttributes fa;
    const cudaError_t e = cudaFuncGetAttributes(&fa, fn);
    if (e != cudaSuccess || (size_t)fa.maxDynamicSharedSizeBytes >= bytes) return e;
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// Host image of a plan's tables, copied to the device in one piece.
struct Image {
    std::vector<unsigned char> buf;
    template <typename T>
    size_t put(const std::vector<T>& x) {
        const size_t off = (buf.size() + 255) / 256 * 256;
        buf.resize(off + std::max<size_t>(x.size(), 1) * sizeof(T) + 64);
        if (!x.empty()) std::memcpy(buf.data() + off, x.data(), x.size() * sizeof(T));
        return off;
    }
    cudaError_t upload(void** d) const {
        cudaError_t e = cudaMalloc(d, buf.size());
        if (e == cudaSuccess) e = cudaMemcpy(*d, buf.data(), buf.size(), cudaMemcpyHostToDevice);
        if (e != cudaSuccess && *d) {
            cudaFree(*d);
            *d = nullptr;
        }
        return e;
    }
};

}  // namespace cg
