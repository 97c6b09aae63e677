// Mixed-precision getrates with the stoichiometric contraction on the
// 5th-generation tensor cores (tcgen05).  Table-driven: one compiled kernel
// serves every mechanism loaded at run time, including 348-species /
// 2163-reaction ones.
//
// Work split of the 128-point kernel (the 32-point one, for large mechanisms and
// small batches, is described where it stands).  A CTA owns a tile of 128 grid
// points -- one point per thread,
// one point per TMEM lane.  For every chunk of 16 reactions each thread
// computes its point's net rates of progress q (the reference's
// rr = kf prod C^nu - kb prod C^nu, reactions/standard.j2:3-19, with the
// third-body factor of third_body.j2:30 and the falloff of troe.j2:9-45)
// and writes them, split exactly into three BF16 parts q = q_hi + q_mid +
// q_lo, into shared memory as the A operand of an MMA whose B operand is
// the chunk's net stoichiometric matrix nu (exact in BF16).  One thread
// issues tcgen05.mma; the products accumulate in FP32 in tensor memory,
// D[point][species] = sum_r q_r nu_rk, which is wdot
// (reactions/standard.j2:21-27).  Two chunk buffers let the tensor core
// accumulate one chunk while the threads compute the next.
//
// Arithmetic.  Exponents are formed in FP64: ln A + b ln T - Ea/(Rc T) and
// the Gibbs sums sum nu G that give Kc (G = log2(exp(smh) Patm/(R0 T))).
// 2^f of the fractional part runs on the SFU (ex2.approx.f32); concentration
// products are FP32 on C * 2^32 (so that they stay clear of FP32 underflow);
// q is FP32 and the accumulation FP32.  PLOG reactions and reactions with
// fractional stoichiometry are evaluated in FP64 and rounded to FP32.
//
// Per-point state: C (FP32) and G (FP64) in shared memory.
// Every mbarrier wait is bounded; a time-out sets the error word.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "cg_math.cuh"
#include "gen_common.cuh"
#include "quad.cuh"
#include "rates_common.cuh"
#include "umma.cuh"

namespace cg {

constexpr int kTile = 128;       // points per CTA tile (TMEM lanes)
constexpr int kChunk = 16;       // reactions per MMA chunk (MMA K)
constexpr int kABytes = kTile * kChunk * 2;   // one BF16 A split tile

// Pre-decoded record of a standard or three-body reaction with at most three
// molecules per side (the common case), built once per plan on the device:
// log2-space Arrhenius constants and the species of each molecule, padded with
// the dummy species ns (C = 1, G = 0), so that the rate needs no decoding.
struct __align__(16) TcFast {
    double l2A, b, th2;          // log2|A|, b, (Ea/Rc) log2 e
    unsigned short sr[3], sp[3]; // reactant / product molecules (species ns = none)
    unsigned char ordf, ordb;    // concentration factors of each side (M included)
    unsigned char flags;         // kFastOn | kFastRev | kFastThird | kFastNeg | kFastFall
    unsigned char neff;          // efficiencies (255: look them up)
    int eff0;                    // first efficiency
    union {
        int aux;                 // falloff row
        int ngen;                // species entries of a general row
    };
};
static_assert(sizeof(TcFast) == 48, "TcFast must stay 48 bytes");
constexpr unsigned kFastOn = 1, kFastRev = 2, kFastThird = 4, kFastNeg = 8;
constexpr unsigned kFastFall = 16;   // falloff with positive A's, decoded for the 32-point kernel only

struct MixedPlan {
    int ns = 0, nr = 0, npad = 0, nhalf = 0, nchunk = 0;
    uint32_t tcols = 0;
    int t128 = 0;           // the 128-point tile fits (Gibbs terms in shared memory)
    size_t smem = 0;
    int grid = 0;
    int group = 4;          // chunks accumulated in FP32 before the FP64 flush
    int nt = 1;             // threads per point (blockDim = 128 nt)
    int hot = 0;            // species with FP64 accumulators in spare tensor-memory columns
    int hot_every = 8;      // chunks between the hot species' FP64 flushes
    const TcFast* fast32 = nullptr;   // the 32-point kernel's records: species as byte offsets
    size_t smem32 = 0;
    int grid32 = 0;
    const int* perm = nullptr;  // accumulator column -> species (-1: padding)
    void* dbuf = nullptr;
    const __nv_bfloat16* nu = nullptr;
    const TcFast* fast = nullptr;
    int* err = nullptr;
};

namespace {

constexpr double kLog2eD = 1.4426950408889634074;
constexpr float kLog2eF = 1.44269504f;
constexpr float kLog10_2F = 0.30103000f;

// 2^e for an integer e, applied in two FP32 steps so that large products
// with small scales (and the reverse) keep their value.
__device__ __forceinline__ float scale2(float m, int e) {
    const int e1 = max(-126, min(e, 127));
    const int e2 = max(-126, min(e - e1, 127));
    return m * __int_as_float((e1 + 127) << 23) * __int_as_float((e2 + 127) << 23);
}

// FP32 q = 2^a * prod * 2^eoff, a in FP64.
__device__ __forceinline__ float rate32(double a, float prod, int eoff) {
    const double magic = 6755399441055744.0;
    const double t = a + magic;
    const int n = __double2loint(t);
    const float f = (float)(a - (t - magic));
    return scale2(cgg::ex2f(f) * prod, n + eoff);
}

struct TileCtx {
    const float* C;      // C * 2^32, one row of points a species
    const double* G;     // log2 Gibbs terms, likewise
    double T, Pv, lnT, lnT2, invT;
    float ctot32, Tf, invTf, lnT2f;
};

// log2 kf of a falloff reaction (Lindemann, Troe, SRI), in FP64 throughout
// (troe.j2:9-45 in the log2 domain).  The FP32 blend that the 53-species
// generated kernels use was measured on JetSurf 2.0 (382 Troe reactions,
// several of them each point's dominant rate): its kf errors reached 5e-6,
// mostly from FP32 exponent arguments in Fcent and the FP32 log10 Pr / f1 chain,
// which put the normwise error of wdot at 7.6e-6 over 2^18 points.  In FP64
// the blend costs about three exp and three log per falloff reaction.
__device__ double falloff_l2(int kind, int flags, const DRxn& R, const DFall& f, double x2, float Ms,
                             const TileCtx& c) {
    constexpr double kLog10_2 = 0.30102999566398119521, kLn2 = 0.69314718055994530942;
    const double ainf = (fma(R.b, c.lnT, R.lnA) - R.theta * c.invT) * kLog2eD;
    const double a0 = (fma(f.b0, c.lnT, f.lnA0) - f.theta0 * c.invT) * kLog2eD;
    const double M = (double)Ms * 2.3283064365386963e-10;   // Ms = M * 2^32
    // log2 Pr and log2 Pr/(1 + Pr), without overflow at either end
    const double l2pr = (a0 - ainf) + cgm::cg_log(M) * kLog2eD;
    const double x = cgm::cg_exp_clamped(-fabs(l2pr) * kLn2);          // min(Pr, 1/Pr)
    const double l2r = fmin(l2pr, 0.0) - cgm::cg_log(1.0 + x) * kLog2eD;
    double l2F = 0.0;
    if (kind == CG_TROE) {
        double Fc = fma(f.p[0], cgm::cg_exp_clamped(-c.T * f.p[1]), f.p[2] * cgm::cg_exp_clamped(-c.T * f.p[3]));
        if (flags & CG_F_TROE_T2) Fc += cgm::cg_exp_clamped(-x2 * c.invT);
        const double lFc = cgm::cg_log10(Fc);
        const double lp = fma(kLog10_2, l2pr, fma(-0.67, lFc, -0.4));
        const double f1 = lp * cgm::cg_rcp(fma(-0.14, lp, fma(-1.27, lFc, 0.75)));
        l2F = lFc * cgm::cg_rcp(fma(f1, f1, 1.0)) / kLog10_2;
    } else if (kind == CG_SRI) {
        const double lp = kLog10_2 * l2pr;
        const double X = cgm::cg_rcp(fma(lp, lp, 1.0));
        const double base = fma(f.p[0], cgm::cg_exp_clamped(-f.p[1] * c.invT), cgm::cg_exp_clamped(-c.T * f.p[2]));
        l2F = (cgm::cg_log(f.p[3]) + fma(X, cgm::cg_log(base), x2 * c.lnT)) * kLog2eD;
    }
    return ainf + (l2r + l2F);
}

// PLOG forward rate in FP64 (plog.j2:4-38).
__device__ double plog_kf64(const DevMech& m, int row, double P, double lnT, double invT) {
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
    double k[2] = {0.0, 0.0};
    const int lev[2] = {la, lb};
    for (int s = 0; s < (la == lb ? 1 : 2); ++s)
        for (int t = __ldg(m.plog_tptr + lev[s]); t < __ldg(m.plog_tptr + lev[s] + 1); ++t) {
            const double4 cc = m.plog_term[t];
            k[s] += cc.w * cgm::cg_exp_clamped(fma(cc.y, lnT, cc.x) - cc.z * invT);
        }
    if (la == lb) return k[0];
    const double a = __ldg(m.plog_lnp + la), b = __ldg(m.plog_lnp + lb);
    const double kl = cgm::cg_log(k[0]);
    return cgm::cg_exp_clamped(kl + (cgm::cg_log(k[1]) - kl) * (cgm::cg_log(P) - a) / (b - a));
}

// FP64 evaluation of reaction r (PLOG, non-integer stoichiometry, falloff
// with negative pre-exponential factors): kept out of line so that the
// common FP32 path keeps few registers.
template <int TS>
__device__ __noinline__ float rate_of_progress_fp64(const DevMech& m, const DRxn& R, int kind, float Ms,
                                                    const TileCtx& c, int tid) {
    const bool compact = (R.flags & kFCompact) != 0;
    {
        double kf;
        if (kind == CG_PLOG) kf = plog_kf64(m, R.aux, c.Pv, c.lnT, c.invT);
        else if (kind <= CG_THIRD_BODY) kf = R.sgn * cgm::cg_exp_clamped(fma(R.b, c.lnT, R.lnA) - R.theta * c.invT);
        else {
            const DFall f = load_fall(m.fall + R.aux);
            kf = R.sgn * exp2(falloff_l2(kind, R.flags, R, f, __ldg(&m.fall2[R.aux].T2), Ms, c));
        }
        const double cs = 2.3283064365386963e-10;   // 2^-32
        double qf = kf, qb = 0.0, g = 0.0;
        {
            if (compact) {
                for (int j = 0; j < R.nre; ++j) {
                    const int s = slot_species(R.sp[j]);
                    qf *= ipow3((double)c.C[s * TS + tid] * cs, slot_nu(R.sp[j]));
                    g = fma((double)slot_nu(R.sp[j]), c.G[s * TS + tid], g);
                }
                double pb = 1.0;
                for (int j = 0; j < R.npr; ++j) {
                    const int s = slot_species(R.sp[3 + j]);
                    pb *= ipow3((double)c.C[s * TS + tid] * cs, slot_nu(R.sp[3 + j]));
                    g = fma(-(double)slot_nu(R.sp[3 + j]), c.G[s * TS + tid], g);
                }
                if (R.flags & CG_F_REVERSIBLE) qb = kf * exp2(g) * pb;
            } else {
                const int gr = R.gen;
                const int r0 = __ldg(m.gen_rptr + gr), r1 = __ldg(m.gen_rptr + gr + 1);
                const int p0 = __ldg(m.gen_pptr + gr), p1 = __ldg(m.gen_pptr + gr + 1);
                for (int j = r0; j < r1; ++j) {
                    const int s = __ldg(m.gen_sp + j);
                    const double nu = __ldg(m.gen_nu + j);
                    qf *= pow((double)c.C[s * TS + tid] * cs, nu);
                    g = fma(nu, c.G[s * TS + tid], g);
                }
                double pb = 1.0;
                for (int j = p0; j < p1; ++j) {
                    const int s = __ldg(m.gen_sp + j);
                    const double nu = __ldg(m.gen_nu + j);
                    pb *= pow((double)c.C[s * TS + tid] * cs, nu);
                    g = fma(-nu, c.G[s * TS + tid], g);
                }
                if (R.flags & CG_F_REVERSIBLE) qb = kf * exp2(g) * pb;
            }
        }
        double rr = qf - qb;
        if (kind == CG_THIRD_BODY) rr *= (double)Ms * cs;
        return (float)rr;
    }
}

// Ms = ctot + sum_e (eff_e - 1) C[sp_e] of reaction r (third_body.j2:18-31) in
// FP32 at point `tid`, the efficiencies taken four at a time so that their
// loads are in flight together; the sum keeps the table's order.
template <int TS>
__device__ __forceinline__ float tc_third_body(const DevMech& m, int e0, int e1, const float* C, float ctot32, int tid) {
    float Ms = ctot32;
    for (int e = e0; e < e1; e += 4) {
        int sp[4];
        float ev[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const bool ok = e + u < e1;
            sp[u] = ok ? __ldg(m.eff_sp + e + u) : 0;
            ev[u] = ok ? (float)__ldg(m.eff_val + e + u) : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float cv = C[sp[u] * TS + tid];
            if (e + u < e1) Ms = fmaf(ev[u], cv, Ms);
        }
    }
    return Ms;
}

template <int TS>
__device__ __forceinline__ float tc_third_body(const DevMech& m, int r, const TileCtx& c, int tid) {
    return tc_third_body<TS>(m, __ldg(m.eff_ptr + r), __ldg(m.eff_ptr + r + 1), c.C, c.ctot32, tid);
}

// Net rate of progress of reaction r at point `tid` of the tile, FP32.
template <int TS>
__device__ float rate_of_progress(const DevMech& m, int r, const TileCtx& c, int tid) {
    const DRxn R = load_rxn(m.rxn + r);
    int kind = CG_STANDARD;
    while (kind < CG_PLOG && r >= m.seg[kind + 1]) ++kind;
    float Ms = 0.0f;
    if (kind >= CG_THIRD_BODY && kind <= CG_SRI) Ms = tc_third_body<TS>(m, r, c, tid);
    const bool compact = (R.flags & kFCompact) != 0;
    const bool neg_falloff = kind >= CG_LINDEMANN && kind <= CG_SRI && (R.flags & (CG_F_A_NEG | CG_F_LOW_NEG));
    if (!compact || kind == CG_PLOG || neg_falloff) return rate_of_progress_fp64<TS>(m, R, kind, Ms, c, tid);
    double a;
    float sgn = 1.0f;
    if (kind <= CG_THIRD_BODY) {
        a = (fma(R.b, c.lnT, R.lnA) - R.theta * c.invT) * kLog2eD;
        sgn = (float)R.sgn;
    } else {
        const DFall f = load_fall(m.fall + R.aux);
        a = falloff_l2(kind, R.flags, R, f, __ldg(&m.fall2[R.aux].T2), Ms, c);
    }
    float cf = 1.0f;
    int of = 0;
    double g = 0.0;
    for (int j = 0; j < R.nre; ++j) {
        const int s = slot_species(R.sp[j]), nu = slot_nu(R.sp[j]);
        const float x = c.C[s * TS + tid];
        cf *= (nu == 1) ? x : (nu == 2 ? x * x : x * x * x);
        of += nu;
        g = fma((double)nu, c.G[s * TS + tid], g);
    }
    if (kind == CG_THIRD_BODY) {
        cf *= Ms;
        of += 1;
    }
    float q = rate32(a, cf, -32 * of);
    if (R.flags & CG_F_REVERSIBLE) {
        float cb = 1.0f;
        int ob = 0;
        for (int j = 0; j < R.npr; ++j) {
            const int s = slot_species(R.sp[3 + j]), nu = slot_nu(R.sp[3 + j]);
            const float x = c.C[s * TS + tid];
            cb *= (nu == 1) ? x : (nu == 2 ? x * x : x * x * x);
            ob += nu;
            g = fma(-(double)nu, c.G[s * TS + tid], g);
        }
        if (kind == CG_THIRD_BODY) {
            cb *= Ms;
            ob += 1;
        }
        q -= rate32(a + g, cb, -32 * ob);
    }
    return sgn * q;
}

// Net rate of progress of a pre-decoded reaction (TcFast) at point `tid`, FP32.
template <int TS>
__device__ __forceinline__ float rate_fast(const DevMech& m, int r, const TcFast& F, const TileCtx& c, int tid) {
    const double a = fma(F.b, c.lnT2, F.l2A) - F.th2 * c.invT;
    float Ms = 1.0f;
    if (F.flags & kFastThird) Ms = tc_third_body<TS>(m, r, c, tid);
    const float cf = c.C[F.sr[0] * TS + tid] * c.C[F.sr[1] * TS + tid] * c.C[F.sr[2] * TS + tid] * Ms;
    float q = rate32(a, cf, -32 * (int)F.ordf);
    if (F.flags & kFastRev) {
        const double g = (c.G[F.sr[0] * TS + tid] + c.G[F.sr[1] * TS + tid] + c.G[F.sr[2] * TS + tid]) -
                         (c.G[F.sp[0] * TS + tid] + c.G[F.sp[1] * TS + tid] + c.G[F.sp[2] * TS + tid]);
        const float cb = c.C[F.sp[0] * TS + tid] * c.C[F.sp[1] * TS + tid] * c.C[F.sp[2] * TS + tid] * Ms;
        q -= rate32(a + g, cb, -32 * (int)F.ordb);
    }
    return (F.flags & kFastNeg) ? -q : q;
}

__device__ __forceinline__ TcFast load_fast(const TcFast* p) {
    const int4* q = reinterpret_cast<const int4*>(p);
    TcFast f;
    int4* d = reinterpret_cast<int4*>(&f);
    d[0] = __ldg(q);
    d[1] = __ldg(q + 1);
    d[2] = __ldg(q + 2);
    return f;
}

// One TcFast per reaction (flags 0 where the generic path is needed).
// Species are stored times `scale` (the 32-point kernel's byte offsets).
__global__ void build_fast_kernel(DevMech m, TcFast* out, int scale) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= m.nr) return;
    const DRxn R = load_rxn(m.rxn + r);
    int kind = CG_STANDARD;
    while (kind < CG_PLOG && r >= m.seg[kind + 1]) ++kind;
    TcFast f;
    f.l2A = R.lnA * kLog2eD;
    f.b = R.b;
    f.th2 = R.theta * kLog2eD;
    f.eff0 = __ldg(m.eff_ptr + r);
    f.neff = (unsigned char)min(__ldg(m.eff_ptr + r + 1) - f.eff0, 255);
    f.aux = R.aux;
    if (!(R.flags & kFCompact) && R.gen >= 0)
        f.ngen = __ldg(m.gen_rptr + R.gen + 1) - __ldg(m.gen_rptr + R.gen) + __ldg(m.gen_pptr + R.gen + 1) -
                 __ldg(m.gen_pptr + R.gen);
    f.flags = 0;
    f.ordf = f.ordb = 0;
    for (int j = 0; j < 3; ++j) f.sr[j] = f.sp[j] = (unsigned short)(m.ns * scale);
    const bool fall = scale > 1 && kind >= CG_LINDEMANN && kind <= CG_SRI && !(R.flags & (CG_F_A_NEG | CG_F_LOW_NEG)) &&
                      R.sgn > 0.0;
    bool ok = (kind == CG_STANDARD || kind == CG_THIRD_BODY || fall) && (R.flags & kFCompact) && R.sgn != 0.0;
    int nf = 0, nb = 0;
    for (int j = 0; ok && j < R.nre; ++j)
        for (int k = 0; k < slot_nu(R.sp[j]); ++k) {
            if (nf == 3) ok = false;
            else f.sr[nf++] = (unsigned short)(slot_species(R.sp[j]) * scale);
        }
    for (int j = 0; ok && j < R.npr; ++j)
        for (int k = 0; k < slot_nu(R.sp[3 + j]); ++k) {
            if (nb == 3) ok = false;
            else f.sp[nb++] = (unsigned short)(slot_species(R.sp[3 + j]) * scale);
        }
    if (ok) {
        const bool third = kind == CG_THIRD_BODY;
        f.ordf = (unsigned char)(nf + (third ? 1 : 0));
        f.ordb = (unsigned char)(nb + (third ? 1 : 0));
        f.flags = (unsigned char)((fall ? kFastFall : kFastOn) | ((R.flags & CG_F_REVERSIBLE) ? kFastRev : 0) | (third ? kFastThird : 0) |
                                  (R.sgn < 0.0 ? kFastNeg : 0));
    }
    out[r] = f;
}

// NT threads share each of the tile's 128 points (blockDim = 128 NT): they
// split the species of the prologue (their partial sums meet in shared
// memory), the 16 reactions of each chunk, and the accumulator columns of
// each flush.  The FP32 sums live in tensor memory, so extra threads cost
// no per-species registers.
template <int NT>
__global__ void __launch_bounds__(kTile * NT, 1)
    getrates_tc_kernel(DevMech m, const __nv_bfloat16* __restrict__ nu, const TcFast* __restrict__ fast, int npad,
                       int nhalf, int nchunk, uint32_t tcols,
                       const double* __restrict__ P, const double* __restrict__ Tg, const double* __restrict__ Y,
                       double* __restrict__ wdot, int64_t ng, int* err, int group,
                       const int* __restrict__ perm, int hot, int hot_every) {
    extern __shared__ __align__(1024) unsigned char sm[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int pt = tid & (kTile - 1), sub = tid >> 7;          // point of the tile, share of its work
    const int ns = m.ns;
    unsigned char* sA = sm;                                    // [2 buffers][3 splits][128 x 16] BF16
    unsigned char* sB = sm + 6 * kABytes;                      // [2 buffers][npad x 16] BF16
    const int rows = ns + 1;                                   // species + the dummy row of TcFast
    float* sC = reinterpret_cast<float*>(sB + 2 * npad * 32);  // [rows][128]
    double* sG = reinterpret_cast<double*>(sC + rows * kTile);  // [rows][128]
    double* sRed = sG + rows * kTile;                          // [NT][128] partial sums
    uint64_t* mbar = reinterpret_cast<uint64_t*>(sRed + NT * kTile);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 2);
    if (tid == 0) {
        um::mbar_init(&mbar[0], 1);
        um::mbar_init(&mbar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) um::tmem_alloc(tslot, tcols);
    um::fence_before_sync();
    __syncthreads();
    um::fence_after_sync();
    const uint32_t tbase = *tslot;
    uint32_t parity[2] = {0u, 0u};
    bool pending[2] = {false, false};
    bool ok = true;
    const uint32_t idesc = um::idesc_bf16(kTile, nhalf);
    const int nh = npad / nhalf;
    const int64_t ntiles = (ng + kTile - 1) / kTile;
    for (int64_t tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
        const int64_t i = tile * kTile + pt;
        const bool act = i < ng;
        TileCtx c;
        c.C = sC;
        c.G = sG;
        // inputs are read once: streaming loads, so that they do not push the
        // stoichiometry image out of L2
        c.T = act ? __ldcs(Tg + i) : 1000.0;
        c.Pv = act ? __ldcs(P + i) : kPatm;
        c.lnT = cgm::cg_log(c.T);
        c.invT = 1.0 / c.T;
        c.lnT2 = c.lnT * kLog2eD;
        c.Tf = (float)c.T;
        c.invTf = (float)c.invT;
        c.lnT2f = (float)c.lnT2;
        // Y -> C (ytoc.j2), stored as C * 2^32 in FP32; species k is handled
        // by the thread with sub = k % NT
        double part = 0.0;
        for (int k = sub; k < ns; k += NT) {
            const double yk = (act ? __ldcs(Y + (int64_t)k * ng + i) : 1.0) * __ldg(m.inv_mw + k);
            sG[k * kTile + pt] = yk;
            part += yk;
        }
        sRed[sub * kTile + pt] = part;
        __syncthreads();
        double csum = 0.0;
        for (int q = 0; q < NT; ++q) csum += sRed[q * kTile + pt];
        const double facs = c.Pv / (kR0 * csum * c.T) * 4294967296.0;
        part = 0.0;
        for (int k = sub; k < ns; k += NT) {
            const double cc = sG[k * kTile + pt] * facs;
            sC[k * kTile + pt] = (float)cc;
            part += cc;
        }
        __syncthreads();
        sRed[sub * kTile + pt] = part;
        __syncthreads();
        double ctot = 0.0;
        for (int q = 0; q < NT; ++q) ctot += sRed[q * kTile + pt];
        c.ctot32 = (float)ctot;
        // G = log2(exp(smh) Patm/(R0 T)) (exp_g.j2), FP64
        const double lpfac2 = -6.35856916300311 - c.lnT2;   // log2(Patm/R0) - log2 T
        for (int k = sub; k < ns; k += NT)
            sG[k * kTile + pt] = fma(species_smh(m.thermo, k, c.T, c.lnT, c.invT), kLog2eD, lpfac2);
        if (sub == 0) {
            sC[ns * kTile + pt] = 1.0f;     // dummy species of TcFast: a factor 1 ...
            sG[ns * kTile + pt] = 0.0;      // ... and no Gibbs term
        }
        __syncthreads();
        bool first_group = true;
        int nhot = 0;                    // hot flushes so far in this tile
        for (int ch = 0; ch < nchunk && ok; ++ch) {
            const int buf = ch & 1;
            if (pending[buf]) {
                ok = um::mbar_wait(&mbar[buf], parity[buf]);
                parity[buf] ^= 1u;
                pending[buf] = false;
                if (!ok) break;
            }
            // the chunk's stoichiometry, B operand [npad x 16], canonical layout
            const uint4* src = reinterpret_cast<const uint4*>(nu + (int64_t)ch * npad * kChunk);
            uint4* dst = reinterpret_cast<uint4*>(sB + buf * npad * 32);
            for (int q = tid; q < npad * 2; q += kTile * NT) dst[q] = __ldg(src + q);
            // q for the chunk's reactions -> A operands (hi, mid, lo).  The
            // thread with share `sub` takes kPer consecutive reactions, so that
            // its BF16 values of a row leave in one 8- or 16-byte store per
            // split instead of one 2-byte store per reaction
            unsigned char* a0 = sA + buf * 3 * kABytes;
            constexpr int kPer = kChunk / NT, kWords = kPer / 4;
            static_assert(kChunk % NT == 0 && kPer % 4 == 0, "each share takes whole 4-reaction words");
            const int j0 = sub * kPer;
            uint64_t ph[kWords], pm[kWords], pl[kWords];
#pragma unroll
            for (int w = 0; w < kWords; ++w) ph[w] = pm[w] = pl[w] = 0ull;
#pragma unroll 1
            for (int u = 0; u < kPer; ++u) {
                const int r = ch * kChunk + j0 + u;
                float q = 0.0f;
                if (r < m.nr) {
                    const TcFast F = load_fast(fast + r);
                    // this thread's next record moves into L1 meanwhile (no registers held)
                    if (u + 1 < kPer && r + 1 < m.nr) asm volatile("prefetch.global.L1 [%0];" ::"l"(fast + r + 1));
                    q = (F.flags & kFastOn) ? rate_fast<kTile>(m, r, F, c, pt) : rate_of_progress<kTile>(m, r, c, pt);
                }
                if (!act) q = 0.0f;
                const __nv_bfloat16 h = __float2bfloat16_rn(q);
                const float r1 = q - __bfloat162float(h);
                const __nv_bfloat16 md = __float2bfloat16_rn(r1);
                const __nv_bfloat16 lo = __float2bfloat16_rn(r1 - __bfloat162float(md));
                const int sh = 16 * (u & 3);
#pragma unroll
                for (int w = 0; w < kWords; ++w)
                    if (w == (u >> 2)) {
                        ph[w] |= (uint64_t)__bfloat16_as_ushort(h) << sh;
                        pm[w] |= (uint64_t)__bfloat16_as_ushort(md) << sh;
                        pl[w] |= (uint64_t)__bfloat16_as_ushort(lo) << sh;
                    }
            }
#pragma unroll
            for (int w = 0; w < kWords; ++w) {
                const uint32_t off = um::kmajor_offset(pt, j0 + 4 * w, kChunk);   // 8-byte aligned
                *reinterpret_cast<uint64_t*>(a0 + off) = ph[w];
                *reinterpret_cast<uint64_t*>(a0 + kABytes + off) = pm[w];
                *reinterpret_cast<uint64_t*>(a0 + 2 * kABytes + off) = pl[w];
            }
            um::fence_proxy_async();
            um::fence_before_sync();
            __syncthreads();
            const bool group_start = (ch % group) == 0;
            if (tid == 0) {
                um::fence_after_sync();
                const uint32_t bb = um::smem_addr(sB + buf * npad * 32);
                for (int s = 0; s < 3; ++s) {
                    const uint64_t ad = um::desc_kmajor(um::smem_addr(a0 + s * kABytes), kChunk, 0);
                    for (int h = 0; h < nh; ++h)
                        um::mma_bf16(tbase + (uint32_t)(h * nhalf), ad,
                                     um::desc_kmajor(bb + (uint32_t)(h * nhalf * 32), kChunk, 0), idesc,
                                     (!group_start || s > 0) ? 1u : 0u);
                }
                um::commit(&mbar[buf]);
            }
            pending[buf] = true;
            const bool group_end = (ch % group) == group - 1 || ch == nchunk - 1;
            if (hot > 0 && !group_end && (ch % hot_every) == hot_every - 1) {
                // hot flush: the FP32 sums of the most-touched species (columns
                // 0 .. hot-1) move into their FP64 accumulators (columns npad +
                // 2j, +1) and restart from zero, so that FP32 never sums more
                // than hot_every chunks of them; tensor-memory traffic only
                for (int b = 0; b < 2; ++b)
                    if (pending[b]) {
                        ok = um::mbar_wait(&mbar[b], parity[b]) && ok;
                        parity[b] ^= 1u;
                        pending[b] = false;
                    }
                um::fence_after_sync();
                if (ok) {
                    for (int blk = warp >> 2; blk < hot / 16; blk += NT) {
                        float v[16];
                        uint32_t d[32];
                        um::tmem_ld16(um::tmem_lane_addr(tbase, warp & 3, 16 * blk), v);
                        if (nhot > 0) um::tmem_ld32(um::tmem_lane_addr(tbase, warp & 3, npad + 32 * blk), d);
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const double a = (nhot > 0 ? __hiloint2double((int)d[2 * j + 1], (int)d[2 * j]) : 0.0) +
                                             (double)v[j];
                            d[2 * j] = (uint32_t)__double2loint(a);
                            d[2 * j + 1] = (uint32_t)__double2hiint(a);
                        }
                        um::tmem_st32(um::tmem_lane_addr(tbase, warp & 3, npad + 32 * blk), d);
                        uint32_t z[16];
#pragma unroll
                        for (int j = 0; j < 16; ++j) z[j] = 0u;
                        um::tmem_st16(um::tmem_lane_addr(tbase, warp & 3, 16 * blk), z);
                    }
                    um::tmem_wait_st();
                }
                ++nhot;
                um::fence_before_sync();
                __syncthreads();
            }
            if (group_end) {
                // end of a group of reactions: wait for its MMAs, then add the
                // FP32 partial sums into the FP64 output; the NT warps that
                // share a lane quadrant split the columns
                for (int b = 0; b < 2; ++b)
                    if (pending[b]) {
                        ok = um::mbar_wait(&mbar[b], parity[b]) && ok;
                        parity[b] ^= 1u;
                        pending[b] = false;
                    }
                um::fence_after_sync();
                if (ok) {
                    for (int col = 16 * (warp >> 2); col < npad; col += 16 * NT) {
                        float v[16];
                        uint32_t d[32];
                        um::tmem_ld16(um::tmem_lane_addr(tbase, warp & 3, col), v);
                        const bool h64 = col < hot && nhot > 0;
                        if (h64) um::tmem_ld32(um::tmem_lane_addr(tbase, warp & 3, npad + 2 * col), d);
                        if (act)
                            for (int j = 0; j < 16; ++j) {
                                const int sp = __ldg(perm + col + j);
                                if (sp >= 0) {
                                    double x = (double)v[j];
                                    if (h64) x += __hiloint2double((int)d[2 * j + 1], (int)d[2 * j]);
                                    double* w = wdot + (int64_t)sp * ng + i;
                                    // first (often only) group: a streaming store
                                    if (first_group) __stcs(w, x);
                                    else *w += x;
                                }
                            }
                    }
                }
                first_group = false;
                um::fence_before_sync();
                __syncthreads();
            }
        }
        um::fence_before_sync();
        __syncthreads();
    }
    if (!ok && lane == 0) atomicExch(err, 1);
    __syncthreads();
    if (warp == 0) um::tmem_dealloc(tbase, tcols);
}

// ------------------------------------------------------------ 32-point tile
//
// One point per lane and one reaction per warp: every lane of a warp runs the
// same reaction (no divergence, records read once per warp), and the tile's
// C (FP32) and G (FP64) fit in shared memory for every mechanism that the mixed
// mode takes (352 species), where a 128-point tile holds G up to 126 species
// only and had to read it from L2 for every molecule beyond.  The 16 warps take
// the 32 reactions of two chunks, two each; lane p's rates are row p of the A
// operands.  The MMAs stay M = 128 (the tensor memory's lanes): rows 32..127
// read whatever follows in shared memory, and nobody reads their sums.  A batch
// of 20011 points is 5 rounds of 626 tiles instead of two waves of 157.  The
// order of the contraction's sums -- reactions in K, chunks, splits, hot flushes --
// is the 128-point kernel's.  The prologue's sums over species (16 parts), ctot, the
// falloff (q_exp, q_rcp) and its Gibbs sum are not, in FP64: a rate whose FP32
// rounding that tips differs by an ulp, so the two kernels agree to rounding
// (far inside the mixed mode's 1e-6), not bit for bit.
// Bound by latency (41 % of issue slots; FP64 chains, shared loads, records
// from L1) with 17 warps of 96 registers.  Measured on B200: JetSurf 2.0, 20011
// points 2.30 -> 1.12 ms, 256 points 1.11 -> 0.22 ms; 348/2163, 20011 points
// 1.71 -> 0.89 ms, 65536 points 3.43 -> 2.47 ms.
constexpr int kTP = 32, kTWarps = 16;
constexpr int kA32 = 1024;             // bytes of a split's 32 rows

// A tile's per-point values that only the slow path reads, in shared memory.
struct Tile32 {
    double T[kTP], P[kTP], lnT[kTP], invT[kTP];
    float ctot[kTP];
    double tab[16];
};

// M of a pre-decoded reaction.
__device__ __forceinline__ float third_body32(const DevMech& m, int r, const TcFast& F, float ctot32, const float* sC) {
    const int lane = threadIdx.x & 31;
    const int e1 = F.neff < 255 ? F.eff0 + F.neff : __ldg(m.eff_ptr + r + 1);
    return tc_third_body<kTP>(m, F.eff0, e1, sC, ctot32, lane);
}

__device__ __forceinline__ float c_at(const char* C, unsigned off) {
    return *reinterpret_cast<const float*>(C + off);
}
__device__ __forceinline__ double g_at(const char* G, unsigned off) {
    return *reinterpret_cast<const double*>(G + 2 * off);
}

// q = 2^a cf - 2^(a + g) cb of a pre-decoded reaction (offsets of 128-byte rows
// of C, twice that of G).  pow2: a species' square is formed first, as
// rate_of_progress does.
__device__ __forceinline__ float net32(const TcFast& F, double a, float Ms, const char* C, const char* G, bool pow2) {
    const float x0 = c_at(C, F.sr[0]), x1 = c_at(C, F.sr[1]), x2 = c_at(C, F.sr[2]);
    float cf = x0 * x1 * x2;
    if (pow2 && F.sr[1] == F.sr[2]) cf = x0 * (x1 * x2);
    float q = rate32(a, cf * Ms, -32 * (int)F.ordf);
    if (F.flags & kFastRev) {
        const double g = (g_at(G, F.sr[0]) + g_at(G, F.sr[1]) + g_at(G, F.sr[2])) -
                         (g_at(G, F.sp[0]) + g_at(G, F.sp[1]) + g_at(G, F.sp[2]));
        const float y0 = c_at(C, F.sp[0]), y1 = c_at(C, F.sp[1]), y2 = c_at(C, F.sp[2]);
        float cb = y0 * y1 * y2;
        if (pow2 && F.sp[1] == F.sp[2]) cb = y0 * (y1 * y2);
        q -= rate32(a + g, cb * Ms, -32 * (int)F.ordb);
    }
    return (F.flags & kFastNeg) ? -q : q;
}

// An elementary or three-body reaction.
__device__ __forceinline__ float rate_common32(const DevMech& m, int r, const TcFast& F, double lnT2, double invT,
                                               float ctot32, const float* sC, const double* sG) {
    const int lane = threadIdx.x & 31;
    const float Ms = (F.flags & kFastThird) ? third_body32(m, r, F, ctot32, sC) : 1.0f;
    return net32(F, fma(F.b, lnT2, F.l2A) - F.th2 * invT, Ms, reinterpret_cast<const char*>(sC + lane),
                 reinterpret_cast<const char*>(sG + lane), false);
}

// A reaction with general stoichiometry that is no falloff and no PLOG, FP64
// (rate_of_progress_fp64 with one reaction per warp): each lane fetches one
// entry of the reaction's row, so the row is one load deep instead of two per
// entry.
__device__ __noinline__ float rate_general32(const DevMech& m, int r, int kind, float Ms, TileCtx c) {
    const int lane = threadIdx.x & 31;
    const DRxn R = load_rxn(m.rxn + r);
    const int r0 = __ldg(m.gen_rptr + R.gen), r1 = __ldg(m.gen_rptr + R.gen + 1);
    const int p0 = __ldg(m.gen_pptr + R.gen), p1 = __ldg(m.gen_pptr + R.gen + 1);
    const int nr = r1 - r0, n = nr + p1 - p0, at = lane < nr ? r0 + lane : p0 + (lane - nr);
    const int sp = lane < n ? __ldg(m.gen_sp + at) : 0;
    const double nu = lane < n ? __ldg(m.gen_nu + at) : 0.0;
    const double kf = R.sgn * cgm::cg_exp_clamped(fma(R.b, c.lnT, R.lnA) - R.theta * c.invT);
    const double cs = 2.3283064365386963e-10;   // 2^-32
    double qf = kf, pb = 1.0, g = 0.0;
    for (int j = 0; j < n; ++j) {
        const int k = __shfl_sync(0xffffffffu, sp, j);
        const double v = __shfl_sync(0xffffffffu, nu, j);
        const double x = (double)c.C[k * kTP + lane] * cs, y = v == 1.0 ? x : pow(x, v);
        if (j < nr) qf *= y;
        else pb *= y;
        g = fma(j < nr ? v : -v, c.G[k * kTP + lane], g);
    }
    const double qb = (R.flags & CG_F_REVERSIBLE) ? kf * exp2(g) * pb : 0.0;
    double rr = qf - qb;
    if (kind == CG_THIRD_BODY) rr *= (double)Ms * cs;
    return (float)rr;
}

// A reaction without a pre-decoded form.  Out of line, like the falloff, and
// with its context in shared memory, so that the common path keeps its values
// in registers (inline, they went through local memory: 374 instructions a
// reaction).
__device__ __noinline__ float rate_other32(const DevMech& m, const TcFast* fast, int r, const Tile32* t,
                                           const float* sC, const double* sG) {
    const int lane = threadIdx.x & 31;
    TileCtx c;
    c.C = sC;
    c.G = sG;
    c.T = t->T[lane];
    c.Pv = t->P[lane];
    c.lnT = t->lnT[lane];
    c.invT = t->invT[lane];
    c.ctot32 = t->ctot[lane];
    const TcFast F = load_fast(fast + r);
    const DRxn R = load_rxn(m.rxn + r);
    if ((R.flags & kFCompact) || r >= m.seg[CG_LINDEMANN] || F.ngen > 32) return rate_of_progress<kTP>(m, r, c, lane);
    return rate_general32(m, r, r >= m.seg[CG_THIRD_BODY] ? CG_THIRD_BODY : CG_STANDARD,
                          r >= m.seg[CG_THIRD_BODY] ? third_body32(m, r, F, c.ctot32, sC) : 0.0f, c);
}

// log of both values, the one's chain beside the other's.
__device__ __forceinline__ void log_pair(double (&x)[2]) {
    const double y0 = cgm::cg_log_of_normal(x[0]), y1 = cgm::cg_log_of_normal(x[1]);
    const bool s0 = !cgm::cg_log_normal(x[0]), s1 = !cgm::cg_log_normal(x[1]);
    if (s0 || s1) {
        x[0] = s0 ? cgm::cg_log_special(x[0]) : y0;
        x[1] = s1 ? cgm::cg_log_special(x[1]) : y1;
        return;
    }
    x[0] = y0;
    x[1] = y1;
}

// Two falloff reactions of one kind (STEP 0: one, twice), falloff_l2's blend with
// the quad kernels' exp, each step of one beside the same step of the other: a
// chain of FP64 logarithms, exponentials and loads bounds them (JetSurf 2.0,
// 20011 points: 1.57 ms one after the other, 1.49 ms so).
template <int STEP>
__device__ __noinline__ float2 falloff_pair32(const DevMech& m, const TcFast* fast, int r, int kind, const Tile32* t,
                                              const float* sC, const double* sG) {
    const int lane = threadIdx.x & 31;
    const double T = t->T[lane], lnT = t->lnT[lane], invT = t->invT[lane];
    const double* tab = t->tab;
    constexpr double kLog10_2 = 0.30102999566398119521, kLn2 = 0.69314718055994530942;
    float Ms[2];
    {
        int e0[2], n[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const TcFast F = load_fast(fast + r + j * STEP);
            e0[j] = F.eff0;
            n[j] = F.neff < 255 ? F.neff : __ldg(m.eff_ptr + r + j * STEP + 1) - F.eff0;
            Ms[j] = t->ctot[lane];
        }
        for (int e = 0; e < max(n[0], n[1]); e += 4) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                int sp[4];
                float ev[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const bool ok = e + u < n[j];
                    sp[u] = ok ? __ldg(m.eff_sp + e0[j] + e + u) : 0;
                    ev[u] = ok ? (float)__ldg(m.eff_val + e0[j] + e + u) : 0.0f;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float cv = sC[sp[u] * kTP + lane];
                    if (e + u < n[j]) Ms[j] = fmaf(ev[u], cv, Ms[j]);
                }
            }
        }
    }
    double ainf[2], l2pr[2], x[2], l2r[2], l2F[2] = {0.0, 0.0};
    const DFall* fr[2];
    int fl[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const DRxn R = load_rxn(m.rxn + r + j * STEP);
        fr[j] = m.fall + R.aux;
        fl[j] = R.flags;
        const double2 f0 = __ldg(reinterpret_cast<const double2*>(fr[j]));
        ainf[j] = (fma(R.b, lnT, R.lnA) - R.theta * invT) * kLog2eD;
        const double a0 = (fma(f0.y, lnT, f0.x) - __ldg(&fr[j]->theta0) * invT) * kLog2eD;
        l2pr[j] = a0 - ainf[j];
        x[j] = (double)Ms[j] * 2.3283064365386963e-10;
    }
    log_pair(x);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        l2pr[j] = l2pr[j] + x[j] * kLog2eD;
        x[j] = 1.0 + q_exp(fmax(-fabs(l2pr[j]) * kLn2, kQMinArg), tab);   // 1 + min(Pr, 1/Pr)
    }
    log_pair(x);
#pragma unroll
    for (int j = 0; j < 2; ++j) l2r[j] = fmin(l2pr[j], 0.0) - x[j] * kLog2eD;
    if (kind == CG_TROE) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const double2 p01 = __ldg(reinterpret_cast<const double2*>(fr[j]->p));
            const double2 p23 = __ldg(reinterpret_cast<const double2*>(fr[j]->p) + 1);
            const double x2 = __ldg(&m.fall2[fr[j] - m.fall].T2);
            double Fc = fma(p01.x, q_exp(fmax(-T * p01.y, kQMinArg), tab), p23.x * q_exp(fmax(-T * p23.y, kQMinArg), tab));
            const double e2 = q_exp(fmax(-x2 * invT, kQMinArg), tab);
            x[j] = (fl[j] & CG_F_TROE_T2) ? Fc + e2 : Fc;
        }
        log_pair(x);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const double lFc = x[j] * 0.4342944819032518;                // cg_log10
            const double lp = fma(kLog10_2, l2pr[j], fma(-0.67, lFc, -0.4));
            const double f1 = lp * q_rcp(fma(-0.14, lp, fma(-1.27, lFc, 0.75)));
            l2F[j] = lFc * q_rcp(fma(f1, f1, 1.0)) / kLog10_2;
        }
    } else if (kind == CG_SRI) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const DFall f = load_fall(fr[j]);
            const double lp = kLog10_2 * l2pr[j];
            const double X = q_rcp(fma(lp, lp, 1.0));
            const double base = fma(f.p[0], q_exp(fmax(-f.p[1] * invT, kQMinArg), tab),
                                    q_exp(fmax(-T * f.p[2], kQMinArg), tab));
            const double x2 = __ldg(&m.fall2[fr[j] - m.fall].T2);
            l2F[j] = (cgm::cg_log(f.p[3]) + fma(X, cgm::cg_log(base), x2 * lnT)) * kLog2eD;
        }
    }
    float q[2];
#pragma unroll
    for (int j = 0; j < 2; ++j)
        q[j] = net32(load_fast(fast + r + j * STEP), ainf[j] + (l2r[j] + l2F[j]), 1.0f,
                     reinterpret_cast<const char*>(sC + lane), reinterpret_cast<const char*>(sG + lane), true);
    return make_float2(q[0], q[1]);
}

// The two reactions r, r + 1 of a warp when one of them has no common form, or
// does not exist.
__device__ __noinline__ float2 rate_pair32(const DevMech& m, const TcFast* fast, int r, const Tile32* t,
                                           const float* sC, const double* sG) {
    const int lane = threadIdx.x & 31;
    float q[2] = {0.0f, 0.0f};
    auto kind_of = [&](int k) {
        int kind = CG_LINDEMANN;
        while (kind < CG_SRI && k >= m.seg[kind + 1]) ++kind;
        return kind;
    };
    if (r + 1 < m.nr && (load_fast(fast + r).flags & load_fast(fast + r + 1).flags & kFastFall)) {
        const int kind = kind_of(r);
        if (r + 1 < m.seg[kind + 1]) return falloff_pair32<1>(m, fast, r, kind, t, sC, sG);
    }
    for (int j = 0; j < 2; ++j) {
        if (r + j >= m.nr) break;
        const TcFast F = load_fast(fast + r + j);
        if (F.flags & kFastFall) {
            q[j] = falloff_pair32<0>(m, fast, r + j, kind_of(r + j), t, sC, sG).x;
            continue;
        }
        if (!(F.flags & kFastOn)) {
            q[j] = rate_other32(m, fast, r + j, t, sC, sG);
            continue;
        }
        q[j] = rate_common32(m, r + j, F, t->lnT[lane] * kLog2eD, t->invT[lane], t->ctot[lane], sC, sG);
    }
    return make_float2(q[0], q[1]);
}

// The most-touched species' FP32 sums move into their FP64 accumulators
// (tensor memory lanes 0..31), by the issuing warp.  Out of line, like the
// function after it: 48 registers of columns beside a loop's values would
// spill to local memory, whose 512 x 370 bytes do not stay in the L1 that the
// tile leaves (83 spills a pair of chunks cost 10k cycles).
__device__ __noinline__ void flush_hot32(int nhot, uint32_t tbase, int npad, int hot) {
    for (int blk = 0; blk < hot / 16; ++blk) {
        float v[16];
        uint32_t d[32];
        um::tmem_ld16(um::tmem_lane_addr(tbase, 0, 16 * blk), v);
        if (nhot > 0) um::tmem_ld32(um::tmem_lane_addr(tbase, 0, npad + 32 * blk), d);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const double a = (nhot > 0 ? __hiloint2double((int)d[2 * j + 1], (int)d[2 * j]) : 0.0) + (double)v[j];
            d[2 * j] = (uint32_t)__double2loint(a);
            d[2 * j + 1] = (uint32_t)__double2hiint(a);
        }
        um::tmem_st32(um::tmem_lane_addr(tbase, 0, npad + 32 * blk), d);
        uint32_t z[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) z[j] = 0u;
        um::tmem_st16(um::tmem_lane_addr(tbase, 0, 16 * blk), z);
    }
    um::tmem_wait_st();
}

// The sums of a group leave tensor memory for wdot.  w: this point's wdot, or
// NULL.
__device__ __noinline__ void flush32(bool first_group, int nhot, uint32_t tbase, int warp, int npad,
                 int hot, const int* __restrict__ perm, double* w, int64_t ng) {
    for (int col = 16 * (warp >> 2); col < npad; col += 4 * kTWarps) {
        float v[16];
        uint32_t d[32];
        um::tmem_ld16(um::tmem_lane_addr(tbase, 0, col), v);
        const bool h64 = col < hot && nhot > 0;
        if (h64) um::tmem_ld32(um::tmem_lane_addr(tbase, 0, npad + 2 * col), d);
        if (!w) continue;
        int sp[16];
#pragma unroll
        for (int j = 0; j < 4; ++j) reinterpret_cast<int4*>(sp)[j] = __ldg(reinterpret_cast<const int4*>(perm + col) + j);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            if (sp[j] < 0) continue;
            double x = (double)v[j];
            if (h64) x += __hiloint2double((int)d[2 * j + 1], (int)d[2 * j]);
            double* o = w + (int64_t)sp[j] * ng;
            if (first_group) __stcs(o, x);
            else *o += x;
        }
    }
}

// 16 warps compute, a 17th loads the stoichiometry, issues the MMAs and moves
// the hot species' sums.  The compute warps meet only at a tile's prologue: a
// pair's operands are handed over by mbarriers (full: one arrival a warp; done:
// the MMAs' commit), so a warp runs up to two pairs ahead of the slowest.  The
// 17th warp's turn is the other half of the pipeline: with descriptors built for
// every MMA (2000 cycles a pair) and the hot sums moved by compute warps (3900
// cycles every four pairs) a pair of elementary reactions took 2.9 us, now 2.1
// (348 species); with a block barrier each pair, 3.5.
__global__ void __launch_bounds__(32 * (kTWarps + 1), 1)
    getrates_tc32_kernel(const __grid_constant__ DevMech m, const __nv_bfloat16* __restrict__ nu,
                         const TcFast* __restrict__ fast, int npad, int nhalf, int nchunk, uint32_t tcols,
                         const double* __restrict__ P, const double* __restrict__ Tg, const double* __restrict__ Y,
                         double* __restrict__ wdot, int64_t ng, int* err, int group, const int* __restrict__ perm,
                         int hot, int hot_every) {
    extern __shared__ __align__(1024) unsigned char sm[];
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int ns = m.ns, rows = ns + 1;
    unsigned char* sA = sm;                                     // [2 buffers][2 chunks][3 splits][32 x 16] BF16
    unsigned char* sB = sA + 12 * kA32;                         // [2 buffers][2 chunks][npad x 16] BF16
    // (the A operands' rows 32..127 run into sB, at most 3 KB of it and of sG)
    double* sG = reinterpret_cast<double*>(sB + 4 * npad * 32);    // [rows][32]
    float* sC = reinterpret_cast<float*>(sG + rows * kTP);      // [rows][32]
    double* sRed = reinterpret_cast<double*>(sC + rows * kTP);  // [16][32]
    Tile32* sT = reinterpret_cast<Tile32*>(sRed + kTWarps * kTP);
    uint64_t* full = reinterpret_cast<uint64_t*>(sT + 1);       // [2] A written
    uint64_t* done = full + 2;                                  // [2] MMAs done
    uint64_t* bfull = full + 4;                                 // [2] B loaded
    uint64_t* flushed = full + 6;                               // sums taken out of tensor memory
    uint32_t* tslot = reinterpret_cast<uint32_t*>(full + 7);
    if (tid == 0) {
        for (int j = 0; j < 2; ++j) {
            um::mbar_init(&full[j], kTWarps);
            um::mbar_init(&done[j], 1);
            um::mbar_init(&bfull[j], 1);
        }
        um::mbar_init(flushed, kTWarps / 4);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < 16) sT->tab[tid] = kQExpTab[tid];
    if (warp == 0) um::tmem_alloc(tslot, tcols);
    um::fence_before_sync();
    __syncthreads();
    um::fence_after_sync();
    const uint32_t tbase = *tslot;
    const int npair = (nchunk + 1) / 2;
    const int64_t ntiles = (ng + kTP - 1) / kTP;
    // A wait that runs out clears ok; the warp goes on without waiting (and the
    // issuing warp without loads and MMAs), so that every warp reaches the end.
    bool ok = true;
    uint32_t n = 0, nflush = 0;        // pairs and flushes so far, of all tiles
    auto wait = [&](uint64_t* bar, uint32_t use) { ok = ok && um::mbar_wait(bar, use & 1u); };
    // chunks so far in the group and since the last hot flush, after nc more
    // of them: group and hot_every are even, so a flush falls on the end of a
    // pair (hot flushes: one group per tile)
    int gpos = 0, hpos = 0;
    auto flush_after = [&](int ch_end, int nc, bool& hot_end) {
        gpos += nc;
        hpos += nc;
        const bool group_end = gpos == group || ch_end == nchunk;
        hot_end = hot > 0 && !group_end && hpos == hot_every;
        if (group_end) gpos = 0;
        if (group_end || hot_end) hpos = 0;
        return group_end || hot_end;
    };
    if (warp == kTWarps) {
        const uint32_t idesc = um::idesc_bf16(kTile, nhalf);
        const int nh = npad / nhalf;
        // descriptors of the first operands; others lie a multiple of 16 bytes further
        const uint64_t ad0 = um::desc_kmajor(um::smem_addr(sA), kChunk, 0);
        const uint64_t bd0 = um::desc_kmajor(um::smem_addr(sB), kChunk, 0);
        const uint32_t bstep = (uint32_t)(npad * 32) >> 4, hstep = (uint32_t)(nhalf * 32) >> 4;
        auto load = [&](int pr, uint32_t k) {                   // pair pr of a tile, pair k of all
            const uint32_t bytes = (uint32_t)(min(2, nchunk - 2 * pr) * npad * 32);
            um::mbar_expect_tx(&bfull[k & 1], bytes);
            um::bulk_g2s(sB + (k & 1) * 2 * npad * 32, nu + (int64_t)2 * pr * npad * kChunk, bytes, &bfull[k & 1]);
        };
        const bool any = (int64_t)blockIdx.x < ntiles && npair > 0;
        bool inflight = any;
        if (any && lane == 0) load(0, 0);
        for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
            int nhot = 0;
            for (int pr = 0; pr < npair; ++pr, ++n) {
                const uint32_t buf = n & 1;
                const int ch0 = 2 * pr, nc = min(2, nchunk - ch0);
                const bool start = gpos == 0;
                // the other buffers are free when the last pair's MMAs are done
                if (n > 0) wait(&done[buf ^ 1], (n - 1) >> 1);
                const bool more = pr + 1 < npair || tile + gridDim.x < ntiles;
                if (inflight) ok = um::mbar_wait(&bfull[buf], (n >> 1) & 1u) && ok;   // even after a time-out
                ok = __all_sync(0xffffffffu, ok);
                inflight = ok && more;
                if (inflight && lane == 0) load(pr + 1 < npair ? pr + 1 : 0, n + 1);
                __syncwarp();
                wait(&full[buf], n >> 1);
                ok = __all_sync(0xffffffffu, ok);
                um::fence_after_sync();
                if (lane == 0) {
#pragma unroll
                    for (int cc = 0; cc < 2; ++cc) {
                        if (cc >= nc || !ok) break;
                        const uint64_t ad = ad0 + (buf * 2 + cc) * 3 * (kA32 >> 4), bd = bd0 + (buf * 2 + cc) * bstep;
#pragma unroll
                        for (int s = 0; s < 3; ++s) {
                            const uint32_t acc = (!start || cc > 0 || s > 0) ? 1u : 0u;
                            um::mma_bf16(tbase, ad + s * (kA32 >> 4), bd, idesc, acc);
                            if (nh > 1) um::mma_bf16(tbase + (uint32_t)nhalf, ad + s * (kA32 >> 4), bd + hstep, idesc, acc);
                        }
                    }
                    um::commit(&done[buf]);
                }
                __syncwarp();
                bool hot_end;
                if (flush_after(ch0 + nc, nc, hot_end)) {
                    if (hot_end) {
                        wait(&done[buf], n >> 1);
                        ok = __all_sync(0xffffffffu, ok);
                        um::fence_after_sync();
                        if (ok) flush_hot32(nhot, tbase, npad, hot);
                        ++nhot;
                        um::fence_before_sync();
                        __syncwarp();
                    } else {
                        wait(flushed, nflush);
                        ++nflush;
                    }
                    um::fence_after_sync();
                }
            }
        }
    } else {
        const int rsub = (warp >> 3) * kChunk + 2 * (warp & 7);     // this warp's two reactions of a pair
        for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
            const int64_t i = tile * kTP + lane;
            const bool act = i < ng;
            const double T = act ? __ldcs(Tg + i) : 1000.0, Pv = act ? __ldcs(P + i) : kPatm;
            const double lnT = cgm::cg_log(T), invT = 1.0 / T, lnT2 = lnT * kLog2eD;
            um::bar_sync(1, 32 * kTWarps);                      // the last tile's rates are done
            double part = 0.0;
#pragma unroll 8
            for (int k = warp; k < ns; k += kTWarps) {
                asm volatile("prefetch.global.L1 [%0];" ::"l"(m.thermo + 16 * k));
                const double yk = (act ? __ldcs(Y + (int64_t)k * ng + i) : 1.0) * __ldg(m.inv_mw + k);
                sG[k * kTP + lane] = yk;
                part += yk;
            }
            sRed[warp * kTP + lane] = part;
            um::bar_sync(1, 32 * kTWarps);
            double csum = 0.0;
#pragma unroll
            for (int q = 0; q < kTWarps; ++q) csum += sRed[q * kTP + lane];
            const double facs = Pv / (kR0 * csum * T) * 4294967296.0;
            const float ctot32 = (float)(csum * facs);
            if (warp == 0) {
                sT->T[lane] = T;
                sT->P[lane] = Pv;
                sT->lnT[lane] = lnT;
                sT->invT[lane] = invT;
                sT->ctot[lane] = ctot32;
                sC[ns * kTP + lane] = 1.0f;
                sG[ns * kTP + lane] = 0.0;
            }
            const double lpfac2 = -6.35856916300311 - lnT2;     // log2(Patm/R0) - log2 T
#pragma unroll 4
            for (int k = warp; k < ns; k += kTWarps) {
                sC[k * kTP + lane] = (float)(sG[k * kTP + lane] * facs);
                const double* th = m.thermo + 16 * k;
                th += T < __ldg(th) ? 1 : 8;
                double cf[7];
#pragma unroll
                for (int j = 0; j < 7; ++j) cf[j] = __ldg(th + j);
                sG[k * kTP + lane] = fma(smh_poly(cf, T, lnT, invT), kLog2eD, lpfac2);
            }
            um::bar_sync(1, 32 * kTWarps);
            bool first_group = true;
            int nhot = 0;
            for (int pr = 0; pr < npair; ++pr, ++n) {
                const uint32_t buf = n & 1;
                const int ch0 = 2 * pr, nc = min(2, nchunk - ch0), r0 = ch0 * kChunk + rsub;
                // (records come from L1, where the last pair's turn has put them: held in
                // registers across the calls below they would go through local memory)
                const TcFast F0 = load_fast(fast + min(r0, m.nr - 1)), F1 = load_fast(fast + min(r0 + 1, m.nr - 1));
                float q0, q1;
                if ((F0.flags & F1.flags & kFastOn) && r0 + 1 < m.nr) {
                    q0 = rate_common32(m, r0, F0, lnT2, invT, ctot32, sC, sG);
                    q1 = rate_common32(m, r0 + 1, F1, lnT2, invT, ctot32, sC, sG);
                } else {
                    const float2 q = rate_pair32(m, fast, r0, sT, sC, sG);
                    q0 = q.x;
                    q1 = q.y;
                }
                if (lane < 2 && r0 + 2 * kChunk + lane < m.nr)
                    asm volatile("prefetch.global.L1 [%0];" ::"l"(fast + r0 + 2 * kChunk + lane));
                if (!act) q0 = q1 = 0.0f;
                // q = hi + mid + lo in BF16
                uint32_t w[3];
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const __nv_bfloat16 b0 = __float2bfloat16_rn(q0), b1 = __float2bfloat16_rn(q1);
                    w[j] = (uint32_t)__bfloat16_as_ushort(b0) | (uint32_t)__bfloat16_as_ushort(b1) << 16;
                    q0 -= __bfloat162float(b0);
                    q1 -= __bfloat162float(b1);
                }
                if (n > 1) wait(&done[buf], (n - 2) >> 1);      // the buffer's last MMAs
                unsigned char* a0 = sA + (buf * 2 + (warp >> 3)) * 3 * kA32 +
                                    um::kmajor_offset(lane, 2 * (warp & 7), kChunk);
#pragma unroll
                for (int j = 0; j < 3; ++j) *reinterpret_cast<uint32_t*>(a0 + j * kA32) = w[j];
                um::fence_proxy_async();
                __syncwarp();
                if (lane == 0) um::mbar_arrive(&full[buf]);
                bool hot_end;
                if (!flush_after(ch0 + nc, nc, hot_end)) continue;
                if (hot_end) {
                    ++nhot;
                    continue;
                }
                // the tile's sums are in lanes 0..31: the warps of that quadrant take
                // them out while the others go on
                if ((warp & 3) == 0) {
                    wait(&done[buf], n >> 1);
                    ok = __all_sync(0xffffffffu, ok);
                    um::fence_after_sync();
                    if (ok) flush32(first_group, nhot, tbase, warp, npad, hot, perm, act ? wdot + i : nullptr, ng);
                    um::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) um::mbar_arrive(flushed);
                }
                first_group = false;
            }
        }
    }
    if (!ok && lane == 0) atomicExch(err, 1);
    um::fence_before_sync();
    __syncthreads();
    if (warp == 0) um::tmem_dealloc(tbase, tcols);
}

const void* kernel_for(int nt) {
    return nt == 4 ? (const void*)getrates_tc_kernel<4>
                   : nt == 2 ? (const void*)getrates_tc_kernel<2> : (const void*)getrates_tc_kernel<1>;
}

template <int NT>
cudaError_t launch_tc(const MixedPlan* p, const DevMech& m, const double* P, const double* T, const double* Y,
                      double* wdot, int64_t ng, int64_t grid, cudaStream_t s) {
    getrates_tc_kernel<NT><<<(unsigned)grid, kTile * NT, p->smem, s>>>(m, p->nu, p->fast, p->npad, p->nhalf, p->nchunk,
                                                                       p->tcols, P, T, Y, wdot, ng, p->err, p->group,
                                                                       p->perm, p->hot, p->hot_every);
    return cudaGetLastError();
}

}  // namespace

// ---------------------------------------------------------------- host side
cudaError_t mixed_prepare(const DevMech& m, const cg_mech_view& v, int device, MixedPlan** out) {
    *out = nullptr;
    const int ns = m.ns, nr = m.nr;
    int npad = (ns + 31) / 32 * 32;
    if (npad > 512) return cudaErrorNotSupported;     // TMEM holds 512 FP32 columns per lane
    const int nhalf = npad <= 256 ? npad : npad / 2;
    uint32_t tcols = 32;
    while ((int)tcols < npad) tcols <<= 1;
    const int nchunk = (nr + kChunk - 1) / kChunk;
    // the largest share count is planned for; the [nt][128] partial-sum slots follow the state
    const size_t rows = (size_t)ns + 1;                       // + the dummy row of TcFast
    const size_t base = 6 * (size_t)kABytes + 2 * (size_t)npad * 32 + rows * kTile * 4 + 4 * kTile * 8 + 32;
    const size_t with_g = base + rows * kTile * 8;
    DeviceLimits dev;
    cudaError_t e = device_limits(device, &dev);
    if (e != cudaSuccess) return e;
    const size_t limit = dev.smem_block;
    // up to 352 species; the 32-point tile then fits too (198 KB)
    const size_t t32 = 12 * (size_t)kA32 + 4 * (size_t)npad * 32 + rows * kTP * 12 + kTWarps * kTP * 8 + sizeof(Tile32) + 64;
    if (base > limit || t32 > limit) return cudaErrorNotSupported;
    MixedPlan* p = new MixedPlan();
    p->ns = ns;
    p->nr = nr;
    p->npad = npad;
    p->nhalf = nhalf;
    p->nchunk = nchunk;
    p->tcols = tcols;
    p->t128 = with_g <= limit ? 1 : 0;
    // FP32 accumulation runs over `group` chunks (16 reactions each) before
    // the partial sums are added into the FP64 output: 64 reactions for small
    // mechanisms (GRI30 needs it for 1e-6), the whole mechanism for large
    // ones, whose output does not fit in L2 and would otherwise be read back
    // from DRAM at every flush (348/2163: 3.5e-7 with one flush)
    p->group = npad <= 128 ? 4 : nchunk;
    p->smem = p->t128 ? with_g : base;
    // resident CTAs per SM, limited by shared memory and by 512 TMEM columns
    int per_sm = (int)(dev.smem_sm / (p->smem + 1024));
    per_sm = std::min(per_sm, (int)(512 / tcols));
    per_sm = std::max(per_sm, 1);
    // threads per point: the most (4, 2, 1) whose registers still let per_sm
    // CTAs share the SM's register file
    p->nt = 1;
    for (int nt : {4, 2}) {
        cudaFuncAttributes fa;
        if (!p->t128 || cudaFuncGetAttributes(&fa, kernel_for(nt)) != cudaSuccess) continue;
        if ((long)per_sm * kTile * nt * fa.numRegs <= dev.regs_sm &&
            per_sm * kTile * nt <= dev.threads_sm) {
            p->nt = nt;
            break;
        }
    }
    p->grid = dev.sms * per_sm;
    p->smem32 = t32;
    p->grid32 = dev.sms;
    // nu chunks in the canonical K-major layout: B[n][k] = nu of species n in reaction 16*chunk + k
    std::vector<float> nuf((size_t)ns * nr, 0.0f);
    const int32_t* rp = (const int32_t*)v.a[CG_RPTR];
    const int32_t* pp = (const int32_t*)v.a[CG_PPTR];
    const int32_t* rsp = (const int32_t*)v.a[CG_RSP];
    const int32_t* psp = (const int32_t*)v.a[CG_PSP];
    const double* rnu = (const double*)v.a[CG_RNU];
    const double* pnu = (const double*)v.a[CG_PNU];
    for (int r = 0; r < nr; ++r) {
        for (int j = rp[r]; j < rp[r + 1]; ++j) nuf[(size_t)rsp[j] * nr + r] -= (float)rnu[j];
        for (int j = pp[r]; j < pp[r + 1]; ++j) nuf[(size_t)psp[j] * nr + r] += (float)pnu[j];
    }
    // accumulator columns: for large mechanisms (one FP64 flush per tile) the
    // species most reactions touch come first, and up to 48 of them (what the
    // spare tensor-memory columns hold as FP64, in multiples of 16) get FP64
    // accumulators flushed every hot_every chunks; otherwise file order
    std::vector<int> perm(npad, -1);
    for (int n = 0; n < ns; ++n) perm[n] = n;
    if (p->group == nchunk && nchunk > p->hot_every) {
        std::vector<int> nnz(ns, 0);
        for (int n = 0; n < ns; ++n)
            for (int r = 0; r < nr; ++r) nnz[n] += nuf[(size_t)n * nr + r] != 0.0f;
        std::stable_sort(perm.begin(), perm.begin() + ns, [&](int a, int b) { return nnz[a] > nnz[b]; });
        p->hot = std::min(48, std::min(((int)tcols - npad) / 2, ns) / 16 * 16);
    }
    std::vector<__nv_bfloat16> img((size_t)nchunk * npad * kChunk, __float2bfloat16(0.0f));
    bool exact = true;
    for (int ch = 0; ch < nchunk; ++ch)
        for (int n = 0; n < ns; ++n)
            for (int k = 0; k < kChunk; ++k) {
                const int r = ch * kChunk + k;
                if (r >= nr) continue;
                const float x = nuf[(size_t)perm[n] * nr + r];
                const __nv_bfloat16 b = __float2bfloat16(x);
                if (__bfloat162float(b) != x) exact = false;
                const size_t off = ((size_t)(n >> 3) * (kChunk * 16) + (k >> 3) * 128 + (n & 7) * 16 + (k & 7) * 2) / 2;
                img[(size_t)ch * npad * kChunk + off] = b;
            }
    if (!exact) {
        delete p;
        return cudaErrorNotSupported;                  // coefficients not exact in BF16
    }
    const size_t img_bytes = (img.size() * sizeof(__nv_bfloat16) + 255) / 256 * 256;
    const size_t fast_bytes = ((size_t)nr * sizeof(TcFast) + 255) / 256 * 256;
    const size_t perm_bytes = ((size_t)npad * sizeof(int) + 255) / 256 * 256;
    const size_t bytes = img_bytes + 2 * fast_bytes + perm_bytes + 256;
    e = cudaMalloc(&p->dbuf, bytes);
    if (e == cudaSuccess) e = cudaMemcpy(p->dbuf, img.data(), img.size() * sizeof(__nv_bfloat16), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset((char*)p->dbuf + bytes - 256, 0, 256);
    if (e == cudaSuccess)
        e = cudaMemcpy((char*)p->dbuf + img_bytes + 2 * fast_bytes, perm.data(), perm.size() * sizeof(int),
                       cudaMemcpyHostToDevice);
    if (e == cudaSuccess && p->t128)
        e = cudaFuncSetAttribute(kernel_for(p->nt), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p->smem);
    if (e != cudaSuccess) {
        if (p->dbuf) cudaFree(p->dbuf);
        delete p;
        return e;
    }
    p->nu = (const __nv_bfloat16*)p->dbuf;
    p->fast = (const TcFast*)((char*)p->dbuf + img_bytes);
    p->fast32 = (const TcFast*)((char*)p->dbuf + img_bytes + fast_bytes);
    p->perm = (const int*)((char*)p->dbuf + img_bytes + 2 * fast_bytes);
    if (nr > 0) {
        build_fast_kernel<<<(nr + 127) / 128, 128>>>(m, (TcFast*)p->fast, 1);
        build_fast_kernel<<<(nr + 127) / 128, 128>>>(m, (TcFast*)p->fast32, kTP * 4);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaDeviceSynchronize();
        if (e != cudaSuccess) {
            cudaFree(p->dbuf);
            delete p;
            return e;
        }
    }
    p->err = (int*)((char*)p->dbuf + bytes - 256);
    *out = p;
    return cudaSuccess;
}

void mixed_release(MixedPlan* p) {
    if (!p) return;
    if (p->dbuf) cudaFree(p->dbuf);
    delete p;
}

// What a caller of chemgen_getrates_ws is asked for: what mechanisms beyond the
// 128-point tile needed when it kept their Gibbs terms in global scratch.  No
// kernel uses it any more; the size stays, so that programs that ask for it,
// allocate it and pass it see no change.
size_t mixed_workspace_bytes(const MixedPlan* p, int64_t ng) {
    if (!p || p->t128) return 0;
    int64_t tiles = (ng + kTile - 1) / kTile;
    int64_t grid = std::min<int64_t>(tiles, p->grid);
    return (size_t)grid * (p->ns + 1) * kTile * sizeof(double);
}

cudaError_t launch_getrates_mixed(const MixedPlan* p, const DevMech& m, const double* P, const double* T,
                                  const double* Y, double* wdot, int64_t ng, cudaStream_t s) {
    if (ng <= 0) return cudaSuccess;
    // the kernel's shared-memory limit is this plan's, set under one lock with
    // the launch (a plan made later for a smaller mechanism sets it lower)
    static std::mutex mu;
    // Mechanisms whose Gibbs terms fit beside the 128-point tile run the faster
    // of the two.  On B200 at 53/325 a round of 32-point tiles takes 40 us and a
    // wave of 128-point tiles, one to an SM, 121 us, with 60 PLOG reactions 57 and
    // 171: there one or two rounds against a wave, or five against two, take the
    // 32-point kernel.  Smaller mechanisms have several 128-point tiles to an SM and a
    // wave for many more rounds: 9/21, 12 and 29 us, two rounds at most.  Larger
    // ones always run 32-point tiles (348/2163: a round 0.17 ms, a wave 0.82 ms).
    const int64_t rounds = (ng + (int64_t)kTP * p->grid32 - 1) / ((int64_t)kTP * p->grid32);
    const int64_t waves = (ng + (int64_t)kTile * p->grid - 1) / ((int64_t)kTile * p->grid);
    if (!p->t128 || (double)rounds * 0.35 <= (double)waves) {
        const unsigned g32 = (unsigned)std::min<int64_t>((ng + kTP - 1) / kTP, p->grid32);
        std::lock_guard<std::mutex> lk(mu);
        const cudaError_t e = cudaFuncSetAttribute(getrates_tc32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)p->smem32);
        if (e != cudaSuccess) return e;
        getrates_tc32_kernel<<<g32, 32 * (kTWarps + 1), p->smem32, s>>>(m, p->nu, p->fast32, p->npad, p->nhalf, p->nchunk,
                                                                  p->tcols, P, T, Y, wdot, ng, p->err, p->group,
                                                                  p->perm, p->hot, p->hot_every);
        return cudaGetLastError();
    }
    const int64_t grid = std::min<int64_t>((ng + kTile - 1) / kTile, p->grid);
    std::lock_guard<std::mutex> lk(mu);
    const cudaError_t e =
        cudaFuncSetAttribute(kernel_for(p->nt), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p->smem);
    if (e != cudaSuccess) return e;
    switch (p->nt) {
        case 4: return launch_tc<4>(p, m, P, T, Y, wdot, ng, grid, s);
        case 2: return launch_tc<2>(p, m, P, T, Y, wdot, ng, grid, s);
        default: return launch_tc<1>(p, m, P, T, Y, wdot, ng, grid, s);
    }
}

int mixed_error_flag(const MixedPlan* p) {
    int v = 0;
    if (!p || cudaMemcpy(&v, p->err, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    return v;
}

}  // namespace cg
