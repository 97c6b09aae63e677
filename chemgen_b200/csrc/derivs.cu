// Analytic derivatives of getrates: the dense Jacobian d wdot / d(T, Y) and
// the adjoint (vector-Jacobian product), table-driven so that one compiled
// kernel serves every mechanism.
//
// The reference has no derivative code (its torch prototype
// chemgen/chemistry_nn.py:15-85 never ran); these kernels differentiate the
// rate law of reactions/*.j2:
//     wdot_k = sum_r nu_kr q_r,   q_r = m_r (qf_r - qb_r),   C = C(T, Y)
// with
//     dC_m/dY_j  = (ctot delta_mj - C_m) / (W_j S),  S = sum_j Y_j / W_j,
//     dC_m/dT    = -C_m / T,   dM/dC_m = 1 + (eff_m - 1),
//     d ln kf/dT = (b + theta/T) / T   (theta = Ea/Rc),
//     d ln kb/dT = d ln kf/dT + sum nu_r dE_r - sum nu_p dE_p,
//     dE_k       = d ln(exp(smh_k) Patm/(R0 T))/dT = d smh_k/dT - 1/T,
//     falloff:   d ln kf = d ln kinf + g (d ln k0 - d ln kinf + d ln M) + d ln F|_Pr,
//                g = 1/(1 + Pr) + d ln F / d ln Pr.
// Mass-action derivatives use the product of the other factors, so species
// at zero concentration keep exact derivatives.
//
// Layouts: J[(k*(ns+1) + c)*ng + i], column c = 0 for T and 1 + j for Y_j;
// adjoint outputs gT[i], gY[j*ng + i], gP[i].  Per-point state (C, EGp, dE
// and, for the Jacobian, the dense-M vector A) lives in a scratch buffer of
// 4*ns*ng doubles laid out [array][species][point].
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <utility>
#include <vector>

#include "deriv_common.cuh"

namespace cg {
namespace {

template <bool JAC, typename JT>
__global__ void __launch_bounds__(128) deriv_kernel(DevMech m, const double* __restrict__ P, const double* __restrict__ Tg,
                                                    const double* __restrict__ Y, const double* __restrict__ G,
                                                    JT* __restrict__ J, double* __restrict__ gT, double* __restrict__ gY,
                                                    double* __restrict__ gP, double* __restrict__ scratch, int64_t ng) {
    const int ns = m.ns;
    const int64_t ncol = ns + 1;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ng; i += (int64_t)gridDim.x * blockDim.x) {
        DState st{scratch + i, scratch + (int64_t)ns * ng + i, scratch + (int64_t)2 * ns * ng + i,
                  scratch + (int64_t)3 * ns * ng + i, ng, ng};
        const double T = Tg[i], Pv = P[i];
        PointT pt;
        pt.T = T;
        pt.lnT = cgm::cg_log(T);
        pt.invT = 1.0 / T;
        double S = 0.0;
        for (int k = 0; k < ns; ++k) {
            const double c = Y[(int64_t)k * ng + i] * __ldg(m.inv_mw + k);
            st.C[k * st.s] = c;
            S += c;
        }
        const double fac = Pv / (kR0 * S * T);
        double ctot = 0.0;
        for (int k = 0; k < ns; ++k) {
            const double c = st.C[k * st.s] * fac;
            st.C[k * st.s] = c;
            ctot += c;
        }
        const double pfac = kPatm / (kR0 * T);
        for (int k = 0; k < ns; ++k) {
            const double* th = m.thermo + 16 * k;
            const double* c = (T < __ldg(th)) ? th + 1 : th + 8;
            double cc[7];
            for (int j = 0; j < 7; ++j) cc[j] = __ldg(c + j);
            const double smh = smh_poly(cc, T, pt.lnT, pt.invT);
            st.E[k * st.s] = cgm::cg_exp_clamped(smh) * pfac;
            // d smh/dT - 1/T
            const double dp = fma(fma(fma(4.0 * cc[5], T, 3.0 * cc[4]), T, 2.0 * cc[3]), T, cc[2]);
            st.D[k * st.s] = dp + fma(cc[6], pt.invT, cc[1]) * pt.invT - pt.invT;
            st.A[k * st.s] = 0.0;
        }
        if (JAC) {
            JT* Jp = J + i;
            for (int64_t c = 0; c < (int64_t)ns * ncol; ++c) Jp[c * ng] = (JT)0;
        } else {
            for (int k = 0; k < ns; ++k) gY[(int64_t)k * ng + i] = 0.0;   // holds C-bar until the end
        }
        double tb = 0.0, ab = 0.0, pb = 0.0;
        const double lnP = cgm::cg_log(Pv);
        for (int r = 0; r < m.nr; ++r) {
            Side re, pr;
            RxnGrad rg;
            const DRxn R = load_rxn(m.rxn + r);
            reaction_grad<16>(m, r, R, pt, ctot, Pv, lnP, st, re, pr, rg);
            const int kind = rg.kind, nd = rg.nd;
            const double dqdT = rg.dqdT, dqdM = rg.dqdM;
            const bool usesM = rg.usesM;
            const int* dsp = rg.dsp;
            const double* dqc = rg.dqc;
            if (JAC) {
                JT* Jp = J + i;
                // rows: every species of the reaction with its net coefficient contribution
                for (int side = 0; side < 2; ++side) {
                    const Side& s = side ? pr : re;
                    const double sg = side ? 1.0 : -1.0;
                    for (int kk = 0; kk < s.n; ++kk) {
                        const int k = s.sp[kk];
                        const double nu = sg * s.nu[kk];
                        Jp[(int64_t)(k * ncol) * ng] += (JT)(nu * dqdT);
                        for (int j = 0; j < nd; ++j) Jp[(int64_t)(k * ncol + 1 + dsp[j]) * ng] += (JT)(nu * dqc[j]);
                        if (usesM) {
                            st.A[k * st.s] = fma(nu, dqdM, st.A[k * st.s]);
                            for (int e = __ldg(m.eff_ptr + r); e < __ldg(m.eff_ptr + r + 1); ++e)
                                Jp[(int64_t)(k * ncol + 1 + __ldg(m.eff_sp + e)) * ng] +=
                                    (JT)(nu * __ldg(m.eff_val + e) * dqdM);
                        }
                    }
                }
            } else {
                double gq = 0.0;
                for (int j = 0; j < re.n; ++j) gq = fma(-re.nu[j], G[(int64_t)re.sp[j] * ng + i], gq);
                for (int j = 0; j < pr.n; ++j) gq = fma(pr.nu[j], G[(int64_t)pr.sp[j] * ng + i], gq);
                tb = fma(gq, dqdT, tb);
                for (int j = 0; j < nd; ++j) gY[(int64_t)dsp[j] * ng + i] = fma(gq, dqc[j], gY[(int64_t)dsp[j] * ng + i]);
                if (usesM) {
                    ab = fma(gq, dqdM, ab);
                    for (int e = __ldg(m.eff_ptr + r); e < __ldg(m.eff_ptr + r + 1); ++e) {
                        const int64_t o = (int64_t)__ldg(m.eff_sp + e) * ng + i;
                        gY[o] = fma(gq * dqdM, __ldg(m.eff_val + e), gY[o]);
                    }
                }
                if (kind == CG_PLOG) pb = fma(gq, rg.qnet * rg.dlkf_lnP / Pv, pb);
            }
        }
        const double iS = 1.0 / S;
        if (JAC) {
            JT* Jp = J + i;
            for (int k = 0; k < ns; ++k) {
                const double ak = st.A[k * st.s];
                double rk = ak * ctot;
                for (int j = 0; j < ns; ++j) rk = fma((double)Jp[(int64_t)(k * ncol + 1 + j) * ng], st.C[j * st.s], rk);
                Jp[(int64_t)(k * ncol) * ng] = (JT)((double)Jp[(int64_t)(k * ncol) * ng] - rk * pt.invT);
                for (int j = 0; j < ns; ++j) {
                    const int64_t o = (int64_t)(k * ncol + 1 + j) * ng;
                    Jp[o] = (JT)(fma(ctot, (double)Jp[o] + ak, -rk) * __ldg(m.inv_mw + j) * iS);
                }
            }
        } else {
            double rho = 0.0;
            for (int k = 0; k < ns; ++k) {
                const double cb = gY[(int64_t)k * ng + i] + ab;
                gY[(int64_t)k * ng + i] = cb;
                rho = fma(cb, st.C[k * st.s], rho);
            }
            for (int k = 0; k < ns; ++k) {
                const int64_t o = (int64_t)k * ng + i;
                gY[o] = fma(ctot, gY[o], -rho) * __ldg(m.inv_mw + k) * iS;
            }
            gT[i] = tb - rho * pt.invT;
            if (gP) gP[i] = fma(rho, 1.0 / Pv, pb);
        }
    }
}

// ------------------------------------------------ row-owner Jacobian kernel
//
// J written once.  A persistent CTA owns a tile of 32 points (one per lane,
// so every lane of a warp evaluates the same reaction and nothing diverges)
// and keeps the tile's C, EGp and dE in shared memory.  Warp w owns the rows
// k = w, w + W, ...: for row k it walks the reactions that change species k
// (a per-species list of (reaction, net nu), built once per mechanism),
// evaluates each reaction's rate derivatives for its 32 points and adds
// nu * dq into the row, held in a [ns + 1][32] shared-memory buffer of its
// own; then it applies the chain rule through C(T, Y) (file header) and
// stores the row's ns + 1 columns, one coalesced 32-point store each.  A
// reaction is evaluated once per species it changes (about four times), in
// exchange for J never being read back from memory.
constexpr int kJTile = 32;
constexpr int kJMaxWarps = 8;

template <typename JT>
__global__ void __launch_bounds__(32 * kJMaxWarps, 1)
    jac_rows_kernel(DevMech m, const int* __restrict__ lptr, const int* __restrict__ lrx,
                    const double* __restrict__ lnu, const int* __restrict__ lrow, const double* __restrict__ P,
                    const double* __restrict__ Tg,
                    const double* __restrict__ Y, JT* __restrict__ J, int64_t ng, double* __restrict__ kcache) {
    extern __shared__ double smem[];
    const int ns = m.ns, ncol = ns + 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    double* sC = smem;
    double* sE = sC + ns * kJTile;
    double* sD = sE + ns * kJTile;
    double* sRed = sD + ns * kJTile;                               // [kJMaxWarps][32]
    double* row = sRed + kJMaxWarps * kJTile + (size_t)warp * ncol * kJTile + lane;   // this warp's [ncol][32]
    const int64_t ntiles = (ng + kJTile - 1) / kJTile;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int64_t i = tile * kJTile + lane;
        const bool act = i < ng;
        const double T = act ? Tg[i] : 1000.0;
        const double Pv = act ? P[i] : kPatm;
        PointT pt;
        pt.T = T;
        pt.lnT = cgm::cg_log(T);
        pt.invT = 1.0 / T;
        double part = 0.0;
        for (int k = warp; k < ns; k += nw) {
            const double c = (act ? Y[(int64_t)k * ng + i] : 1.0) * __ldg(m.inv_mw + k);
            sC[k * kJTile + lane] = c;
            part += c;
        }
        sRed[warp * kJTile + lane] = part;
        __syncthreads();
        double S = 0.0;
        for (int w = 0; w < nw; ++w) S += sRed[w * kJTile + lane];
        const double fac = Pv / (kR0 * S * T);
        const double pfac = kPatm / (kR0 * T);
        part = 0.0;
        for (int k = warp; k < ns; k += nw) {
            const double c = sC[k * kJTile + lane] * fac;
            sC[k * kJTile + lane] = c;
            part += c;
            const double* th = m.thermo + 16 * k;
            const double* cf = (T < __ldg(th)) ? th + 1 : th + 8;
            double cc[7];
#pragma unroll
            for (int j = 0; j < 7; ++j) cc[j] = __ldg(cf + j);
            sE[k * kJTile + lane] = cgm::cg_exp_clamped(smh_poly(cc, T, pt.lnT, pt.invT)) * pfac;
            const double dp = fma(fma(fma(4.0 * cc[5], T, 3.0 * cc[4]), T, 2.0 * cc[3]), T, cc[2]);
            sD[k * kJTile + lane] = dp + fma(cc[6], pt.invT, cc[1]) * pt.invT - pt.invT;
        }
        __syncthreads();                     // S read by every warp before sRed is reused
        sRed[warp * kJTile + lane] = part;
        __syncthreads();
        double ctot = 0.0;
        for (int w = 0; w < nw; ++w) ctot += sRed[w * kJTile + lane];
        const double lnP = cgm::cg_log(Pv);
        const DState st{sC + lane, sE + lane, sD + lane, nullptr, kJTile, kJTile};
        const double iS = 1.0 / S;
        // phase 1: every reaction once, into this CTA's slice [nr][kDC][32]
        // (a few hundred KB: it stays in L2): a compact reaction's rate
        // derivatives, which the rows then only gather, or another reaction's
        // rate constants, from which each row that needs it evaluates them
        double* kc = kcache + (int64_t)blockIdx.x * m.nr * kDC * kJTile;
        for (int r = warp; r < m.nr; r += nw) {
            const DRxn R = load_rxn(m.rxn + r);
            double* o = kc + (int64_t)r * kDC * kJTile + lane;
            if (R.flags & kFCompact) {
                SideT<3> re, pr;
                RxnGradT<3> g;
                reaction_grad<3>(m, r, R, pt, ctot, Pv, lnP, st, re, pr, g);
                o[0] = g.dqdT;
                o[32] = g.dqdM;
#pragma unroll
                for (int j = 0; j < 6; ++j) o[(2 + j) * kJTile] = g.dqc[j];
                continue;
            }
            int kind = CG_STANDARD;
            while (kind < CG_PLOG && r >= m.seg[kind + 1]) ++kind;
            double kf, kb, dlkf, gM, M, dlp;
            reaction_k(m, r, R, kind, pt, ctot, Pv, lnP, st, kf, kb, dlkf, gM, M, dlp);
            o[0] = kf;
            o[32] = kb;
            o[64] = dlkf;
            o[96] = gM;
            o[128] = M;
        }
        __syncthreads();
        // rows t = warp, warp + nw, ...: species lrow[t], dealt out so that the
        // warps' lists are about equally long and reach the barrier together
        for (int t = warp; t < ns; t += nw) {
            const int k = __ldg(lrow + t);
            for (int c = 0; c < ncol; ++c) row[c * kJTile] = 0.0;
            double ak = 0.0;
            const int e1 = __ldg(lptr + k + 1);
            for (int e = __ldg(lptr + k); e < e1; ++e) {
                const int r = __ldg(lrx + e);
                const double nu = __ldg(lnu + e);
                const DRxn R = load_rxn(m.rxn + r);
                double dqdT, dqdM;
                bool usesM;
                const double* kr = kc + (int64_t)r * kDC * kJTile + lane;
                if (R.flags & kFCompact) {
                    // the derivatives from phase 1; the slots' species as
                    // reaction_grad<3> lays them out
                    SideT<3> re, pr;
                    load_sides3(R, re, pr);
                    const bool rev = (R.flags & CG_F_REVERSIBLE) != 0;
                    int dsp[6];
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        dsp[j] = j < re.n ? re.sp[j] : 0;
                        dsp[3 + j] = (rev && j < pr.n) ? pr.sp[j] : 0;
                    }
                    double dq[6];
#pragma unroll
                    for (int j = 0; j < 6; ++j) dq[j] = kr[(2 + j) * kJTile];
#pragma unroll
                    for (int j = 0; j < 6; ++j) row[(1 + dsp[j]) * kJTile] = fma(nu, dq[j], row[(1 + dsp[j]) * kJTile]);
                    dqdT = kr[0];
                    dqdM = kr[32];
                    int kind = CG_STANDARD;
                    while (kind < CG_PLOG && r >= m.seg[kind + 1]) ++kind;
                    usesM = kind >= CG_THIRD_BODY && kind <= CG_SRI;
                } else {
                    Side re, pr;
                    RxnGrad g;
                    reaction_grad<16, true>(m, r, R, pt, ctot, Pv, lnP, st, re, pr, g, kr);
                    for (int j = 0; j < g.nd; ++j)
                        row[(1 + g.dsp[j]) * kJTile] = fma(nu, g.dqc[j], row[(1 + g.dsp[j]) * kJTile]);
                    dqdT = g.dqdT;
                    dqdM = g.dqdM;
                    usesM = g.usesM;
                }
                row[0] = fma(nu, dqdT, row[0]);
                if (usesM) {
                    // dM/dC_j = 1 + (eff_j - 1): the 1 goes to every column (ak), the rest is sparse
                    ak = fma(nu, dqdM, ak);
                    for (int f = __ldg(m.eff_ptr + r); f < __ldg(m.eff_ptr + r + 1); ++f)
                        row[(1 + __ldg(m.eff_sp + f)) * kJTile] =
                            fma(nu * __ldg(m.eff_val + f), dqdM, row[(1 + __ldg(m.eff_sp + f)) * kJTile]);
                }
            }
            // chain rule through C(T, Y): rk = sum_j dwdot_k/dC_j C_j
            double rk = ak * ctot;
            for (int j = 0; j < ns; ++j) rk = fma(row[(1 + j) * kJTile], sC[j * kJTile + lane], rk);
            if (act) {
                // streaming stores: J is never read back, so its lines go
                // first when L2 needs room and the tile's rate-constant cache
                // stays resident instead of being written back to DRAM
                JT* Jr = J + (int64_t)k * ncol * ng + i;
                __stcs(Jr, (JT)(row[0] - rk * pt.invT));
                for (int j = 0; j < ns; ++j)
                    __stcs(Jr + (int64_t)(1 + j) * ng,
                           (JT)(fma(ctot, row[(1 + j) * kJTile] + ak, -rk) * __ldg(m.inv_mw + j) * iS));
            }
        }
        __syncthreads();                     // the tile's state stays until every row is done
    }
}

}  // namespace

// Row-owner Jacobian plan: per-species (reaction, net nu) lists.
struct JacPlan {
    int warps = 0;
    size_t smem = 0;
    int grid = 0;
    const int* lptr = nullptr;
    const int* lrx = nullptr;
    const double* lnu = nullptr;
    const int* lrow = nullptr;  // species of row slot t (warp t % warps)
    void* dbuf = nullptr;
};

cudaError_t jac_prepare(const DevMech& m, const cg_mech_view& v, int device, JacPlan** out) {
    *out = nullptr;
    const int ns = m.ns, nr = m.nr;
    DeviceLimits dev;
    cudaError_t e = device_limits(device, &dev);
    if (e != cudaSuccess) return e;
    const size_t fixed = (size_t)3 * ns * kJTile * 8 + (size_t)kJMaxWarps * kJTile * 8;
    const size_t per_warp = (size_t)(ns + 1) * kJTile * 8;
    if (fixed + 2 * per_warp > dev.smem_block) return cudaErrorNotSupported;
    const int warps = (int)std::min<size_t>(kJMaxWarps, (dev.smem_block - fixed) / per_warp);
    const int32_t* rp = (const int32_t*)v.a[CG_RPTR];
    const int32_t* pp = (const int32_t*)v.a[CG_PPTR];
    const int32_t* rsp = (const int32_t*)v.a[CG_RSP];
    const int32_t* psp = (const int32_t*)v.a[CG_PSP];
    const double* rnu = (const double*)v.a[CG_RNU];
    const double* pnu = (const double*)v.a[CG_PNU];
    std::vector<std::vector<std::pair<int, double>>> lists(ns);
    std::vector<double> net(ns, 0.0);
    for (int r = 0; r < nr; ++r) {
        for (int j = rp[r]; j < rp[r + 1]; ++j) net[rsp[j]] -= rnu[j];
        for (int j = pp[r]; j < pp[r + 1]; ++j) net[psp[j]] += pnu[j];
        for (int j = rp[r]; j < rp[r + 1]; ++j)
            if (net[rsp[j]] != 0.0) {
                lists[rsp[j]].push_back({r, net[rsp[j]]});
                net[rsp[j]] = 0.0;
            }
        for (int j = pp[r]; j < pp[r + 1]; ++j)
            if (net[psp[j]] != 0.0) {
                lists[psp[j]].push_back({r, net[psp[j]]});
                net[psp[j]] = 0.0;
            }
    }
    std::vector<int> lptr(ns + 1, 0), lrx;
    std::vector<double> lnu;
    for (int k = 0; k < ns; ++k) {
        for (const auto& x : lists[k]) {
            lrx.push_back(x.first);
            lnu.push_back(x.second);
        }
        lptr[k + 1] = (int)lrx.size();
    }
    // row slots: warp w takes slots w, w + warps, ...; species dealt out
    // longest list first, each to the warp with the least work so far among
    // those with a free slot (a row costs its list plus the chain rule)
    std::vector<int> order(ns);
    for (int k = 0; k < ns; ++k) order[k] = k;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return lists[a].size() > lists[b].size(); });
    std::vector<std::vector<int>> warp_rows(warps);
    std::vector<long> load(warps, 0);
    for (int k : order) {
        int best = -1;
        for (int w = 0; w < warps; ++w) {
            const int cap = (ns - w + warps - 1) / warps;
            if ((int)warp_rows[w].size() < cap && (best < 0 || load[w] < load[best])) best = w;
        }
        warp_rows[best].push_back(k);
        load[best] += (long)lists[k].size() + ns;
    }
    std::vector<int> lrow(ns);
    for (int w = 0; w < warps; ++w)
        for (size_t j = 0; j < warp_rows[w].size(); ++j) lrow[j * warps + w] = warp_rows[w][j];
    const size_t b_ptr = ((ns + 1) * sizeof(int) + 255) / 256 * 256;
    const size_t b_rx = (std::max<size_t>(lrx.size(), 1) * sizeof(int) + 255) / 256 * 256;
    const size_t b_nu = (std::max<size_t>(lnu.size(), 1) * sizeof(double) + 255) / 256 * 256;
    const size_t b_row = (size_t)ns * sizeof(int);
    JacPlan* p = new JacPlan();
    p->warps = warps;
    p->smem = fixed + (size_t)warps * per_warp;
    p->grid = dev.sms;
    e = cudaMalloc(&p->dbuf, b_ptr + b_rx + b_nu + b_row);
    char* d = (char*)p->dbuf;
    if (e == cudaSuccess) e = cudaMemcpy(d, lptr.data(), lptr.size() * sizeof(int), cudaMemcpyHostToDevice);
    if (e == cudaSuccess && !lrx.empty()) e = cudaMemcpy(d + b_ptr, lrx.data(), lrx.size() * sizeof(int), cudaMemcpyHostToDevice);
    if (e == cudaSuccess && !lnu.empty())
        e = cudaMemcpy(d + b_ptr + b_rx, lnu.data(), lnu.size() * sizeof(double), cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaMemcpy(d + b_ptr + b_rx + b_nu, lrow.data(), b_row, cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(jac_rows_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p->smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(jac_rows_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p->smem);
    if (e != cudaSuccess) {
        if (p->dbuf) cudaFree(p->dbuf);
        delete p;
        return e;
    }
    p->lptr = (const int*)d;
    p->lrx = (const int*)(d + b_ptr);
    p->lnu = (const double*)(d + b_ptr + b_rx);
    p->lrow = (const int*)(d + b_ptr + b_rx + b_nu);
    *out = p;
    return cudaSuccess;
}

void jac_release(JacPlan* p) {
    if (!p) return;
    if (p->dbuf) cudaFree(p->dbuf);
    delete p;
}

size_t jac_rows_workspace_bytes(const JacPlan* p, const DevMech& m, int64_t ng) {
    const int64_t tiles = (ng + kJTile - 1) / kJTile;
    const int64_t grid = std::min<int64_t>(tiles, p->grid);
    return (size_t)grid * m.nr * kDC * kJTile * sizeof(double);
}

cudaError_t launch_jacobian_rows(const JacPlan* p, const DevMech& m, int precision, const double* P, const double* T,
                                 const double* Y, void* J, int64_t ng, double* scratch, size_t scratch_bytes,
                                 cudaStream_t s) {
    if (ng <= 0) return cudaSuccess;
    const int64_t tiles = (ng + kJTile - 1) / kJTile;
    const unsigned grid = (unsigned)std::min<int64_t>(tiles, p->grid);
    if (!scratch || scratch_bytes < jac_rows_workspace_bytes(p, m, ng)) return cudaErrorInvalidValue;
    const unsigned threads = 32u * (unsigned)p->warps;
    // the kernel's shared-memory limit is this plan's, set under one lock with
    // the launch (a plan made later for a smaller mechanism sets it lower)
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    cudaError_t e = precision == 0 ? cudaFuncSetAttribute(jac_rows_kernel<double>,
                                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p->smem)
                                   : cudaFuncSetAttribute(jac_rows_kernel<float>,
                                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p->smem);
    if (e != cudaSuccess) return e;
    if (precision == 0)
        jac_rows_kernel<double><<<grid, threads, p->smem, s>>>(m, p->lptr, p->lrx, p->lnu, p->lrow, P, T, Y,
                                                               (double*)J, ng, scratch);
    else
        jac_rows_kernel<float><<<grid, threads, p->smem, s>>>(m, p->lptr, p->lrx, p->lnu, p->lrow, P, T, Y,
                                                              (float*)J, ng, scratch);
    return cudaGetLastError();
}

size_t deriv_workspace_bytes(int ns, int64_t ng) { return (size_t)4 * ns * ng * sizeof(double); }

cudaError_t launch_jacobian(const DevMech& m, int precision, const double* P, const double* T, const double* Y,
                            void* J, int64_t ng, double* scratch, int sm_count, cudaStream_t s) {
    if (ng <= 0) return cudaSuccess;
    int64_t blocks = (ng + 127) / 128;
    if (blocks > (int64_t)sm_count * 16) blocks = (int64_t)sm_count * 16;
    if (precision == 0)
        deriv_kernel<true, double><<<(unsigned)blocks, 128, 0, s>>>(m, P, T, Y, nullptr, (double*)J, nullptr, nullptr,
                                                                   nullptr, scratch, ng);
    else
        deriv_kernel<true, float><<<(unsigned)blocks, 128, 0, s>>>(m, P, T, Y, nullptr, (float*)J, nullptr, nullptr,
                                                                  nullptr, scratch, ng);
    return cudaGetLastError();
}

cudaError_t launch_vjp(const DevMech& m, const double* P, const double* T, const double* Y, const double* G, double* gT,
                       double* gY, double* gP, int64_t ng, double* scratch, int sm_count, cudaStream_t s) {
    if (ng <= 0) return cudaSuccess;
    int64_t blocks = (ng + 127) / 128;
    if (blocks > (int64_t)sm_count * 16) blocks = (int64_t)sm_count * 16;
    deriv_kernel<false, double><<<(unsigned)blocks, 128, 0, s>>>(m, P, T, Y, G, nullptr, gT, gY, gP, scratch, ng);
    return cudaGetLastError();
}

}  // namespace cg
