"""The calls that a user of this framework makes, as timed cases.

Every case goes through the package's public entry points: getrates on CUDA
tensors (both layouts, both arithmetic modes), the analytic Jacobian, the
differentiable getrates, getrates on host arrays, and the surrogate with its
per-point fallback.  The mechanisms are the ones of tests/golden: H2 (9
species / 23 reactions), GRI30 (53 / 322), a synthetic 53 / 325 set, a
synthetic 348 / 2163 set and JetSurf 2.0 (348 / 2158).  States have the
workload's distributions: T ~ U(300, 2500) K, P log-uniform over 1..40 atm,
Y ~ Dirichlet(0.5).
"""
import functools
import json
import math
import os

import numpy as np
import torch

from chemgen_b200 import GpuMechanism, getrates
from chemgen_b200.mechanism import Mechanism
from chemgen_b200.surrogate import Surrogate, SurrogateGetrates

ATM = 1013250.0             # dyne/cm^2
R0 = 8.314510e07            # erg/(mol K)
RC = 1.9872155832           # cal/(mol K)
GOLDEN = os.path.join("tests", "golden")

H2, GRI30, C53, C348, JETSURF = "h2_burke", "gri30", "synthetic_53_325", "synthetic_348_2163", "jetsurf2"
SMALL = (H2, GRI30, C53)    # mechanisms with generated kernels
LARGE = (C348, JETSURF)     # mechanisms on the table-driven kernels


def listed():
    return [
        # one small partition of a reacting-flow solver with hydrogen
        # chemistry: the smallest call, one launch
        dict(name="h2_fp64_1000", kind="rates", mech=H2, mode="fp64", ng=1000, layout="species_major"),
        # a 16^3 block of cells with a 53-species mechanism, FP64: a solver's
        # per-block call
        dict(name="c53_fp64_4096", kind="rates", mech=C53, mode="fp64", ng=4096, layout="species_major"),
        # an ordinary subdomain of ragged size, real GRI30, mixed precision
        dict(name="gri30_mixed_100003", kind="rates", mech=GRI30, mode="mixed", ng=100003, layout="species_major"),
        # a whole GPU's grid (bench.py's workload), both arithmetic modes
        dict(name="c53_fp64_1m", kind="rates", mech=C53, mode="fp64", ng=1 << 20, layout="species_major"),
        dict(name="c53_mixed_1m", kind="rates", mech=C53, mode="mixed", ng=1 << 20, layout="species_major"),
        # large-fuel chemistry: FP64 over a large grid, and mixed precision on
        # a small ragged subdomain of the real mechanism
        dict(name="c348_fp64_128k", kind="rates", mech=C348, mode="fp64", ng=1 << 17, layout="species_major"),
        dict(name="jetsurf_mixed_20011", kind="rates", mech=JETSURF, mode="mixed", ng=20011, layout="species_major"),
        # the Jacobian of an implicit integrator: a large batch in FP64, and a
        # small ragged one stored in FP32 for a preconditioner
        dict(name="c53_jacobian_fp64_64k", kind="jacobian", mech=C53, precision="fp64", ng=1 << 16),
        dict(name="gri30_jacobian_fp32_5003", kind="jacobian", mech=GRI30, precision="fp32", ng=5003),
        # training through the rates in PyTorch: forward and backward with
        # batch-first tensors
        dict(name="c53_autograd_32k", kind="autograd", mech=C53, mode="fp64", ng=1 << 15, layout="point_major"),
        # a host code's call: pinned host arrays in and out
        dict(name="c53_host_mixed_200k", kind="host", mech=C53, mode="mixed", ng=200000),
        # the learned surrogate with its per-point fallback, about 0.2 % of the
        # points going to the exact kernel
        dict(name="c53_surrogate_1m", kind="surrogate", mech=C53, ng=1 << 20),
    ]


def _log_int(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, n))


def draw(rng):
    kind = rng.choice(["rates", "rates", "rates", "rates_large", "rates_large", "jacobian", "jacobian", "autograd",
                       "host", "surrogate"])
    if kind == "rates":
        return dict(kind="rates", mech=rng.choice(SMALL), mode=rng.choice(["fp64", "mixed"]),
                    ng=_log_int(rng, 256, 1 << 20),
                    layout=rng.choice(["species_major", "species_major", "species_major", "point_major"]))
    if kind == "rates_large":
        return dict(kind="rates", mech=rng.choice(LARGE), mode=rng.choice(["fp64", "mixed"]),
                    ng=_log_int(rng, 256, 1 << 16), layout="species_major")
    if kind == "jacobian":
        return dict(kind="jacobian", mech=rng.choice(SMALL), precision=rng.choice(["fp64", "fp32"]),
                    ng=_log_int(rng, 256, 1 << 16))
    if kind == "autograd":
        return dict(kind="autograd", mech=rng.choice(SMALL), mode=rng.choice(["fp64", "mixed"]),
                    ng=_log_int(rng, 256, 1 << 16), layout=rng.choice(["species_major", "point_major"]))
    if kind == "host":
        return dict(kind="host", mech=rng.choice(SMALL), mode=rng.choice(["fp64", "mixed"]),
                    ng=_log_int(rng, 1024, 200000))
    return dict(kind="surrogate", mech=C53, ng=_log_int(rng, 4096, 1 << 20))


# ------------------------------------------------------------------ inputs
def _device():
    return torch.device("cuda", torch.cuda.current_device())


@functools.lru_cache(maxsize=None)
def _data(mech):
    """The mechanism's description as plain data."""
    return json.loads(str(np.load(os.path.join(GOLDEN, mech + ".npz"))["mech"]))


@functools.lru_cache(maxsize=None)
def _handle(mech):
    """One handle per mechanism, kept by the program as a solver keeps it."""
    return GpuMechanism(Mechanism.from_json(json.dumps(_data(mech))), device=_device().index,
                        generated=mech in SMALL)


def _states(mech, ng, seed, layout="species_major"):
    g = torch.Generator(device=_device()).manual_seed(seed)
    f = dict(generator=g, device=_device(), dtype=torch.float64)
    ns = len(_data(mech)["species"])
    T = 300.0 + 2200.0 * torch.rand(ng, **f)
    P = ATM * torch.exp(torch.rand(ng, **f) * math.log(40.0))
    Y = torch.randn((ns, ng), **f).square_()        # gamma(1/2): Dirichlet(0.5) once normalised
    Y /= Y.sum(dim=0, keepdim=True)
    return P, T, (Y.t().contiguous() if layout == "point_major" else Y)


@functools.lru_cache(maxsize=None)
def _gate(mech):
    """The surrogate with its gate, with seeded weights (a trained network's
    shapes and the same work per point); the tolerance is the one that about
    0.2 % of the points miss."""
    gm = _handle(mech)
    sur = Surrogate(gm, seed=7, device=_device().index)
    P, T, Y = _states(mech, 1 << 16, 99)
    W = gm.getrates(P, T, Y)
    ln = torch.log(W.norm(dim=0).clamp_min(1e-300))
    x = torch.log(Y.clamp_min(1e-30) * sur.inv_mw[:, None])
    x -= torch.logsumexp(x, dim=0, keepdim=True)
    sur.norm[6], sur.norm[7] = round(float(x.mean()), 6), round(1.0 / float(x.std()), 6)
    sur.lnorm[0], sur.lnorm[1] = round(float(ln.mean()), 3), round(float(ln.std()), 3)
    _, est = sur.predict(P, T, Y)
    return SurrogateGetrates(sur, tol=10.0 ** float(torch.quantile(est.double(), 0.998)))


def prepare(case, seed):
    kind, mech, ng = case["kind"], case["mech"], case["ng"]
    st = dict(case, gm=_handle(mech))
    st["P"], st["T"], st["Y"] = _states(mech, ng, seed, case.get("layout", "species_major"))
    if kind == "autograd":
        g = torch.Generator(device=_device()).manual_seed(seed + 1)
        st["G"] = torch.randn(st["Y"].shape, generator=g, device=_device(), dtype=torch.float64)
        for k in ("P", "T", "Y"):
            st[k].requires_grad_(True)
    elif kind == "host":
        for k in ("P", "T", "Y"):
            st[k] = st[k].cpu().pin_memory()
        st["out"] = torch.empty_like(st["Y"], pin_memory=True)
    elif kind == "surrogate":
        st["gate"] = _gate(mech)
    return st


# --------------------------------------------------------------------- run
def run(st):
    kind, gm, P, T, Y = st["kind"], st["gm"], st["P"], st["T"], st["Y"]
    if kind == "rates":
        return gm.getrates(P, T, Y, mode=st["mode"], layout=st["layout"])
    if kind == "jacobian":
        return gm.jacobian(P, T, Y, precision=st["precision"])
    if kind == "autograd":
        w = getrates(gm, P, T, Y, mode=st["mode"], layout=st["layout"])
        gP, gT, gY = torch.autograd.grad(w, (P, T, Y), st["G"])
        return {"wdot": w.detach(), "gP": gP, "gT": gT, "gY": gY}
    if kind == "host":
        return gm.getrates_host(P, T, Y, out=st["out"], mode=st["mode"])
    return st["gate"](P, T, Y)


# -------------------------------------------------------------------- work
def _rate_flops(mech):
    """Additions and multiplications of one point's rates, an exp, a log or a
    reciprocal counted as 20."""
    d = _data(mech)
    f = 36 * len(d["species"])
    for r in d["reactions"]:
        nre, npr = sum(r["reactants"].values()), sum(r["products"].values())
        f += 24 + nre + 1 + 2 * (len(r["reactants"]) + len(r["products"]))
        if r["reversible"]:
            f += nre + 2 * npr + 22
        if r["kind"] in ("third_body", "troe"):
            f += 2 * len(r["efficiencies"]) + 1
        if r["kind"] == "troe":
            f += 24 + 140
    return f


def work(case):
    ns, ng = len(_data(case["mech"])["species"]), case["ng"]
    rates = _rate_flops(case["mech"]) * ng
    states = (2 + ns) * 8 * ng
    if case["kind"] == "jacobian":
        size = 8 if case["precision"] == "fp64" else 4
        return {"bytes": states + ns * (ns + 1) * size * ng, "flops": 2 * rates + 4 * ns * (ns + 1) * ng}
    if case["kind"] == "autograd":
        # P, T, Y and the cotangent read; wdot and the three gradients written
        return {"bytes": 2 * states + 2 * ns * 8 * ng, "flops": 3 * rates}
    if case["kind"] == "surrogate":
        return {"bytes": states + ns * 8 * ng, "flops": 2 * (64 * 256 + 2 * 256 * 256 + 256 * 64) * ng}
    return {"bytes": states + ns * 8 * ng, "flops": rates}


# ------------------------------------------------------------------- exact
class _Tables:
    """The rate law's coefficients as FP64 tensors, a row per species or reaction."""

    def __init__(self, mech, dev):
        d = _data(mech)
        t = lambda x: torch.tensor(x, dtype=torch.float64, device=dev)     # noqa: E731
        sp, rx = d["species"], d["reactions"]
        idx = {s["name"]: k for k, s in enumerate(sp)}
        self.ns, self.nr = len(sp), len(rx)
        self.mw = t([s["mw"] for s in sp])
        self.tmid = t([s["t_ranges"][1] for s in sp])
        self.nasa = t([[s["nasa_low"], s["nasa_high"]] for s in sp])
        most = int(max(max(sum(r["reactants"].values()), sum(r["products"].values())) for r in rx))

        def molecules(side):
            m = [idx[s] for s, nu in side.items() for _ in range(int(nu))]
            return m + [self.ns] * (most - len(m))                         # row ns: a factor 1
        self.re = torch.tensor([molecules(r["reactants"]) for r in rx], device=dev)
        self.pr = torch.tensor([molecules(r["products"]) for r in rx], device=dev)
        self.rev = t([1.0 if r["reversible"] else 0.0 for r in rx])[:, None]
        self.arh = t([r["arh"] for r in rx])
        net = np.zeros((self.ns, self.nr))
        for j, r in enumerate(rx):
            for s, nu in r["reactants"].items():
                net[idx[s], j] -= nu
            for s, nu in r["products"].items():
                net[idx[s], j] += nu
        self.net = t(net)
        m = [j for j, r in enumerate(rx) if r["kind"] != "standard"]
        eff = np.zeros((len(m), self.ns))
        for i, j in enumerate(m):
            for s, e in rx[j]["efficiencies"].items():
                eff[i, idx[s]] = e
        self.eff = t(eff)
        third = [i for i, j in enumerate(m) if rx[j]["kind"] == "third_body"]
        fall = [i for i, j in enumerate(m) if rx[j]["kind"] == "troe"]
        self.m_third, self.m_fall = (torch.tensor(v, dtype=torch.long, device=dev) for v in (third, fall))
        self.r_third, self.r_fall = (torch.tensor([m[i] for i in v], dtype=torch.long, device=dev)
                                     for v in (third, fall))
        tr = [rx[m[i]] for i in fall]
        self.low = t([r["low"] for r in tr]).reshape(-1, 3)
        self.troe = t([list(r["troe"][:3]) + [r["troe"][3] if len(r["troe"]) == 4 else 0.0] for r in tr]).reshape(-1, 4)
        self.has_t2 = (self.troe[:, 3:4] != 0.0).to(torch.float64)

    @staticmethod
    def ln_k(a, T):
        return torch.log(a[:, 0:1]) + a[:, 1:2] * torch.log(T) - a[:, 2:3] / (RC * T)

    def rates(self, P, T, Y):
        """wdot [ns, n] of P [n], T [n], Y [ns, n]."""
        C = Y / self.mw[:, None]
        C = C * P / (R0 * C.sum(dim=0) * T)
        ctot = C.sum(dim=0)
        ones = torch.ones_like(T)[None]
        a = torch.where((T < self.tmid[:, None])[..., None], self.nasa[:, None, 0], self.nasa[:, None, 1])
        g = (a[..., 6] - a[..., 0] + a[..., 0] * torch.log(T) + a[..., 1] / 2 * T + a[..., 2] / 6 * T ** 2
             + a[..., 3] / 12 * T ** 3 + a[..., 4] / 20 * T ** 4 - a[..., 5] / T) + torch.log(ATM / (R0 * T))
        Cx, gx = torch.cat([C, ones]), torch.cat([g, 0.0 * ones])
        lnk = self.ln_k(self.arh, T)
        M = ctot + self.eff @ C
        if self.r_fall.numel():
            lp = self.ln_k(self.low, T) + torch.log(M[self.m_fall]) - lnk[self.r_fall]
            p = self.troe
            fc = (1.0 - p[:, 0:1]) * torch.exp(-T / p[:, 1:2]) + p[:, 0:1] * torch.exp(-T / p[:, 2:3]) \
                + self.has_t2 * torch.exp(-p[:, 3:4] / T)
            lf = torch.log10(fc)
            u = lp / math.log(10.0) - 0.4 - 0.67 * lf
            f1 = u / (0.75 - 1.27 * lf - 0.14 * u)
            lnf = math.log(10.0) * lf / (1.0 + f1 ** 2)
            blend = lnf - torch.nn.functional.softplus(-lp, threshold=1e9)
            lnk = lnk.index_add(0, self.r_fall, blend)
        q = torch.exp(lnk) * Cx[self.re].prod(dim=1)
        lnkb = lnk + gx[self.re].sum(dim=1) - gx[self.pr].sum(dim=1)
        q = q - self.rev * torch.exp(torch.where(self.rev > 0, lnkb, 0.0)) * Cx[self.pr].prod(dim=1)
        if self.r_third.numel():
            f = torch.ones_like(q).index_copy(0, self.r_third, M[self.m_third])
            q = q * f
        return self.net @ q


def exact(case, seed):
    kind, mech, ng = case["kind"], case["mech"], case["ng"]
    if kind == "surrogate":
        return None                     # a network's outputs: there is no exact value of them
    P, T, Y = _states(mech, ng, seed)
    tab = _Tables(mech, P.device)
    step = max(1, (1 << 22) // tab.nr)
    point_major = case.get("layout") == "point_major"
    if kind in ("rates", "host"):
        W = torch.empty_like(Y)
        for i in range(0, ng, 4 * step):
            s = slice(i, i + 4 * step)
            W[:, s] = tab.rates(P[s], T[s], Y[:, s])
        return W.t().contiguous() if point_major else W.cpu() if kind == "host" else W
    if kind == "jacobian":
        J = torch.empty((tab.ns, tab.ns + 1, ng), dtype=torch.float64, device=P.device)
        for i in range(0, ng, step):
            s = slice(i, i + step)
            t, y = T[s].clone().requires_grad_(True), Y[:, s].clone().requires_grad_(True)
            w = tab.rates(P[s], t, y)
            for k in range(tab.ns):
                J[k, 0, s], J[k, 1:, s] = torch.autograd.grad(w[k].sum(), (t, y), retain_graph=True)
        return J
    g = torch.Generator(device=P.device).manual_seed(seed + 1)
    G = torch.randn((ng, tab.ns) if point_major else (tab.ns, ng), generator=g, device=P.device, dtype=torch.float64)
    G = G.t().contiguous() if point_major else G
    out = {"wdot": torch.empty_like(Y), "gP": torch.empty_like(P), "gT": torch.empty_like(T), "gY": torch.empty_like(Y)}
    for i in range(0, ng, step):
        s = slice(i, i + step)
        p, t, y = (x.clone().requires_grad_(True) for x in (P[s], T[s], Y[:, s]))
        w = tab.rates(p, t, y)
        out["gP"][s], out["gT"][s], out["gY"][:, s] = torch.autograd.grad(w, (p, t, y), G[:, s])
        out["wdot"][:, s] = w.detach()
    if point_major:
        for k in ("wdot", "gY"):
            out[k] = out[k].t().contiguous()
    return out
