"""The eight-point-tile kernels (four reactions to a warp) at the sizes where
they can go wrong: part tiles, one point, several chunks of reactions, owners
with long lists, reactions without a pre-decoded form."""
import numpy as np
import pytest

from chemgen_b200 import pack, synthetic
from chemgen_b200.runtime import GpuMechanism
from oracle import oracle

pytestmark = pytest.mark.gpu
TOL_FP64 = 1e-10          # the FP64 kernels' bar (rounding of ~300-term sums is 1e-13)


def _cuda(*arrays):
    import torch
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


def _check(mech, ng, seed=0):
    blob = pack.pack(mech).to_blob()
    P, T, Y = synthetic.states(mech.ns, ng, seed=seed)
    w = GpuMechanism(blob).getrates(*_cuda(P, T, Y)).cpu().numpy()
    r = oracle.rates(blob, P, T, Y, mech.nr)
    e = oracle.errors(w, r["wdot"], r["S"])
    assert e["norm_max"] <= TOL_FP64 and e["gross_max"] <= TOL_FP64, e


@pytest.mark.parametrize("ng", [1, 7, 8, 9, 8 * 148 * 3 + 5])
def test_part_tiles(ng):
    _check(synthetic.gri_shape(), ng, seed=ng)


def test_several_chunks_of_reactions():
    # the rates of 4200 reactions (268 KB for eight points) take two chunks
    _check(synthetic.synthetic_mechanism(120, 4200, 40, 60, seed=9), 41)


@pytest.mark.parametrize("ns", [434, 435, 437, 438])
def test_the_largest_mechanisms_without_a_workspace(ns):
    # up to 437 species the FP64 call needs no workspace and the counted call works
    import torch
    from chemgen_b200.runtime import lib
    mech = synthetic.synthetic_mechanism(ns, 500, 20, 20, seed=1)
    blob = pack.pack(mech).to_blob()
    gm = GpuMechanism(blob)
    ng = 21
    P, T, Y = synthetic.states(mech.ns, ng, seed=2)
    Pt, Tt, Yt = _cuda(P, T, Y)
    W, count = torch.zeros_like(Yt), torch.tensor([ng], device="cuda")
    st = lib().chemgen_getrates_counted(gm._h, Pt.data_ptr(), Tt.data_ptr(), ng, Yt.data_ptr(), W.data_ptr(),
                                        count.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert (gm.workspace_bytes(ng) == 0, st) == ((True, 0) if ns <= 437 else (False, 6))
    r = oracle.rates(blob, P, T, Y, mech.nr)
    for w in [gm.getrates(Pt, Tt, Yt)] + ([W] if st == 0 else []):
        e = oracle.errors(w.cpu().numpy(), r["wdot"], r["S"])
        assert e["norm_max"] <= TOL_FP64, e


def test_every_kind_and_general_stoichiometry():
    # PLOG, SRI, Lindemann; a negative and a zero pre-exponential factor,
    # fractional coefficients and four molecules on a side take the generic path
    mech = synthetic.synthetic_mechanism(60, 200, 12, 12, seed=6, n_lindemann=6, n_sri=6, n_plog=6)
    rx = [r for r in mech.reactions if r.kind == "standard"]
    rx[0].arh = (-rx[0].arh[0],) + rx[0].arh[1:]
    rx[1].arh = (0.0,) + rx[1].arh[1:]
    s = mech.species_names
    rx[2].reactants, rx[2].products = {s[0]: 1.0, s[1]: 1.0}, {s[2]: 0.5, s[3]: 1.5}
    rx[2].reversible = False
    rx[3].reactants, rx[3].products = {s[4]: 1.0}, {s[5]: 2.0, s[6]: 1.0, s[7]: 1.0}
    rx[3].reversible = False
    _check(mech, 83)


def _cold(seed=7):
    # irreversible reactions of small activation energy, which stay finite near
    # 0 K, and states down to 2 mK
    import dataclasses
    mech = synthetic.synthetic_mechanism(6, 12, 0, 0, seed=seed, frac_reversible=0.0)
    theta = [0.0, 0.01, 0.02, 0.1, 0.5, 2.0, -0.05, 8.0, 0.0, 30.0, 0.03, 1.0]
    mech.reactions = [dataclasses.replace(r, arh=(1e3, 0.0 if i % 2 else 0.7, theta[i] * 1.9872155832))
                      for i, r in enumerate(mech.reactions)]
    P, T, Y = synthetic.states(6, 13, seed=seed)
    T[:] = [0.002, 0.003, 0.01, 0.02, 0.05, 0.1, 0.19, 0.2, 0.21, 0.5, 3.0, 40.0, 300.0]
    return mech, P, T, Y


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_temperatures_near_zero(mode):
    # 1/T up to 500 per K reaches the rates unchanged: FP64 tiles (through the
    # counted call) and 32-point mixed tiles
    import torch
    from chemgen_b200.runtime import lib
    mech, P, T, Y = _cold()
    blob = pack.pack(mech).to_blob()
    gm = GpuMechanism(blob)
    Pt, Tt, Yt = _cuda(P, T, Y)
    if mode == "fp64":
        W, count = torch.zeros_like(Yt), torch.tensor([len(T)], device="cuda")
        assert lib().chemgen_getrates_counted(gm._h, Pt.data_ptr(), Tt.data_ptr(), len(T), Yt.data_ptr(), W.data_ptr(),
                                              count.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    else:
        W = gm.getrates(Pt, Tt, Yt, mode=mode)
    r = oracle.rates(blob, P, T, Y, mech.nr)
    assert np.isfinite(r["wdot"]).all()
    assert oracle.errors(W.cpu().numpy(), r["wdot"], r["S"])["norm_max"] <= (TOL_FP64 if mode == "fp64" else 1e-6)


def test_derivatives_at_temperatures_near_zero():
    # dq/dT = q (b + theta / T - n) / T for n reactant molecules, at constant Y and P
    mech, P, T, Y = _cold()
    gm = GpuMechanism(mech)
    Pt, Tt, Yt = _cuda(P, T, Y)
    J = gm.jacobian(Pt, Tt, Yt).cpu().numpy()
    C = Y / np.array([s.mw for s in mech.species])[:, None]
    C *= P / (8.314510e+07 * T * C.sum(0))
    ref = np.zeros_like(Y)
    for r in mech.reactions:
        A, b, Ea = r.arh
        th = Ea / 1.9872155832
        q = A * T ** b * np.exp(-th / T)
        for s, nu in r.reactants.items():
            q = q * C[mech.species_names.index(s)] ** nu
        d = q * (b + th / T - sum(r.reactants.values())) / T
        for side, sign in ((r.reactants, -1.0), (r.products, 1.0)):
            for s, nu in side.items():
                ref[mech.species_names.index(s)] += sign * nu * d
    assert (np.abs(J[:, 0] - ref).max(0) / np.abs(ref).max(0)).max() <= 1e-9


def _derivatives(mech, ng, seed=0, states=None):
    """(Jacobian, adjoint) of the kernels and of autograd through the FP64 law."""
    import torch
    from oracle import torch_ref
    P, T, Y = _cuda(*(states or synthetic.states(mech.ns, ng, seed=seed)))
    gm = GpuMechanism(mech)
    G = torch.randn(mech.ns, ng, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))
    p, t, y = (x.clone().requires_grad_(True) for x in (P, T, Y))
    w = torch_ref.getrates(mech, p, t, y)
    gP, gT, gY = torch.autograd.grad(w, (p, t, y), G, retain_graph=True)
    J = torch.empty(mech.ns, mech.ns + 1, ng, dtype=torch.float64, device="cuda")
    for k in range(mech.ns):
        J[k, 0], J[k, 1:] = torch.autograd.grad(w[k].sum(), (t, y), retain_graph=True)
    return (gm.jacobian(P, T, Y), gm.jacobian(P, T, Y, precision="fp32").double(), gm.vjp(P, T, Y, G)), (J, (gT, gY, gP))


def _rel(x, ref):
    # per point, relative to the point's largest value (columns of J by column T and the rest)
    d = (x - ref).abs().reshape(-1, ref.shape[-1]).amax(0)
    return float((d / ref.abs().reshape(-1, ref.shape[-1]).amax(0).clamp_min(1e-300)).max())


@pytest.mark.parametrize("name,ng", [("all_kinds", 1), ("all_kinds", 19), ("one_cta", 17), ("chunks", 9)])
def test_derivatives_of_every_kind(name, ng):
    # 1e-9: the bar of the derivative tests; FP32 storage 1e-6 (half an ulp is 6e-8)
    mech = {"all_kinds": synthetic.all_kinds,
            # rows for one CTA per SM: 24 warps, 32 for FP32 storage
            "one_cta": lambda: synthetic.synthetic_mechanism(30, 330, 30, 10, seed=3, n_lindemann=10, n_sri=10,
                                                             n_plog=10),
            "chunks": lambda: synthetic.synthetic_mechanism(30, 900, 30, 30, seed=3)}[name]()
    (J64, J32, v), (J, r) = _derivatives(mech, ng, seed=ng)
    for sl in (slice(0, 1), slice(1, None)):
        assert _rel(J64[:, sl], J[:, sl]) <= 1e-9
        assert _rel(J32[:, sl], J[:, sl]) <= 1e-6
    gT, gY, gP = v
    assert _rel(gY, r[1]) <= 1e-9
    assert _rel(gT[None], r[0][None]) <= 1e-7 and _rel(gP[None], r[2][None]) <= 1e-7


def test_plog_reactions():
    # two and three molecules on a side, one way, fractional (the general form),
    # a single pressure, two entries at one pressure; pressures below, between and
    # above the levels
    mech = synthetic.synthetic_mechanism(14, 50, 4, 4, seed=11, n_plog=14)
    s = mech.species_names
    rx = [r for r in mech.reactions if r.kind == "plog"]
    rx[0].reactants, rx[0].products, rx[0].reversible = {s[0]: 2.0, s[1]: 1.0}, {s[2]: 1.0, s[3]: 1.0}, False
    rx[1].reactants, rx[1].products, rx[1].reversible = {s[4]: 1.0}, {s[5]: 1.0, s[6]: 1.0, s[7]: 1.0}, False
    rx[2].reactants, rx[2].products, rx[2].reversible = {s[8]: 1.0}, {s[9]: 0.5, s[10]: 1.5}, False
    rx[3].plog = rx[3].plog[:1]
    rx[4].plog = sorted(rx[4].plog + [rx[4].plog[0]])
    _check(mech, 37, seed=3)
    P, T, Y = synthetic.states(mech.ns, 27, seed=4)
    P[:] = np.geomspace(1e2, 1e10, 27)
    (J64, J32, v), (J, r) = _derivatives(mech, 27, states=(P, T, Y))
    assert _rel(J64, J) <= 1e-9 and _rel(J32, J) <= 1e-6
    assert _rel(v[1], r[1]) <= 1e-9
    assert _rel(v[0][None], r[0][None]) <= 1e-7 and _rel(v[2][None], r[2][None]) <= 1e-7


def test_plog_reactions_cost_little_more_than_others():
    # 8 of 40 reactions: the adjoint takes under 1.6 times that of 40 without PLOG
    # (it took over twice as long when they were evaluated out of line)
    import torch
    from conftest import load_golden
    import dataclasses
    mech = load_golden("synthetic_plog_15_40")[0]
    plain = dataclasses.replace(mech, reactions=[
        dataclasses.replace(r, kind="standard", plog=None, arh=tuple(r.plog[0][1:])) if r.kind == "plog" else r
        for r in mech.reactions])
    P, T, Y = _cuda(*synthetic.states(mech.ns, 200000, seed=2))
    G = torch.ones_like(Y)

    def us(m):
        gm = GpuMechanism(m)
        t = []
        for _ in range(12):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            gm.vjp(P, T, Y, G)
            b.record()
            b.synchronize()
            t.append(a.elapsed_time(b))
        return min(t[2:])
    assert us(mech) < 1.6 * us(plain)


def test_derivatives_where_a_third_body_is_zero():
    # a species without efficiency alone: M = 0, and nothing divides by it
    mech = synthetic.synthetic_mechanism(10, 24, 10, 0, seed=5)
    for r in mech.reactions:
        if r.kind == "third_body":
            r.efficiencies = {**r.efficiencies, "S3": -1.0}
    P, T, Y = synthetic.states(mech.ns, 9, seed=1)
    Y[:] = 0.0
    Y[3] = 1.0
    (J64, J32, v), (J, r) = _derivatives(mech, 9, states=(P, T, Y))
    # (column T is zero but for rounding: relative to the rest)
    assert _rel(J64, J) <= 1e-9 and _rel(J32, J) <= 1e-6
    assert _rel(v[1], r[1]) <= 1e-9


def test_derivatives_where_a_falloff_has_no_collider():
    # M = 0 of Lindemann reactions: the rate is zero, its derivative by M is
    # k0 (prod C - prod C / Kc), and nothing divides by M.  Against autograd
    mech = synthetic.synthetic_mechanism(10, 24, 0, 0, seed=5, n_lindemann=10)
    for r in mech.reactions:
        if r.kind == "lindemann":
            r.efficiencies = {**r.efficiencies, "S3": -1.0}
            r.reactants, r.products, r.reversible = {"S3": 2.0}, {"S1": 1.0, "S3": 1.0}, False
    P, T, Y = synthetic.states(mech.ns, 9, seed=1)
    Y[:] = 0.0
    Y[3] = 1.0
    (J64, J32, v), (J, r) = _derivatives(mech, 9, states=(P, T, Y))
    assert bool((J[1].abs().amax(0) > 0).all())
    assert _rel(J64, J) <= 1e-9 and _rel(J32, J) <= 1e-6
    assert _rel(v[1], r[1]) <= 1e-9


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
@pytest.mark.parametrize("name", ["gri30", "h2_burke", "synthetic_53_325", "all_kinds"])
def test_small_batches_and_remainders_equal_the_generated_kernel(name, mode):
    # a batch of one wave runs the generated kernel, its first points alone the
    # tile kernel, and a wave plus a few points both: the same arithmetic, with
    # FP64 mode's sums in another order (1e-12 covers 300 terms of rounding; a mixed
    # rate off by one FP32 ulp would show as 6e-8)
    from conftest import load_golden
    mech = synthetic.all_kinds() if name == "all_kinds" else load_golden(name)[0]
    gm = GpuMechanism(mech, generated=True)
    assert gm.kernel_kind(mode) == "generated"
    wave = 148 * 512
    P, T, Y = _cuda(*synthetic.states(mech.ns, wave + 77, seed=4))

    def run(a, b):
        return gm.getrates(P[a:b].contiguous(), T[a:b].contiguous(), Y[:, a:b].contiguous(), mode=mode)
    ref = run(0, wave)
    for n in (1, 8 * 148, 8 * 148 + 1, 3001):
        assert _rel(run(0, n), ref[:, :n]) <= 1e-12, n
    both = run(0, wave + 77)
    assert _rel(both[:, :wave], ref) <= 1e-12
    assert _rel(both[:, wave:], run(wave, wave + 77)) <= 1e-12
    if mode == "mixed":
        # the mixed tile kernel repeats the generated one to the last bit
        assert all(bool((run(0, n) == ref[:, :n]).all()) for n in (1, 1184, 1185, 3001))


@pytest.mark.parametrize("name,waves,n,tiles", [
    ("h2_burke", 0, 1000, True), ("h2_burke", 0, 8192, False), ("h2_burke", 1, 500, False), ("all_kinds", 0, 4000, True), ("all_kinds", 0, 16000, False),
    ("gri30", 0, 20000, True), ("gri30", 0, 30000, False), ("all_kinds", 1, 2000, True), ("all_kinds", 1, 12000, False)])
def test_which_kernel_a_batch_of_a_generated_mechanism_runs_on(name, waves, n, tiles):
    # the FP64 tile kernel adds in another order than the generated one, so its bits
    # tell which of them ran: the last n points of a batch against the same points
    # in a whole wave (the generated kernel's)
    import torch
    from chemgen_b200 import emit_cuda as E
    from conftest import load_golden
    mech = synthetic.all_kinds() if name == "all_kinds" else load_golden(name)[0]
    gm = GpuMechanism(mech, generated=True)
    wave = (E.choose_block(mech.ns, False, E.use_tmem(mech.ns, False)) *
            torch.cuda.get_device_properties(0).multi_processor_count)
    P, T, Y = _cuda(*synthetic.states(mech.ns, wave + n, seed=8))
    k = n + waves * wave                                   # the batch, and the wave that ends where it does

    def run(a, b):
        return gm.getrates(P[a:b].contiguous(), T[a:b].contiguous(), Y[:, a:b].contiguous())
    w, ref = run(0, k)[:, k - n:], run(k - wave if waves else 0, k if waves else wave)
    ref = ref[:, wave - n:] if waves else ref[:, :n]
    assert bool((w == ref).all()) == (not tiles)
    assert _rel(w, ref) <= 1e-12


@pytest.mark.parametrize("name,ng,pinned", [("gri30", 60000, False), ("synthetic_plog_15_40", 50000, True)])
def test_host_calls_that_gain_nothing_from_chunks_take_one(name, ng, pinned):
    # pageable arrays and small states: one chunk, so the generated kernel serves all
    # of it and the FP64 bits are the device call's (chunks of 8192 points run on the
    # tile kernel)
    import torch
    from conftest import load_golden
    mech = load_golden(name)[0]
    gm = GpuMechanism(mech, generated=True)
    P, T, Y = synthetic.states(mech.ns, ng, seed=9)
    w = gm.getrates(*_cuda(P, T, Y)).cpu()
    if pinned:
        P, T, Y = (torch.from_numpy(x).pin_memory() for x in (P, T, Y))
    out = torch.empty(mech.ns, ng, dtype=torch.float64, pin_memory=pinned)
    gm.getrates_host(P, T, Y, out=out if pinned else out.numpy())
    assert torch.equal(out, w)


@pytest.mark.parametrize("ng", [1, 31, 33, 32 * 148 + 7])
def test_mixed_32_point_tiles(ng):
    # part tiles and more tiles than SMs on the 32-point tensor-core kernel; 1e-6
    # is the mixed kernels' bar
    from conftest import load_golden
    mech = load_golden("jetsurf2")[0]
    blob = pack.pack(mech).to_blob()
    P, T, Y = synthetic.states(mech.ns, ng, seed=ng)
    w = GpuMechanism(blob).getrates(*_cuda(P, T, Y), mode="mixed").cpu().numpy()
    idx = np.unique(np.concatenate([np.arange(min(ng, 40)), np.arange(max(0, ng - 40), ng)]))
    r = oracle.rates(blob, P[idx], T[idx], np.ascontiguousarray(Y[:, idx]), mech.nr)
    assert oracle.errors(w[:, idx], r["wdot"], r["S"])["norm_max"] <= 1e-6


@pytest.mark.parametrize("kinds", [(5, 0, 0), (0, 1, 4), (3, 3, 3), (40, 33, 30)])
def test_mixed_32_point_tiles_falloff(kinds):
    # pairs of one falloff kind, pairs across two kinds and single ones; 1e-6 as above
    n_lind, n_troe, n_sri = kinds
    mech = synthetic.synthetic_mechanism(40, 60 + sum(kinds), 7, n_troe, seed=2, n_lindemann=n_lind, n_sri=n_sri)
    blob = pack.pack(mech).to_blob()
    P, T, Y = synthetic.states(mech.ns, 45, seed=1)
    w = GpuMechanism(blob).getrates(*_cuda(P, T, Y), mode="mixed").cpu().numpy()
    r = oracle.rates(blob, P, T, Y, mech.nr)
    assert oracle.errors(w, r["wdot"], r["S"])["norm_max"] <= 1e-6


@pytest.mark.parametrize("ns,nr", [(53, 325), (10, 60), (126, 200)])
def test_mixed_tiles_of_32_and_128_points_agree(ns, nr):
    # the same points in a batch of one 32-point round and in one of a whole
    # 128-point wave.  Their FP64 values differ in rounding, which can tip the FP32
    # rounding of up to three concentrations, M, 2^f, the products and the sum: eight
    # times 1.2e-7 of the gross rate S
    import torch
    mech = synthetic.synthetic_mechanism(ns, nr, 9, 9, seed=4, n_lindemann=3, n_sri=3, n_plog=3)
    blob = pack.pack(mech).to_blob()
    gm = GpuMechanism(blob)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    P, T, Y = _cuda(*synthetic.states(ns, 4 * 128 * sms, seed=3))
    n = 32 * sms - 5
    w = gm.getrates(P[:n].contiguous(), T[:n].contiguous(), Y[:, :n].contiguous(), mode="mixed")
    ref = gm.getrates(P, T, Y, mode="mixed")[:, :n]
    r = oracle.rates(blob, P[:n].cpu().numpy(), T[:n].cpu().numpy(), Y[:, :n].contiguous().cpu().numpy(), mech.nr)
    S = torch.from_numpy(r["S"]).cuda()
    assert float(((w - ref).abs() / S.clamp_min(1e-300)).max()) <= 1e-6


@pytest.mark.parametrize("rows,cols", [(1 << 19, 1), (1, 1 << 19), (9893, 53), (53, 9893), (8129, 65), (348, 1507)])
def test_transposed_copies(rows, cols):
    # tiles of 64 x 64: whole, part and single-row ones; the values are moved, not computed
    import torch
    from chemgen_b200.runtime import transposed
    x = torch.arange(rows * cols, dtype=torch.float64, device="cuda").reshape(rows, cols)
    assert torch.equal(transposed(x), x.t())
    out = torch.empty(cols, rows, dtype=torch.float64, device="cuda")
    assert transposed(x, out) is out and torch.equal(out, x.t())
    assert torch.equal(transposed(x[:, ::2]), x[:, ::2].t())


def test_a_handle_is_made_in_a_few_milliseconds():
    # plans and tables of 348/2158; querying every property of the device for each
    # plan took 23 ms in all, the plans themselves take 7
    import time
    from conftest import load_golden
    blob = pack.pack(load_golden("jetsurf2")[0]).to_blob()
    t = []
    for _ in range(6):
        t0 = time.perf_counter()
        gm = GpuMechanism(blob)
        t.append(time.perf_counter() - t0)
        gm.close()
    assert min(t[1:]) < 12e-3, t


def test_split_calls_from_two_threads_on_streams_of_their_own():
    # a wave on the generated kernel and 5000 points on the tiles, from two threads
    # of one handle; and with point-major tensors into a ragged out=
    import threading
    import torch
    from chemgen_b200 import emit_cuda as E
    from conftest import load_golden
    mech = load_golden("gri30")[0]
    gm = GpuMechanism(mech, generated=True)
    n = 5000 + (E.choose_block(mech.ns, False, E.use_tmem(mech.ns, False)) *
                torch.cuda.get_device_properties(0).multi_processor_count)
    data = [_cuda(*synthetic.states(mech.ns, n, seed=s)) for s in (1, 2)]
    ref = [gm.getrates(*d) for d in data]
    out = torch.empty(n, mech.ns, dtype=torch.float64, device="cuda")
    assert gm.getrates(data[0][0], data[0][1], data[0][2].t().contiguous(), layout="point_major", out=out) is out
    assert torch.equal(out, ref[0].t())
    torch.cuda.synchronize()
    bad = []

    def work(k):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for _ in range(10):
                w = gm.getrates(*data[k])
                s.synchronize()
                if not torch.equal(w, ref[k]):
                    bad.append(k)
    th = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    [t.start() for t in th]
    [t.join() for t in th]
    assert not bad
