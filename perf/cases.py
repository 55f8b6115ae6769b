"""The work a user of the line-strength library has it do, as cases that can be timed.

A case is a dict: its kind (which public entry points it calls) and its sizes.  The inputs
follow the synthetic workloads of this repository (``synth``): rotational-vibrational bases
of N_v vibrational functions per (K, tau), symmetry classes of a rule, a vibrational dipole
that decays away from its diagonal, dense eigenvectors of unit norm, energies spread over
0 to 8000 cm^-1.  Everything a seed decides (dipole, eigenvectors, energies, level subsets,
loss gradients) differs from seed to seed; bases, expansion tables and the jobs of a plan
depend on sizes only.

Kinds:
  pair      one block pair, (J'', Gamma'') -> (J', Gamma'), through ``Engine.run_pair`` on
            resident eigenvectors; the amplitudes stay on the device (``amp_device``)
  lines     every component pair of a degenerate block pair, then its line strengths
  stream    what a line-list job does per block pair: both eigenvector sets from page-locked
            host memory, the run, S and A back into page-locked host memory
  text      the line list of a run as text in page-locked host memory
  plan      many uneven block pairs as one grouped plan
  adjoint   forward and gradient of a loss over line strengths with respect to the dipole
  dropin    the kernel-level calls of one lower state: expansion, one half line strength
            launch per upper K block, expansion and dot product per upper state
"""
from __future__ import annotations

import ctypes
import functools
import math
import os
import sys
from fractions import Fraction

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gain-mpi_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import gainls  # noqa: E402
import synth  # noqa: E402

SPLIT, PLAIN = "split", "plain"
# the symmetry pairs each rule runs: lower Gamma, upper Gamma
_GAMMAS = {"full": (0, 0), "c4": (0, 1), "c4m": (0, 1), "c4r": (0, 1), "c3e": (2, 2)}


def listed():
    return [
        # The smallest calls: 50 states of J = 0 against every state of J = 1, whole basis
        # (the repository's smallest named workload).  Latency and launches count.
        dict(name="pair_small", kind="pair", rule="full", path=SPLIT, nv=200, JI=0, JF=1, low=50, up=600, subset=False),
        # An ordinary pair of a many-pair sweep (N_v = 200, as in the sweep benchmark).
        dict(name="pair_medium", kind="pair", rule="c4", path=SPLIT, nv=200, JI=10, JF=11, low=550, up=1200, subset=False),
        # Odd sizes, mixing expansions, scattered subsets of the levels.
        dict(name="pair_ragged_mixed", kind="pair", rule="c4m", path=SPLIT, nv=333, JI=7, JF=6, low=777, up=1001,
             subset=True),
        # The rotational-symmetry form: the matrix is dense in K.
        dict(name="pair_rotsym", kind="pair", rule="c4r", path=SPLIT, nv=301, JI=5, JF=6, low=640, up=900, subset=False),
        # The largest: the headline benchmark's pair, 2000 x 12000 transitions at N_v = 2000.
        dict(name="pair_large", kind="pair", rule="c4", path=SPLIT, nv=2000, JI=10, JF=11, low=2000, up=12000,
             subset=False),
        # The reference's own FP64 method, which checks and near-threshold lines run on.
        dict(name="pair_plain", kind="pair", rule="c4", path=PLAIN, nv=800, JI=6, JF=7, low=96, up=3000, subset=False),
        # Degenerate symmetries: four component pairs and the lines that combine them.
        dict(name="lines_degenerate", kind="lines", rule="c3e", path=SPLIT, nv=250, JI=4, JF=5, low=300, up=1000,
             subset=False),
        # A line-list job's step for one pair, host memory to host memory.
        dict(name="stream_pair", kind="stream", rule="c4", path=SPLIT, nv=1000, JI=10, JF=11, low=1000, up=6000,
             subset=False),
        # The line list itself as text, intensity column included.
        dict(name="text_lines", kind="text", rule="c4", path=PLAIN, nv=600, JI=10, JF=11, low=1000, up=3600,
             subset=False),
        # Every allowed pair of J = 0..5 as one plan: 52 pairs of 50 to 1100 functions.
        dict(name="plan_sweep", kind="plan", rule="c4", nv=400, jmax=5, elow=4000),
        # A refinement step's forward and gradient on the tensor cores.
        dict(name="adjoint_split", kind="adjoint", rule="c4", path=SPLIT, nv=600, JI=4, JF=5, low=1350, up=1650,
             subset=False, precision="split"),
        # One lower state through the kernel-level calls, as the reference's driver makes them.
        dict(name="dropin_state", kind="dropin", rule="c4", nv=600, JI=10, JF=11, up=32),
    ]


def _log(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair", "pair", "pair", "pair", "lines", "stream", "text", "plan", "adjoint", "dropin"])
    if kind == "plan":
        return dict(kind="plan", rule=rng.choice(["c4", "c4m"]), nv=_log(rng, 24, 300), jmax=rng.randint(2, 5),
                    elow=rng.randint(1500, 6000))
    JI = rng.randint(1, 9)
    JF = JI + rng.choice([-1, 0, 1, 1])
    if kind == "dropin":
        return dict(kind="dropin", rule="c4", nv=_log(rng, 40, 600), JI=JI, JF=JF, up=_log(rng, 4, 48))
    rule = {"lines": "c3e", "stream": "c4", "text": "c4", "adjoint": "c4"}.get(kind) or rng.choice(
        ["full", "c4", "c4", "c4m", "c4r"])
    path = PLAIN if kind == "text" or (kind == "pair" and rng.random() < 0.2) else SPLIT
    top = {"full": 150, "c4": 1200, "c4m": 500, "c4r": 300, "c3e": 300}[rule]
    if path == PLAIN or kind == "adjoint":
        top = min(top, 100 if rule == "c4r" else 500)
    nv = _log(rng, 25, top)
    nI, nF = _block_size(rule, JI, nv), _block_size(rule, JF, nv)
    low = min(nI, _log(rng, 16, 1500 if path == SPLIT else 24 if rule == "c4r" else 200))
    up = min(nF, _log(rng, 48, 6000))
    c = dict(kind=kind, rule=rule, path=path, nv=nv, JI=JI, JF=JF, low=low, up=up,
             subset=kind == "pair" and rng.random() < 0.4)
    if kind == "adjoint":
        c["precision"] = rng.choice(["split", "split", "f64", "f32"])
    return c


# ------------------------------------------------------------------ tables that sizes decide
@functools.lru_cache(maxsize=64)
def _tables(rule, J, nv):
    b = synth.make_rotsym_basis(J, nv) if rule == "c4r" else synth.make_basis(J, nv)
    return b, synth.inflation_of(b, rule, synth.nsym_of(rule))


@functools.lru_cache(maxsize=256)
def _block_size(rule, J, nv):
    return int(_tables(rule, J, nv)[1].Ntot[_GAMMAS[rule][0]])


# ------------------------------------------------------------------------- seeded inputs
def _generator(seed, *tags):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + sum(int(t) * 7919 ** (k + 1) for k, t in enumerate(tags))) % (1 << 62))
    return g


def _vectors(seed, J, gamma, levels, n):
    """Dense unit rows, as the columns of the Q factor of a Gaussian matrix are."""
    v = torch.randn((levels, n), generator=_generator(seed, 1, J, gamma), dtype=torch.float64, device="cuda")
    return v / v.norm(dim=1, keepdim=True)


def _dipole(seed, nv):
    """[3][i][f], symmetric, decaying away from the diagonal."""
    a = torch.randn((3, nv, nv), generator=_generator(seed, 2), dtype=torch.float64, device="cuda")
    i = torch.arange(nv, device="cuda", dtype=torch.float64)
    a = a * (0.5 * torch.exp(-(i[:, None] - i[None, :]).abs() / 20.0))
    return (0.5 * (a + a.transpose(1, 2))).contiguous()


def _energies(seed, J, gamma, n):
    return np.sort(np.random.default_rng([seed, 3, J, gamma]).uniform(0.0, 8000.0, n))


def _wigner(seed, JI, JF):
    n = 3 * (2 * JI + 1) * (2 * JF + 1)
    return 0.5 * np.random.default_rng([seed, 4, JI, JF]).uniform(-1.0, 1.0, n)


def _levels(case, seed, side, have, want):
    if not case["subset"]:
        return np.arange(want, dtype=np.int32)
    r = np.random.default_rng([seed, 5, side])
    return np.sort(r.choice(have, want, replace=False)).astype(np.int32)


def _pair_inputs(case, seed):
    """What one pair needs, before any of it reaches the library (prepare and exact share it)."""
    rule, nv, JI, JF = case["rule"], case["nv"], case["JI"], case["JF"]
    gI, gF = _GAMMAS[rule]
    (bI, iI), (bF, iF) = _tables(rule, JI, nv), _tables(rule, JF, nv)
    nI, nF = int(iI.Ntot[gI]), int(iF.Ntot[gF])
    low, up = min(case["low"], nI), min(case["up"], nF)
    haveI, haveF = (nI, nF) if case["subset"] else (low, up)
    same = (JI, gI) == (JF, gF)      # one block on both sides: both level lists index it
    if same:
        haveI = haveF = max(haveI, haveF)
    return dict(gI=gI, gF=gF, bI=bI, iI=iI, bF=bF, iF=iF, same=same,
                vI=_vectors(seed, JI, gI, haveI, nI), vF=_vectors(seed, JF, gF, haveF, nF),
                eI=_energies(seed, JI, gI, haveI), eF=_energies(seed, JF, gF, haveF), mu=_dipole(seed, nv),
                lo=_levels(case, seed, 0, haveI, low), up=_levels(case, seed, 1, haveF, up))


# ---------------------------------------------------------------------------------- prepare
def _upload_tables(eng, jind, b, inf):
    eng.upload_basis(jind, b.J, b.K, b.tau, b.vib, b.kblock, b.kstart)
    eng.upload_inflation(jind, inf.icontr, inf.ijterms, b.dimen, inf.maxcoeff, inf.matsize, inf.N, inf.repres, inf.Ntot,
                         inf.sdeg)


def _pinned(t):
    p = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    p.copy_(t)
    return p.numpy()


def prepare(case, seed):
    torch.cuda.init()
    return {"plan": _prepare_plan, "dropin": _prepare_dropin}.get(case["kind"], _prepare_pair)(case, seed)


def _prepare_pair(case, seed):
    x = _pair_inputs(case, seed)
    kind, rule, nv, JI, JF = case["kind"], case["rule"], case["nv"], case["JI"], case["JF"]
    gI, gF, lo, up = x["gI"], x["gF"], x["lo"], x["up"]
    eng = gainls.Engine(max(11, JI, JF), synth.nsym_of(rule), int(synth.degen_of(rule).max()))
    jI, jF = 0, 0 if JF == JI else 1
    _upload_tables(eng, jI, x["bI"], x["iI"])
    if jF != jI:
        _upload_tables(eng, jF, x["bF"], x["iF"])
    eng.upload_dipole(x["mu"].cpu().numpy().reshape(-1), nv, 0, nv, nv)
    if rule == "c4r":
        eng.upload_wigner(jI, jF, 2 * JI + 1, 2 * JF + 1, 1, _wigner(seed, JI, JF))
    s = dict(case=case, eng=eng, job=(jI, gI, jF, gF), lo=lo, up=up, eI=x["eI"][lo], eF=x["eF"][up],
             path=gainls.PATH_SPLIT if case["path"] == SPLIT else gainls.PATH_PLAIN_FP64)
    if kind == "stream":   # the vectors wait in page-locked host memory, S and A come back to it
        s["hI"], s["hF"] = _pinned(x["vI"]), _pinned(x["vF"])
        s["S"], s["A"] = (_pinned(torch.zeros(len(lo), len(up), dtype=torch.float64)) for _ in range(2))
        return s
    for (j, g, v) in ((jI, gI, x["vI"]),) if x["same"] else ((jI, gI, x["vI"]), (jF, gF, x["vF"])):
        eng.upload_eigvecs_device(j, g, v.data_ptr(), v.shape[0], v.shape[1])
    if kind == "lines":
        d = synth.degen_of(rule)
        s["ndeg"] = (int(d[gI]), int(d[gF]))
        s["filters"] = _filters(rule)
    if kind == "text":     # the amplitudes are there; the list is written from them
        eng.run_pair(*s["job"], lo, up, s["path"])
        s["out"] = _pinned(torch.zeros(96 * len(lo) * len(up), dtype=torch.uint8))
    if kind == "adjoint":
        r = torch.randn((len(lo), len(up)), generator=_generator(seed, 6), dtype=torch.float64, device="cuda")
        s["dL_dS"] = r.cpu().numpy()
        s["ndip"] = 3 * nv * nv
    return s


def _filters(rule, elow=1e9, maxJ=40):
    sel = synth.selection_of(rule)
    return gainls.make_filters([1.0] * synth.nsym_of(rule), sel, synth.igamma_pair_of(sel), synth.degen_of(rule),
                               (0.0, float(elow)), (-1e9, 1e9), (-1e9, 1e9), 0.0, maxJ)


def _plan_jobs(case):
    """(tables per J, jobs): every pair the library's own state selection allows.  The energies
    are the same for every seed, so that the jobs have the same sizes."""
    rule, nv, nsym = case["rule"], case["nv"], synth.nsym_of(case["rule"])
    tables = [_tables(rule, J, nv) for J in range(case["jmax"] + 1)]
    en, J_, g_, lev = [], [], [], []
    for J, (_, inf) in enumerate(tables):
        for g in range(nsym):
            n = int(inf.Ntot[g])
            en.append(_energies(0, J, g, n))
            J_ += [J] * n
            g_ += [g] * n
            lev += list(range(n))
    en = np.concatenate(en)
    o = np.argsort(en, kind="stable")
    J_, g_, lev = np.asarray(J_)[o], np.asarray(g_)[o], np.asarray(lev)[o]
    table = gainls.state_table(en[o], J_, J_, g_, np.ones_like(g_), lev)
    jobs = gainls.plan_pairs(_filters(rule, case["elow"], case["jmax"]), table)
    jobs = [(a, b, c, d, np.asarray(lo, np.int32), np.asarray(up, np.int32)) for a, b, c, d, lo, up in jobs]
    return tables, jobs


def _prepare_plan(case, seed):
    tables, jobs = _plan_jobs(case)
    nv, nsym = case["nv"], synth.nsym_of(case["rule"])
    eng = gainls.Engine(11, nsym, 1)
    eng.upload_dipole(_dipole(seed, nv).cpu().numpy().reshape(-1), nv, 0, nv, nv)
    for J, (b, inf) in enumerate(tables):
        _upload_tables(eng, J, b, inf)
        for g in range(nsym):
            n = int(inf.Ntot[g])
            if n:
                v = _vectors(seed, J, g, n, n)
                eng.upload_eigvecs_device(J, g, v.data_ptr(), n, n)
    return dict(case=case, eng=eng, plan=gainls.Plan(eng, jobs), shapes=[(len(j[4]), len(j[5])) for j in jobs])


def _prepare_dropin(case, seed):
    nv, JI, JF = case["nv"], case["JI"], case["JF"]
    gI, gF = _GAMMAS["c4"]
    (bI, iI), (bF, iF) = _tables("c4", JI, nv), _tables("c4", JF, nv)
    up = min(case["up"], int(iF.Ntot[gF]))
    def d(a, t):
        return torch.from_numpy(np.ascontiguousarray(a, t)).cuda()

    s = dict(case=case, gI=gI, gF=gF, bI=bI, bF=bF, iI=iI, iF=iF, up=up, mu=_dipole(seed, nv),
             vI=_vectors(seed, JI, gI, 1, int(iI.Ntot[gI])), vF=_vectors(seed, JF, gF, up, int(iF.Ntot[gF])),
             threej=d(gainls.threej_table(11), np.float64),
             prim=torch.zeros(bI.dimen, dtype=torch.float64, device="cuda"),
             primF=torch.zeros(bF.dimen, dtype=torch.float64, device="cuda"),
             half=torch.zeros(bF.dimen, dtype=torch.float64, device="cuda"),
             amp=torch.zeros(up, dtype=torch.float64, device="cuda"))
    for side, b, inf, g in (("I", bI, iI, gI), ("F", bF, iF, gF)):
        s["d" + side] = dict(tau=d(b.tau, np.int32), vib=d(b.vib, np.int32), kb=d(b.kblock, np.int32),
                             ij=d(inf.ijterms, np.int32), ic=d(inf.icontr, np.int32), N=d(inf.N[g], np.int32),
                             rp=d(inf.repres[g], np.float64))
    return s


# -------------------------------------------------------------------------------------- run
class _DeviceMatrix:
    """A device matrix of the library as an object torch can view without a copy; it keeps the
    engine or plan that owns the memory alive."""

    def __init__(self, owner, ptr, rows, cols, ld):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=(rows, cols), typestr="<f8", data=(ptr, False), version=2,
                                             strides=(8 * ld, 8))


def _amp(eng, shape):
    ptr, ld = eng.amp_device()
    return torch.as_tensor(_DeviceMatrix(eng, ptr, shape[0], shape[1], ld), device="cuda")


def _plan_amp(plan, q, shape):
    ptr, ld = ctypes.c_void_p(), ctypes.c_int()
    gainls.check(gainls.lib().gain_plan_amp_device(plan.h, q, ctypes.byref(ptr), ctypes.byref(ld)))
    return torch.as_tensor(_DeviceMatrix(plan, ptr.value, shape[0], shape[1], ld.value), device="cuda")


def run(s):
    kind = s["case"]["kind"]
    if kind == "dropin":
        return _run_dropin(s)
    eng = s["eng"]
    if kind == "plan":
        s["plan"].run()
        return [_plan_amp(s["plan"], q, shape) for q, shape in enumerate(s["shapes"])]
    J = s["case"]["JI"], s["case"]["JF"]
    if kind == "text":
        _, n = eng.lines_text_host(s["eI"], s["eF"], *J, s["job"][1], s["job"][3], s["out"], temperature=296.0,
                                   q_part=300.0)
        return {"text": s["out"], "lines": n}     # how many lines are kept depends on the energies
    if kind == "stream":
        eng.upload_eigvecs_async(*s["job"][:2], s["hI"])
        eng.upload_eigvecs_async(*s["job"][2:], s["hF"])
        eng.run_pair(*s["job"], s["lo"], s["up"], s["path"])
        eng.lines(s["eI"], s["eF"], *J, intensity=False, want=("S", "A"), out_S=s["S"], out_A=s["A"])
        return {"S": s["S"], "A": s["A"]}
    if kind == "lines":
        eng.run_pair(*s["job"], s["lo"], s["up"], s["path"], filters=s["filters"])
        r = eng.lines(s["eI"], s["eF"], *J, intensity=False, want=("S", "A"), ndeg=s["ndeg"])
        return {"S": r["S"], "A": r["A"]}
    eng.run_pair(*s["job"], s["lo"], s["up"], s["path"])
    if kind == "adjoint":
        g = eng.adjoint(*s["job"], s["lo"], s["up"], s["dL_dS"], np.zeros(s["ndip"]), precision=s["case"]["precision"])
        return {"dL_dmu": g}
    return _amp(eng, (len(s["lo"]), len(s["up"])))


def _run_dropin(s):
    c, bI, bF, iI, iF, I, F = s["case"], s["bI"], s["bF"], s["iI"], s["iF"], s["dI"], s["dF"]
    st = torch.cuda.current_stream().cuda_stream
    nv, JI, JF = c["nv"], c["JI"], c["JF"]
    gainls.expand(bI.dimen, s["gI"], iI.maxcoeff, 0, 1, int(iI.Ntot[s["gI"]]), I["ij"].data_ptr(), I["ic"].data_ptr(),
                  I["N"].data_ptr(), I["rp"].data_ptr(), s["vI"].data_ptr(), s["prim"].data_ptr(), st)
    for kF in range(JF + 1):
        if kF - 1 > JI:
            continue
        gainls.hls_kblock(int(bF.kblock[kF]), bI.dimen, JI, JF, kF, I["tau"].data_ptr(), F["tau"].data_ptr(),
                          I["vib"].data_ptr(), F["vib"].data_ptr(), int(bF.kstart[kF]), int(bI.kstart[max(kF - 1, 0)]),
                          0, nv, nv, int(bF.kblock[kF]), I["kb"].data_ptr(), s["mu"].data_ptr(), s["prim"].data_ptr(),
                          s["threej"].data_ptr(), s["half"].data_ptr(), 11, nv, st)
    for u in range(s["up"]):
        gainls.expand(bF.dimen, s["gF"], iF.maxcoeff, 0, 1, int(iF.Ntot[s["gF"]]), F["ij"].data_ptr(),
                      F["ic"].data_ptr(), F["N"].data_ptr(), F["rp"].data_ptr(), s["vF"][u].data_ptr(),
                      s["primF"].data_ptr(), st)
        gainls.dot(bF.dimen, s["half"].data_ptr(), s["primF"].data_ptr(), s["amp"][u:].data_ptr(), st)
    return {"half_ls": s["half"], "amp": s["amp"]}


# ------------------------------------------------------------------------------------- work
def work(case):
    """Bytes: every input read once and every output written once.  Flops: the contraction with
    the rotational-dipole matrix (its non-zero K blocks) and the products with the upper
    vectors, each as multiply and add."""
    kind, rule, nv = case["kind"], case["rule"], case["nv"]
    if kind == "plan":
        total = {"bytes": 24.0 * nv * nv, "flops": 0.0}
        sizes = [[int(n) for n in _tables(rule, J, nv)[1].Ntot] for J in range(case["jmax"] + 1)]
        total["bytes"] += sum(8.0 * n * n for blk in sizes for n in blk)
        pair = synth.igamma_pair_of(synth.selection_of(rule))
        for JI in range(case["jmax"]):
            for JF in range(max(0, JI - 1), min(case["jmax"], JI + 1) + 1):
                if JI + JF == 0:
                    continue
                for g, nI in enumerate(sizes[JI]):
                    nF = sizes[JF][int(pair[g])]
                    low = nI * min(1.0, case["elow"] / 8000.0)
                    total["bytes"] += 8.0 * low * nF
                    total["flops"] += 2.0 * low * nF * (nF + nI * min(1.0, 3.0 / (JI + 1)))
        return total
    JI, JF = case["JI"], case["JF"]
    nI = int(_tables(rule, JI, nv)[1].Ntot[_GAMMAS[rule][0]])
    nF = int(_tables(rule, JF, nv)[1].Ntot[_GAMMAS[rule][1]])
    up = min(case["up"], nF)
    low = 1 if kind == "dropin" else min(case["low"], nI)
    if kind == "text":
        lines = 0.9 * low * up
        return {"bytes": 8.0 * low * up + 93.0 * lines, "flops": 30.0 * lines}
    dense = rule == "c4r"
    if kind == "dropin":   # the reference's calls work over primitives
        dI, dF = (2 * JI + 1) * nv, (2 * JF + 1) * nv
        return {"bytes": 24.0 * nv * nv + 8.0 * (2 * dI + dF + nF * up), "flops": 2.0 * nI * dF * min(1.0, 3.0 / (JI + 1)) + 2.0 * up * nF}
    comps = 4 if kind == "lines" else 1
    one = 2.0 * low * nF * (nI * (1.0 if dense else min(1.0, 3.0 / (JI + 1)))) + 2.0 * low * nF * up
    out = 2 if kind in ("lines", "stream") else 1
    w = {"bytes": 24.0 * nv * nv + 8.0 * (low * nI + up * nF + out * low * up), "flops": comps * one}
    if kind == "adjoint":
        w = {"bytes": w["bytes"] + 8.0 * low * up + 24.0 * nv * nv, "flops": 2 * one}
    return w


# ------------------------------------------------------------------------------------ exact
@functools.lru_cache(maxsize=4096)
def _threej(jI, kI, jF, kF):
    """3j(jI 1 jF; kI kF-kI -kF) by Racah's sum over exact rationals."""
    j1, j2, j3, m1, m2, m3 = jI, 1, jF, kI, kF - kI, -kF
    if abs(m2) > 1 or abs(m1) > j1 or abs(m3) > j3 or not abs(j1 - j2) <= j3 <= j1 + j2:
        return 0.0
    f = math.factorial
    tri = Fraction(f(j1 + j2 - j3) * f(j1 - j2 + j3) * f(-j1 + j2 + j3), f(j1 + j2 + j3 + 1))
    sq = tri * f(j1 + m1) * f(j1 - m1) * f(j2 + m2) * f(j2 - m2) * f(j3 + m3) * f(j3 - m3)
    t = Fraction(0)
    for k in range(0, j1 + j2 - j3 + 1):
        a = (j1 + j2 - j3 - k, j1 - m1 - k, j2 + m2 - k, j3 - j2 + m1 + k, j3 - j1 - m2 + k)
        if min(a) >= 0:
            t += Fraction((-1) ** k, f(k) * f(a[0]) * f(a[1]) * f(a[2]) * f(a[3]) * f(a[4]))
    return (-1) ** (j1 - j2 - m3) * float(t) * math.sqrt(sq)


def _expansion(b, inf, g, ideg):
    """(primitives, symmetric functions, coefficients) of the non-zero expansion entries."""
    d, nt, sd = b.dimen, int(inf.Ntot[g]), int(inf.sdeg[g])
    case, ib = inf.icontr[:d], inf.icontr[d:]
    n = inf.N[g][case]
    first = inf.ijterms[g * inf.maxcoeff + case]
    r, c, v = [], [], []
    for i in range(int(n.max(initial=0))):
        p = np.nonzero(n > i)[0]
        r.append(p)
        c.append(first[p] + i)
        v.append(inf.repres[g][first[p] + i + ideg * nt + ib[p].astype(np.int64) * sd * nt])
    return np.concatenate(r), np.concatenate(c), np.concatenate(v)


def _primitive(vecs, exp):
    """Rows of symmetric-function coefficients over the primitives their expansion touches."""
    r, c, v = exp
    sup, pos = np.unique(r, return_inverse=True)
    out = torch.zeros((vecs.shape[0], len(sup)), dtype=torch.float64, device="cuda")
    for lo in range(0, vecs.shape[0], 512):
        x = vecs[lo:lo + 512][:, torch.from_numpy(c).long().cuda()] * torch.from_numpy(v).cuda()
        out[lo:lo + 512].index_add_(1, torch.from_numpy(pos).long().cuda(), x)
    return out, sup


def _factors(bI, bF, rI, rF):
    """Dipole component and rotational factor of primitives rI x rF (the K-block form)."""
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).long().cuda()  # noqa: E731
    kI, tI, kF, tF = t(bI.K[rI])[:, None], t(bI.tau[rI])[:, None], t(bF.K[rF])[None, :], (t(bF.tau[rF]) & 1)[None, :]
    w = torch.zeros((bI.J + 1, bF.J + 1), dtype=torch.float64)
    for a in range(bI.J + 1):
        for c in range(max(0, a - 1), min(bF.J, a + 1) + 1):
            w[a, c] = _threej(bI.J, a, bF.J, c) * (0.70710678118 if a != c and a * c else 1.0)
    w = w.cuda()[kI, kF]
    eq = (kI == kF).long()
    ne, tn = 1 - eq, (tI != tF).long()
    comp = 2 * eq + ne * (1 - tn)
    c = (tF - tI) * eq + (tF - tI) * (kF - kI) * ne * tn - ne * (1 - tn)
    sign = 1 - 2 * ((((kI % 3) * tI + kI) + (kF % 3) * tF) & 1)
    return comp, w * (c * sign)


def _matrix(case, seed, bI, bF, rI, rF, mu):
    """The rotational-dipole matrix over primitives rI x rF, a piece of rows at a time."""
    vF = torch.from_numpy(bF.vib[rF]).long().cuda()[None, :]
    out = torch.empty((len(rI), len(rF)), dtype=torch.float64, device="cuda")
    rot = None
    if case["rule"] == "c4r":
        rot = torch.from_numpy(_wigner(seed, bI.J, bF.J)).cuda().view(2 * bF.J + 1, 2 * bI.J + 1, 3)
    for lo in range(0, len(rI), 512):
        r = rI[lo:lo + 512]
        vI = torch.from_numpy(bI.vib[r]).long().cuda()[:, None]
        if rot is None:
            comp, w = _factors(bI, bF, r, rF)
            out[lo:lo + 512] = w * mu[comp, vI, vF]
        else:
            k = rot[torch.from_numpy(bF.tau[rF]).long().cuda()[None, :], torch.from_numpy(bI.tau[r]).long().cuda()[:, None]]
            out[lo:lo + 512] = sum(k[..., d] * mu[d, vI, vF] for d in range(3))
    return out


def _amplitudes(case, seed, bI, bF, eI, eF, V, U, mu):
    Vp, rI = _primitive(V, eI)
    Up, rF = _primitive(U, eF)
    return (Vp @ _matrix(case, seed, bI, bF, rI, rF, mu)) @ Up.T


def exact(case, seed):
    kind = case["kind"]
    if kind == "text":      # bytes and a count
        return None
    if kind == "plan":
        tables, jobs = _plan_jobs(case)
        mu, out = _dipole(seed, case["nv"]), []
        for jI, gI, jF, gF, lo, up in jobs:
            (bI, iI), (bF, iF) = tables[jI], tables[jF]
            V = _vectors(seed, jI, gI, int(iI.Ntot[gI]), int(iI.Ntot[gI]))[torch.from_numpy(lo).long().cuda()]
            U = _vectors(seed, jF, gF, int(iF.Ntot[gF]), int(iF.Ntot[gF]))[torch.from_numpy(up).long().cuda()]
            out.append(_amplitudes(case, seed, bI, bF, _expansion(bI, iI, gI, 0), _expansion(bF, iF, gF, 0), V, U, mu))
        return out
    if kind == "dropin":
        s = _prepare_dropin(case, seed)
        bI, bF = s["bI"], s["bF"]
        Vp, rI = _primitive(s["vI"], _expansion(bI, s["iI"], s["gI"], 0))
        half = (Vp @ _matrix(case, seed, bI, bF, rI, np.arange(bF.dimen), s["mu"]))[0]
        Up, rF = _primitive(s["vF"], _expansion(bF, s["iF"], s["gF"], 0))
        return {"half_ls": half, "amp": Up @ half[torch.from_numpy(rF).long().cuda()]}
    x = _pair_inputs(case, seed)
    bI, bF, iI, iF, gI, gF = x["bI"], x["bF"], x["iI"], x["iF"], x["gI"], x["gF"]
    vF = x["vI"] if x["same"] else x["vF"]
    V, U = x["vI"][torch.from_numpy(x["lo"]).long().cuda()], vF[torch.from_numpy(x["up"]).long().cuda()]
    if kind in ("lines", "stream"):
        d = synth.degen_of(case["rule"])
        S = torch.zeros((len(x["lo"]), len(x["up"])), dtype=torch.float64, device="cuda")
        for dF in range(int(d[gF])):
            for dI in range(int(d[gI])):
                S += _amplitudes(case, seed, bI, bF, _expansion(bI, iI, gI, dI), _expansion(bF, iF, gF, dF), V, U,
                                 x["mu"]) ** 2
        S /= int(d[gI])
        nu = torch.from_numpy(x["eF"][x["up"]][None, :] - x["eI"][x["lo"]][:, None]).cuda().abs()
        return {"S": S, "A": 3.13618923e-7 * (2 * case["JI"] + 1) * S * nu ** 3}
    if kind == "adjoint":
        r = torch.randn(V.shape[0], U.shape[0], generator=_generator(seed, 6), dtype=torch.float64, device="cuda")
        Vp, rI = _primitive(V, _expansion(bI, iI, gI, 0))
        Up, rF = _primitive(U, _expansion(bF, iF, gF, 0))
        amp = (Vp @ _matrix(case, seed, bI, bF, rI, rF, x["mu"])) @ Up.T
        dM = Vp.T @ ((2.0 * r * amp) @ Up)
        nv, grad = case["nv"], torch.zeros(3 * case["nv"] ** 2, dtype=torch.float64, device="cuda")
        vF = torch.from_numpy(bF.vib[rF]).long().cuda()[None, :]
        for lo in range(0, len(rI), 512):
            comp, w = _factors(bI, bF, rI[lo:lo + 512], rF)
            vI = torch.from_numpy(bI.vib[rI[lo:lo + 512]]).long().cuda()[:, None]
            grad.index_add_(0, (comp * nv * nv + vI * nv + vF).reshape(-1), (w * dM[lo:lo + 512]).reshape(-1))
        return {"dL_dmu": grad.cpu().numpy()}
    return _amplitudes(case, seed, bI, bF, _expansion(bI, iI, gI, 0), _expansion(bF, iF, gF, 0), V, U, x["mu"])
