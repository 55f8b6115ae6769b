"""The residue form of the split path (the default): one BF16 GEMM per modulus, reconstructed
exactly.  Sizes at the edges of its row and column tiles (128, 256), of its exact-accumulation
chunks (384 inner elements) and of the reconstruction's blocks, on CTA pairs and single CTAs."""
import os
import re

import numpy as np
import pytest

JMAX = 11


def test_moduli_are_coprime_and_chunks_stay_exact():
    """Pairwise coprime moduli; a chunk of products of balanced residues plus the running
    residue stays below 2^24; residues are exact in BF16 (8 significant bits)."""
    import math
    src = open(os.path.join(os.path.dirname(__file__), "..", "gain-mpi_gb300", "csrc", "residue.h")).read()
    mods = [int(x) for x in re.search(r"kModuli\[kMaxMod\] = \{([^}]*)\}", src).group(1).split(",")]
    blocks = int(re.search(r"kChunkBlocks = (\d+)", src).group(1))
    assert all(math.gcd(a, b) == 1 for i, a in enumerate(mods) for b in mods[:i])
    for m in mods:
        v = np.arange(-(1 << 24) + 1, 1 << 24, 7, dtype=np.int64)
        q = np.rint(v.astype(np.float64) * np.float64(np.float32(1.0) / np.float32(m)))
        r = np.abs(v - q.astype(np.int64) * m).max()     # the kernel's reduction, exact in binary64
        assert r <= 256 and 64 * blocks * r * r + r < 1 << 24, (m, r)


@pytest.fixture(scope="module")
def problems(built_lib):
    import gainls
    import synth
    out = {}
    for name, (rule, nv, jv) in {"c4": ("c4", 120, (5, 6)), "c4r": ("c4r", 130, (2, 3)), "full": ("full", 48, (3, 4)),
                                 "c4m": ("c4m", 75, (3, 4))}.items():
        g = (0, 0) if rule == "full" else (0, 1)
        p = synth.make_problem(nv, list(jv), rule, blocks=[(jv[0], g[0]), (jv[1], g[1])])
        eng = gainls.Engine(JMAX, p.nsym, 1)
        gainls.upload_problem(eng, p)
        out[name] = (p, eng, g)
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["c4", "c4r", "full", "c4m"])
@pytest.mark.parametrize("sizes", [(1, 1), (5, 127), (128, 128), (129, 129), (127, 257), (256, 256), (257, 391), (10**6, 10**6)])
@pytest.mark.parametrize("pair", ["1", "0"])
def test_residue_form_matches_plain_fp64(problems, name, sizes, pair, monkeypatch):
    """|amp - plain| against the rounding of the operands: each operand row is rounded to 48
    bits of its largest entry (a relative 2^-48 sqrt(N) of its norm, twice), each H entry is
    within the FP64 bound (W + 64) 2^-53 of its rows' norms, and the plain path adds N 2^-53."""
    import gainls
    p, eng, (gI, gF) = problems[name]
    vI, vF = p.blocks[(0, gI)].vecs, p.blocks[(1, gF)].vecs
    lo = np.arange(min(sizes[0], vI.shape[0]), dtype=np.int32)
    up = np.arange(min(sizes[1], vF.shape[0]), dtype=np.int32)[::-1].copy()
    monkeypatch.setenv("GAINLS_GEMM_PAIR", pair)
    eng.run_pair(0, gI, 1, gF, lo, np.arange(vF.shape[0], dtype=np.int32), gainls.PATH_PLAIN_FP64)
    full = eng.fetch_amp().copy()      # every upper state: an orthonormal set, so the rows' norms are those of H
    st = eng.run_pair(0, gI, 1, gF, lo, up, gainls.PATH_SPLIT)
    assert st["status"] == gainls.OK and st["products2"] == st["slices2"] == 13
    amp = eng.fetch_amp()
    N, W = vF.shape[1], 2 * vI.shape[1] + 128
    h = np.linalg.norm(full, axis=1).max()
    mrow = np.sqrt(15.0) * np.sqrt((p.dipole ** 2).sum(axis=(0, 1))).max()     # a row of M: at most 5 of each (K, tau)
    tol = (4 * np.sqrt(N) * 2.0 ** -48 + (N + 64) * 2.0 ** -52) * h + np.sqrt(N) * (W + 64) * 2.0 ** -53 * mrow
    assert np.max(np.abs(amp - full[:, up])) <= tol


@pytest.mark.gpu
@pytest.mark.parametrize("nup", [200, 780])
def test_several_row_panels_equal_one_run(problems, nup, monkeypatch):
    """More output rows than one panel (1024 on single CTAs), reconstructed one and four rows to a
    block: every row equals its own run's bits."""
    import gainls
    p, eng, (gI, gF) = problems["c4"]
    n = p.blocks[(0, gI)].vecs.shape[0]
    up = np.arange(nup, dtype=np.int32) % p.blocks[(1, gF)].vecs.shape[0]
    many = np.arange(2 * 1024 + 130, dtype=np.int32) % n
    eng.run_pair(0, gI, 1, gF, np.arange(n, dtype=np.int32), up, gainls.PATH_SPLIT)
    one = eng.fetch_amp().copy()
    for pair in ("1", "0"):
        monkeypatch.setenv("GAINLS_GEMM_PAIR", pair)
        eng.run_pair(0, gI, 1, gF, many, up, gainls.PATH_SPLIT)
        np.testing.assert_array_equal(eng.fetch_amp(), one[many])


@pytest.mark.gpu
@pytest.mark.parametrize("bits,moduli", [(46, 12), (48, 13), (54, 14), (56, 14)])
def test_other_numbers_of_moduli(problems, bits, moduli, monkeypatch):
    """First-GEMM precisions that take fewer or more moduli than the usual 13: the amplitudes agree
    within the rounding of the lower and band rows to that many bits (H entries that miss the
    FP64 bound are recomputed)."""
    import gainls
    p, eng, (gI, gF) = problems["c4"]
    lo = np.arange(p.blocks[(0, gI)].vecs.shape[0], dtype=np.int32)
    up = np.arange(p.blocks[(1, gF)].vecs.shape[0], dtype=np.int32)
    eng.run_pair(0, gI, 1, gF, lo, up, gainls.PATH_SPLIT)
    ref = eng.fetch_amp().copy()
    monkeypatch.setenv("GAINLS_GEMM1_BITS", str(bits))
    st = eng.run_pair(0, gI, 1, gF, lo, up, gainls.PATH_SPLIT)
    assert st["status"] == gainls.OK and st["slices1"] == moduli
    N, W = up.size, 2 * lo.size + 128
    mrow = np.sqrt(15.0) * np.sqrt((p.dipole ** 2).sum(axis=(0, 1))).max()
    h = np.linalg.norm(ref, axis=1).max()
    # two H errors (each within the FP64 bound of its rows) and two roundings of H to 48 bits
    tol = 2 * (np.sqrt(N) * (W + 64) * 2.0 ** -53 * mrow + 2 * np.sqrt(N) * 2.0 ** -48 * h)
    assert np.max(np.abs(eng.fetch_amp() - ref)) <= tol


@pytest.mark.gpu
def test_scales_and_zero_rows(built_lib):
    """Rows of very different scales, subnormal rows and all-zero rows: amplitudes scale with
    their rows exactly (powers of two) and zero rows give exact zeros."""
    import gainls
    import synth
    p = synth.make_problem(24, [2, 3], "c4", blocks=[(2, 0), (3, 1)])
    vI, vF = p.blocks[(0, 0)].vecs, p.blocks[(1, 1)].vecs
    lo, up = np.arange(vI.shape[0]), np.arange(vF.shape[0])
    eng = gainls.Engine(JMAX, p.nsym, 1)
    gainls.upload_problem(eng, p)
    eng.run_pair(0, 0, 1, 1, lo, up, gainls.PATH_SPLIT)
    ref = eng.fetch_amp().copy()
    e = np.resize([0, -40, 300, -300, 7], vI.shape[0])
    v2 = np.ldexp(vI, e[:, None])
    v2[3] = 0.0
    eng.upload_eigvecs(0, 0, v2)
    eng.run_pair(0, 0, 1, 1, lo, up, gainls.PATH_SPLIT)
    want = np.ldexp(ref, e[:, None])
    want[3] = 0.0
    np.testing.assert_array_equal(eng.fetch_amp(), want)
    eng.upload_eigvecs(0, 0, np.ldexp(vI, -1060))     # subnormal entries, rounded by the input itself
    eng.run_pair(0, 0, 1, 1, lo, up, gainls.PATH_SPLIT)
    got = eng.fetch_amp()
    assert np.max(np.abs(got - np.ldexp(ref, -1060))) <= 2.0 ** -1074 * 64 * vI.shape[1]


@pytest.mark.gpu
def test_plan_refines_flagged_entries_of_every_job(built_lib, monkeypatch):
    """A first GEMM of 40 bits: no H entry certifies FP64-grade, so every job's list is full.  The
    plan's one refinement launch recomputes what the single runs' do, and both agree with the
    plain FP64 path as an FP64 H and a 48-bit second GEMM must (see above)."""
    import gainls
    import synth
    p = synth.make_problem(20, [1, 2, 3], "c4")
    eng = gainls.Engine(JMAX, p.nsym, 1)
    gainls.upload_problem(eng, p)
    filt = gainls.make_filters([1.0] * 4, p.isym_pairs, p.igamma_pair, p.sym_degen, (0.0, 5000.0), (-1e9, 1e9),
                               (-1e9, 1e9), 0.0, 3)
    table = gainls.state_table(p.st_energy, p.st_J, p.st_jind, p.st_gamma, p.st_ndeg, p.st_ilevel)
    jobs = gainls.plan_pairs(filt, table)
    monkeypatch.setenv("GAINLS_GEMM1_BITS", "40")
    plan = gainls.Plan(eng, jobs)
    ps, js, st = plan.run()
    assert st == gainls.OK and all(j["inexact"] > 0 for j in js)
    for q, job in enumerate(jobs):
        one = eng.run_pair(*job, gainls.PATH_SPLIT)
        assert one["inexact"] == js[q]["inexact"]
        eng.run_pair(*job, gainls.PATH_PLAIN_FP64)
        ref = eng.fetch_amp().copy()
        N = p.blocks[(job[2], job[3])].vecs.shape[1]
        mrow = np.sqrt(15.0) * np.sqrt((p.dipole ** 2).sum(axis=(0, 1))).max()
        tol = (4 * np.sqrt(N) * 2.0 ** -48) * np.sqrt(N) * mrow + np.sqrt(N) * (3 * N + 64) * 2.0 ** -52 * mrow
        assert np.max(np.abs(plan.amp(q) - ref)) <= tol
    plan.close()


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols", [(1, 1), (100, 130), (129, 257), (300, 500), (520, 700), (700, 770)])
def test_any_number_of_items_gives_the_same_bits(built_lib, rows, cols, monkeypatch):
    """Inner lengths of two to four chunks and one to five items a unit, odd and even: the items
    alternate between the accumulators, and the last one of an odd number runs alone.  The residues
    are the same integers whatever the tiles, so every amplitude equals the whole block's bits."""
    import gainls
    import synth
    p = synth.make_problem(310, [5, 6], "c4", blocks=[(5, 0), (6, 1)])
    eng = gainls.Engine(JMAX, p.nsym, 1)
    gainls.upload_problem(eng, p)
    nI, nF = p.blocks[(0, 0)].vecs.shape[0], p.blocks[(1, 1)].vecs.shape[0]
    assert nI >= 700 and nF >= 2 * 384 + 1
    eng.run_pair(0, 0, 1, 1, np.arange(nI, dtype=np.int32), np.arange(nF, dtype=np.int32), gainls.PATH_SPLIT)
    whole = eng.fetch_amp().copy()
    lo, up = np.arange(rows, dtype=np.int32), np.arange(cols, dtype=np.int32)
    for pair in ("1", "0"):
        monkeypatch.setenv("GAINLS_GEMM_PAIR", pair)
        eng.run_pair(0, 0, 1, 1, lo, up, gainls.PATH_SPLIT)
        assert np.array_equal(eng.fetch_amp(), whole[:rows, :cols])


@pytest.mark.gpu
@pytest.mark.parametrize("order", ["all", "half", "reversed", "late"])
def test_upper_vectors_arriving_in_parts(built_lib, order, monkeypatch):
    """An asynchronous upload in several parts, the upper side run part by part
    (GAINLS_UPPER_HALVES=force: also when the copy has landed): leading states, in whole tiles,
    with each part; lists that do not ascend or lie in the last part wait for it.  The same bits as
    after one synchronous upload."""
    import torch
    import gainls
    import synth
    p = synth.make_problem(345, [5, 6], "c4", blocks=[(5, 0), (6, 1)])
    eng = gainls.Engine(JMAX, p.nsym, 1)
    gainls.upload_problem(eng, p)
    nI, vu = p.blocks[(0, 0)].vecs.shape[0], p.blocks[(1, 1)].vecs
    n = vu.shape[0]
    assert n >= 1024
    up = {"all": np.arange(n), "half": np.arange(0, n, 2), "reversed": np.arange(n)[::-1],
          "late": np.arange(n - 300, n)}[order].astype(np.int32)
    lo = np.arange(0, nI, 3, dtype=np.int32)
    eng.run_pair(0, 0, 1, 1, lo, up, gainls.PATH_SPLIT)
    one = eng.fetch_amp().copy()
    pin = torch.empty(vu.shape, dtype=torch.float64, pin_memory=True).numpy()
    pin[...] = vu
    monkeypatch.setenv("GAINLS_UPPER_HALVES", "force")
    eng.upload_eigvecs_async(1, 1, pin)
    st = eng.run_pair(0, 0, 1, 1, lo, up, gainls.PATH_SPLIT)
    assert st["kernel_launches"] == {"all": 16, "half": 12, "reversed": 10, "late": 10}[order]
    assert np.array_equal(eng.fetch_amp(), one)


@pytest.mark.gpu
@pytest.mark.parametrize("lead", [256, 512])
def test_a_run_returns_after_the_whole_asynchronous_copy(built_lib, lead):
    """Leading upper states that whole parts of an asynchronous upload hold: the run needs none of
    the rest, but the caller may change the vectors once it returns, so the rest (270 MB here,
    over a millisecond) has to be in place then."""
    import torch
    import gainls
    import synth
    p = synth.make_problem(345, [5, 6], "c4", blocks=[(5, 0), (6, 1)])
    eng = gainls.Engine(JMAX, p.nsym, 1)
    gainls.upload_problem(eng, p)
    nsize, n = p.blocks[(1, 1)].vecs.shape[1], 40000
    pin = torch.empty((n, nsize), dtype=torch.float64, pin_memory=True)
    pin.normal_(generator=torch.Generator().manual_seed(1))
    lo, tail = np.arange(3, dtype=np.int32), np.arange(n - 256, n, dtype=np.int32)
    up = np.arange(lead, dtype=np.int32)
    pin = pin.numpy()
    eng.upload_eigvecs(1, 1, pin)
    eng.run_pair(0, 0, 1, 1, lo, tail, gainls.PATH_SPLIT)
    want = eng.fetch_amp().copy()
    eng.run_pair(0, 0, 1, 1, lo, up, gainls.PATH_SPLIT)     # (the layout and buffers are there)
    eng.upload_eigvecs(1, 1, np.zeros_like(pin))
    eng.upload_eigvecs_async(1, 1, pin)
    eng.run_pair(0, 0, 1, 1, lo, up, gainls.PATH_SPLIT)
    pin[-64:] = 0.0
    eng.run_pair(0, 0, 1, 1, lo, tail, gainls.PATH_SPLIT)
    np.testing.assert_array_equal(eng.fetch_amp(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["c4", "c4r", "full", "c4m"])
def test_narrow_bands_keep_the_bits_of_their_digits(problems, name, monkeypatch):
    """First GEMMs of band widths below 960: their digits hold 8 x 7 = 56 bits of each operand, and
    the residue form holds as many, so a run without options is the run of 56 bits."""
    import gainls
    p, eng, (gI, gF) = problems[name]
    lo = np.arange(p.blocks[(0, gI)].vecs.shape[0], dtype=np.int32)
    up = np.arange(p.blocks[(1, gF)].vecs.shape[0], dtype=np.int32)
    dig = eng.run_pair(0, gI, 1, gF, lo, up, gainls.PATH_SPLIT, slices=6)
    assert dig["beta1"] * dig["slices1"] == 56
    st = eng.run_pair(0, gI, 1, gF, lo, up, gainls.PATH_SPLIT)
    amp = eng.fetch_amp().copy()
    monkeypatch.setenv("GAINLS_GEMM1_BITS", "56")
    want = eng.run_pair(0, gI, 1, gF, lo, up, gainls.PATH_SPLIT)
    assert st["slices1"] == want["slices1"] in (14, 15)
    assert np.array_equal(amp, eng.fetch_amp())


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["c4", "c4r"])
@pytest.mark.parametrize("bits", [56, 57, 62])
def test_more_bits_than_the_planes_hold_are_left_to_the_digits(problems, name, bits, monkeypatch):
    """GAINLS_GEMM1_BITS above 56: a run without options answers as one with a digit configuration
    does, here a refusal (9 x 7 or 8 x 8 bits do not fit the recombination), and a plan too."""
    import gainls
    p, eng, (gI, gF) = problems[name]
    lo, up = np.arange(5, dtype=np.int32), np.arange(7, dtype=np.int32)
    monkeypatch.setenv("GAINLS_GEMM1_BITS", str(bits))
    got = [eng.run_pair(0, gI, 1, gF, lo, up, gainls.PATH_SPLIT, raise_on_error=False, **kw)["status"]
           for kw in (dict(), dict(slices=6))]
    assert got[0] == got[1] == (gainls.OK if bits <= 56 else gainls.ERR_INVALID_ARG)
    for kw in (dict(), dict(slices=6)) if bits > 56 else ():
        with pytest.raises(gainls.GainError) as err:    # (a plan prepares its jobs when it is made)
            gainls.Plan(eng, [(0, gI, 1, gF, lo, up)], **kw)
        assert err.value.status == gainls.ERR_INVALID_ARG
