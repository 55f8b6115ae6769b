"""The residue form's planes take about twice the memory of the digits'.  Where they do not fit,
the run takes digits with the memory a digit run has: an allocation that fails at any point
(GAINLS_RESIDUE_BYTES limits the new memory of an attempt) leaves nothing behind."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

JMAX = 11
LIMITS = [0] + [(1 << k) + (1 << (k - 1)) * h for k in range(17, 28) for h in (0, 1)]


def _problem():
    import synth
    return synth.make_problem(120, [5, 6], "c4", blocks=[(5, 0), (6, 1)])


def _engine(p):
    import gainls
    eng = gainls.Engine(JMAX, p.nsym, 1)
    gainls.upload_problem(eng, p)
    return eng


def _job(p):
    return (0, 0, 1, 1, np.arange(p.blocks[(0, 0)].vecs.shape[0], dtype=np.int32),
            np.arange(p.blocks[(1, 1)].vecs.shape[0], dtype=np.int32))


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_pair_runs_on_digits_where_the_residue_planes_do_not_fit(built_lib, monkeypatch):
    """Limits from nothing to more than the attempt takes: every run gives the bits of a digit run or
    of the residue form, a digit run has the memory of one that never tried, and the same engine
    takes the residue form once there is room."""
    import gainls
    p = _problem()
    job = _job(p)
    _engine(p).run_pair(*job, gainls.PATH_SPLIT)    # (the context and the modules are loaded)

    def run(eng, **kw):
        st = eng.run_pair(*job, gainls.PATH_SPLIT, **kw)
        assert st["status"] == gainls.OK
        return st["products2"], eng.fetch_amp().copy()

    eng = _engine(p)
    before = _free()
    n_dig, digits = run(eng, slices=6)     # the digits a run without room takes
    used = before - _free()
    n_res, residues = run(eng)
    assert (n_dig, n_res) == (21, 13)
    del eng
    seen = set()
    for limit in LIMITS:
        eng = _engine(p)
        monkeypatch.setenv("GAINLS_RESIDUE_BYTES", str(limit))
        before = _free()
        n, amp = run(eng)
        seen.add(n)
        assert np.array_equal(amp, residues if n == n_res else digits)
        if n == n_dig:
            assert before - _free() <= used + (4 << 20)
            # a digit run, then another attempt, in what may be the same addresses; the outputs have
            # their place by now, so the attempt may succeed
            assert np.array_equal(run(eng, slices=6)[1], digits)
            n, amp = run(eng)
            assert np.array_equal(amp, residues if n == n_res else digits)
        monkeypatch.delenv("GAINLS_RESIDUE_BYTES")
        n, amp = run(eng)
        assert n == n_res and np.array_equal(amp, residues)
        del eng
    assert seen == {n_dig, n_res}


@pytest.mark.parametrize("rule,nv,jv", [("c4", 120, (5, 6)), ("c4m", 75, (3, 4))])
def test_a_form_is_chosen_with_room_for_its_outputs(built_lib, rule, nv, jv, monkeypatch):
    """Room for the planes but not for what is written next to them (the refinement lists of 2 x 32 MB
    are the last to be placed): digits, as without room for the planes."""
    import gainls
    import synth
    p = synth.make_problem(nv, list(jv), rule, blocks=[(jv[0], 0), (jv[1], 1)])
    job = _job(p)
    warm = _engine(p)
    warm.run_pair(*job, gainls.PATH_SPLIT, slices=6)
    digits = warm.fetch_amp().copy()
    eng = _engine(p)
    before = _free()
    assert eng.run_pair(*job, gainls.PATH_SPLIT)["products2"] == 13
    residues, used = eng.fetch_amp().copy(), before - _free()
    for short in (16 << 20, 48 << 20, 80 << 20):
        eng = _engine(p)
        monkeypatch.setenv("GAINLS_RESIDUE_BYTES", str(max(used - short, 0)))
        st = eng.run_pair(*job, gainls.PATH_SPLIT)
        assert st["status"] == gainls.OK and st["products2"] == 21
        assert np.array_equal(eng.fetch_amp(), digits)
        monkeypatch.delenv("GAINLS_RESIDUE_BYTES")
        assert eng.run_pair(*job, gainls.PATH_SPLIT)["products2"] == 13
        assert np.array_equal(eng.fetch_amp(), residues)


def test_plan_runs_on_digits_where_the_residue_planes_do_not_fit(built_lib, monkeypatch):
    """A digit run leaves its band planes with the block pair; a plan's attempt at the residue form
    then replaces them and fails at any of its allocations.  The plan runs on digits made anew:
    every job has the bits of a digit plan, or of the residue form where all of it fits."""
    import gainls
    import synth
    p = synth.make_problem(40, [1, 2, 3], "c4")
    filt = gainls.make_filters([1.0] * 4, p.isym_pairs, p.igamma_pair, p.sym_degen, (0.0, 5000.0), (-1e9, 1e9),
                               (-1e9, 1e9), 0.0, 3)
    table = gainls.state_table(p.st_energy, p.st_J, p.st_jind, p.st_gamma, p.st_ndeg, p.st_ilevel)
    jobs = gainls.plan_pairs(filt, table)

    def run(eng, **kw):
        plan = gainls.Plan(eng, jobs, **kw)
        ps, _, st = plan.run()
        amps = [plan.amp(q) for q in range(len(jobs))]
        plan.close()
        assert st == gainls.OK
        return ps["slices2"][0], amps

    def same(a, b):
        return all(np.array_equal(x, y) for x, y in zip(a, b))

    eng = _engine(p)
    n_dig, digits = run(eng, slices=6)
    n_res, residues = run(eng)
    assert (n_dig, n_res) == (6, 13)
    seen = set()
    for limit in LIMITS:
        eng = _engine(p)
        for job in jobs:
            eng.run_pair(*job, gainls.PATH_SPLIT, slices=6)
        monkeypatch.setenv("GAINLS_RESIDUE_BYTES", str(limit))
        n, amps = run(eng)
        monkeypatch.delenv("GAINLS_RESIDUE_BYTES")
        seen.add(n)
        assert same(amps, residues if n == n_res else digits)
        assert same(run(eng)[1], residues)
        del eng
    assert seen == {n_dig, n_res}


def test_adjoint_runs_on_digits_where_the_residue_form_does_not_fit(built_lib, monkeypatch):
    """The tensor-core adjoint at the same limits: the gradient of the FP64 chain to 1e-9 of its
    largest component (what either form is held to), and on digits the memory of one that never
    tried."""
    import gainls
    import synth
    p = synth.make_problem(75, [4, 5], "c4", blocks=[(4, 0), (5, 1)])
    job = _job(p)
    w = np.random.default_rng(5).standard_normal((len(job[4]), len(job[5])))
    g64 = _engine(p).adjoint(*job, w, np.zeros(p.dipole.size))

    def run(eng):     # (behind a plain run: the forward is not part of it)
        eng.run_pair(*job, gainls.PATH_PLAIN_FP64)
        g = eng.adjoint(*job, w, np.zeros(p.dipole.size), precision="split")
        assert np.max(np.abs(g - g64)) <= 1e-9 * np.abs(g64).max()
        return eng.last_adjoint_stats.tensor_flops

    before = _free()
    eng = _engine(p)
    f_res, used_res = run(eng), before - _free()
    del eng
    forms, used_dig = set(), None
    for limit in LIMITS + [used_res - (20 << 20)]:
        before = _free()
        eng = _engine(p)
        monkeypatch.setenv("GAINLS_RESIDUE_BYTES", str(limit))
        f, used = run(eng), before - _free()
        monkeypatch.delenv("GAINLS_RESIDUE_BYTES")
        if limit == 0:
            assert f != f_res
            f_dig, used_dig = f, used
        assert f in (f_dig, f_res)
        if f == f_dig:
            assert used <= used_dig + (4 << 20)
        forms.add(f)
        assert run(eng) == f_res
        del eng
    assert forms == {f_dig, f_res} and f == f_dig    # (the last limit ends in the list of 32 MB)
