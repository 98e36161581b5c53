"""Batched dose solves (lb_batch_*): many independent problems with their own meshes, quadratures,
group counts and beams, solved together, must reproduce the single-problem solver and the FP64
oracle.  Tolerances: 1e-5 relative L2 against the oracle (the stated flux/dose target); against the
single-problem GPU solver the difference is only reduction order inside GMRES (1e-6)."""
import numpy as np
import pytest

import oracle as O
from helpers import rel_l2
from lionbolt_b200 import BatchSolver, MultigroupSolver
from lionbolt_b200 import problems as P

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _small_batch(count=5, seed=7):
    return P.batch_problems(count=count, seed=seed, hmin=3, hmax=6, groups=(1, 3), orders=(8, 12))


def test_batch_matches_single_problem_solver():
    probs = _small_batch()
    assert len({p.NI for p in probs}) > 1 and len({p.G for p in probs}) > 1   # mixed quadratures and groups
    bs = BatchSolver()
    ids = [bs.add_problem(p) for p in probs]
    it = bs.solve(m=20, rtol=1e-8)
    info = bs.info()
    assert info["problems"] == len(probs) and info["graph_launches"] > 0 and info["sweep_threads"] in (512, 1024)
    for pid, prob in zip(ids, probs):
        mg = MultigroupSolver().set_problem(prob)
        it1 = mg.solve("GMRES", m=20, rtol=1e-8)
        f1, d1 = mg.results()
        fb, db = bs.results(pid)
        assert np.all(it[pid, :prob.G] > 0) and np.all(it[pid, prob.G:] == 0)
        assert np.abs(it[pid, :prob.G] - it1).max() <= 1, (it[pid], it1)
        assert rel_l2(db, d1) < 1e-6, pid
        for g in range(prob.G):
            assert rel_l2(fb[g], f1[g]) < 1e-6, (pid, g)


def test_batch_matches_oracle():
    probs = _small_batch(count=3, seed=11)
    bs = BatchSolver()
    ids = [bs.add_problem(p) for p in probs]
    bs.solve(m=20, rtol=1e-8)
    for pid, prob in zip(ids, probs):
        o = O.Oracle(prob.mesh)
        assert o.set_angular(prob.k, prob.w, prob.Ls) == 0
        flux_ref, dose_ref, _ = o.multigroup(prob, "GMRES", m=20, rtol=1e-11)
        fb, db = bs.results(pid)
        assert rel_l2(db, dose_ref) < TOL, pid
        for g in range(prob.G):
            assert rel_l2(fb[g], flux_ref[g]) < TOL, (pid, g)


def test_batch_resolve_is_repeatable():
    probs = _small_batch(count=3, seed=5)
    bs = BatchSolver()
    for p in probs:
        bs.add_problem(p)
    it1 = bs.solve(m=10, rtol=1e-7)
    d1 = [bs.results(i)[1] for i in range(len(probs))]
    it2 = bs.solve(m=10, rtol=1e-7)
    d2 = [bs.results(i)[1] for i in range(len(probs))]
    assert np.array_equal(it1, it2)
    for a, b in zip(d1, d2):
        assert rel_l2(a, b) < 1e-12


def test_batch_info_before_and_after_the_first_solve():
    bs = BatchSolver()
    for p in _small_batch(count=2, seed=3):
        bs.add_problem(p)
    info = bs.info()
    assert info["problems"] == 2 and info["sweep_threads"] == 0 and info["sweep_launches"] == 0
    bs.solve(m=10, rtol=1e-4)
    info = bs.info()
    assert info["sweep_threads"] > 0 and info["sweep_launches"] > 0


def _walk_mesh(kind):
    """Meshes without tile types, by what their directions are walked by."""
    from helpers import jittered
    from lionbolt_b200 import mesh as M
    n = (6, 5, 7)
    box = M.box_mesh(*n, (0, 0, 0), (3.0, 2.5, 3.5), material=lambda c: np.minimum(c[:, 2] / 0.4375, 7).astype(np.int32), Nm=8)
    if kind == "type table":                 # 48 shape and material types: more than tiles have
        return box
    if kind == "split blocks":               # every element a shape of its own, blocks split on cycles
        return jittered(box, 0.035)
    if kind == "member table":               # elements in no order: blocks listed element by element
        p = np.random.default_rng(2).permutation(box.NE)
        node = box.node[p]
        return M.Mesh(rg=box.rg, node=node, neighbors=M.neighbours(node), mat=box.mat[p], Nm=8)
    node = box.node[:5]                      # fewer elements than a block has
    return M.Mesh(rg=box.rg, node=node, neighbors=M.neighbours(node), mat=box.mat[:5], Nm=8)


def _walk_problem(kind, seed):
    m = _walk_mesh(kind)
    k, w = P.quadrature(8, 10)
    r = np.random.default_rng(seed)
    st = r.uniform(0.2, 1.0, size=(1, 8))
    sigs = 0.8 * st[None, :, :, None] * 0.5 ** np.arange(2)
    return P.Problem(kind, m, k, w, 8, 10, 1, 1, st, sigs, 0.2 * st, r.uniform(size=m.NENK), np.array([0.0, 0.0, 1.0]))


def _check_against_single(probs, which):
    bs = BatchSolver()
    for p in probs:
        bs.add_problem(p)
    bs.solve(m=20, rtol=1e-7, maxit=200)
    for i in which:
        mg = MultigroupSolver().set_problem(probs[i])
        mg.solve("GMRES", m=20, rtol=1e-7, maxit=200)
        assert rel_l2(bs.results(i)[1], mg.results()[1]) < 1e-6


@pytest.mark.parametrize("count,team", [(2, 512), (4, 256), (8, 128)])
@pytest.mark.parametrize("kind", ["type table", "split blocks", "member table", "no blocks"])
def test_batched_walks_match_single_solves(kind, count, team, monkeypatch, capfd):
    """Every walk of the batched sweep, by teams of every size (80 directions a problem, 148 SMs): reduction order inside
    GMRES, 1e-6."""
    monkeypatch.setenv("LB_SWEEP_VERBOSE", "1")
    _check_against_single([_walk_problem(kind, s) for s in range(count)], (0, count - 1))
    assert f"block and level walk, {80 * count} directions" in (err := capfd.readouterr().err)
    assert f"teams of {team} threads" in err


def test_batch_of_tiled_and_other_problems_matches_single_solves(monkeypatch, capfd):
    """Two kernels share a sweep: problems with tile types and without, in turns."""
    monkeypatch.setenv("LB_SWEEP_VERBOSE", "1")
    probs = []
    for s, kind in enumerate(("type table", "split blocks", "member table", "no blocks")):
        probs += [_walk_problem(kind, s), P.multigroup_box(n=(4 + s, 4, 6), size=(2.0 + 0.5 * s, 2.0, 3.0), Ng=4, Nc=8, G=2,
                                                           Ls=2, seed=s, slab=(0.5, 1.5))]
    _check_against_single(probs, range(len(probs)))
    err = capfd.readouterr().err
    assert "block tiles, 128 directions" in err and "block and level walk, 320 directions" in err


@pytest.mark.parametrize("count,team", [(2, 512), (4, 256), (8, 128)])
def test_batched_tiles_run_the_teams_they_are_meant_to(count, team, monkeypatch, capfd):
    monkeypatch.setenv("LB_SWEEP_VERBOSE", "1")
    probs = [P.multigroup_box(n=(5, 4, 6), size=(2.5, 2.0, 3.0), Ng=8, Nc=10, G=1, Ls=2, seed=s, slab=(0.5, 1.5))
             for s in range(count)]
    _check_against_single(probs, (0, count - 1))
    err = capfd.readouterr().err
    assert f"block tiles, {80 * count} directions" in err and f"teams of {team} threads" in err
