"""The tile sweep (whole blocks moved through shared memory) on the GPU: the same numbers as the level
schedule, bit for bit, and the oracle's T^-1, at the sizes where its passes and rows change."""
import numpy as np
import pytest

import oracle as O
from helpers import rel_l2
from lionbolt_b200 import AngularClass, TransportOp, XSType
from lionbolt_b200 import mesh as M
from lionbolt_b200 import problems as P

pytestmark = pytest.mark.gpu

TOL = 1e-5                       # FP32 sweep against the FP64 oracle, as in the other sweep tests
LEVELS = 6                       # launch candidate: element levels, 512 threads
TILES = {24: "block tiles"}


def _two(c):
    return (c[:, 0] > 1.0).astype(np.int32)


# hexes per axis: one block; fewer blocks than a warp; a level just over one CTA pass of 128, 256 or 512
# threads (the widest block level of an n^3 box has about 3 n^2 / 4 blocks)
BOXES = [(1, 1, 1), (2, 1, 3), (5, 4, 3), (14, 14, 14), (19, 20, 18), (27, 28, 26)]


def _sweep(monkeypatch, cfg, m, k, w, sigt, q):
    monkeypatch.setenv("LB_SWEEP_CONFIG", str(cfg))
    T = TransportOp().Build(m, AngularClass(k=k, w=w), XSType(sigt, np.zeros((sigt.size, 1))))
    v = q.copy()
    T.MatInv(v)
    T.MatInv(v)                  # the second sweep reads what the first one wrote
    return T, v


@pytest.mark.parametrize("n", BOXES)
@pytest.mark.parametrize("cfg", sorted(TILES))
def test_tile_sweep_is_bit_identical_to_element_levels(cfg, n, monkeypatch):
    m = M.box_mesh(*n, (0, 0, 0), (2.0, 1.5, 2.5), material=_two, Nm=2)
    k, w = P.quadrature(2, 6)
    sigt = np.array([0.3, 1.7])
    q = np.random.default_rng(cfg).uniform(size=m.NENK * len(w))
    T, v = _sweep(monkeypatch, cfg, m, k, w, sigt, q)
    assert T._h.sweep_config()["schedule"] == TILES[cfg]
    _, ref = _sweep(monkeypatch, LEVELS, m, k, w, sigt, q)
    assert np.array_equal(v, ref)
    if m.NE < 5000:
        o = O.Oracle(m)
        assert o.set_angular(k, w, 0) == 0
        o.set_xs(sigt, np.zeros((2, 1)))
        assert rel_l2(v, o.transport_inv(o.transport_inv(q))) < TOL


def test_more_tile_types_than_a_slot_names_take_the_cluster_schedule(monkeypatch):
    """11 materials of 6 shapes give more than 32 tile types: the tile candidates run the cluster schedule instead."""
    m = M.box_mesh(11, 3, 3, (0, 0, 0), (11, 3, 3), material=lambda c: c[:, 0].astype(np.int32), Nm=11)
    k, w = P.quadrature(2, 4)
    sigt = np.linspace(0.1, 2.0, 11)
    q = np.random.default_rng(0).uniform(size=m.NENK * len(w))
    T, v = _sweep(monkeypatch, 24, m, k, w, sigt, q)
    assert T._h.sweep_config()["schedule"].startswith("cluster levels")
    assert np.array_equal(v, _sweep(monkeypatch, LEVELS, m, k, w, sigt, q)[1])


@pytest.mark.parametrize("n,quad,count", [((27, 26, 28), (2, 4), 1), ((19, 20, 18), (4, 8), 10), ((5, 4, 6), (8, 10), 8)])
def test_batched_tile_sweep_matches_single_solves(n, quad, count):
    """Batches whose groups suit teams of 512, 256 and 128 threads per direction (few wide directions, many
    middling ones, many small ones), against the single-problem solver (reduction order inside GMRES: 1e-6)."""
    from lionbolt_b200 import BatchSolver, MultigroupSolver
    probs = [P.multigroup_box(n=n, size=tuple(0.5 * v for v in n), Ng=quad[0], Nc=quad[1], G=1, Ls=2, seed=s,
                              slab=(0.5, 1.5)) for s in range(count)]
    bs = BatchSolver()
    for p in probs:
        bs.add_problem(p)
    bs.solve(m=20, rtol=1e-8)
    for i in {0, count - 1}:
        mg = MultigroupSolver().set_problem(probs[i])
        mg.solve("GMRES", m=20, rtol=1e-8)
        assert rel_l2(bs.results(i)[1], mg.results()[1]) < 1e-6


@pytest.mark.parametrize("amount", [0.0, 0.07])
def test_noalloc_sweep_runs_the_handles_schedule(amount):
    """lb_transport_inv_noalloc on a box (tiles) and on a jittered box (element levels before the autotuner's
    pick, the pick after it): the bits of TransportOp.MatInv, sources in FP32."""
    import ctypes
    import torch
    from helpers import jittered
    m = M.box_mesh(6, 5, 7, (0, 0, 0), (3.0, 2.5, 3.5), material=_two, Nm=2)
    if amount:
        m = jittered(m, amount)
    k, w = P.quadrature(4, 6)
    T = TransportOp().Build(m, AngularClass(k=k, w=w), XSType(np.array([0.3, 1.7]), np.zeros((2, 1))))
    q = np.random.default_rng(3).uniform(size=m.NENK * len(w)).astype(np.float32)

    def noalloc():
        d = torch.from_numpy(q).to("cuda:0")
        torch.cuda.synchronize()
        T._h.call("lb_transport_inv_noalloc", ctypes.c_void_p(d.data_ptr()))
        return d.cpu().numpy().astype(np.float64)

    first = noalloc()
    for _ in range(100):                 # until the autotuner has picked
        ref = q.astype(np.float64)
        T.MatInv(ref)
        if T._h.sweep_config() is not None:
            break
    assert T._h.sweep_config() is not None
    assert np.array_equal(first, ref) and np.array_equal(noalloc(), ref)


# meshes whose levels end before and after the passes of 256 and 512 elements; the smallest has levels of one
# element
RELAY_BOXES = [(1, 1, 1), (3, 2, 2), (9, 8, 10), (24, 25, 23)]


@pytest.mark.parametrize("amount", [0.0, 0.06])
@pytest.mark.parametrize("n", RELAY_BOXES)
@pytest.mark.parametrize("cfg", [25, 26, 27])
def test_level_relay_is_bit_identical_to_element_levels(cfg, n, amount, monkeypatch):
    from helpers import jittered
    m = M.box_mesh(*n, (0, 0, 0), tuple(0.5 * v for v in n), material=_two, Nm=2)
    if amount:
        m = jittered(m, amount)
    k, w = P.quadrature(2, 6)
    sigt = np.array([0.3, 1.7])
    q = np.random.default_rng(cfg).uniform(size=m.NENK * len(w))
    T, v = _sweep(monkeypatch, cfg, m, k, w, sigt, q)
    assert T._h.sweep_config()["schedule"] == ("resident level relay" if cfg == 27 and m.NE <= 14000 else "level relay")
    assert np.array_equal(v, _sweep(monkeypatch, LEVELS, m, k, w, sigt, q)[1])


@pytest.mark.parametrize("group", [1024, 700, 0])
def test_tile_sweep_with_several_passes_in_a_group(group, monkeypatch):
    """Groups of more units than the CTA has threads (levels of up to some 740 here): the second pass starts without a
    barrier, its last warps are part empty."""
    monkeypatch.setenv("LB_CLUSTER_GROUP", str(group))
    m = M.box_mesh(32, 32, 30, (0, 0, 0), (2.0, 1.5, 2.5), material=_two, Nm=2)
    k, w = P.quadrature(2, 6)
    sigt = np.array([0.3, 1.7])
    q = np.random.default_rng(group).uniform(size=m.NENK * len(w))
    T, v = _sweep(monkeypatch, 24, m, k, w, sigt, q)
    assert T._h.sweep_config()["schedule"] == "block tiles"
    assert np.array_equal(v, _sweep(monkeypatch, LEVELS, m, k, w, sigt, q)[1])


@pytest.mark.parametrize("cfg", [24, 25, 27])
@pytest.mark.parametrize("n", [(5, 4, 3), (15, 14, 16)])
def test_more_directions_than_resident_ctas(n, cfg, monkeypatch):
    """320 directions on 148 SMs with two CTAs each: CTAs walk a second direction with the tables and rows of the first
    still in place.  (The larger mesh does not fit the resident relay twice an SM.)"""
    m = M.box_mesh(*n, (0, 0, 0), (2.0, 1.5, 2.5), material=_two, Nm=2)
    k, w = P.quadrature(16, 20)
    sigt = np.array([0.3, 1.7])
    q = np.random.default_rng(cfg).uniform(size=m.NENK * len(w))
    T, v = _sweep(monkeypatch, cfg, m, k, w, sigt, q)
    assert T._h.sweep_config()["schedule"] in ("block tiles", "level relay", "resident level relay")
    assert np.array_equal(v, _sweep(monkeypatch, LEVELS, m, k, w, sigt, q)[1])
