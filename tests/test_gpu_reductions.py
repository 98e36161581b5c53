"""Krylov reductions on the GPU: block partials in rows without padding, summed on the host four columns at a time.  GMRES
whose basis grows past each multiple of four columns, against the FP64 oracle."""
import numpy as np
import pytest

import oracle as O
from helpers import rel_l2
from lionbolt_b200 import AngularClass, BoltzmannOp, XSType
from lionbolt_b200 import mesh as M
from lionbolt_b200 import problems as P

pytestmark = pytest.mark.gpu

TOL = 1e-5                       # as in the other solves; rtol 1e-8 and 1 / (1 - c) = 20 leave two orders of margin


# (restart lengths below 4 stagnate above this tolerance: a restart recomputes the residual with an FP32 sweep)
@pytest.mark.parametrize("m", [4, 5, 8, 15, 30])
def test_gmres_at_the_widths_of_its_partial_rows(m):
    box = M.box_mesh(5, 6, 5, (0, 0, 0), (10.0, 12.0, 10.0))
    k, w = P.quadrature(4, 8)
    sigt, sigs = np.array([1.0]), np.array([[0.95, 0.3]])
    o = O.Oracle(box)
    assert o.set_angular(k, w, 1) == 0
    o.set_xs(sigt, sigs)
    q = np.random.default_rng(4).uniform(size=box.NENK * len(w))
    ref, info = o.boltzmann_solve(q, "GMRES", m=30, rtol=1e-11)
    assert info["status"] == 0
    L = BoltzmannOp(m=m, rtol=1e-8, atol=0.0).Build(box, AngularClass(k=k, w=w), XSType(sigt, sigs))
    out = q.copy()
    L.MatInv(out, solver="GMRES")
    assert L.iters > 1
    assert rel_l2(out, ref) < TOL


def test_batch_with_more_blocks_than_the_reduction_buffers_start_with():
    """2,130 problems, a block each at least: rows of up to 19 values fit the pinned buffer (40,960 values), up to 30 the
    device buffer a handle starts with (65,536), and the full basis of 30 vectors needs a larger one.  Every problem is the
    same, so all results are the same, and they match the single-problem solver (the same Krylov steps to the rounding of
    the sums, 1e-6)."""
    from lionbolt_b200 import BatchSolver, MultigroupSolver
    box = M.box_mesh(4, 2, 2, (0, 0, 0), (80.0, 40.0, 40.0))
    k, w = P.quadrature(2, 4)
    sigs = np.array([[[[0.999 * 0.6 ** l for l in range(3)]]]])
    prob = P.Problem("thick", box, k, w, 2, 4, 1, 2, np.array([[1.0]]), sigs, np.array([[1.0]]),
                     np.random.default_rng(8).uniform(size=box.NENK), np.array([0.0, 0.0, 1.0]))
    mg = MultigroupSolver().set_problem(prob)
    one = mg.solve("GMRES", m=30, rtol=1e-5)
    assert one[0] > 31                                      # the first cycle fills its basis
    flux, dose = mg.results()
    bs = BatchSolver()
    count = 2130
    for _ in range(count):
        bs.add_problem(prob)
    it = bs.solve(m=30, rtol=1e-5)
    assert np.abs(it - one[0]).max() <= 1
    first = bs.results(0)
    assert rel_l2(first[0], flux) < 1e-6 and rel_l2(first[1], dose) < 1e-6
    for p in (1, count // 2, count - 1):
        assert np.array_equal(bs.results(p)[1], first[1])
    bs.close()
