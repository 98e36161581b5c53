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
