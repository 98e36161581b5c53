"""Host vectors to and from the device through the handles' pinned buffers, where they could go wrong."""
import threading

import numpy as np
import pytest

from lionbolt_b200 import BatchSolver
from lionbolt_b200 import mesh as M
from lionbolt_b200 import problems as P

pytestmark = pytest.mark.gpu


def _large_problem(n, seed):
    """Fluxes of more than 4 MB, which go through a batch's shared buffers."""
    box = M.box_mesh(*n, (0, 0, 0), tuple(0.5 * v for v in n))
    k, w = P.quadrature(2, 4)
    r = np.random.default_rng(seed)
    return P.Problem("large", box, k, w, 2, 4, 1, 0, np.array([[0.3]]), np.array([[[[0.1]]]]), np.array([[0.2]]),
                     r.uniform(size=box.NENK), np.array([0.0, 0.0, 1.0]))


def test_threads_read_results_of_different_problems():
    """Each thread reads a problem of its own while another one does the same."""
    bs = BatchSolver()
    sizes = [(28, 28, 29), (29, 28, 28), (28, 29, 30)]
    for s, n in enumerate(sizes):
        bs.add_problem(_large_problem(n, s))
    bs.solve(m=10, rtol=1e-4)
    ref = [bs.results(p) for p in range(len(sizes))]
    bad = []

    def read(p):
        for _ in range(12):
            flux, dose = bs.results(p)
            if not (np.array_equal(flux, ref[p][0]) and np.array_equal(dose, ref[p][1])):
                bad.append(p)

    threads = [threading.Thread(target=read, args=(p,)) for p in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
