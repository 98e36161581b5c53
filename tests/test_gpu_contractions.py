"""The tcgen05 contractions on the GPU against the FP64 oracle, at the shapes where their tensor-memory layout changes:
M2D with two A buffers, with one, and with the directions in two parts; D2M with four A stages and with fewer; node counts
that are no multiple of the 128-node tile, and several tiles per CTA."""
import ctypes

import numpy as np
import pytest

import oracle as O
from helpers import rel_l2
from lionbolt_b200 import AngularClass, ScatteringOp, XSType
from lionbolt_b200 import mesh as M
from lionbolt_b200 import problems as P

pytestmark = pytest.mark.gpu

TOL = 1e-5                       # split-BF16 contractions reproduce FP32, as in the other contraction tests

# (hexes per axis, polar, azimuthal, Legendre order)
SHAPES = [
    ((1, 1, 1), 2, 4, 1),        # a single ragged tile, 8 directions, 4 moments
    ((13, 14, 15), 4, 8, 1),     # 3 to 4 tiles per CTA, NM padded from 4 to 16
    ((3, 2, 5), 8, 28, 3),       # 224 directions at P3: the most with two A buffers
    ((13, 14, 15), 8, 30, 3),    # 240: one A buffer
    ((3, 2, 5), 16, 16, 3),      # 256: the first in two parts
    ((13, 14, 15), 12, 14, 2),   # 9 moments of 16
    ((13, 14, 15), 12, 24, 5),   # 288 at P5 in two parts of 144
    ((13, 14, 15), 8, 20, 7),    # 160 at P7: the most with two A buffers and 96-column A stages
    ((3, 2, 5), 8, 26, 7),       # 208: the most in one part
    ((13, 14, 15), 12, 18, 7),   # 216: in two parts
]


@pytest.mark.parametrize("n,Ng,Nc,L", SHAPES)
def test_contractions_at_the_edges_of_their_tensor_memory_layout(n, Ng, Nc, L):
    _check(n, Ng, Nc, L)


# M2D with A in shared memory, where A in tensor memory would take another part of the directions: one part instead of two,
# the most directions that one holds, two parts instead of three, and with per-thread moment loads where the ring does not fit
SHARED_A = [
    ((3, 2, 5), 12, 18, 5),      # 216 at P5: the fewest that take a part more
    ((13, 14, 15), 16, 16, 5),   # 256 at P5
    ((13, 14, 15), 12, 36, 5),   # 432 at P5 in two parts of 224, the second with fewer directions
    ((3, 2, 5), 16, 32, 7),      # 512 at P7: the most, all of it
    ((13, 14, 15), 12, 18, 7),   # 216 at P7
    ((3, 2, 5), 12, 20, 4),      # 240 at P4
    ((13, 14, 15), 16, 32, 1),   # 512 at P1
]


@pytest.mark.parametrize("n,Ng,Nc,L", SHARED_A)
def test_m2d_with_its_first_operand_in_shared_memory(n, Ng, Nc, L):
    _check(n, Ng, Nc, L)


def _check(n, Ng, Nc, L):
    torch = pytest.importorskip("torch")
    m = M.box_mesh(*n, (0, 0, 0), (2.0, 1.5, 2.5), material=lambda c: (c[:, 2] > 1.0).astype(np.int32), Nm=2)
    k, w = P.quadrature(Ng, Nc)
    sigt = np.array([0.3, 0.81])
    sigs = np.array([[0.27 * 0.7 ** l for l in range(L + 1)], [0.6 * 0.9 ** l for l in range(L + 1)]])
    o = O.Oracle(m)
    assert o.set_angular(k, w, L) == 0
    o.set_xs(sigt, sigs)
    x = np.random.default_rng(Ng * Nc + L).normal(size=m.NENK * len(w)).astype(np.float32)
    ref = o.scatter_apply(x.astype(np.float64))
    K = ScatteringOp().Build(m, AngularClass(k=k, w=w), XSType(sigt, sigs))
    lib, h = K._h.lib, K._h.h
    psi = torch.from_numpy(x).to("cuda:0")
    phi = torch.zeros((L + 1) ** 2 * m.NENK, dtype=torch.float64, device="cuda:0")
    out = torch.zeros_like(psi)
    torch.cuda.synchronize()
    assert lib.lb_d2m_device(h, ctypes.c_void_p(psi.data_ptr()), ctypes.c_void_p(phi.data_ptr())) == 0
    assert lib.lb_m2d_device(h, ctypes.c_void_p(phi.data_ptr()), ctypes.c_void_p(out.data_ptr())) == 0
    assert lib.lb_synchronize(h) == 0
    got = out.cpu().numpy().astype(np.float64).reshape(len(w), m.NENK)
    ref = ref.reshape(got.shape)
    assert rel_l2(got, ref) < TOL
    # no node tile and no direction is off by itself
    for t in range(0, m.NENK, 128):
        assert rel_l2(got[:, t:t + 128], ref[:, t:t + 128]) < 10 * TOL
    for d in range(len(w)):
        assert rel_l2(got[d], ref[d]) < 10 * TOL
