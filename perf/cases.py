"""Performance cases of the transport-solve library: what its users run, through the public entry points.

A case is a dict of plain values.  Its "kind" names the call:

  dose         MultigroupSolver: new cross sections and beam into a kept solver (lb_mg_update_inputs),
               GMRES(20) to 1e-6 over all groups, fluence and dose back on the host
  batch        BatchSolver: several uneven dose problems solved together
  solve        BoltzmannOp.MatInv on a host angular vector (the reference's OpL%MatInv)
  matvec       BoltzmannOp.MatVec on a host angular vector
  transport    TransportOp.MatInv on a host angular vector (one sweep)
  application  one operator application on device arrays: M2D, sweep, D2M
  m2d, d2m     the two scattering contractions alone, on device arrays
  beam         first-collision data of a planar beam (ray walk through the mesh)
  gradient     loss and gradient of the learned preconditioner's network on host samples

Meshes are box meshes of nx x ny x nz hexes split into 6 tets (the benchmark's geometry, 0.5 cm hexes),
with "jitter" > 0 boxes whose interior nodes are moved, so that no two elements share a shape.  The
operator handle of a geometry (mesh, quadrature, sweep schedule, tuned launch shape) is what a user's
program keeps between solves: it is built once and shared by the states of the case; what differs from
state to state (cross sections, sources, beams, moments) enters with every pass.
"""
import ctypes
import math

import numpy as np
import torch

from lionbolt_b200 import AngularClass, BatchSolver, BoltzmannOp, MultigroupSolver, ScatteringOp, TransportOp, XSType
from lionbolt_b200 import mesh as M
from lionbolt_b200 import problems as P
from lionbolt_b200._lib import as_f64, dptr

CELL = 0.5          # hex edge (cm)
MESH_SEED = 20261203
RESTART, RTOL = 20, 1e-6


def listed():
    return [
        # the smallest complete solve (6,000 tets, 80 directions, one group, P3): launches and latency
        dict(name="dose_6k", kind="dose", nx=10, ny=10, nz=10, Ng=8, Nc=10, G=1, Ls=3, jitter=0.0),
        # an ordinary planning-sized solve with the benchmark's physics (96,000 tets, 288 directions, P5)
        dict(name="dose_96k", kind="dose", nx=20, ny=20, nz=40, Ng=12, Nc=24, G=4, Ls=5, jitter=0.0),
        # the benchmark's mesh and quadrature (768,000 tets, 288 directions, P5), its first groups
        dict(name="dose_768k", kind="dose", nx=40, ny=40, nz=80, Ng=12, Nc=24, G=3, Ls=5, jitter=0.0),
        # a mesh without repeated element shapes (as from a mesh generator), S12-like quadrature
        dict(name="dose_jittered_47k", kind="dose", nx=19, ny=18, nz=23, Ng=12, Nc=14, G=2, Ls=3, jitter=0.12),
        # independent problems of uneven size and quadrature solved together
        dict(name="batch_8", kind="batch", count=8, hmin=8, hmax=20, Gmax=4, mix=3),
        # the reference's within-group call on host vectors, small (6,000 tets, 80 directions)
        dict(name="solve_6k", kind="solve", nx=10, ny=10, nz=10, Ng=8, Nc=10, Ls=3, jitter=0.0),
        # one operator application on a host angular vector
        dict(name="matvec_25k", kind="matvec", nx=16, ny=15, nz=17, Ng=12, Nc=14, Ls=3, jitter=0.0),
        # one operator application on device arrays, ragged box, S8-like quadrature with many directions
        dict(name="application_58k", kind="application", nx=21, ny=19, nz=24, Ng=16, Nc=18, Ls=3, jitter=0.0),
        # the scattering contractions at the benchmark's size (3,072,000 nodes, 288 directions, P5)
        dict(name="m2d_768k", kind="m2d", nx=40, ny=40, nz=80, Ng=12, Nc=24, Ls=5, jitter=0.0),
        dict(name="d2m_768k", kind="d2m", nx=40, ny=40, nz=80, Ng=12, Nc=24, Ls=5, jitter=0.0),
        # ray-traced first-collision data of a slanted 5 x 5 cm beam (96,000 tets, 384,000 rays)
        dict(name="beam_96k", kind="beam", nx=20, ny=20, nz=40, Ng=4, Nc=8, width=5.0, tilt=15.0),
        # forward and backward of the per-cell network on a training batch
        dict(name="gradient_16k", kind="gradient", n=16384),
    ]


QUADRATURES = ((4, 8), (6, 12), (8, 10), (8, 16), (12, 14), (12, 24), (16, 18))


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("dose", "dose", "dose", "batch", "solve", "matvec", "transport", "application", "application",
                       "m2d", "d2m", "beam", "gradient"))
    if kind == "gradient":
        return dict(kind=kind, n=logint(200, 60000))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(3, 10), hmin=8, hmax=rng.randint(12, 22), Gmax=rng.randint(2, 5),
                    mix=rng.randrange(1000))
    # hexes per axis from the geometric mean and two aspect ratios
    top = {"dose": 36, "solve": 14, "matvec": 17, "transport": 17, "application": 34, "m2d": 40, "d2m": 40, "beam": 36}[kind]
    base = math.exp(rng.uniform(math.log(6), math.log(top)))
    a, b = rng.uniform(-0.35, 0.35), rng.uniform(-0.35, 0.35)
    n = [max(4, int(round(base * math.exp(t)))) for t in (a, b, -a - b)]
    c = dict(kind=kind, nx=n[0], ny=n[1], nz=n[2])
    if kind == "beam":
        c.update(Ng=4, Nc=8, width=round(rng.uniform(1.0, 8.0), 3), tilt=round(rng.uniform(0.0, 40.0), 2))
        return c
    c["Ng"], c["Nc"] = rng.choice(QUADRATURES)
    if kind == "dose":
        c["G"] = rng.randint(1, 3)
    c["Ls"] = rng.choice((1, 2, 3, 3, 4, 5, 5, 7) if kind in ("m2d", "d2m", "application") else (2, 3, 3, 5))
    c["jitter"] = 0.0 if kind in ("m2d", "d2m") or rng.random() < 0.7 else round(rng.uniform(0.02, 0.15), 3)
    return c


# ---- geometry and the operator a program keeps for it ------------------------------------------------
_kept = {}


def _keep(key, build):
    """The kept value of `key`; the values of other geometries are let go first."""
    if key not in _kept:
        for old in [k for k in _kept if k[0] != key[0]]:
            del _kept[old]
        _kept[key] = build()
    return _kept[key]


def _geo(case):
    return tuple(case.get(k) for k in ("nx", "ny", "nz", "Ng", "Nc", "jitter"))


def _base_problem(case):
    """The problem of a case before a seed changes its cross sections: the benchmark's physics (slab of a
    denser material, log-uniform cross sections, downscatter, beam 15 degrees off axis) on the case's box."""
    def build():
        n = (case["nx"], case["ny"], case["nz"])
        z = lambda t: CELL * round(t * n[2])
        slab = (z(0.125), max(z(0.175), z(0.125) + CELL))
        prob = P.multigroup_box(n=n, size=tuple(CELL * v for v in n), Ng=case["Ng"], Nc=case["Nc"], G=case.get("G", 1),
                                Ls=case.get("Ls", 3), seed=MESH_SEED, slab=slab, name="box")
        if case.get("jitter"):
            rg = prob.mesh.rg.copy()
            inner = np.all((rg > rg.min(axis=0) + 1e-9) & (rg < rg.max(axis=0) - 1e-9), axis=1)
            rg[inner] += CELL * case["jitter"] * np.random.default_rng(5).uniform(-1, 1, size=(int(inner.sum()), 3))
            m = prob.mesh
            prob.mesh = M.Mesh(rg=rg, node=m.node, neighbors=m.neighbors, mat=m.mat, Nm=m.Nm)
            s = prob.sigt[0]
            layers = [(0.0, slab[0], s[0]), (slab[0], slab[1], s[1]), (slab[1], CELL * n[2], s[0])]
            prob.unc = P.beam_uncollided(prob.mesh, prob.beam_dir, (0.5 * CELL * n[0], 0.5 * CELL * n[1]), (5.0, 5.0), layers)
        return prob
    return _keep((_geo(case), "problem", case.get("G", 1), case.get("Ls", 3)), build)


def _scaled(prob, seed):
    """Cross sections and beam of a seed: every group's scaled by a factor of its own (the scattering ratios
    stay), and the uncollided fluence exp(-tau) of the beam with group 0's factor."""
    f = np.exp(np.random.default_rng(seed).uniform(np.log(0.75), np.log(1.35), size=prob.G))
    return dict(sigt=as_f64(prob.sigt * f[:, None]), sigs=as_f64(prob.sigs * f[:, None, None, None]),
                dd=as_f64(prob.dd * f[:, None]), unc=as_f64(np.where(prob.unc > 0, np.abs(prob.unc) ** f[0], 0.0)),
                beam_dir=as_f64(prob.beam_dir))


def _within(prob, inp):
    """Within-group cross sections of the angular kinds: the group's transfer is the whole scattering."""
    sig = inp["sigt"][0]
    ls = np.arange(prob.Ls + 1)
    return as_f64(sig), as_f64(0.9 * sig[:, None] * 0.8 ** ls[None, :])


def _tuned(op, sweep):
    """Runs sweeps until the handle has picked its launch shape (its first sweeps time the candidates)."""
    for _ in range(200):
        if op._h.sweep_config() is not None:
            break
        sweep()
    return op


def _operator(cls, case):
    def build():
        prob = _base_problem(case)
        t, s = _within(prob, _scaled(prob, 0))
        kw = dict(m=RESTART, rtol=RTOL, atol=0.0) if cls is BoltzmannOp else {}
        op = cls(**kw).Build(prob.mesh, AngularClass(k=prob.k, w=prob.w), XSType(t, s))
        if cls in (BoltzmannOp, TransportOp):
            v = np.ones(prob.mesh.NENK * prob.NI)
            _tuned(op, lambda: (op.MatInv if cls is TransportOp else op.MatVec)(v.copy()))
        return op
    return _keep((_geo(case), cls.__name__, case.get("Ls", 3)), build)


def _solver(case):
    def build():
        mg = MultigroupSolver().set_problem(_base_problem(case))
        return _tuned(mg, lambda: mg.solve(m=RESTART, rtol=RTOL))
    return _keep((_geo(case), "mg", case["G"], case["Ls"]), build)


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _normal(shape, seed, scale=None, dtype=torch.float64):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    x = torch.randn(*shape, dtype=dtype, device="cuda", generator=g)
    return x if scale is None else x.mul_(scale)


def _moment_scale(Ls):
    """Flux moments fall off with their order: 0.8^l for the 2 l + 1 moments of order l."""
    return torch.tensor([0.8 ** l for l in range(Ls + 1) for _ in range(2 * l + 1)], dtype=torch.float64, device="cuda")[:, None]


def _batch_problems(case, seed):
    """Sizes, quadratures and beams from the case's mix; cross sections from the seed."""
    geo = np.random.default_rng(case["mix"])
    probs = [P.batch_problem(geo, i, hmin=case["hmin"], hmax=case["hmax"], groups=(1, case["Gmax"])) for i in range(case["count"])]
    for i, p in enumerate(probs):
        inp = _scaled(p, seed * 64 + i)
        p.sigt, p.sigs, p.dd, p.unc = inp["sigt"], inp["sigs"], inp["dd"], inp["unc"]
    return probs


def _beam(case):
    """Beam plane 2 cm before the box, tilted in the x-z plane, aimed at the centre of the z = 0 face."""
    t = math.radians(case["tilt"])
    axis = np.array([math.sin(t), 0.0, math.cos(t)])
    e1 = np.array([math.cos(t), 0.0, -math.sin(t)])
    e2 = np.array([0.0, 1.0, 0.0])
    sx, sy = CELL * case["nx"], CELL * case["ny"]
    # far enough back that the whole plane of the field lies before the mesh
    back = 2.0 + math.tan(t) * (sx + sy)
    origin = np.array([0.5 * sx, 0.5 * sy, 0.0]) - back * axis
    return origin, axis, e1, e2


def _samples(n, seed):
    r = np.random.default_rng(seed)
    x = r.standard_normal((n, 19)).astype(np.float32)
    x[:, 16:] = r.uniform(0.01, 1.0, size=(n, 3)).astype(np.float32)
    t = (0.3 * r.standard_normal((n, 16))).astype(np.float32)
    w = r.uniform(0.1, 1.0, size=n).astype(np.float32)
    p = np.concatenate([(r.uniform(-1, 1, size=a * b) * math.sqrt(3.0 / b)).astype(np.float32) if b else
                        (0.05 * r.standard_normal(a)).astype(np.float32)
                        for a, b in ((64, 19), (64, 0), (64, 64), (64, 0), (16, 64), (16, 0))])
    return x, t, w, p


def prepare(case, seed):
    kind = case["kind"]
    if kind == "gradient":
        x, t, w, p = _samples(case["n"], seed)
        op = TransportOp().lp_set_weights(p)
        return dict(kind=kind, op=op, x=x, t=t, w=w)
    if kind == "batch":
        probs = _batch_problems(case, seed)
        bs = BatchSolver()
        for p in probs:
            bs.add_problem(p)
        return dict(kind=kind, bs=bs, n=len(probs))
    if kind == "beam":
        prob = _base_problem(case)
        op = _operator(ScatteringOp, case)
        sig = np.random.default_rng(seed).uniform(0.02, 0.5) * np.array([1.0, 2.7])
        return dict(kind=kind, op=op, beam=_beam(case), width=case["width"], attn=as_f64(sig[:prob.mesh.Nm]))
    prob = _base_problem(case)
    inp = _scaled(prob, seed)
    if kind == "dose":
        return dict(kind=kind, mg=_solver(case), inp=inp)
    NENK, NI, nm = prob.mesh.NENK, prob.NI, (case["Ls"] + 1) ** 2
    if kind in ("solve", "matvec", "transport"):
        q = np.random.default_rng(seed).uniform(size=NENK * NI)
        op = _operator(TransportOp if kind == "transport" else BoltzmannOp, case)
        return dict(kind=kind, op=op, xs=XSType(*_within(prob, inp)), q=q, v=np.empty_like(q))
    s = dict(kind=kind, op=_operator(ScatteringOp, case))
    if kind in ("m2d", "application"):
        s["phi"] = _normal((nm, NENK), seed, _moment_scale(case["Ls"]))
        s["psi"] = torch.empty(NI, NENK, dtype=torch.float32, device="cuda")
    else:
        s["psi"] = _normal((NI, NENK), seed, dtype=torch.float32)
    if kind in ("d2m", "application"):
        s["out"] = torch.empty(nm, NENK, dtype=torch.float64, device="cuda")
    return s


def run(s):
    kind = s["kind"]
    if kind == "dose":
        i, mg = s["inp"], s["mg"]
        mg._h.call("lb_mg_update_inputs", dptr(i["sigt"]), dptr(i["sigs"]), dptr(i["dd"]), dptr(i["unc"]), dptr(i["beam_dir"]))
        mg.solve(m=RESTART, rtol=RTOL)
        flux, dose = mg.results()
        return dict(flux=flux, dose=dose)
    if kind == "batch":
        s["bs"].solve(m=RESTART, rtol=RTOL)
        return [s["bs"].results(p) for p in range(s["n"])]
    op = s["op"]
    if kind == "gradient":
        loss, g = op.lp_loss_grad(s["x"], s["t"], s["w"])
        return dict(loss=np.float32(loss), grad=g)      # both are sums of 32-bit terms
    if kind == "beam":
        return op.beam_uncollided(*s["beam"], s["width"], s["width"], s["attn"])
    if kind in ("solve", "matvec", "transport"):
        op.set_xs(s["xs"])
        np.copyto(s["v"], s["q"])    # the operators work in place
        return (op.MatVec if kind == "matvec" else op.MatInv)(s["v"])
    h = op._h
    if kind == "d2m":
        h.call("lb_d2m_device", _ptr(s["psi"]), _ptr(s["out"]))
        return s["out"]
    h.call("lb_m2d_device", _ptr(s["phi"]), _ptr(s["psi"]))
    if kind == "m2d":
        return s["psi"]
    h.call("lb_transport_inv_noalloc", _ptr(s["psi"]))
    h.call("lb_d2m_device", _ptr(s["psi"]), _ptr(s["out"]))
    return dict(psi=s["psi"], phi=s["out"])


def work(case):
    kind = case["kind"]
    if kind == "gradient":
        n, par = case["n"], 6480
        return dict(bytes=4.0 * n * (19 + 16 + 1) + 8.0 * par, flops=6.0 * n * par)
    if kind == "batch":
        tot = dict(bytes=0.0, flops=0.0)
        geo = np.random.default_rng(case["mix"])
        for i in range(case["count"]):
            p = P.batch_problem(geo, i, hmin=case["hmin"], hmax=case["hmax"], groups=(1, case["Gmax"]))
            w = _dose_work(p.mesh.NENK, p.NI, p.nm, p.G)
            tot = {k: tot[k] + w[k] for k in tot}
        return tot
    NENK = 24 * case["nx"] * case["ny"] * case["nz"]
    NI, nm = case["Ng"] * case["Nc"], (case.get("Ls", 3) + 1) ** 2
    if kind == "beam":
        # every element's 4 nodes read and its 4 values written; a face-plane test per face of a crossed tet
        return dict(bytes=NENK * (8.0 + 4.0 + 8.0), flops=NENK * 40.0)
    if kind == "dose":
        return _dose_work(NENK, NI, nm, case["G"])
    gemm = 2.0 * NENK * NI * nm
    upd = 60.0 / 4.0 * NENK * NI      # about 60 operations per element and direction of a sweep
    if kind == "m2d":
        return dict(bytes=NENK * (8.0 * nm + 4.0 * NI), flops=gemm)
    if kind == "d2m":
        return dict(bytes=NENK * (8.0 * nm + 4.0 * NI), flops=gemm)
    if kind == "application":
        return dict(bytes=NENK * (16.0 * nm + 4.0 * NI), flops=2 * gemm + upd)
    # host angular vectors: FP64 in and out
    calls = dict(transport=0, matvec=1, solve=3)[kind]
    return dict(bytes=16.0 * NENK * NI, flops=calls * 2 * gemm + max(1, calls) * upd)


def _dose_work(NENK, NI, nm, G):
    """A group takes at least its right-hand side, the initial residual and two Arnoldi steps: four
    applications, each with one pass over the angular vector (read and written) and one moment vector in
    and out; the fluence and dose come back."""
    app = NENK * (8.0 * NI + 16.0 * nm)
    return dict(bytes=G * 4 * app + 8.0 * NENK * (G + 1), flops=G * 4 * NENK * NI * (4.0 * nm + 15.0))


# ---- the same results in 64 bits, from the equations -------------------------------------------------
def _harmonics(Ls, k):
    """Real orthonormal spherical harmonics Y[i][l l + l + m] (cosines for m > 0, sines for m < 0)."""
    ct = k[:, 2]
    st = np.sqrt(np.maximum(0.0, 1 - ct * ct))
    ph = np.arctan2(k[:, 1], k[:, 0])
    leg = {(0, 0): np.ones_like(ct)}
    for m in range(1, Ls + 1):
        leg[m, m] = leg[m - 1, m - 1] * (2 * m - 1) * st
    for m in range(Ls):
        leg[m + 1, m] = (2 * m + 1) * ct * leg[m, m]
    for m in range(Ls + 1):
        for l in range(m + 2, Ls + 1):
            leg[l, m] = ((2 * l - 1) * ct * leg[l - 1, m] - (l + m - 1) * leg[l - 2, m]) / (l - m)
    Y = np.zeros((len(k), (Ls + 1) ** 2))
    for l in range(Ls + 1):
        for m in range(-l, l + 1):
            a = abs(m)
            c = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - a) / math.factorial(l + a))
            t = 1.0 if m == 0 else math.sqrt(2.0) * (np.cos(a * ph) if m > 0 else np.sin(a * ph))
            Y[:, l * l + l + m] = c * leg[l, a] * t
    return Y


FACES = ((0, 1, 2), (0, 1, 3), (0, 2, 3), (1, 2, 3))


class _Transport64:
    """T^-1 of the linear-DG upwind discretisation on tetrahedra in FP64, all directions at once, level by
    level of the upwind order.  With c_f = k . n_f A_f / V, mass-eliminated element system
      r_k = q_k - sum over inflow faces of c_f P_f psi_up,  T = sigma I - convection + outflow faces,
      P_f(k,k') = 2 (k = k' in f), 1/3 (k in f, k' in f), -4/3 (k not in f, k' in f)."""

    def __init__(self, mesh, k, w, Ls):
        dev = "cuda"
        rg, node = torch.tensor(mesh.rg, device=dev), torch.tensor(mesh.node.astype(np.int64), device=dev)
        self.NE, self.NI, self.Ls = mesh.NE, len(k), Ls
        NE, NI = self.NE, self.NI
        X = rg[node]                                                        # [NE, 4, 3]
        vol = torch.linalg.det(X[:, 1:] - X[:, :1]).abs() / 6
        S = torch.empty(NE, 4, 3, dtype=torch.float64, device=dev)
        for f, (a, b, c) in enumerate(FACES):
            n = torch.linalg.cross(X[:, b] - X[:, a], X[:, c] - X[:, a]) / 2
            s = torch.sign((n * (X[:, a] - X.mean(dim=1))).sum(1, keepdim=True))
            S[:, f] = s * n / vol[:, None]
        nrm = S / S.norm(dim=2, keepdim=True)
        K = torch.tensor(np.asarray(k, dtype=np.float64), device=dev)
        self.k, self.S, self.mat = K, S, torch.tensor(mesh.mat.astype(np.int64), device=dev)
        self.nbr = torch.tensor(mesh.neighbors.astype(np.int64), device=dev)
        # local index, in the neighbour, of each node of each face
        self.perm = torch.zeros(NE, 4, 3, dtype=torch.int64, device=dev)
        back = torch.zeros(NE, 4, dtype=torch.int64, device=dev)
        for f, nodes in enumerate(FACES):
            nb = self.nbr[:, f].clamp(min=0)
            for j, a in enumerate(nodes):
                self.perm[:, f, j] = (node[nb] == node[:, a:a + 1]).to(torch.int64).argmax(dim=1)
            back[:, f] = (self.nbr[nb] == torch.arange(NE, device=dev)[:, None]).to(torch.int64).argmax(dim=1)
        # upwind levels of all (direction, element) pairs
        up = torch.zeros(NI, NE, dtype=torch.uint8, device=dev)
        out = torch.zeros(NI, NE, dtype=torch.uint8, device=dev)
        for f in range(4):
            kn = K @ nrm[:, f].T
            up |= ((kn < -2.220446049250313e-16) & (self.nbr[:, f] >= 0)[None, :]).to(torch.uint8) << f
            out |= (~(kn < 0)).to(torch.uint8) << f
        self.up, self.out = up.reshape(-1), out.reshape(-1)
        cnt = sum(((self.up >> f) & 1).to(torch.int32) for f in range(4))
        cur = torch.nonzero(cnt == 0).reshape(-1)
        self.levels = []
        one = torch.ones(1, dtype=torch.int32, device=dev)
        while cur.numel():
            self.levels.append(cur.to(torch.int32))
            e, base = cur % NE, cur - cur % NE
            nxt = []
            for f in range(4):
                nb = self.nbr[e, f]
                to = base + nb.clamp(min=0)
                hit = (nb >= 0) & (((self.up[to] >> back[e, f].to(torch.uint8)) & 1) == 1)
                to = to[hit]
                cnt.index_add_(0, to, -one.expand(to.numel()))
                nxt.append(to)
            nxt = torch.unique(torch.cat(nxt))
            cur = nxt[cnt[nxt] == 0]
        Y = torch.tensor(_harmonics(Ls, np.asarray(k)), device=dev)
        self.Y, self.D = Y, (Y * torch.tensor(np.asarray(w), device=dev)[:, None]).T.contiguous()
        self.lofj = torch.tensor([l for l in range(Ls + 1) for _ in range(2 * l + 1)], device=dev)

    def sweep(self, q, sigt):
        """T^-1 q for q [NI, NENK], in place."""
        NE = self.NE
        psi = q.reshape(-1, 4)
        sig = torch.tensor(np.asarray(sigt), device="cuda")
        for lev in self.levels:
            for idx in lev.split(4_000_000):
                idx = idx.to(torch.int64)
                e = idx % NE
                base = idx - e
                c = (self.k[idx // NE][:, None, :] * self.S[e]).sum(2)                # [n, 4]
                up, out = self.up[idx], self.out[idx]
                r = psi[idx].clone()
                co = torch.zeros_like(c)
                for f, nodes in enumerate(FACES):
                    on = ((up >> f) & 1).to(torch.float64)
                    u = psi[base + self.nbr[e, f].clamp(min=0)].gather(1, self.perm[e, f])   # [n, 3]
                    t = on * c[:, f]
                    U = u.sum(1)
                    for j, a in enumerate(nodes):
                        r[:, a] -= t * (5.0 / 3.0 * u[:, j] + U / 3.0)
                    r[:, 3 - f] += t * 4.0 / 3.0 * U
                    co[:, f] = ((out >> f) & 1).to(torch.float64) * c[:, f]
                # T = d I + a 1^T + 1 b^T, inverted through its 2 x 2 capacitance matrix
                Ct = co.sum(1, keepdim=True)
                d = sig[self.mat[e]][:, None] + 5.0 / 3.0 * Ct
                a = 5.0 / 3.0 * (c - co).flip(1)
                b = (Ct - co.flip(1)) / 3.0
                e00, e11 = d[:, 0] + a.sum(1), d[:, 0] + b.sum(1)
                ba = (a * b).sum(1)
                v0, v1 = r.sum(1), (b * r).sum(1)
                det = e00 * e11 - 4.0 * ba
                z0 = (e11 * v0 - 4.0 * v1) / det
                z1 = (e00 * v1 - ba * v0) / det
                psi[idx] = (r - a * z0[:, None] - z1[:, None]) / d
        return q

    def sigma(self, sigs, phi):
        """Sigma phi: moment j times sigma_l(j) of every node's material; sigs [Nm][Ls + 1]."""
        s = torch.tensor(np.asarray(sigs), device="cuda")[self.mat][:, self.lofj].T       # [nm, NE]
        return (phi.reshape(phi.shape[0], self.NE, 4) * s[:, :, None]).reshape(phi.shape)

    def m2d(self, mom):
        return self.Y @ mom

    def d2m(self, psi):
        return self.D @ psi

    def solve(self, b, sigt, sigs, tol=1e-11, most=60):
        """phi of (I - D T^-1 M Sigma) phi = b by GMRES without restarts."""
        op = lambda x: x - self.d2m(self.sweep(self.m2d(self.sigma(sigs, x)), sigt))
        beta = float(b.norm())
        V, H = [b / beta], np.zeros((most + 1, most))
        for j in range(most):
            w = op(V[j])
            for _ in range(2):
                for i, v in enumerate(V):
                    t = float((v * w).sum())
                    H[i, j] += t
                    w = w - t * v
            H[j + 1, j] = float(w.norm())
            g = np.zeros(j + 2)
            g[0] = beta
            y = np.linalg.lstsq(H[:j + 2, :j + 1], g, rcond=None)[0]
            if np.linalg.norm(H[:j + 2, :j + 1] @ y - g) <= tol * beta:
                break
            V.append(w / H[j + 1, j])
        return sum(float(t) * v for t, v in zip(y, V))


def _dose64(mesh, k, w, Ls, sigt, sigs, dd, unc, beam_dir):
    T = _Transport64(mesh, k, w, Ls)
    dev = "cuda"
    u = torch.tensor(unc, device=dev)
    yb = torch.tensor(_harmonics(Ls, np.asarray(beam_dir)[None, :])[0], device=dev)
    first = yb[:, None] * u[None, :]
    node_mat = T.mat.repeat_interleave(4)
    phis, flux, dose = [], [], torch.zeros_like(u)
    for g in range(sigt.shape[0]):
        src = T.sigma(sigs[0, g], first)
        for gp in range(g):
            src = src + T.sigma(sigs[gp, g], phis[gp])
        b = T.d2m(T.sweep(T.m2d(src), sigt[g]))
        phis.append(T.solve(b, sigt[g], sigs[g, g]))
        fl = math.sqrt(4 * math.pi) * phis[-1][0] + (u if g == 0 else 0.0)
        flux.append(fl)
        dose += torch.tensor(dd[g], device=dev)[node_mat] * fl
    return torch.stack(flux).cpu().numpy(), dose.cpu().numpy()


def _beam64(mesh, case, attn):
    """exp(-tau) of the straight ray from each of the 4 quadrature points of an element to the beam plane,
    tau from the lengths inside the box and inside its slab layer, projected onto the linear basis."""
    origin, axis, e1, e2 = _beam(case)
    a, b = (5 + 3 * math.sqrt(5)) / 20, (5 - math.sqrt(5)) / 20
    Q = np.einsum("qk,ekd->eqd", np.full((4, 4), b) + (a - b) * np.eye(4), mesh.rg[mesh.node])
    u = Q - origin
    inside = (np.abs(u @ e1) <= 0.5 * case["width"]) & (np.abs(u @ e2) <= 0.5 * case["width"])
    lo, hi = mesh.rg.min(axis=0), mesh.rg.max(axis=0)
    length = u @ axis
    d = -axis
    far = np.full(length.shape, np.inf)            # distance at which the ray leaves the box
    for i in range(3):
        if abs(d[i]) > 1e-14:
            far = np.minimum(far, ((hi[i] if d[i] > 0 else lo[i]) - Q[..., i]) / d[i])
    far = np.minimum(far, length)
    slab = mesh.centroids()[mesh.mat == 1][:, 2]
    h = CELL
    z0, z1 = math.floor(slab.min() / h) * h, math.ceil(slab.max() / h) * h
    zend = Q[..., 2] + far * d[2]
    in_slab = np.clip(np.minimum(Q[..., 2], z1) - np.maximum(zend, z0), 0.0, None) / abs(d[2])
    tau = attn[0] * (far - in_slab) + attn[1] * in_slab
    phi = np.where(inside, np.exp(-tau), 0.0)
    return (math.sqrt(5) * phi + 0.25 * (1 - math.sqrt(5)) * phi.sum(axis=1, keepdims=True)).ravel()


def _gradient64(x, t, w, p):
    p = torch.tensor(p.astype(np.float64), requires_grad=True)
    part = torch.split(p, [64 * 19, 64, 64 * 64, 64, 16 * 64, 16])
    a = torch.tensor(x.astype(np.float64))
    for W, b, rows in ((part[0], part[1], 64), (part[2], part[3], 64)):
        a = torch.relu(a @ W.reshape(rows, -1).T + b)
    y = a @ part[4].reshape(16, 64).T + part[5]
    loss = (torch.tensor(w.astype(np.float64))[:, None] * (y - torch.tensor(t.astype(np.float64))) ** 2).sum() / (2 * len(x))
    loss.backward()
    return float(loss.detach()), p.grad.numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "gradient":
        loss, g = _gradient64(*_samples(case["n"], seed))
        return dict(loss=np.float64(loss), grad=g)
    if kind == "batch":
        return [_dose64(p.mesh, p.k, p.w, p.Ls, p.sigt, p.sigs, p.dd, p.unc, p.beam_dir) for p in _batch_problems(case, seed)]
    prob = _base_problem(case)
    m = prob.mesh
    if kind == "beam":
        sig = np.random.default_rng(seed).uniform(0.02, 0.5) * np.array([1.0, 2.7])
        return _beam64(m, case, sig)
    # the device kinds keep the operator's cross sections (seed 0) from call to call
    inp = _scaled(prob, seed if kind in ("dose", "solve", "matvec", "transport") else 0)
    if kind == "dose":
        if m.NE * prob.NI * prob.G > 120e6:
            return None                     # minutes of 64-bit sweeps
        flux, dose = _dose64(m, prob.k, prob.w, prob.Ls, inp["sigt"], inp["sigs"], inp["dd"], inp["unc"], inp["beam_dir"])
        return dict(flux=flux, dose=dose)
    sigt, sigs = _within(prob, inp)
    NENK, NI, nm = m.NENK, prob.NI, prob.nm
    lofj = np.array([l for l in range(prob.Ls + 1) for _ in range(2 * l + 1)])
    if kind in ("m2d", "d2m"):
        Y = torch.tensor(_harmonics(prob.Ls, prob.k), device="cuda")
        if kind == "d2m":
            psi = _normal((NI, NENK), seed, dtype=torch.float32)
            D = (Y * torch.tensor(prob.w, device="cuda")[:, None]).T.contiguous()
            return torch.cat([D @ c.double() for c in psi.split(1 << 18, dim=1)], dim=1)
        phi = _normal((nm, NENK), seed, _moment_scale(prob.Ls))
        phi *= torch.tensor(sigs[m.mat][:, lofj].T.copy(), device="cuda").repeat_interleave(4, dim=1)
        return Y @ phi
    T = _Transport64(m, prob.k, prob.w, prob.Ls)
    if kind == "application":
        psi = T.sweep(T.m2d(T.sigma(sigs, _normal((nm, NENK), seed, _moment_scale(prob.Ls)))), sigt)
        return dict(psi=psi, phi=T.d2m(psi))
    q = torch.tensor(np.random.default_rng(seed).uniform(size=NENK * NI), device="cuda").reshape(NI, NENK)
    if kind == "transport":
        return T.sweep(q, sigt).reshape(-1)
    if kind == "matvec":
        return (q - T.sweep(T.m2d(T.sigma(sigs, T.d2m(q))), sigt)).reshape(-1)
    b = T.d2m(T.sweep(q.clone(), sigt))
    phi = T.solve(b, sigt, sigs)
    return T.sweep(T.m2d(T.sigma(sigs, phi)) + q, sigt).reshape(-1)
