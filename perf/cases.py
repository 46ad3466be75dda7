"""Workloads the engine is timed on, through its public Python entry points.

Each case is one call sequence that a program using the engine makes again and
again; `listed()` holds the ones that are followed over time and `draw()` gives
others of the same ranges.  The fields of a case:

  kind       "host"   MechSystemSolver.backwardEulerHost: the host keeps x and v
                      in page-locked arrays and makes one call per time step
             "run"    setState, `steps` BackwardEuler steps, getState
             "update" updateStressAndStiffness with the scalar CRS values, what
                      a host with its own direct solver calls every step
             "pack"   FemPack of uneven beams: setStates, setActive when only a
                      share of the models has work, backwardEuler, getStates
  elem       "tet", "hex" or "quadtet" (ten-node tetrahedra)
  material   "linear" (corotated), "neo" (NeoHookean) or "mooney" (MooneyRivlin,
             soft incompressibility AUTO, which is NODAL on these meshes)
  nx, ny, nz grid cells;  steps, h, tol: the time integration
  mixed      FP32 tangent and matrix, FP64 forces and PCG vectors
  models, sizes_seed, large, active, refine: packs (number of beams, the draw of
             their sizes, the share of long ones, the share with work, sweeps)

Mixed-precision cases take one step per pass: their FP32 tangent rounds the
positions, so a last-bit difference of one step's result moves the next step's
matrix by FP32 round-off and longer runs can only be compared at that level.
"""
import math

import numpy as np
import torch

from artisynth_core_b200 import _lib as L
from artisynth_core_b200.femmodel import (FemModel3d, FemPack, LinearMaterial, MechSystemSolver,
                                          MooneyRivlinMaterial, NeoHookeanMaterial)

ELEM = {"tet": L.ELEM_TET, "hex": L.ELEM_HEX, "quadtet": L.ELEM_QUADTET}
# material parameters, box of the mesh (m) and fixed face of the single models
LINEAR = dict(E=1e5, nu=0.33)
NEO = dict(E=5e4, nu=0.45)
MOONEY = dict(c10=1000.0, c01=500.0, kappa=1e5)
GRAVITY = (0.0, 0.0, -9.81)
ALPHA = 2.0  # mass damping (the engine's default); stiffness damping stays 0


def _single(name, kind, elem, material, nx, ny, nz, steps=1, h=0.005, tol=1e-10, mixed=False):
    return dict(name=name, kind=kind, elem=elem, material=material, nx=nx, ny=ny, nz=nz, steps=steps, h=h, tol=tol,
                mixed=mixed)


def _pack(name, models, sizes_seed, large=0.0, active=1.0, refine=0, mixed=True, steps=1, tol=1e-10):
    return dict(name=name, kind="pack", elem="tet", material="neo", models=models, sizes_seed=sizes_seed, large=large,
                active=active, refine=refine, mixed=mixed, steps=steps, h=0.01, tol=tol)


def listed():
    return [
        # the smallest call: a 200-tet corotated beam, one step from host state (interactive simulation)
        _single("tet_beam_linear_step", "host", "tet", "linear", 10, 2, 2, h=0.01, tol=1e-12),
        # a small non-linear beam stepped ten times (the size of the equivalence tests)
        _single("tet_beam_small_run", "run", "tet", "neo", 6, 3, 2, steps=10, tol=1e-12),
        # the benchmark's hex beam, one step per call from host state, and the same beam left to run
        _single("hex_beam_step", "host", "hex", "neo", 40, 10, 10),
        _single("hex_beam_run", "run", "hex", "neo", 40, 10, 10, steps=20),
        # forces, stiffness blocks and CRS values of that beam for the host's direct solver
        _single("hex_beam_update", "update", "hex", "neo", 40, 10, 10),
        # quadratic elements, odd sizes
        _single("quadtet_beam_run", "run", "quadtet", "neo", 11, 5, 4, steps=10),
        # nearly incompressible tissue block, ordinary and the benchmark's size
        _single("tet_block_run", "run", "tet", "mooney", 21, 11, 9, steps=10, h=0.01),
        _single("tet_block_large_run", "run", "tet", "mooney", 60, 30, 30, steps=5, h=0.01),
        _single("tet_block_large_mixed_step", "run", "tet", "mooney", 60, 30, 30, h=0.01, mixed=True),
        # parameter sweep: the benchmark's 256 uneven beams, mixed precision
        _pack("pack256_mixed_step", 256, 3),
        # a smaller sweep with one refinement sweep (results at FP64 level), and one in plain FP64
        _pack("pack48_refined_step", 48, 5, refine=1),
        # a served pack: some models ten times longer, two thirds of them with a request in this tick
        _pack("served64_tick", 64, 4, large=0.1, active=0.66, mixed=False, steps=2),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the listed ones' ranges."""
    kind = rng.choice(["host", "run", "run", "update", "pack", "pack"])
    if kind == "pack":
        refine = rng.choice([0, 0, 1])
        mixed = refine == 1 or rng.random() < 0.6
        c = _pack("", _log_int(rng, 6, 200), rng.randint(10, 10**6), large=rng.choice([0.0, 0.1]),
                  active=rng.choice([1.0, 1.0, 0.5]), refine=refine, mixed=mixed, steps=1 if mixed else rng.randint(1, 3),
                  tol=10 ** rng.uniform(-12, -10))
        del c["name"]
        return c
    elem, material = rng.choice([("tet", "linear"), ("tet", "neo"), ("hex", "neo"), ("hex", "neo"), ("quadtet", "neo"),
                                 ("tet", "mooney"), ("tet", "mooney")])
    if kind == "update" and material == "mooney":
        material = "neo"
    top = {"hex": 48, "quadtet": 16, "tet": 52}[elem]
    nx = _log_int(rng, 4, top)
    ny = max(2, int(nx * rng.uniform(0.2, 0.5)))
    nz = max(2, int(nx * rng.uniform(0.2, 0.5)))
    mixed = kind in ("host", "run") and material != "linear" and rng.random() < 0.25
    steps = 1 if kind != "run" or mixed else rng.randint(2, 12 if nx < 30 else 4)
    c = _single("", kind, elem, material, nx, ny, nz, steps, rng.choice([0.005, 0.01]), 10 ** rng.uniform(-12, -10),
                mixed)
    del c["name"]
    return c


# ------------------------------------------------------------------ the inputs
TET_CELL = {0: [(0, 1, 2, 5), (0, 2, 3, 7), (0, 5, 7, 4), (2, 7, 5, 6), (0, 2, 7, 5)],
            1: [(1, 2, 3, 6), (1, 3, 0, 4), (1, 6, 4, 5), (3, 4, 6, 7), (1, 3, 4, 6)]}
TET_EDGES = [(0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3)]


def _grid(elem, nx, ny, nz, wx, wy, wz, jitter, rng):
    """Node positions (interior ones jittered) and connectivity of a box of cells: one hexahedron, or five
    tetrahedra whose diagonals alternate from cell to cell, with edge midpoints for the ten-node ones."""
    k, j, i = np.meshgrid(np.arange(nz + 1), np.arange(ny + 1), np.arange(nx + 1), indexing="ij")
    x = np.stack([i.ravel() * (wx / nx) - wx / 2, j.ravel() * (wy / ny) - wy / 2, k.ravel() * (wz / nz) - wz / 2], 1)
    inner = ((i > 0) & (i < nx) & (j > 0) & (j < ny) & (k > 0) & (k < nz)).ravel()
    x += inner[:, None] * rng.uniform(-jitter, jitter, x.shape) * np.array([wx / nx, wy / ny, wz / nz])
    ck, cj, ci = (a.ravel() for a in np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij"))

    def node(a, b, c):
        return (ci + a) + (nx + 1) * ((cj + b) + (ny + 1) * (ck + c))

    corners = np.stack([node(0, 0, 0), node(1, 0, 0), node(1, 1, 0), node(0, 1, 0),
                        node(0, 0, 1), node(1, 0, 1), node(1, 1, 1), node(0, 1, 1)], 1)
    if elem == "hex":  # the engine's hexes list the +z face first
        return x, np.ascontiguousarray(corners[:, [4, 5, 6, 7, 0, 1, 2, 3]], dtype=np.int32)
    odd = (ci + cj + ck) % 2
    conn = np.empty((len(ci), 5, 4), dtype=np.int64)
    for parity, tets in TET_CELL.items():
        conn[odd == parity] = corners[odd == parity][:, np.array(tets)]
    conn = conn.reshape(-1, 4)
    e = x[conn[:, 1:]] - x[conn[:, :1]]
    flip = np.linalg.det(e) < 0
    conn[flip] = conn[flip][:, [0, 2, 1, 3]]
    if elem == "quadtet":
        pairs = np.sort(conn[:, np.array(TET_EDGES)], axis=2).reshape(-1, 2)
        uniq, inv = np.unique(pairs, axis=0, return_inverse=True)
        conn = np.concatenate([conn, inv.reshape(-1, 6) + len(x)], 1)
        x = np.concatenate([x, 0.5 * (x[uniq[:, 0]] + x[uniq[:, 1]])])
    return x, np.ascontiguousarray(conn, dtype=np.int32)


def _smooth(rest, span, rng, size):
    """A smooth vector field of the given magnitude that vanishes at the lower end of axis 0 of `span`."""
    out = np.zeros_like(rest)
    axis, lo, length = span
    ramp = (rest[:, axis] - lo) / length
    for _ in range(4):
        wave = rng.uniform(-2.0, 2.0, 3) * math.pi / length
        out += np.sin(rest @ wave + rng.uniform(0, 2 * math.pi))[:, None] * rng.uniform(-1, 1, 3)
    return out * (ramp * size / 4)[:, None]


def _one(elem, material, params, cells, widths, rng, h, fix_axis=0):
    """One model's arrays: mesh, fixed nodes, a smoothly deformed and moving state."""
    rest, conn = _grid(elem, *cells, *widths, 0.04, rng)
    lo = -widths[fix_axis] / 2
    fixed = rest[:, fix_axis] <= lo + 1e-9
    span = (fix_axis, lo, widths[fix_axis])
    # half a per cent of the thickness; the tissue block resists volume changes a hundred times more than shear
    size = (0.0005 if material == "mooney" else 0.005) * min(widths)
    x0 = rest + _smooth(rest, span, rng, size)
    v0 = _smooth(rest, span, rng, size / h)
    v0[fixed] = 0.0
    x0[fixed] = rest[fixed]
    return dict(elem=elem, material=material, params=params, rest=rest, conn=conn, fixed=fixed, x0=x0, v0=v0,
                density=1050.0 if material == "mooney" else 1000.0)


def _inputs(case, seed):
    rng = np.random.default_rng([int(seed) & 0x7FFFFFFF, 17])
    if case["kind"] != "pack":
        params = {"linear": LINEAR, "neo": NEO, "mooney": MOONEY}[case["material"]]
        cells = (case["nx"], case["ny"], case["nz"])
        # beams of 25 mm cells, a tissue block of 5 mm cells held at its base
        cell = 0.005 if case["material"] == "mooney" else 0.025
        return [_one(case["elem"], case["material"], params, cells, tuple(cell * c for c in cells), rng, case["h"],
                     2 if case["material"] == "mooney" else 0)]
    # uneven beams of 50 mm cells; sizes and materials belong to the case, the state to the seed
    sizes = np.random.default_rng(case["sizes_seed"])
    out = []
    for _ in range(case["models"]):
        n = int(sizes.integers(4, 61))
        if case["large"] and sizes.random() < case["large"]:
            n = int(sizes.integers(80, 121))
        m = int(sizes.integers(2, 9))
        params = dict(E=float(10 ** sizes.uniform(3, 6)), nu=float(sizes.uniform(0.30, 0.49)))
        out.append(_one("tet", "neo", params, (n, m, m), (0.05 * n, 0.05 * m, 0.05 * m), rng, case["h"]))
    return out


def _active(case):
    mask = np.random.default_rng(case["sizes_seed"] + 1).random(case["models"]) < case["active"]
    mask[0] = True
    return mask


def _material(d):
    p = d["params"]
    if d["material"] == "linear":
        return LinearMaterial(p["E"], p["nu"], True)
    if d["material"] == "neo":
        return NeoHookeanMaterial(p["E"], p["nu"])
    return MooneyRivlinMaterial(p["c10"], p["c01"], 0.0, 0.0, 0.0, p["kappa"])


def _model(d):
    m = FemModel3d()
    m.setMesh(ELEM[d["elem"]], d["rest"], d["conn"], d["fixed"])
    m.setMaterial(_material(d))
    m.setDensity(d["density"])
    m.setMassDamping(ALPHA)
    m.setGravity(np.array(GRAVITY))
    return m


class State:
    """What the program holds between calls: the built engine and its arrays."""


def prepare(case, seed):
    data = _inputs(case, seed)
    s = State()
    s.case = case
    prec = L.PREC_MIXED if case["mixed"] else L.PREC_FP64
    if case["kind"] == "pack":
        options = {L.OPT_REFINE: case["refine"]} if case["refine"] else {}
        s.pack = FemPack([_model(d) for d in data], precision=prec, options=options)
        s.pack.engine()
        s.x0 = [d["x0"] for d in data]
        s.v0 = [d["v0"] for d in data]
        s.active = _active(case) if case["active"] < 1 else None
        return s
    d = data[0]
    s.model = _model(d)
    s.model.setPrecision(prec)
    s.model.engine()
    s.solver = MechSystemSolver(s.model, tol=case["tol"])
    s.x0, s.v0 = d["x0"], d["v0"]
    if case["kind"] == "host":
        n3 = 3 * len(d["rest"])
        s.x = torch.empty(n3, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()
        s.v = torch.empty(n3, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()
        s.x0f, s.v0f = s.x0.reshape(-1).copy(), s.v0.reshape(-1).copy()
    return s


def run(s):
    c = s.case
    if c["kind"] == "host":
        s.x[:] = s.x0f
        s.v[:] = s.v0f
        s.solver.backwardEulerHost(c["h"], s.x, s.v)
        return s.x, s.v
    if c["kind"] == "run":
        s.model.setState(s.x0, s.v0)
        s.solver.backwardEuler(c["h"], c["steps"])
        return s.model.getState()
    if c["kind"] == "update":
        return s.model.updateStressAndStiffness(s.x0, want_crs=True)
    s.pack.setStates(s.x0, s.v0)
    if s.active is not None:
        s.pack.setActive(s.active)
    s.pack.backwardEuler(c["h"], c["steps"], tol=c["tol"])
    states = s.pack.getStates()
    # the models' arrays are slices of one array for x and one for v
    return states[0][0].base, states[0][1].base


def work(case):
    """Bytes and operations of one pass: state in and out, mesh, rest data and the solve matrix (or the stiffness
    arrays) once per step, the element arithmetic; the iterations of the solve are not counted."""
    nip = {"tet": 1, "hex": 8, "quadtet": 4}[case["elem"]]
    nen = {"tet": 4, "hex": 8, "quadtet": 10}[case["elem"]]
    if case["kind"] == "pack":
        cells = sum(n * m * m for n, m in _pack_cells(case))
        nodes = sum((n + 1) * (m + 1) ** 2 for n, m in _pack_cells(case))
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
        nodes = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
    elems = cells * (1 if case["elem"] == "hex" else 5)
    if case["elem"] == "quadtet":
        nodes += 6 * cells
    blocks = nodes + cells * {"tet": 12, "hex": 26, "quadtet": 170}[case["elem"]]
    mesh = elems * (4 * nen + 72 * nip)
    flops = elems * nip * (400 + 80 * nen * (nen + 1) // 2)
    if case["kind"] == "update":
        return {"bytes": 48 * nodes + mesh + 144 * blocks, "flops": flops}
    per_step = 96 * nodes + mesh + (36 if case["mixed"] else 72) * blocks
    return {"bytes": case["steps"] * per_step, "flops": case["steps"] * (flops + 18 * blocks)}


def _pack_cells(case):
    sizes = np.random.default_rng(case["sizes_seed"])
    out = []
    for _ in range(case["models"]):
        n = int(sizes.integers(4, 61))
        if case["large"] and sizes.random() < case["large"]:
            n = int(sizes.integers(80, 121))
        m = int(sizes.integers(2, 9))
        sizes.uniform(3, 6), sizes.uniform(0.30, 0.49)
        out.append((n, m))
    return out


# ------------------------------------------------------- the same in plain torch
def _gradients(elem):
    """dN/ds at the integration points (nip, nen, 3) and the points' weights."""
    if elem == "tet":
        return np.array([[[-1, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]]], dtype=float), np.array([1 / 6.0])
    if elem == "hex":
        node = np.array([[-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1], [-1, -1, -1], [1, -1, -1], [1, 1, -1],
                         [-1, 1, -1]], dtype=float)
        g = np.empty((8, 8, 3))
        for k, p in enumerate(node / math.sqrt(3.0)):
            t = 1 + node * p
            g[k] = np.stack([node[:, 0] * t[:, 1] * t[:, 2], node[:, 1] * t[:, 0] * t[:, 2],
                             node[:, 2] * t[:, 0] * t[:, 1]], 1) / 8
        return g, np.ones(8)
    a, b = 0.58541020, 0.13819660
    dl = np.array([[-1, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]], dtype=float)
    g = np.empty((4, 10, 3))
    for k in range(4):
        c = [a if k == q + 1 else b for q in range(3)]
        lam = np.array([1 - sum(c)] + c)
        g[k, :4] = (4 * lam - 1)[:, None] * dl
        for q, (i, j) in enumerate(TET_EDGES):
            g[k, 4 + q] = 4 * (lam[i] * dl[j] + lam[j] * dl[i])
    return g, np.full(4, 0.25 / 6)


def _density(material, F, p):
    """Strain energy per rest volume (the deviatoric part for MooneyRivlin)."""
    J = torch.linalg.det(F)
    B = F @ F.transpose(-1, -2)
    I1 = B.diagonal(dim1=-2, dim2=-1).sum(-1)
    if material == "neo":
        mu = p[..., 0] / (2 * (1 + p[..., 1]))
        lam = p[..., 0] * p[..., 1] / ((1 - 2 * p[..., 1]) * (1 + p[..., 1]))
        lj = torch.log(J)
        return 0.5 * mu * (I1 - 3) - mu * lj + 0.5 * lam * lj * lj
    I2 = 0.5 * (I1 * I1 - (B * B).sum((-1, -2)))
    return p[..., 0] * (I1 * J ** (-2 / 3) - 3) + p[..., 1] * (I2 * J ** (-4 / 3) - 3)


class _Plain:
    """The models of a case as one set of arrays in 64 bits: forces, element stiffness, BackwardEuler steps."""

    def __init__(self, data, device):
        def t(a):
            return torch.as_tensor(np.ascontiguousarray(a), device=device)

        self.elem, self.material = data[0]["elem"], data[0]["material"]
        off = np.cumsum([0] + [len(d["rest"]) for d in data])
        self.rest = t(np.concatenate([d["rest"] for d in data]))
        self.conn = t(np.concatenate([d["conn"].astype(np.int64) + o for d, o in zip(data, off)]))
        self.free = t(~np.concatenate([d["fixed"] for d in data]))
        p = {"linear": ("E", "nu"), "neo": ("E", "nu"), "mooney": ("c10", "c01")}[self.material]
        self.prm = t(np.concatenate([np.tile([d["params"][k] for k in p], (len(d["conn"]), 1)) for d in data]))
        self.kappa = data[0]["params"].get("kappa")
        g, w = _gradients(self.elem)
        self.g, self.w = t(g), t(w)
        J0 = torch.einsum("enr,knc->ekrc", self.rest[self.conn], self.g)
        self.iJ0 = torch.linalg.inv(J0)
        self.dv0 = torch.linalg.det(J0) * self.w
        nen = self.conn.shape[1]
        n = len(self.rest)
        share = (self.dv0.sum(1) * data[0]["density"] / nen)[:, None].expand(-1, nen)
        self.mass = torch.zeros(n, dtype=torch.float64, device=device).index_add_(0, self.conn.reshape(-1),
                                                                                share.reshape(-1))
        if self.material == "mooney":
            self.vol0 = self._node_volume(self.rest)
        if self.material == "linear":
            self._linear_rest()

    def _linear_rest(self):
        E, nu = self.prm[:, 0], self.prm[:, 1]
        lam, mu = E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
        G = torch.einsum("knc,ekcr->eknr", self.g, self.iJ0)
        eye = torch.eye(3, dtype=torch.float64, device=G.device)
        K = torch.einsum("eknr,ekms,ek->enrms", G, G, self.dv0 * lam[:, None])
        K += torch.einsum("ekns,ekmr,ek->enrms", G, G, self.dv0 * mu[:, None])
        K += torch.einsum("eknq,ekmq,ek,rs->enrms", G, G, self.dv0 * mu[:, None], eye)
        self.K0 = K

    def _node_volume(self, x):
        e = x[self.conn]
        v = torch.linalg.det(e[:, 1:] - e[:, :1]) / 24
        return torch.zeros(len(x), dtype=x.dtype, device=x.device).index_add_(
            0, self.conn.reshape(-1), v[:, None].expand(-1, 4).reshape(-1))

    def assemble(self, x):
        """Element forces (E, nen, 3) and stiffness (E, nen, 3, nen, 3); for NODAL incompressibility also the
        elements' volume gradients and the nodes' moduli, whose rank-one terms are kept apart."""
        xe = x[self.conn]
        nen = xe.shape[1]
        self.vg = self.kp = None
        if self.material == "linear":
            F = torch.einsum("enr,nc,ecs->ers", xe, self.g[0], self.iJ0[:, 0])
            U, _, Vh = torch.linalg.svd(F)
            s = torch.ones(len(F), 3, dtype=F.dtype, device=F.device)
            s[:, 2] = torch.linalg.det(U @ Vh)
            R = U @ (s[:, :, None] * Vh)
            local = torch.einsum("esr,ens->enr", R, xe) - self.rest[self.conn]
            f = torch.einsum("ers,ens->enr", R, torch.einsum("enrms,ems->enr", self.K0, local))
            return f, torch.einsum("era,enamb,esb->enrms", R, self.K0, R)
        pe = torch.zeros(len(xe), dtype=x.dtype, device=x.device)
        if self.material == "mooney":
            J = self._node_volume(x) / self.vol0
            zero = torch.zeros_like(J)
            pn = torch.where(self.free, self.kappa * (J - 1), zero)
            self.kp = torch.where(self.free, self.kappa / self.vol0, zero)
            pe = pn[self.conn].mean(1)

        def energy(z, iJ0, dv0, prm, p):
            z = z.reshape(nen, 3)
            F = torch.einsum("nr,knc->krc", z, self.g) @ iJ0
            out = (_density(self.material, F, prm) * dv0).sum()
            if self.material == "mooney":
                out = out + p * torch.linalg.det(z[1:] - z[:1]) / 6
            return out

        grad = torch.func.vmap(torch.func.grad(energy))
        hess = torch.func.vmap(torch.func.hessian(energy))
        fs, Ks, step = [], [], 60000 if nen == 4 else 4000
        for a in range(0, len(xe), step):
            arg = (xe[a:a + step].reshape(-1, 3 * nen), self.iJ0[a:a + step], self.dv0[a:a + step],
                   self.prm[a:a + step], pe[a:a + step])
            fs.append(grad(*arg))
            Ks.append(hess(*arg))
        if self.material == "mooney":
            def vol(z):
                z = z.reshape(4, 3)
                return torch.linalg.det(z[1:] - z[:1]) / 6
            self.vg = torch.func.vmap(torch.func.grad(vol))(xe.reshape(-1, 12)).reshape(-1, 4, 3)
        return torch.cat(fs).reshape(-1, nen, 3), torch.cat(Ks).reshape(-1, nen, 3, nen, 3)

    def step(self, x, v, h, mask):
        """One BackwardEuler step of the nodes in `mask`."""
        n, flat = len(x), self.conn.reshape(-1)
        nen = self.conn.shape[1]
        f, K = self.assemble(x)
        gravity = torch.tensor(GRAVITY, dtype=x.dtype, device=x.device)

        def scatter(ye):
            return torch.zeros(n, ye.shape[-1], dtype=x.dtype, device=x.device).index_add_(0, flat,
                                                                                       ye.reshape(n_slots, -1))

        n_slots = flat.numel()
        live = (self.free & mask)[:, None].to(x.dtype)
        m = self.mass[:, None]
        b = (m * v + h * (m * gravity - scatter(f))) * live
        K2 = K.reshape(-1, 3 * nen, 3 * nen)

        def apply(u):
            ye = torch.bmm(K2, u[self.conn].reshape(-1, 3 * nen, 1)).reshape(-1, nen, 3)
            if self.vg is not None:
                dn = scatter((self.vg * u[self.conn]).sum((1, 2))[:, None, None].expand(-1, nen, 1) / 4)
                t = (self.kp[:, None] * dn)[self.conn].sum(1) / 4
                ye = ye + self.vg * t[:, :, None]
            return ((1 + h * ALPHA) * m * u + h * h * scatter(ye)) * live

        i = torch.arange(nen, device=x.device)
        Dd = scatter(K[:, i, :, i, :].permute(1, 0, 2, 3).reshape(-1, nen, 9)).reshape(n, 3, 3) * h * h
        eye = torch.eye(3, dtype=x.dtype, device=x.device)
        P = torch.linalg.inv(Dd + ((1 + h * ALPHA) * self.mass)[:, None, None] * eye)
        sol = torch.zeros_like(b)
        for _ in range(3):  # residual replacement: the last rounds bring it to round-off
            r = b - apply(sol)
            z = torch.bmm(P, r[:, :, None])[:, :, 0]
            p, rz = z.clone(), (r * z).sum()
            stop = 1e-14 * b.norm()
            for it in range(6000):
                if it % 16 == 0 and r.norm() <= stop:
                    break
                q = apply(p)
                alpha = rz / (p * q).sum()
                sol += alpha * p
                r -= alpha * q
                z = torch.bmm(P, r[:, :, None])[:, :, 0]
                rz, old = (r * z).sum(), rz
                p = z + (rz / old) * p
        on = live > 0
        v1 = torch.where(on, sol, v)
        return torch.where(on, x + h * v1, x), v1


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    data = _inputs(case, seed)
    s = _Plain(data, device)
    x = torch.as_tensor(np.concatenate([d["x0"] for d in data]), device=device)
    v = torch.as_tensor(np.concatenate([d["v0"] for d in data]), device=device)
    if case["kind"] == "update":
        return _exact_update(s, x)
    mask = torch.ones(len(x), dtype=torch.bool, device=device)
    if case["kind"] == "pack" and case["active"] < 1:
        mask = torch.as_tensor(np.repeat(_active(case), [len(d["rest"]) for d in data]), device=device)
    for _ in range(case["steps"]):
        x, v = s.step(x, v, case["h"], mask)
    if case["kind"] == "run":
        return x, v
    return x.reshape(-1), v.reshape(-1)


def _exact_update(s, x):
    """Forces, stiffness blocks in block-row order over the free nodes, and the scalar rows' values."""
    f, K = s.assemble(x)
    n, nen = len(x), s.conn.shape[1]
    fn = torch.zeros(n, 3, dtype=x.dtype, device=x.device).index_add_(0, s.conn.reshape(-1), f.reshape(-1, 3))
    if s.material == "linear":  # formed for the free nodes only
        fn = fn * s.free[:, None]
    idx = torch.cumsum(s.free, 0) - 1
    idx = torch.where(s.free, idx, torch.full_like(idx, -1))
    R = int(s.free.sum())
    row = idx[s.conn][:, :, None].expand(-1, nen, nen).reshape(-1)
    col = idx[s.conn][:, None, :].expand(-1, nen, nen).reshape(-1)
    keep = (row >= 0) & (col >= 0)
    uniq, inv = torch.unique(row[keep] * R + col[keep], return_inverse=True)
    blocks = K.permute(0, 1, 3, 2, 4).reshape(-1, 9)[keep]
    B = torch.zeros(len(uniq), 9, dtype=x.dtype, device=x.device).index_add_(0, inv, blocks).reshape(-1, 3, 3)
    brow = torch.div(uniq, R, rounding_mode="floor")
    # scalar row 3 br + r holds the r-th rows of its blocks side by side
    order = (brow[:, None, None] * 3 + torch.arange(3, device=x.device)[None, :, None]).expand(-1, 3, 3)
    at = torch.argsort(order.reshape(-1) * 1, stable=True)
    return fn, B, B.reshape(-1)[at]
