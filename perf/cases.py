"""The workloads whose speed is followed: Flux Reconstruction solves through the public Python API.

A case is a dict of plain values; `prepare` sets a solver up on the GPU from a
deck, a mesh and a seeded initial state, as a program does once per solve, and
`run` is one pass of that program's loop (steps, a residual with its norm, or a
batch).  Outputs are the solver's own device arrays.  `exact` is the same
computation in plain 64-bit torch on structured grids, written from the
scheme's definition.
"""
import math
import os
import shutil
import tempfile

import numpy as np
import torch

import flurrypp_b200 as fb
from flurrypp_b200.decks import channel_case, write_deck
from flurrypp_b200.meshgen import channel_bump, write_gmsh

GAMMA = 1.4
CHAR, SLIP_WALL, SYMMETRY, PERIODIC = 1, 8, 12, 0


def _case(kind, nx, ny=0, nz=0, order=3, steps=1, precision="fp64", call="run", roe=0, perturb=0.0, members=0):
    return {"kind": kind, "nx": nx, "ny": ny or nx, "nz": nz, "order": order, "steps": steps,
            "precision": precision, "call": call, "roe": roe, "perturb": perturb, "members": members}


def listed():
    named = {
        # one update() of a very small 2-D vortex: a program that steps by hand
        # (monitoring, coupling) pays the host path and every launch each step
        "vortex2d_p3_8_update": _case("vortex", 8, call="update"),
        # the reference's 2-D vortex benchmark size: latency of graph-replayed steps
        "vortex2d_p3_32": _case("vortex", 32, steps=20),
        # mid-size 2-D run with the Roe flux on an odd, non-square grid
        "vortex2d_p4_roe_odd": _case("vortex", 201, 149, order=4, steps=4, roe=1),
        # large 2-D run in the precision form
        "vortex2d_p2_384_mixed": _case("vortex", 384, order=2, steps=4, precision="mixed"),
        # the headline: 3-D Euler Taylor-Green vortex, 32^3 hexes, P3, both forms
        "tgv3d_p3_32": _case("tgv", 32, nz=32, steps=4),
        "tgv3d_p3_32_mixed": _case("tgv", 32, nz=32, steps=4, precision="mixed"),
        # general (non-affine) hexes in an odd number, quadratic elements
        "tgv3d_p2_27_perturbed": _case("tgv", 27, nz=27, order=2, steps=4, perturb=0.05),
        # viscous: Navier-Stokes Taylor-Green vortex, P4, perturbed hexes, both forms
        "ns_tgv3d_p4_24": _case("ns", 24, nz=24, order=4, steps=2, perturb=0.05),
        "ns_tgv3d_p4_24_mixed": _case("ns", 24, nz=24, order=4, steps=2, precision="mixed", perturb=0.05),
        # steady solve as the solve server runs it: channel bump, walls and far
        # field, local time steps, P-multigrid, ten driver steps between checks
        "channel_p3_48_pmg": _case("channel", 48, 16, steps=10),
        # residual evaluation and its norm on a wall-bounded 3-D duct of odd sizes
        "duct3d_p3_residual": _case("duct", 41, 21, 17, call="residual", perturb=0.05),
        # many small cases of orders 2..5 advanced together
        "batch24_vortex_mixed": _case("batch", 8, 96, order=5, steps=10, precision="mixed", members=24),
    }
    return [dict(c, name=n) for n, c in named.items()]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["vortex", "vortex", "tgv", "tgv", "ns", "channel", "duct", "batch"])
    precision = rng.choice(["fp64", "mixed"])
    steps = rng.randint(1, 6)
    if kind == "vortex":
        order = rng.randint(1, 5)
        nx = _log(rng, 6, 900 // (order + 1))
        ny = max(5, min(900 // (order + 1), int(nx * rng.uniform(0.6, 1.4))))
        return _case(kind, nx, ny, order=order, steps=steps, precision=precision,
                     call=rng.choice(["run", "run", "update"]), roe=rng.choice([0, 0, 1]))
    if kind == "tgv":
        order = rng.randint(1, 4)
        n = _log(rng, 4, 110 // (order + 1))
        return _case(kind, n, max(4, n + rng.randint(-3, 2)), max(4, n + rng.randint(-3, 2)), order, min(steps, 4),
                     precision, perturb=rng.choice([0.0, 0.05]))
    if kind == "ns":
        order = rng.randint(2, 4)
        n = _log(rng, 4, 100 // (order + 1))
        return _case(kind, n, max(4, n + rng.randint(-2, 2)), n, order, min(steps, 2), precision, perturb=0.05)
    if kind == "channel":
        nx = _log(rng, 24, 96)
        return _case(kind, nx, nx // 3, order=rng.randint(1, 4), steps=10)
    if kind == "duct":
        order = rng.randint(1, 4)
        n = _log(rng, 6, 120 // (order + 1))
        return _case(kind, n, max(4, n // 2 + rng.randint(0, 3)), max(4, n // 2 + rng.randint(-1, 2)), order, steps,
                     precision, call=rng.choice(["run", "residual"]), perturb=0.05)
    return _case(kind, 8, rng.randint(24, 96), order=5, steps=10, precision=precision, members=rng.randint(6, 24))


# --- inputs ------------------------------------------------------------------

def _members(case, seed):
    """The vortex cases of a batch: sizes and orders belong to the case, the fields to the seed."""
    r = np.random.default_rng(case["members"] * 1000 + case["ny"])
    return [_case("vortex", int(r.integers(case["nx"], case["ny"] + 1)), order=int(r.integers(2, case["order"] + 1)),
                  steps=case["steps"], precision=case["precision"]) for _ in range(case["members"])]


def _box(case):
    if case["kind"] == "vortex":
        return [(-5.0, 5.0), (-5.0, 5.0)]
    if case["kind"] == "duct":
        return [(0.0, 2.0), (0.0, 1.0), (0.0, 1.0)]
    return [(0.0, 2 * math.pi)] * 3


def _sizes(case):
    return [case["nx"], case["ny"]] + ([case["nz"]] if case["nz"] else [])


def _vertices(case, seed):
    """Vertex grid [nx+1, ny+1(, nz+1), nd] of a structured mesh."""
    n = _sizes(case)
    if case["kind"] == "channel":
        nx, ny = n
        xs = np.linspace(-1.5, 1.5, nx + 1)
        yb = _bump_height(seed) * np.exp(-25.0 * xs * xs)
        t = np.arange(ny + 1) / ny
        return np.stack([np.broadcast_to(xs[:, None], (nx + 1, ny + 1)), yb[:, None] + (0.8 - yb[:, None]) * t], -1)
    box = _box(case)
    axes = [np.linspace(a, b, m + 1) for (a, b), m in zip(box, n)]
    v = np.stack(np.meshgrid(*axes, indexing="ij"), -1)
    if case["perturb"]:
        h = np.array([(b - a) / m for (a, b), m in zip(box, n)])
        inner = tuple(slice(1, m) for m in n)
        r = np.random.default_rng([seed, 7])
        v[inner] += r.uniform(-case["perturb"], case["perturb"], v[inner].shape) * h
    return v


def _bump_height(seed):
    return float(np.random.default_rng([seed, 3]).uniform(0.02, 0.1))


def _field(case, seed, x):
    """Seeded initial state at positions x [..., nd] (conserved variables)."""
    r = np.random.default_rng([seed, 11])
    nd = x.shape[-1]
    X = [x[..., d] for d in range(nd)]
    kind = case["kind"]
    if kind == "vortex":
        eps, xc, yc = r.uniform(1, 5), r.uniform(-2, 2), r.uniform(-2, 2)
        mach = r.uniform(0.2, 0.6)
        dx, dy = X[0] - xc, X[1] - yc
        dx, dy = dx - 10 * torch.round(dx / 10), dy - 10 * torch.round(dy / 10)
        f = eps / (2 * math.pi) * torch.exp(0.5 * (1 - dx * dx - dy * dy))
        T = 1 - (GAMMA - 1) / (2 * GAMMA) * f * f
        rho = T ** (1 / (GAMMA - 1))
        vel, p = [mach * math.sqrt(GAMMA) - f * dy, f * dx], rho * T
    elif kind in ("tgv", "ns"):
        # Mach 0.1 Taylor-Green vortex with two weak seeded modes on top
        ph = r.uniform(0, 2 * math.pi, 6)
        p0, V = (1.0, 0.1 * math.sqrt(GAMMA)) if kind == "tgv" else (1 / (GAMMA * 0.01), 1.0)
        s, c = torch.sin, torch.cos
        vel = [V * (s(X[0]) * c(X[1]) * c(X[2]) + 0.05 * s(X[1] + ph[0]) * c(X[2] + ph[1])),
               V * (-c(X[0]) * s(X[1]) * c(X[2]) + 0.05 * s(X[2] + ph[2]) * c(X[0] + ph[3])),
               V * 0.05 * s(X[0] + ph[4]) * c(X[1] + ph[5])]
        rho = torch.ones_like(X[0])
        p = p0 + V * V / 16 * (c(2 * X[0]) + c(2 * X[1])) * (c(2 * X[2]) + 2)
    else:  # free stream with a weak seeded disturbance
        c0 = [r.uniform(-0.5, 0.5) if kind == "channel" else r.uniform(0.5, 1.5)] + list(r.uniform(0.3, 0.5, nd - 1))
        bump = torch.exp(-8 * sum((X[d] - c0[d]) ** 2 for d in range(nd)))
        rho = 1 + 0.02 * bump
        vel = [_mach(case) * (1 + 0.1 * bump)] + [0.02 * bump * (d + 1) for d in range(nd - 1)]
        p = (1 + 0.02 * bump) / GAMMA
    E = p / (GAMMA - 1) + 0.5 * rho * sum(v * v for v in vel)
    return torch.stack([rho] + [rho * v for v in vel] + [E], -1)


def _mach(case):
    return 0.35


def _dt(case):
    """A fixed step well inside the stability limit."""
    speed = {"vortex": 3.5, "tgv": 1.4, "ns": 11.0, "duct": 1.6}[case["kind"]]
    h = min((b - a) / m for (a, b), m in zip(_box(case), _sizes(case)))
    return 0.1 * h / ((2 * case["order"] + 1) * speed)


def _points(case, seed):
    """Solution-point positions [nS, nE, nd] in the solver's layout, from the mesh's vertices."""
    g = _Grid(case, seed, "cpu", metrics=False)
    return g.to_layout(g.pos)


def _initial(case, seed):
    return _field(case, seed, _points(case, seed)).numpy()


def _deck_options(case):
    nd = len(_sizes(case))
    o = dict(nDims=nd, order=case["order"], riemannType=case["roe"], dt=repr(_dt(case)), rhoBound=1,
             uBound=_mach(case), pBound=repr(1 / GAMMA), resType=2)
    if case["kind"] == "ns":
        o.update(viscous=1, Re=1600, MachBound=0.1, prandtl=0.71, fixVis=1, LDG_tau=0.1, LDG_penFact=0.5,
                 TBound=291.15, TGas=291.15, MachWall=0)
    if not case["perturb"]:
        o.update(meshType=1)
        for name, m, (a, b) in zip("xyz", _sizes(case), _box(case)):
            o.update({"n" + name: m, name + "min": repr(a), name + "max": repr(b)})
    return o


def _mesh(case, seed):
    """A caller-owned mesh of linear hexes, boundary faces listed by their vertices."""
    v = _vertices(case, seed)
    n = _sizes(case)
    vid = np.arange(v[..., 0].size).reshape(v.shape[:-1])
    c = lambda a, b, d: vid[a:a + n[0], b:b + n[1], d:d + n[2]].reshape(-1)
    c2v = np.stack([c(0, 0, 0), c(1, 0, 0), c(1, 1, 0), c(0, 1, 0), c(0, 0, 1), c(1, 0, 1), c(1, 1, 1), c(0, 1, 1)], 1)
    faces, codes = [], []
    for d in range(3):
        for side in (0, -1):
            g = np.take(vid, side, axis=d)
            q = np.stack([g[:-1, :-1], g[1:, :-1], g[1:, 1:], g[:-1, 1:]], -1).reshape(-1, 4)
            faces.append(q)
            codes.append(np.full(len(q), _boundaries(case)[d]))
    period = [b - a for a, b in _box(case)] if case["kind"] != "duct" else [1e300] * 3
    return {"xv": v.reshape(-1, 3), "c2v": c2v, "bnd_face_verts": np.concatenate(faces),
            "bnd_face_bc": np.concatenate(codes), "period": period}


def _boundaries(case):
    """Boundary condition of each axis (both of its sides)."""
    return {"channel": [CHAR, SLIP_WALL], "duct": [CHAR, SLIP_WALL, SYMMETRY]}.get(case["kind"], [PERIODIC] * 3)


class _View:
    """A solver's device array as an object torch can wrap; keeps the solver alive."""

    def __init__(self, solver, name):
        ptr, size = solver.device_ptr(name)
        wide = size == 8 * math.prod(solver.shape)
        self.solver = solver
        self.__cuda_array_interface__ = {"shape": solver.shape, "typestr": "<f8" if wide else "<f4",
                                         "data": (ptr, False), "version": 2}


def _solver(case, seed):
    tmp = tempfile.mkdtemp(prefix="fr_case_")
    try:
        path = os.path.join(tmp, "case.deck")
        opts = {"precision": fb.FR_PREC_MIXED if case["precision"] == "mixed" else fb.FR_PREC_FP64}
        if case["kind"] == "channel":
            msh = os.path.join(tmp, "bump.msh")
            write_gmsh(msh, channel_bump(case["nx"], case["ny"], _bump_height(seed)))
            s = fb.Solver(channel_case(path, msh, case["order"], _mach(case)), **opts)
        else:
            write_deck(path, **_deck_options(case))
            s = fb.Solver(path, mesh=_mesh(case, seed) if case["perturb"] else None, **opts)
    finally:
        shutil.rmtree(tmp, ignore_errors=True)
    s.set_state(_initial(case, seed))
    return s


def prepare(case, seed):
    if case["kind"] == "batch":
        solvers = [_solver(m, seed * 100 + i) for i, m in enumerate(_members(case, seed))]
        return {"case": case, "batch": fb.Batch(solvers),
                "out": [torch.as_tensor(_View(s, "U_spts"), device="cuda") for s in solvers]}
    s = _solver(case, seed)
    name = "divF_0" if case["call"] == "residual" else "U_spts"
    return {"case": case, "solver": s, "out": torch.as_tensor(_View(s, name), device="cuda")}


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        state["batch"].run(case["steps"])
        state["batch"].gather()
        return state["out"]
    s = state["solver"]
    if case["call"] == "residual":
        s.calc_residual(0)
        return {"divF": state["out"], "norm": s.residual_norm(2)}
    if case["call"] == "update":
        s.update()
    else:
        s.run(case["steps"])
    return state["out"]


def _stages(case):
    """(order, stages per pass) of every level of a pass."""
    P, steps = case["order"], case["steps"]
    if case["call"] == "residual":
        return [(P, 1)]
    if case["call"] == "update":
        return [(P, 4)]
    if case["kind"] == "channel":
        # update and the cycle's residual; per coarse level its source residual,
        # 2 x 2 smoothing updates and the residual restricted further
        return [(P, 5 * steps)] + [(q, (17 + (q > 0)) * steps) for q in range(P)]
    return [(P, 4 * steps)]


def work(case):
    """Per stage: the state read once and written once, the metrics (nd^2 + 1
    values a point) read once; the operators applied line by line."""
    if case["kind"] == "batch":
        each = [work(m) for m in _members(case, 0)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    n = _sizes(case)
    nd, word = len(n), 4 if case["precision"] == "mixed" else 8
    nb = fl = 0
    for P, stages in _stages(case):
        N, E, F = P + 1, math.prod(n), nd + 2
        pts, fpts = N ** nd, 2 * nd * N ** (nd - 1)
        nb += stages * E * pts * (2 * F + nd * nd + 1) * word
        line = 2 * N * F * nd * pts + 4 * N * F * fpts  # derivative, extrapolation of flux and state
        point = 2 * F * nd * nd + 8 * nd * F + 4 * F + 4 * nd * F
        face = 30 + 10 * nd * F
        visc = (2 * N * F * nd * pts + 2 * nd * N * F * fpts + 150 * pts + 200 * fpts // 2) if case["kind"] == "ns" else 0
        fl += stages * E * (line + pts * point + fpts // 2 * face + visc)
    return {"bytes": float(nb), "flops": float(fl)}


# --- the same in plain 64-bit torch -------------------------------------------

def _legendre(n, x):
    c = np.zeros(max(n, 0) + 1)
    c[-1] = 1.0 if n >= 0 else 0.0
    return np.polynomial.legendre.legval(x, c)


def _dlegendre(n, x):
    c = np.zeros(max(n, 0) + 1)
    c[-1] = 1.0 if n >= 0 else 0.0
    return np.polynomial.legendre.legval(x, np.polynomial.legendre.legder(c)) if n > 0 else np.zeros_like(x)


def _lagrange(nodes, x):
    """[len(x), len(nodes)] values of the Lagrange basis."""
    V = np.stack([_legendre(n, np.asarray(x, float)) for n in range(len(nodes))], -1)
    W = np.stack([_legendre(n, nodes) for n in range(len(nodes))], -1)
    return V @ np.linalg.inv(W)


class _Grid:
    """Flux Reconstruction (DG correction, Gauss-Legendre points) on a structured
    grid of linear quads or hexes.  Arrays are [elements x,y(,z), points x,y(,z), ...];
    a face belongs to the lower-numbered element as its left side."""

    def __init__(self, case, seed, device, order=None, metrics=True):
        self.case, self.dev = case, device
        self.n = _sizes(case)
        self.nd = nd = len(self.n)
        self.F = nd + 2
        P = case["order"] if order is None else order
        self.P, self.N = P, P + 1
        x, w = np.polynomial.legendre.leggauss(self.N)
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=device)
        W = np.stack([_legendre(n, x) for n in range(self.N)], -1)
        dV = np.stack([_dlegendre(n, x) for n in range(self.N)], -1)
        self.x, self.w = x, t(w)
        self.D, self.E = t(dV @ np.linalg.inv(W)), t(_lagrange(x, [-1.0, 1.0]))
        # divergence correction per outward jump at side 0 / 1 (Radau polynomials)
        gl = 0.5 * (-1.0) ** P * (_dlegendre(P, x) - _dlegendre(P + 1, x))
        gr = 0.5 * (_dlegendre(P, x) + _dlegendre(P + 1, x))
        self.corr = [t(-gl), t(gr)]
        v = t(_vertices(case, seed))
        self.corner = {}
        for bits in np.ndindex(*[2] * nd):
            self.corner[bits] = v[tuple(slice(b, b + m) for b, m in zip(bits, self.n))]
        self.pos = self.map([x] * nd)[0]
        if not metrics:
            return
        J = self.map([x] * nd)[1]
        self.JG = self.adjugate(J)
        self.det = sum(J[0][a] * self.JG[0][a] for a in range(nd))
        self.face = {}
        for d in range(nd):
            for s in (0, 1):
                at = [x] * nd
                at[d] = np.array([-1.0 if s == 0 else 1.0])
                JG = self.adjugate(self.map(at)[1])
                nv = (2 * s - 1) * torch.stack([JG[d][a].squeeze(nd + d) for a in range(nd)], -1)
                dA = nv.norm(dim=-1)
                self.face[d, s] = (nv / dA[..., None], dA)
        self.bc = _boundaries(case)[:nd]
        self.free = {"rho": 1.0, "v": [_mach(case)] + [0.0] * (nd - 1), "p": 0.7142857143 if case["kind"] == "channel" else 1 / GAMMA}
        self.wave, self.source = {}, 0.0

    def map(self, at):
        """Positions and d(position)/d(reference) [axis][component] at a tensor of points."""
        nd = self.nd
        pos, J = 0.0, [0.0] * nd
        for bits, c in self.corner.items():
            w = [torch.as_tensor((1 + (2 * b - 1) * np.asarray(r)) / 2, device=self.dev) for b, r in zip(bits, at)]
            g = [torch.full_like(w[d], (2 * b - 1) / 2) for d, b in enumerate(bits)]
            for e in range(-1, nd):
                f = [g[d] if d == e else w[d] for d in range(nd)]
                m = f[0]
                for q in f[1:]:
                    m = m[..., None] * q
                val = c.reshape(c.shape[:nd] + (1,) * nd + (nd,)) * m[..., None]
                if e < 0:
                    pos = pos + val
                else:
                    J[e] = J[e] + val
        return pos, [[J[d][..., a] for a in range(nd)] for d in range(nd)]

    def adjugate(self, J):
        """JG[d][a] = det * d(xi_d)/d(x_a) from J[d][a] = d(x_a)/d(xi_d)."""
        if self.nd == 2:
            return [[J[1][1], -J[1][0]], [-J[0][1], J[0][0]]]
        out = []
        for d in range(3):
            p, q = J[(d + 1) % 3], J[(d + 2) % 3]
            out.append([p[(a + 1) % 3] * q[(a + 2) % 3] - p[(a + 2) % 3] * q[(a + 1) % 3] for a in range(3)])
        return out

    # layouts: the solver's [point (x fastest)][element][field]
    def _perm(self):
        nd = self.nd
        ele = list(range(nd))  # element numbering, slowest axis first
        if self.case["kind"] == "channel":
            ele = ele[::-1]
        elif nd == 3 and not self.case["perturb"]:
            ele = [2, 0, 1]  # the deck's generated hexes
        return [2 * nd - 1 - d for d in range(nd)] + ele + [2 * nd]

    def to_layout(self, a):
        return a.permute(self._perm()).reshape(self.N ** self.nd, -1, a.shape[-1])

    def from_layout(self, a):
        perm = self._perm()
        full = self.n + [self.N] * self.nd + [a.shape[-1]]
        inv = [perm.index(i) for i in range(len(perm))]
        return a.reshape([full[p] for p in perm]).permute(inv).contiguous()

    def lines(self, M, a, d):
        """M applied along point axis d."""
        return torch.movedim(torch.tensordot(a, M, dims=([self.nd + d], [1])), -1, self.nd + d)

    def trace(self, a, d, s):
        return torch.tensordot(a, self.E[s], dims=([self.nd + d], [0]))

    def lift(self, q, d, s):
        """Correction of the outward jump q at face (d, s), over the element's points."""
        shape = [1] * (q.dim() + 1)
        shape[self.nd + d] = self.N
        return q.unsqueeze(self.nd + d) * self.corr[s].reshape(shape)

    def opposite(self, tr, d, s):
        """The neighbour's trace at face (d, s)."""
        return torch.roll(tr[d, 1 - s], -1 if s == 1 else 1, dims=d)

    def at_end(self, d, s):
        sl = [slice(None)] * self.nd
        sl[d] = slice(self.n[d] - 1, None) if s == 1 else slice(0, 1)
        return tuple(sl)

    def own_left(self, d, s):
        """Whether this side is the left one, per element (broadcastable)."""
        m = torch.full(self.n, s == 1, device=self.dev)
        m[self.at_end(d, s)] = s == 0 if self.bc[d] == PERIODIC else True
        return m

    def prim(self, U):
        nd = self.nd
        v = [U[..., d + 1] / U[..., 0] for d in range(nd)]
        return U[..., 0], v, (GAMMA - 1) * (U[..., nd + 1] - 0.5 * U[..., 0] * sum(q * q for q in v))

    def flux(self, U):
        rho, v, p = self.prim(U)
        out = []
        for d in range(self.nd):
            f = [rho * v[d]] + [rho * v[d] * v[a] + (p if a == d else 0) for a in range(self.nd)]
            out.append(torch.stack(f + [(U[..., -1] + p) * v[d]], -1))
        return out

    def ghost(self, code, U, n):
        rho, v, p = self.prim(U)
        nd = self.nd
        vn = sum(v[d] * n[..., d] for d in range(nd))
        if code in (SLIP_WALL, SYMMETRY):
            vr = [v[d] - 2 * vn * n[..., d] for d in range(nd)]
            return torch.stack([rho] + [rho * q for q in vr] + [U[..., -1]], -1)
        vb = self.free["v"]
        vnb = sum(vb[d] * n[..., d] for d in range(nd))
        g1 = GAMMA - 1
        cl, cb = torch.sqrt(GAMMA * p / rho), math.sqrt(GAMMA * self.free["p"] / self.free["rho"])
        fast = vnb.abs() >= cb
        rl = torch.where(fast & (vn >= 0), vnb + 2 / g1 * cb, vn + 2 / g1 * cl)
        rb = torch.where(fast & (vn < 0), vn - 2 / g1 * cl, vnb - 2 / g1 * cb)
        c = 0.25 * g1 * (rl - rb)
        into = vn < 0
        s = torch.where(into, torch.full_like(p, self.free["rho"] ** GAMMA / self.free["p"]), rho ** GAMMA / p)
        r = (c * c / GAMMA * s) ** (1 / g1)
        pr, vbar = c * c * r / GAMMA, 0.5 * (rl + rb)
        vr = [torch.where(into, vb[d] + (vbar - vnb) * n[..., d], v[d] + (vbar - vn) * n[..., d]) for d in range(nd)]
        return torch.stack([r] + [r * q for q in vr] + [pr / g1 + 0.5 * r * sum(q * q for q in vr)], -1)

    def rusanov(self, L, R, n):
        FL, FR = self.flux(L), self.flux(R)
        f = sum(n[..., d:d + 1] * (FL[d] + FR[d]) for d in range(self.nd))
        eig = torch.maximum(*[sum(n[..., d] * v[d] for d in range(self.nd)).abs()
                              + torch.sqrt(torch.clamp(GAMMA * p / r, min=0)) for r, v, p in (self.prim(L), self.prim(R))])
        return 0.5 * (f - eig[..., None] * (R - L)), eig

    def roe(self, L, R, n):
        """Roe's flux with an entropy fix (2-D): 0.5 (FL + FR - |A| dU) by wave strengths."""
        (rl, vl, pl), (rr, vr, pr) = self.prim(L), self.prim(R)
        g1 = GAMMA - 1
        hl, hr = (L[..., 3] + pl) / rl, (R[..., 3] + pr) / rr
        q = torch.sqrt(rr / rl)
        mean = lambda a, b: (a + q * b) / (1 + q)
        u, v, h = mean(vl[0], vr[0]), mean(vl[1], vr[1]), mean(hl, hr)
        nx, ny = n[..., 0], n[..., 1]
        un, k = u * nx + v * ny, 0.5 * (u * u + v * v)
        a2 = g1 * (h - k)
        a = torch.sqrt(a2)
        unl, unr = vl[0] * nx + vl[1] * ny, vr[0] * nx + vr[1] * ny
        eps = 0.5 * ((unl - unr).abs() + (torch.sqrt(GAMMA * pl / rl) - torch.sqrt(GAMMA * pr / rr)).abs())
        fix = lambda w: torch.where(w < 2 * eps, 0.25 * w * w / eps + eps, w)
        l0, lp, lm = fix(un.abs()), fix((un + a).abs()), fix((un - a).abs())
        d = R - L
        dp = g1 * (k * d[..., 0] - u * d[..., 1] - v * d[..., 2] + d[..., 3])
        dm = nx * d[..., 1] + ny * d[..., 2] - un * d[..., 0]  # rho * d(un)
        s0, sp, sm = l0 * (d[..., 0] - dp / a2), lp * 0.5 * (dp / a2 + dm / a), lm * 0.5 * (dp / a2 - dm / a)
        tang = [l0 * (d[..., 1] - u * d[..., 0] - dm * nx), l0 * (d[..., 2] - v * d[..., 0] - dm * ny)]
        diss = torch.stack([s0 + sp + sm,
                            s0 * u + sp * (u + a * nx) + sm * (u - a * nx) + tang[0],
                            s0 * v + sp * (v + a * ny) + sm * (v - a * ny) + tang[1],
                            s0 * k + sp * (h + a * un) + sm * (h - a * un) + u * tang[0] + v * tang[1]], -1)
        FL, FR = self.flux(L), self.flux(R)
        return 0.5 * (sum(n[..., e:e + 1] * (FL[e] + FR[e]) for e in range(2)) - diss)

    def viscous(self, U, g):
        """Viscous flux of the reference solver in 3-D (its own shear terms, its flux.cpp)."""
        mu, pr = self.mu, 0.71
        rho, (u, v, w) = U[..., 0], [U[..., d + 1] / U[..., 0] for d in range(3)]
        e = U[..., 4] / rho - 0.5 * (u * u + v * v + w * w)
        dv = [[(g[d][..., a + 1] - g[d][..., 0] * q) / rho for a, q in enumerate((u, v, w))] for d in range(3)]
        de = []
        for d in range(3):
            dk = 0.5 * (u * u + v * v + w * w) * g[d][..., 0] + rho * (u * dv[d][0] + v * dv[d][1] + w * dv[d][2])
            de.append((g[d][..., 4] - dk - g[d][..., 0] * e) / rho)
        div = (dv[0][0] + dv[1][1] + dv[2][2]) / 3
        xx, yy, zz = (2 * mu * (dv[a][a] - div) for a in range(3))
        xy, xz, yz = mu * (dv[1][0] + dv[0][1]), mu * (dv[2][0] + dv[0][1]), mu * (dv[2][0] + dv[1][1])
        kq = mu / pr * GAMMA
        z = torch.zeros_like(rho)
        return [torch.stack([z, -xx, -xy, -zz, -(u * xx + v * xy + w * xz + kq * de[0])], -1),
                torch.stack([z, -xy, -yy, -yz, -(u * xy + v * yy + w * yz + kq * de[1])], -1),
                torch.stack([z, -xz, -yz, -zz, -(u * xz + v * yz + w * zz + kq * de[2])], -1)]

    def faces(self):
        return [(d, s) for d in range(self.nd) for s in (0, 1)]

    def residual(self, U):
        nd, ns = self.nd, self.case["kind"] == "ns"
        tr = {f: self.trace(U, *f) for f in self.faces()}
        F = self.flux(U)
        if ns:
            self.mu, beta, tau = 1.0 / 1600, 0.5, 0.1
            gr = [self.lines(self.D, U, d) for d in range(nd)]
            pen = {}
            for d, s in self.faces():
                n = self.face[d, s][0]
                up = n[..., 0] + n[..., 1] + math.sqrt(2.0) * n[..., 2]
                pen[d, s] = torch.where(up < 0, -beta, beta)[..., None]  # changes sign with the side, as (own - other) does
                o = self.opposite(tr, d, s)
                jump = 0.5 * (tr[d, s] + o) - pen[d, s] * (tr[d, s] - o) - tr[d, s]
                gr[d] = gr[d] + self.lift((2 * s - 1) * jump, d, s)
            g = [sum(self.JG[d][a][..., None] * gr[d] for d in range(nd)) / self.det[..., None] for a in range(nd)]
            F = [a + b for a, b in zip(self.viscous(U, g), F)]
            vt = {f: self.viscous(tr[f], [self.trace(q, *f) for q in g]) for f in self.faces()}
        Fr = [sum(self.JG[d][a][..., None] * F[a] for a in range(nd)) for d in range(nd)]
        div = sum(self.lines(self.D, Fr[d], d) for d in range(nd))
        for d, s in self.faces():
            n, dA = self.face[d, s]
            own, other = tr[d, s], self.opposite(tr, d, s)
            end = self.at_end(d, s)
            if self.bc[d] != PERIODIC:
                other[end] = self.ghost(self.bc[d], own[end], n[end])
            Fn, eig = self.rusanov(own, other, n)
            if self.case["roe"]:
                Fn = self.roe(own, other, n)
            left = self.own_left(d, s).reshape(self.n + [1] * (nd - 1))
            if (d, s) in self.wave:
                self.wave[d, s] = torch.where(left, eig, self.wave[d, s])
            if ns:
                ov = [torch.roll(q, -1 if s == 1 else 1, dims=d) for q in vt[d, 1 - s]]
                lf, sg = left[..., None], torch.where(left, 1.0, -1.0)[..., None]
                L = [torch.where(lf, a, b) for a, b in zip(vt[d, s], ov)]
                R = [torch.where(lf, b, a) for a, b in zip(vt[d, s], ov)]
                nl = n * sg
                # the reference pairs the left y-flux with the right z-flux here (its face.cpp)
                sd = nl[..., :1] * (L[0] - R[0]) + nl[..., 1:2] * (L[1] - R[1]) + nl[..., 2:] * (L[1] - R[2])
                dU = (own - other) * sg
                c = 0.0
                for a in range(nd):
                    na = nl[..., a:a + 1]
                    c = c + na * (0.5 * (L[a] + R[a]) + pen[d, s] * sg * na * sd + tau * na * dU)
                Fn = Fn + sg * c
            q = Fn * dA[..., None] - (2 * s - 1) * self.trace(Fr[d], d, s)
            div = div + self.lift(q, d, s)
        return div

    def first_wave(self, U):
        for f in self.faces():
            n = self.face[f][0]
            r, v, p = self.prim(self.trace(U, *f))
            self.wave[f] = sum(v[d] * n[..., d] for d in range(self.nd)).abs() + torch.sqrt(GAMMA * p / r)

    def local_dt(self):
        limit = [1.393, 0.464, 0.235, 0.1453, 0.100, 0.0736][self.P]
        vol, surf = self.det, 0.0
        for _ in range(self.nd):
            vol = vol @ self.w
        for f in self.faces():
            a = self.wave[f] * self.face[f][1]
            for _ in range(self.nd - 1):
                a = a @ self.w
            surf = surf + a
        return (0.5 * limit * 2 * vol / surf).reshape(self.n + [1] * (self.nd + 1))

    def step(self, U, dt, first=False):
        if dt is None:
            if first:
                self.first_wave(U)
            dt = self.local_dt()
        out, V, first_div = U, U, None
        for a, b in ((0.5, 1 / 6), (0.5, 1 / 3), (1.0, 1 / 3), (None, 1 / 6)):
            k = self.residual(V)
            first_div = k if first_div is None else first_div
            k = (k + self.source) / self.det[..., None] * dt
            out = out - b * k
            V = U - a * k if a else None
        return out


def _multigrid(grids, low, U):
    """One P-multigrid V-cycle below the finest grid (two smoothing steps a level)."""
    P = len(grids) - 1

    def between(a, b, V):
        M = torch.as_tensor(_lagrange(a.x, b.x), device=a.dev)
        for d in range(a.nd):
            V = a.lines(M, V, d)
        return V

    state, kept = {}, {}
    V, res = U, grids[P].residual(U)
    for q in range(P - 1, low - 1, -1):
        g = grids[q]
        V, res = between(grids[q + 1], g, V), between(grids[q + 1], g, res)
        kept[q] = V
        g.source = res - g.residual(V)
        for _ in range(2):
            V = g.step(V, None)
        state[q] = V
        if q > low:
            res = g.residual(V) + g.source
    for q in range(low, P):
        g = grids[q]
        for _ in range(2):
            state[q] = g.step(state[q], None)
        up = between(g, grids[q + 1], state[q] - kept[q])
        state[q + 1] = (state[q + 1] if q + 1 < P else U) + up
    return state[P]


def _exact_one(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = _Grid(case, seed, dev)
    U = g.from_layout(torch.as_tensor(_initial(case, seed), device=dev))
    if case["call"] == "residual":
        k = g.residual(U)
        q = k * k / g.det[..., None]
        for _ in range(g.nd):
            q = torch.tensordot(q, g.w, dims=([g.nd], [0]))
        return {"divF": g.to_layout(k), "norm": torch.sqrt(q.reshape(-1, g.F).sum(0)).cpu().numpy()}
    if case["kind"] != "channel":
        for _ in range(1 if case["call"] == "update" else case["steps"]):
            U = g.step(U, _dt(case))
        return g.to_layout(U)
    grids = [_Grid(case, seed, dev, order=q) for q in range(case["order"])] + [g]
    free = g.free
    rest = torch.tensor([1.0, free["v"][0], 0.0, free["p"] / (GAMMA - 1) + 0.5 * free["v"][0] ** 2], dtype=torch.float64, device=dev)
    for c in grids[:-1]:  # coarse levels take their first wave speeds from the free stream
        c.first_wave(rest.expand(c.n + [c.N] * 2 + [4]))
    for i in range(case["steps"]):
        U = g.step(U, None, first=i == 0)
        U = _multigrid(grids, 0, U)
    return g.to_layout(U)


def exact(case, seed):
    if case["kind"] == "batch":
        return [_exact_one(m, seed * 100 + i) for i, m in enumerate(_members(case, seed))]
    return _exact_one(case, seed)
