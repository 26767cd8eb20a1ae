"""What is timed: explicit finite-volume steps as a program using this package takes them.

A case names a mesh (``n`` squares or hexes a side, split into triangles or tetrahedra by the
package's own seeded generators), a solver with its options, the number of steps between two
looks at the result, and how the program drives the solver:

* ``graph``: ``advance(steps, graph=True)``, the device loop of a long run;
* ``advance``: ``advance(steps)`` (shallow water has no graph option);
* ``loop``: the driver loop of a manapy script, ``stepper`` / ``compute_fluxes`` /
  ``compute_new_val`` once per step;
* ``unsteady``: the same loop with new face velocities given from pinned host memory before
  every step, as a program coupled to a flow solver does.

``prepare`` builds the domain, the variables and the solver from the seed (vertex jitter,
diagonals and numbering of the mesh, velocity, initial state, source); ``run`` takes the steps
and returns the state in the mesh's own cell numbering, on the device.  ``exact`` computes the
same steps with plain torch operations in 64 bits from the mesh's vertices and elements.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import manapy_b200 as M
from manapy_b200 import meshgen

GRAV = 9.81
GAMMA = 1.4
DIFFUSION = {2: (1e-3, 5e-4, 0.0), 3: (1e-3, 1e-3, 5e-4)}

_BASE = {"kind": "advdiff", "dim": 2, "n": 100, "order": 2, "diffusion": True, "precision": "fp64", "bc": "dirichlet",
         "source": False, "walls": "neumann", "mode": "graph", "steps": 10}


def _case(name=None, **kw):
    c = dict(_BASE, **kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # a script's first try on a small mesh: one step of manapy's own loop, launch latency only
        _case("tri-loop-1k", n=24, mode="loop", steps=1),
        # the first-order run on 20,000 triangles (the C1 workload), all of its 200 steps
        _case("tri-o1-20k", n=100, order=1, steps=200),
        # a mid-size second-order run with a source term, ragged size
        _case("tri-o2-63k", n=177, source=True, steps=20),
        # the flagship: 2M triangles, second order + diffusion (the C2 workload)
        _case("tri-o2-2m", n=1000, steps=10),
        # velocities from another code before every step
        _case("tri-unsteady-180k", n=300, mode="unsteady", steps=2),
        # pure advection (AdvectionSolver), sides of several kinds
        _case("tri-advec-245k", kind="advec", n=350, diffusion=False, bc="mixed", steps=10),
        # FP32 state with compensated sums
        _case("tri-fp32c-500k", n=500, precision="fp32c", steps=10),
        # tetrahedra: a small mesh, and one beyond the L2 cache (the C4 workload's physics)
        _case("tet-o2-16k", dim=3, n=14, bc="mixed", steps=20),
        _case("tet-o2-384k", dim=3, n=40, steps=5),
        # shallow water: a dam break over a bump on 1.3M triangles (the C3 workload's physics), and
        # a closed basin at second order
        _case("sw-o1-1.3m", kind="sw", n=800, order=1, diffusion=False, mode="advance", steps=10),
        _case("sw-o2-45k", kind="sw", n=150, order=2, diffusion=False, walls="reflective", mode="advance", steps=10),
        # compressible Euler, 720,000 triangles (the E1 workload's physics)
        _case("euler-720k", kind="euler", n=600, order=1, diffusion=False, steps=24),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["advdiff", "advdiff", "advdiff", "advec", "sw", "sw", "euler"])
    if kind in ("advdiff", "advec"):
        dim = rng.choice([2, 2, 3])
        n = _log_int(rng, 16, 900) if dim == 2 else _log_int(rng, 4, 38)
        mode = rng.choice(["graph", "graph", "loop", "unsteady"])
        c = _case(kind=kind, dim=dim, n=n, order=rng.choice([1, 2, 2]), diffusion=kind == "advdiff",
                  precision=rng.choice(["fp64", "fp64", "fp32c"]), bc=rng.choice(["dirichlet", "mixed"]),
                  source=rng.random() < 0.3, mode=mode)
    elif kind == "sw":
        order = rng.choice([1, 1, 2])
        c = _case(kind="sw", n=_log_int(rng, 16, 700), order=order, diffusion=False,
                  precision=rng.choice(["fp64", "fp32c"]) if order == 1 else "fp64",
                  walls=rng.choice(["neumann", "reflective"]), mode=rng.choice(["advance", "loop"]))
    else:
        c = _case(kind="euler", n=_log_int(rng, 16, 560), order=1, diffusion=False, mode=rng.choice(["graph", "loop"]))
    # as many steps as keep the pass below the largest listed one
    most = max(1, int(8e6 / (_cells(c) * (4 if c["dim"] == 3 else 2 if c["kind"] == "sw" else 1))))
    few = 4 if c["mode"] in ("loop", "unsteady") else 48
    c["steps"] = rng.randint(1, min(most, few))
    return c


def _cells(c):
    return 2 * c["n"] ** 2 if c["dim"] == 2 else 6 * c["n"] ** 3


def work(case):
    """Compulsory traffic of the steps: per cell-update every input and output array once
    (32-bit indices, 64-bit reals; state reals of 8 bytes, or 4 with FP32 state), nothing
    intermediate."""
    c = case
    if c["kind"] == "sw":
        b, f = (152.4 if c["order"] == 1 else 176.4), (400 if c["order"] == 1 else 600)
        state = 7
    elif c["kind"] == "euler":
        b, f, state = 136.2, 300, 10
    else:
        b = {(2, 1, True): 146.6, (2, 2, True): 198.8, (2, 1, False): 48.2, (2, 2, False): 114.4,
             (3, 1, True): 177.5, (3, 2, True): 265.9, (3, 1, False): 56.3, (3, 2, False): 161.3}[
                 (c["dim"], c["order"], bool(c["diffusion"]))]
        f = (60 if c["order"] == 1 else 150) + (90 if c["diffusion"] else 0)
        f *= 2 if c["dim"] == 3 else 1
        state = 2
        if c["source"]:
            b += 8
    if c["precision"] == "fp32c":
        b -= 4 * state
    u = float(_cells(c)) * c["steps"]
    return {"bytes": b * u, "flops": f * u}


# ------------------------------------------------------------------ inputs from the seed

def _mesh(case, seed):
    if case["dim"] == 2:
        return meshgen.square_triangles(case["n"], seed=seed)
    return meshgen.cube_tetrahedra(case["n"], seed=seed)


def _bc(case):
    sides = ["in", "out", "upper", "bottom"] + (["front", "back"] if case["dim"] == 3 else [])
    if case["bc"] == "dirichlet":
        return {s: "dirichlet" for s in sides}, {s: (1.0 if s == "in" else 0.0) for s in sides}
    bc = {"in": "dirichlet", "out": "neumann", "upper": "nonslip", "bottom": "neumann", "front": "nonslip",
          "back": "neumann"}
    return {s: bc[s] for s in sides}, {"in": 1.0}


def _params(seed):
    r = np.random.default_rng(seed + 1000)
    return {"x0": r.uniform(0.35, 0.65, 3), "amp": r.uniform(0.5, 2.0), "speed": r.uniform(0.5, 1.5),
            "ang": r.uniform(0.1, 1.4), "ratio": r.uniform(1.3, 2.5), "bump": r.uniform(0.05, 0.15)}


def _velocity(case, p, fc):
    """Face velocity: a rotating field (2D) or a uniform one (3D)."""
    x, y = fc[:, 0], fc[:, 1]
    s = p["speed"]
    if case["dim"] == 2:
        return [s * np.sin(np.pi * x) * np.cos(np.pi * y), -s * np.cos(np.pi * x) * np.sin(np.pi * y), np.zeros(len(x))]
    return [np.full(len(x), s * math.cos(p["ang"])), np.full(len(x), s * math.sin(p["ang"])), np.full(len(x), 0.25 * s)]


def _scalar(case, p, cc):
    d2 = sum((cc[:, k] - p["x0"][k]) ** 2 for k in range(case["dim"]))
    return p["amp"] * np.exp(-d2 / 0.02)


def _source(p, cc):
    return 0.3 * np.sin(2 * np.pi * cc[:, 0]) * p["amp"]


def _sw_state(p, cc):
    x, y = cc[:, 0], cc[:, 1]
    h = np.where(x < p["x0"][0], p["ratio"], 1.0)
    hc = h * 0.2 * np.exp(-((x - 0.5) ** 2 + (y - p["x0"][1]) ** 2) / 0.05)
    Z = p["bump"] * np.exp(-((x - 0.7) ** 2 + (y - 0.5) ** 2) / 0.02)
    return [h, np.zeros(len(x)), np.zeros(len(x)), hc, Z]


def _euler_state(p, cc):
    x, y = cc[:, 0], cc[:, 1]
    rho = 1.0 + 0.2 * np.sin(2 * np.pi * x) * np.cos(2 * np.pi * y)
    P = 1.0 + 0.3 * p["amp"] * np.exp(-40 * ((x - p["x0"][0]) ** 2 + (y - p["x0"][1]) ** 2))
    u = 0.3 * np.cos(np.pi * y)
    v = 0.2 * np.sin(np.pi * x)
    return [rho, P, rho * u, rho * v, P / (GAMMA - 1) + 0.5 * rho * (u * u + v * v)]


def prepare(case, seed):
    dom = M.Domain(dim=case["dim"], mesh=_mesh(case, seed))
    p = _params(seed)
    cc = dom.cells.center
    s = {"case": case, "dom": dom}
    if case["kind"] in ("advdiff", "advec"):
        bc, values = _bc(case)
        w = M.Variable(domain=dom, BC=bc, values=values)
        vel = [M.Variable(domain=dom) for _ in range(3)]
        faces = _velocity(case, p, dom.faces.center)
        for var, a in zip(vel, faces):
            var.face = a
            var.interpolate_facetocell()
        w.cell = _scalar(case, p, cc)
        conf = dict(order=case["order"], cfl=0.8, precision=case["precision"])
        if case["kind"] == "advdiff":
            D = DIFFUSION[case["dim"]]
            S = M.AdvectionDiffusionSolver(w, vel=tuple(vel), conf=M.Struct(Dxx=D[0], Dyy=D[1], Dzz=D[2], **conf))
        else:
            S = M.AdvectionSolver(w, vel=tuple(vel), conf=M.Struct(**conf))
        if case["source"]:
            w.source = _source(p, cc)
        s.update(S=S, vars=[w], vel=vel)
        if case["mode"] == "unsteady":
            # two velocity fields in pinned memory, given in turn
            s["faces"] = [[torch.from_numpy(np.ascontiguousarray(f * a)).pin_memory() for a in faces[:case["dim"]]]
                          for f in (1.0, 0.9)]
    elif case["kind"] == "sw":
        vs = [M.Variable(domain=dom) for _ in range(5)]
        for var, a in zip(vs, _sw_state(p, cc)):
            var.cell = a
        S = M.ShallowWaterSolver(vs[0], hvel=(vs[1], vs[2]), hc=vs[3], Z=vs[4],
                                 conf=M.Struct(order=case["order"], cfl=0.4, grav=GRAV, walls=case["walls"],
                                               precision=case["precision"]))
        s.update(S=S, vars=vs[:4])
    else:
        vs = [M.Variable(domain=dom) for _ in range(5)]
        for var, a in zip(vs, _euler_state(p, cc)):
            var.cell = a
        s.update(S=M.EulerSolver(*vs, conf=M.Struct(cfl=0.4, gamma=GAMMA)), vars=vs)
    return s


def run(s):
    case, S = s["case"], s["S"]
    steps, mode = case["steps"], case["mode"]
    if mode == "graph":
        S.advance(steps, graph=True)
    elif mode == "advance":
        S.advance(steps)
    else:
        for k in range(steps):
            if mode == "unsteady":
                for var, a in zip(s["vel"], s["faces"][k % 2]):
                    var.face = a
                    var.interpolate_facetocell()
            S.stepper()
            if case["kind"] != "euler":
                S.compute_fluxes()      # the Euler step forms its fluxes in compute_new_val
            S.compute_new_val()
    dm = s["dom"].device_mesh
    return [dm.to_host_order("cell", v.dev("cell")) for v in s["vars"]]


# ------------------------------------------------------------------ the same steps in plain torch

def _add(n, idx, val):
    return torch.zeros(n, dtype=torch.float64, device=val.device).index_add_(0, idx, val)


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=1)


def _dot(a, b):
    return (a * b).sum(1)


class _Geometry:
    """Connectivity and geometry of a triangle or tetrahedron mesh, on ``dev``."""

    def __init__(self, case, seed, dev):
        el, vx = _mesh(case, seed)
        dim = self.dim = case["dim"]
        k = dim + 1
        cn = torch.from_numpy(el[:, :k].astype(np.int64)).to(dev)
        vx = torch.from_numpy(vx).to(dev)
        X = vx[:, :dim]
        nc, nn = len(cn), len(X)
        self.nc, self.nn, self.cn, self.X = nc, nn, cn, X
        P = X[cn]
        self.cc = P.sum(1) / k
        if dim == 2:
            a, b = P[:, 0] - P[:, 1], P[:, 0] - P[:, 2]
            self.vol = 0.5 * (a[:, 0] * b[:, 1] - b[:, 0] * a[:, 1]).abs()
            loc = torch.tensor([[0, 1], [1, 2], [2, 0]], device=dev)
        else:
            self.vol = _dot(P[:, 1] - P[:, 0], _cross(P[:, 2] - P[:, 0], P[:, 3] - P[:, 0])).abs() / 6
            loc = torch.tensor([[0, 1, 2], [2, 3, 0], [0, 1, 3], [3, 1, 2]], device=dev)
        # faces: node tuples in descending order; first cell = the smaller cell number
        pf = cn[:, loc].reshape(-1, dim).sort(dim=1, descending=True).values
        key = pf[:, 0]
        for j in range(1, dim):
            key = key * nn + pf[:, j]
        uk, inv, cnt = torch.unique(key, return_inverse=True, return_counts=True)
        nf = self.nf = len(uk)
        order = torch.sort(inv, stable=True).indices
        start = torch.cumsum(cnt, 0) - cnt
        owner = order // k
        self.c0 = owner[start]
        self.inner = cnt == 2
        self.c1 = torch.where(self.inner, owner[(start + 1).clamp(max=len(owner) - 1)], torch.full_like(start, -1))
        self.cf = inv.reshape(nc, k)
        fn = self.fn = pf[order[start]]
        self.fc = X[fn].mean(1)
        if dim == 2:
            A, B = X[fn[:, 0]], X[fn[:, 1]]
            N = torch.stack([A[:, 1] - B[:, 1], B[:, 0] - A[:, 0]], 1)
        else:
            N = 0.5 * _cross(X[fn[:, 1]] - X[fn[:, 0]], X[fn[:, 2]] - X[fn[:, 0]])
        flip = _dot(self.cc[self.c0] - self.fc, N) > 0
        self.N = torch.where(flip[:, None], -N, N)
        self.mes = self.N.square().sum(1).sqrt()
        self.bf = torch.nonzero(~self.inner).flatten()
        self.side = torch.zeros(nf, dtype=torch.long, device=dev)
        self.side[self.bf] = self._sides(vx[:, 3].long())
        # ghost centres: the cell centre mirrored at the face
        n = self.N / self.mes[:, None]
        d = _dot(self.fc - self.cc[self.c0], n)
        self.gc = self.cc[self.c0] + 2 * d[:, None] * n

    def _sides(self, tag):
        """The side of every boundary face: its vertices' tag, or where they differ (at an edge of the
        cube) the last of 4, 3, 6, 5 among them, as manapy names faces."""
        t = tag[self.fn[self.bf]]
        s = t[:, 0].clone()
        for k in (4, 3, 6, 5):
            s = torch.where((t == k).any(1), torch.full_like(s, k), s)
        return torch.where((t == t[:, :1]).all(1), t[:, 0], s)

    def _pairs(self, items, item_node, drop_self):
        """Distinct (cell, item) pairs that share a vertex; ``item_node``: the vertices of the items."""
        node = item_node.flatten()
        of = items.repeat_interleave(item_node.shape[1])
        order = torch.sort(node, stable=True).indices
        node, of = node[order], of[order]
        cnt = torch.bincount(node, minlength=self.nn)
        start = torch.cumsum(cnt, 0) - cnt
        cell = torch.arange(self.nc, device=node.device).repeat_interleave(self.cn.shape[1])
        v = self.cn.flatten()
        rep = cnt[v]
        i = cell.repeat_interleave(rep)
        off = torch.arange(len(i), device=node.device) - (torch.cumsum(rep, 0) - rep).repeat_interleave(rep)
        j = of[start[v].repeat_interleave(rep) + off]
        big = max(self.nc, self.nf)
        u = torch.unique(i * big + j)
        i, j = u // big, u % big
        if drop_self:
            keep = i != j
            i, j = i[keep], j[keep]
        return i, j

    def stencil(self):
        """The least-squares stencil: vertex neighbours, and the ghosts of boundary faces at a vertex."""
        self.si, self.sj = self._pairs(torch.arange(self.nc, device=self.cn.device), self.cn, True)
        self.gi, self.gf = self._pairs(self.bf, self.fn[self.bf], False)
        self.sd = self.cc[self.sj] - self.cc[self.si]
        self.gd = self.gc[self.gf] - self.cc[self.gi]
        dim = self.dim
        m = torch.zeros(self.nc, dim, dim, dtype=torch.float64, device=self.cn.device)
        m.index_add_(0, self.si, self.sd[:, :, None] * self.sd[:, None, :])
        m.index_add_(0, self.gi, self.gd[:, :, None] * self.gd[:, None, :])
        self.minv = torch.linalg.inv(m)

    def gradient(self, w, g):
        r = torch.zeros(self.nc, self.dim, dtype=torch.float64, device=w.device)
        r.index_add_(0, self.si, self.sd * (w[self.sj] - w[self.si])[:, None])
        r.index_add_(0, self.gi, self.gd * (g[self.gf] - w[self.gi])[:, None])
        return (self.minv @ r[:, :, None])[:, :, 0]

    def limiter(self, w, g, grad):
        other = torch.where(self.inner, w[self.c1.clamp(min=0)], g)
        a, b = w[self.c0][self.cf], other[self.cf]
        hi = torch.maximum(torch.maximum(a, b).max(1).values, w)
        lo = torch.minimum(torch.minimum(a, b).min(1).values, w)
        d = ((self.fc[self.cf] - self.cc[:, None, :]) * grad[:, None, :]).sum(2)
        room = torch.where(d > 0, (hi - w)[:, None], (lo - w)[:, None]) / d
        eps = 1e-8 if self.dim == 2 else 1e-10
        psi = torch.where(d.abs() < eps, torch.ones_like(d), room.clamp(max=1.0))
        return psi.min(1).values.clamp(max=1.0)

    def vertex_weights(self):
        nv = self.dim + 1
        node = torch.cat([self.cn.flatten(), self.fn[self.bf].flatten()])
        src = torch.cat([torch.arange(self.nc, device=node.device).repeat_interleave(nv),
                         self.nc + self.bf.repeat_interleave(self.dim)])
        pts = torch.cat([self.cc, self.gc])[src] - self.X[node]
        m = torch.zeros(self.nn, self.dim, self.dim, dtype=torch.float64, device=node.device)
        m.index_add_(0, node, pts[:, :, None] * pts[:, None, :])
        R = torch.zeros(self.nn, self.dim, dtype=torch.float64, device=node.device).index_add_(0, node, pts)
        lam = -torch.linalg.solve(m, R[:, :, None])[:, :, 0]
        num = torch.bincount(node, minlength=self.nn).double()
        den = num + _dot(lam, R)
        self.vn, self.vs = node, src
        self.va = (1 + _dot(lam[node], pts)) / den[node]

    def to_vertices(self, w, g):
        return _add(self.nn, self.vn, self.va * torch.cat([w, g])[self.vs])

    def diamond(self, D):
        """D grad(w) . N of every face as a linear form: coefficients of the face's vertices and of
        the right minus the left value."""
        N = self.N
        v1 = self.cc[self.c0]
        v2 = torch.where(self.inner[:, None], self.cc[self.c1.clamp(min=0)], self.gc)
        D = torch.tensor(D[:self.dim], dtype=torch.float64, device=N.device)
        DN = D * N
        air = _dot(N, v2 - v1)
        if self.dim == 2:
            # grad w . e = dw along v1 -> v2 and along the face: solved in the face's frame
            A, B = self.X[self.fn[:, 0]], self.X[self.fn[:, 1]]
            t, e = B - A, v2 - v1
            det = t[:, 0] * e[:, 1] - t[:, 1] * e[:, 0]
            # grad = (dwt * perp(e) - dwe * perp(t)) / det, perp(a) = (a_y, -a_x)
            pt = torch.stack([t[:, 1], -t[:, 0]], 1)
            pe = torch.stack([e[:, 1], -e[:, 0]], 1)
            ct, ce = _dot(pe, DN) / det, -_dot(pt, DN) / det
            self.dv = [-ct, ct]
            self.dw = ce
        else:
            Q = [self.X[self.fn[:, k]] for k in range(3)]
            flip = _dot(_cross(Q[1] - Q[0], Q[2] - Q[0]), N) < 0
            e = v2 - v1
            # w along e, and the vertex values: grad . N-part from e, tangential part from the vertices
            i, j = torch.where(flip, 2, 1), torch.where(flip, 1, 2)
            Qs = torch.stack(Q, 1)
            r = torch.arange(self.nf, device=N.device)
            Q2, Q3 = Qs[r, i], Qs[r, j]
            f1 = 0.5 * _cross(Q3 - Q2, v1 - v2)
            f2 = 0.5 * _cross(Q[0] - Q3, v1 - v2)
            a, b = _dot(f1, DN) / air, _dot(f2, DN) / air
            # (V_0 - V_3) a + (V_2 - V_3) b in the oriented order (0, i, j)
            self.dv = [a, torch.where(flip, -a - b, b), torch.where(flip, b, -a - b)]
            self.dw = _dot(N, DN) / air

    def diffusive(self, w, other, vert):
        v = self.dw * (other - w[self.c0])
        for k in range(self.dim):
            v = v + self.dv[k] * vert[self.fn[:, k]]
        return v

    def gather(self, F):
        """Minus the outward sum of the face fluxes of every cell."""
        r = -_add(self.nc, self.c0, F)
        return r.index_add_(0, self.c1[self.inner], F[self.inner])


def _exact_scalar(case, seed, g, p):
    dev = g.cc.device
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(dev)  # noqa: E731
    cc = np.concatenate([g.cc.cpu().numpy(), np.zeros((g.nc, 3 - g.dim))], 1)
    fc = np.concatenate([g.fc.cpu().numpy(), np.zeros((g.nf, 3 - g.dim))], 1)
    w = to(_scalar(case, p, cc))
    src = to(_source(p, cc)) if case["source"] else torch.zeros_like(w)
    V = torch.stack([to(a) for a in _velocity(case, p, fc)[:g.dim]], 1)
    D = DIFFUSION[g.dim] if case["kind"] == "advdiff" else (0.0, 0.0, 0.0)
    bc, values = _bc(case)
    name = {1: "in", 2: "out", 3: "upper", 4: "bottom", 5: "front", 6: "back"}
    if case["order"] == 2:
        g.stencil()
    if case["diffusion"]:
        g.vertex_weights()
        g.diamond(D)

    def ghosts(w):
        out = torch.zeros(g.nf, dtype=torch.float64, device=dev)
        wi = w[g.c0]
        for t, s in name.items():
            if s in bc:
                v = {"dirichlet": torch.full_like(wi, values.get(s, 0.0)), "neumann": wi, "nonslip": -wi}[bc[s]]
                out = torch.where(g.side == t, v, out)
        return out

    def time_step(V):
        u = V[g.cf].sum(1) / g.cf.shape[1]
        N = g.N[g.cf]
        lam = (u[:, None, :] * N).sum(2).abs().sum(1) + (sum(D) * g.mes[g.cf].square()).sum(1) / g.vol
        return torch.where(lam > 0, 0.8 * g.vol / lam, torch.full_like(lam, 1e6)).min().clamp(max=1e6)

    for k in range(case["steps"]):
        U = V * (1.0, 0.9)[k % 2] if case["mode"] == "unsteady" else V
        dt = time_step(U)
        gh = ghosts(w)
        s = _dot(U, g.N)
        left, right = w[g.c0], torch.where(g.inner, w[g.c1.clamp(min=0)], gh)
        other = right
        if case["order"] == 2:
            grad = g.gradient(w, gh)
            grad = grad * g.limiter(w, gh, grad)[:, None]
            left = left + _dot(grad[g.c0], g.fc - g.cc[g.c0])
            c1 = g.c1.clamp(min=0)
            right = torch.where(g.inner, right + _dot(grad[c1], g.fc - g.cc[c1]), right)
        rez = g.gather(s * torch.where(s >= 0, left, right))
        if case["diffusion"]:
            rez = rez - g.gather(g.diffusive(w, other, g.to_vertices(w, gh)))
        w = w + dt * (rez / g.vol + src)
    return [w]


def _srnh(l, r, n, mes, grav):
    """SRNH flux of (h, hu, hv, hc) with the eigenvalues u - c, u + c, 0 and u of its Roe matrix."""
    hl, hul, hvl, hcl, Zl = l
    hr, hur, hvr, hcr, Zr = r
    nx, ny = n[:, 0], n[:, 1]
    sl, sr = hl.sqrt(), hr.sqrt()
    roe = lambda a, b: (a / hl * sl + b / hr * sr) / (sl + sr)  # noqa: E731
    uh, vh, ch = roe(hul, hur), roe(hvl, hvr), roe(hcl, hcr)
    u, v = (uh * nx + vh * ny) / mes, (vh * nx - uh * ny) / mes
    rot = lambda a, b: ((a * nx + b * ny) / mes, (b * nx - a * ny) / mes)  # noqa: E731
    (ul, vl), (ur, vr) = rot(hul, hvl), rot(hur, hvr)
    c = (grav * (hl + hr) / 2).sqrt()
    a, b = u + c, u - c
    sgn = lambda x: torch.where(x.abs() < 1e-10, torch.zeros_like(x), x.sign())  # noqa: E731
    sa, sb, s0 = sgn(a), sgn(b), sgn(u)
    ia = torch.where(sa == 0, torch.zeros_like(a), sa / a)
    ib = torch.where(sb == 0, torch.zeros_like(b), sb / b)
    d0, d1, d2, d3, d4 = hr - hl, ur - ul, vr - vl, hcr - hcl, Zr - Zl
    dh = ((sb * a - sa * b) * d0 + (sa - sb) * d1) / (2 * c) + 0.5 * c * (ia - ib) * d4
    dq = (a * b * (sb - sa) * d0 + (a * sa - b * sb) * d1) / (2 * c) + 0.5 * c * (sa - sb) * d4
    dv = v * dh + s0 * (d2 - v * d0)
    dc = ch * dh + s0 * (d3 - ch * d0)
    h, q, t, hc = (hl + hr) / 2 - dh / 2, (ul + ur) / 2 - dq / 2, (vl + vr) / 2 - dv / 2, (hcl + hcr) / 2 - dc / 2
    un, vn = (q * nx - t * ny) / mes, (q * ny + t * nx) / mes
    qs = nx * un + ny * vn
    p = 0.5 * grav * h * h
    return [qs, qs * un / h + p * nx, qs * vn / h + p * ny, qs * hc / h]


def _exact_sw(case, seed, g, p):
    dev = g.cc.device
    cc = np.concatenate([g.cc.cpu().numpy(), np.zeros((g.nc, 1))], 1)
    q = [torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(dev) for a in _sw_state(p, cc)]
    Z = q[4]
    if case["order"] == 2:
        g.stencil()
    c1 = torch.where(g.inner, g.c1, g.c0)
    mine = torch.arange(g.nc, device=dev)[:, None]
    out = torch.where(g.c0[g.cf] == mine, 1.0, -1.0)
    nf = g.N[g.cf] * out[:, :, None].double()              # outward normals of the local faces
    inner = g.inner[g.cf]
    # the neighbours across inner faces, moved to the front of the row; manapy reads slot j of
    # that list for local face j, and its padding as the last cell
    nb = torch.where(g.c0[g.cf] == mine, g.c1[g.cf], g.c0[g.cf])
    order = torch.sort((~inner).long(), dim=1, stable=True).indices
    fid = torch.gather(nb, 1, order)
    fid = torch.where(torch.arange(3, device=dev)[None] < inner.sum(1)[:, None], fid, torch.full_like(fid, g.nc - 1))
    b = g.X[g.cn[:, 1]]
    for _ in range(case["steps"]):
        h, hu, hv, hc = q[:4]
        N, mes = g.N[g.cf], g.mes[g.cf]
        un = ((hu / h)[:, None] * N[..., 0] + (hv / h)[:, None] * N[..., 1]).abs()
        dt = (0.4 * g.vol / ((un / mes + (GRAV * h).sqrt()[:, None]) * mes).sum(1)).min().clamp(max=1e6)
        left = [a[g.c0] for a in q]
        right = [a[c1] for a in q]
        if case["walls"] == "reflective":
            k = 2 * (left[1] * g.N[:, 0] + left[2] * g.N[:, 1]) / g.mes.square()
            right[1] = torch.where(g.inner, right[1], left[1] - k * g.N[:, 0])
            right[2] = torch.where(g.inner, right[2], left[2] - k * g.N[:, 1])
        if case["order"] == 2:
            gh, gc = h[g.c0], hc[g.c0]
            dh, dc = g.gradient(h, gh), g.gradient(hc, gc)
            psi = g.limiter(hc, gc, dc)[:, None]
            for a, d in ((0, psi * dh), (3, psi * dc)):
                left[a] = left[a] + _dot(d[g.c0], g.fc - g.cc[g.c0])
                right[a] = torch.where(g.inner, right[a] + _dot(d[c1], g.fc - g.cc[c1]), right[a])
        rez = [g.gather(F) for F in _srnh(left, right, g.N, g.mes, GRAV)]
        # the bathymetry source
        hp = torch.where(inner, h[fid], h[:, None])
        zp = torch.where(inner, Z[fid], Z[:, None])
        S = nf
        m = hp[:, :, None] * S                              # rows j: (mata_j, matb_j)
        hm = 0.5 * (h[:, None] + hp)
        rhs = (hm.square()[:, :, None] * S).sum(1)
        sysm = torch.cat([torch.ones(g.nc, 1, 3, dtype=torch.float64, device=dev), m.transpose(1, 2)], 1)
        H = torch.linalg.solve(sysm, torch.cat([3 * h[:, None], rhs], 1)[:, :, None])[:, :, 0]
        z = (Z + h)[:, None] - H
        G = g.cc
        n0 = torch.stack([G[:, 1] - b[:, 1], -(G[:, 0] - b[:, 0])], 1)
        n1, n2 = n0 - S[:, 1], n0 + S[:, 0]
        e = lambda a, i: a[:, i, None]  # noqa: E731
        s = (0.5 * e(H, 0) * (e(zp, 0) * S[:, 0] + e(z, 1) * n0 - e(z, 2) * n2)
             + 0.5 * e(H, 1) * (e(zp, 1) * S[:, 1] - e(z, 0) * n0 + e(z, 2) * n1)
             + 0.5 * e(H, 2) * (e(zp, 2) * S[:, 2] + e(z, 0) * n2 - e(z, 1) * n1))
        s = -GRAV * s
        q = [h + dt * rez[0] / g.vol, hu + dt * (rez[1] + s[:, 0]) / g.vol, hv + dt * (rez[2] + s[:, 1]) / g.vol,
             hc + dt * rez[3] / g.vol, Z]
    return q[:4]


def _exact_euler(case, seed, g, p):
    dev = g.cc.device
    cc = np.concatenate([g.cc.cpu().numpy(), np.zeros((g.nc, 1))], 1)
    q = [torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(dev) for a in _euler_state(p, cc)]
    c1 = torch.where(g.inner, g.c1, g.c0)
    n = g.N / g.mes[:, None]
    nx, ny = n[:, 0], n[:, 1]
    for _ in range(case["steps"]):
        rho, P, mu, mv, E = q
        N, mes = g.N[g.cf], g.mes[g.cf]
        c = (GAMMA * (P / rho).abs()).sqrt()[:, None]
        un = ((mu[:, None] * N[..., 0] + mv[:, None] * N[..., 1]) / rho[:, None]).abs() / mes
        dt = (0.4 * g.vol / ((un + c) * mes).sum(1)).min()
        L, R = [a[g.c0] for a in q], [a[c1] for a in q]

        def flux(s):
            r, p_, a, b, e = s
            qn = a * nx + b * ny
            return [qn, a * qn / r + p_ * nx, b * qn / r + p_ * ny, (e + p_) * qn / r]

        # manapy's right normal momentum takes the left cell's rhov
        ql, qr = L[2] * nx + L[3] * ny, R[2] * nx + L[3] * ny
        cl, cr = (GAMMA * L[1] / L[0]).sqrt(), (GAMMA * R[1] / R[0]).sqrt()
        S = torch.maximum((ql / L[0]).abs() + cl, (qr / R[0]).abs() + cr)
        rez = [g.gather((0.5 * (fl + fr) - 0.5 * S * (R[k] - L[k])) * g.mes)
               for fl, fr, k in zip(flux(L), flux(R), (0, 2, 3, 4))]
        rho, mu, mv, E = (a + dt * r / g.vol for a, r in zip((rho, mu, mv, E), rez))
        q = [rho, (GAMMA - 1) * (E - 0.5 * (mu * mu + mv * mv) / rho), mu, mv, E]
    return q


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = _Geometry(case, seed, dev)
    fn = {"sw": _exact_sw, "euler": _exact_euler}.get(case["kind"], _exact_scalar)
    return fn(case, seed, g, _params(seed))
