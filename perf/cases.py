"""Performance cases of the spectral-element time step, through the package's public calls.

A user of this library builds a mesh with its model, attaches sources and
receivers, and then advances the wavefield in runs of a few dozen to a few
thousand steps, reading the seismograms after each.  A pass here is one such
run on a problem that is already set up: `steps` time steps, then the samples
they recorded (and the wavefield, where a snapshot is taken).  Two further
calls that such programs spend time in are a group of small meshes advanced
together and the estimate of the stable time step of a new mesh.

Every case is a dict of plain values:

  kind     "run" | "shots" | "group" | "dt"
  shape    "hex" | "quad" | "tri" | "tet", order its polynomial order
  physics  "acoustic" | "elastic" | "ti" (transversely isotropic) | "coupled"
           (fluid over solid quadrilaterals)
  nel      elements along an edge (hex: nel^3, quad: nel^2, tri: 2 nel^2,
           tet: 6 nel^3); a group's largest member
  jitter   interior vertices moved by up to this fraction of the spacing
           (general instead of parallelepiped elements)
  fp64     double-precision problem
  steps    time steps of a pass ("dt": power iterations)
  shots    shots of a batched problem, members of a group
  nrec     receivers (all shots share them)
  snapshot the displacement is read back too

`exact` integrates the same equations in 64 bits with dense reference-element
operators in plain torch and its own node numbering.
"""
import math

import numpy as np
import torch

from salvus_b200 import core

DIM = {"hex": 3, "quad": 2, "tri": 2, "tet": 3}
SHAPE = {"hex": core.HEX, "quad": core.QUAD, "tri": core.TRI, "tet": core.TET}
LENGTH = 1.0e4
VP, VS, RHO = 4000.0, 2300.0, 2500.0


def _case(kind, shape, order, physics, nel, steps, nrec, jitter=0.0, fp64=False, shots=1,
          snapshot=False, name=None):
    c = dict(kind=kind, shape=shape, order=order, physics=physics, nel=nel, steps=steps, nrec=nrec,
             jitter=jitter, fp64=fp64, shots=shots, snapshot=snapshot)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one shot on a 40 x 40 section (the smallest model anybody runs): every
        # step is a handful of launches; 100 steps leave a ragged remainder
        _case("run", "quad", 4, "acoustic", 40, 100, 16, name="quad acoustic 40"),
        # a forward-modelling job on a large 2-D section, advanced in chunks
        _case("run", "quad", 4, "acoustic", 400, 64, 8, name="quad acoustic 400"),
        # anisotropic 2-D elastic modelling on an unstructured, odd-sized mesh
        # of a higher order
        _case("run", "quad", 6, "elastic", 301, 20, 16, jitter=0.15, name="quad elastic 301 N6"),
        # a small 3-D elastic job of a serving stream: one 32-step chunk, the
        # samples and a wavefield snapshot
        _case("run", "hex", 4, "elastic", 16, 32, 8, snapshot=True, name="hex elastic 16"),
        # the large 3-D elastic run: one shot through a 64^3 cube
        _case("run", "hex", 4, "elastic", 64, 32, 64, name="hex elastic 64"),
        # a mesh with topography: general hexahedra, odd size
        _case("run", "hex", 4, "elastic", 27, 32, 16, jitter=0.15, name="hex distorted 27"),
        # transversely isotropic rock at a higher order
        _case("run", "hex", 5, "ti", 18, 32, 16, name="hex ti 18 N5"),
        # a double-precision run (reference solutions)
        _case("run", "hex", 4, "elastic", 22, 20, 16, fp64=True, name="hex fp64 22"),
        # shot batching: every shot of a survey over one velocity model
        _case("shots", "quad", 4, "acoustic", 200, 16, 16, shots=256, name="shots 256 x quad 200"),
        # many small models of uneven size advanced together
        _case("group", "quad", 4, "acoustic", 90, 32, 8, shots=16, name="group 16 quads"),
        # unstructured triangles (P3), topography in 2-D
        _case("run", "tri", 3, "acoustic", 317, 32, 16, jitter=0.15, name="tri acoustic 317"),
        # unstructured tetrahedra (P3), elastic
        _case("run", "tet", 3, "elastic", 27, 12, 64, jitter=0.15, name="tet elastic 27"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    steps = rng.choice([8, 13, 20, 32, 33, 50])
    nrec = rng.choice([1, 4, 16, 37, 64])
    what = rng.choice(["quad", "quad", "hex", "hex", "hex", "tri", "tet", "shots", "group", "dt"])
    jitter = rng.choice([0.0, 0.0, 0.1, 0.17])
    if what == "quad":
        order = rng.randint(1, 10)
        return _case("run", "quad", order, rng.choice(["acoustic", "elastic", "coupled"]),
                     _log_int(rng, 6, 1600 // order), steps, nrec, jitter, rng.random() < 0.25,
                     snapshot=rng.random() < 0.2)
    if what == "hex":
        order = rng.randint(1, 6)
        return _case("run", "hex", order, rng.choice(["acoustic", "elastic", "elastic", "ti"]),
                     _log_int(rng, 3, 140 // order), steps, nrec, jitter, rng.random() < 0.25,
                     snapshot=rng.random() < 0.2)
    if what == "tri":
        return _case("run", "tri", 3, "acoustic", _log_int(rng, 10, 380), steps, nrec, 0.15,
                     rng.random() < 0.25)
    if what == "tet":
        return _case("run", "tet", 3, rng.choice(["acoustic", "elastic", "elastic"]),
                     _log_int(rng, 3, 26), min(steps, 20), nrec, 0.15, rng.random() < 0.2)
    if what == "shots":
        order = rng.randint(2, 5)
        return _case("shots", "quad", order, "acoustic", _log_int(rng, 20, 400 // order),
                     min(steps, 20), 16, jitter, shots=rng.choice([8, 32, 50, 96, 200]))
    if what == "group":
        shape = rng.choice(["quad", "hex"])
        return _case("group", shape, 4, "acoustic" if shape == "quad" else "elastic",
                     rng.randint(30, 120) if shape == "quad" else rng.randint(5, 16),
                     rng.choice([32, 40]), 8, shots=rng.randint(4, 24))
    return _case("dt", "hex", 4, "elastic", _log_int(rng, 4, 20), rng.choice([40, 60, 100]), 0)


# ---------------------------------------------------------------- models
def _lattice(nel, dim, jitter, rng):
    ax = np.linspace(0.0, LENGTH, nel + 1)
    pts = np.stack([g.ravel() for g in np.meshgrid(*[ax] * dim, indexing="ij")[::-1]], axis=1)
    if jitter:
        h = LENGTH / nel
        inner = (pts > 0.5 * h) & (pts < LENGTH - 0.5 * h)
        pts = pts + inner * rng.uniform(-jitter * h, jitter * h, pts.shape)
    return pts


def _cells(shape, n):
    """Vertex order of the library's elements: see salvus_mesh_desc."""
    if DIM[shape] == 2:
        j, i = (x.ravel() for x in np.meshgrid(np.arange(n), np.arange(n), indexing="ij"))
        v = lambda a, b: (j + b) * (n + 1) + i + a  # noqa: E731
        if shape == "quad":
            return np.stack([v(0, 0), v(1, 0), v(1, 1), v(0, 1)], axis=1)
        two = np.stack([v(0, 0), v(1, 0), v(1, 1), v(0, 0), v(1, 1), v(0, 1)], axis=1)
        return two.reshape(-1, 3)
    k, j, i = (x.ravel() for x in np.meshgrid(*[np.arange(n)] * 3, indexing="ij"))
    v = lambda a, b, c: ((k + c) * (n + 1) + j + b) * (n + 1) + i + a  # noqa: E731
    if shape == "hex":
        return np.stack([v(0, 0, 0), v(0, 1, 0), v(1, 1, 0), v(1, 0, 0),
                         v(0, 0, 1), v(1, 0, 1), v(1, 1, 1), v(0, 1, 1)], axis=1)
    # six tetrahedra around each cube's main diagonal, det[v2-v0; v1-v0; v3-v0] > 0
    c = [v(q & 1, (q >> 1) & 1, q >> 2) for q in range(8)]
    six = [(0, 3, 1, 7), (0, 1, 5, 7), (0, 2, 3, 7), (0, 6, 2, 7), (0, 5, 4, 7), (0, 4, 6, 7)]
    return np.stack([c[q] for t in six for q in t], axis=1).reshape(-1, 4)


def _orient(V, C):
    """Tetrahedra in the library's orientation."""
    x = V[C]
    det = np.einsum("ij,ij->i", x[:, 2] - x[:, 0], np.cross(x[:, 1] - x[:, 0], x[:, 3] - x[:, 0]))
    C[det < 0] = C[det < 0][:, [0, 2, 1, 3]]
    return C


def _inside(V, C, elements, rng):
    """A point well inside each of these elements."""
    vx = V[C[elements]]
    w = rng.uniform(0.5, 1.5, vx.shape[:2])
    return np.einsum("mv,mvx->mx", w / w.sum(axis=1, keepdims=True), vx)


def _model(case, seed, nel=None):
    """Mesh, material and acquisition of one case: plain arrays."""
    rng = np.random.default_rng(seed)
    shape, nel, dim, phys = case["shape"], nel or case["nel"], DIM[case["shape"]], case["physics"]
    V = _lattice(nel, dim, case["jitter"], rng)
    C = _cells(shape, nel)
    if shape == "tet":
        C = _orient(V, C)
    # a smooth model: 10 % variation over one to three wavelengths
    k = rng.integers(1, 4, size=(3, dim)) * (2 * np.pi / LENGTH)
    ph = rng.uniform(0, 2 * np.pi, 3)
    pert = 1.0 + 0.1 * np.mean(np.cos(V @ k.T + ph), axis=1)
    vp, vs, rho = VP * pert, VS * pert, RHO * pert
    if phys == "acoustic":
        par = [vp]
    elif phys == "ti":  # RHO VPV VPH VSV VSH ETA
        par = [rho, vp, vp * math.sqrt(1.16), vs, vs * math.sqrt(1.12), 0.9 + 0 * vp]
    elif dim == 3:
        par = [rho, vp, vs]
    else:  # RHO C11 C13 C33 C55, weakly anisotropic
        c33, c55 = rho * vp ** 2, rho * vs ** 2
        par = [rho, 1.2 * c33, c33 - 2 * c55, c33, c55]
    par = np.stack([p[C] for p in par])
    if phys == "coupled":  # FLUID VP RHO C11 C13 C33 C55: water over rock
        fluid = np.repeat(V[C].mean(axis=1)[:, 1:2] > 0.6 * LENGTH, 4, axis=1) * 1.0
        par = np.stack([fluid, 0 * fluid + 1500.0, np.where(fluid > 0, 1000.0, par[0]), *par[1:]])
    comps = 1 if phys == "acoustic" else 3 if phys == "coupled" else dim
    # stable time step: the GLL spacing (the simplices' node spacing) over the
    # fastest speed, reduced for moved vertices
    if shape in ("hex", "quad"):
        x = _gll(case["order"])[0]
        dt = 0.3 * (x[1] - x[0]) / 2 * (1 - 2.5 * case["jitter"])
    else:
        dt = 0.01 if shape == "tri" else 0.004
    dt *= LENGTH / nel / (VP * 1.1 * math.sqrt(1.2))
    f0 = 1.0 / (25 * dt)  # the wavelet acts within a pass
    n_src = case["shots"] if case["kind"] == "shots" else 1
    spots = _inside(V, C, rng.integers(len(C) // 4, len(C) - len(C) // 4, n_src), rng)
    sources = []
    for s, where in enumerate(spots):
        amp = f0 ** 2 * (LENGTH / nel / case["order"]) ** dim
        src = dict(location=where, center_freq=f0, time_delay=0.5 / f0, amplitude=amp, shot=s)
        if comps == 1:
            src["direction"] = [1.0]
        elif phys == "coupled":
            src.update(direction=[0.0, 0.6, 0.8], amplitude=amp * RHO)
        else:
            m = rng.standard_normal(6 if dim == 3 else 3)
            src.update(moment_tensor=m, amplitude=amp * RHO * LENGTH / nel)
        sources.append(src)
    receivers = _inside(V, C, rng.integers(0, len(C), case["nrec"]), rng)
    wave = (rng.integers(1, 5, size=(comps, dim)) * (2 * np.pi / LENGTH),
            rng.uniform(0, 2 * np.pi, comps))
    return dict(V=V, C=C, par=par, comps=comps, dt=dt, sources=sources, receivers=receivers,
                wave=wave, shot_phase=rng.uniform(0, 2 * np.pi, case["shots"]))


def _initial(md, xyz, which):
    """Displacement (which = 0) and velocity (1) at the nodes: standing waves, [G][c]."""
    k, ph = (torch.as_tensor(w, dtype=torch.float64, device=xyz.device) for w in md["wave"])
    w = VP * float(md["wave"][0].max())
    return torch.sin(xyz @ k.T + ph) if which == 0 else 0.3 * w * torch.cos(xyz @ k.T - ph)


def _setup(case, md):
    """Mesh and problem as a program creates them, with a wavefield under way."""
    phys = {"acoustic": core.ACOUSTIC, "ti": core.ELASTIC3D, "coupled": core.COUPLED2D,
            "elastic": core.ELASTIC2D if DIM[case["shape"]] == 2 else core.ELASTIC3D}[case["physics"]]
    need64 = case["fp64"] or case["kind"] == "dt"
    mesh = core.Mesh(SHAPE[case["shape"]], case["order"], phys, md["V"], md["C"], md["par"],
                     flags=0 if need64 else core.MESH_FP32_ONLY)
    if case["kind"] == "dt":
        return mesh, None
    shots = case["shots"] if case["kind"] == "shots" else 1
    p = core.Problem(mesh, core.FP64 if case["fp64"] else core.FP32, dt=md["dt"], n_shots=shots)
    for s in md["sources"]:
        p.add_source(**s)
    for r in md["receivers"]:
        p.add_receiver(r)
    if shots > 1:
        p.set_seismogram_capacity(256)
    xyz = torch.from_numpy(mesh.node_coords())
    u = _initial(md, xyz, 0).numpy()
    for s in range(shots):  # every shot its own amplitude
        p.set_field("u", u if shots == 1 else u * math.cos(md["shot_phase"][s]), shot=s)
    if shots == 1:
        p.set_field("v", _initial(md, xyz, 1).numpy())
    return mesh, p


def _member_edges(case):
    n = case["shots"]
    return [max(2, case["nel"] * (k + 2) // (n + 1)) for k in range(n)]


def prepare(case, seed):
    if case["kind"] == "group":
        pairs = [_setup(case, _model(case, seed * 100 + k, nel))
                 for k, nel in enumerate(_member_edges(case))]
        group = core.Group([p for _, p in pairs])
        return dict(case=case, pairs=pairs, group=group)
    md = _model(case, seed)
    mesh, p = _setup(case, md)
    if p is not None:
        p.prepare_run(case["steps"])
    return dict(case=case, mesh=mesh, p=p, seed=seed)


def _samples(case, p):
    """What the last run recorded, in the precision that the problem computes in."""
    n = case["steps"]
    s = p.seismograms(p.step_index - n, n)
    return s if case["fp64"] else s.astype(np.float32)


def run(state):
    case = state["case"]
    if case["kind"] == "dt":
        return state["mesh"].max_eigenvalue(case["steps"], seed=1 + state["seed"])
    if case["kind"] == "group":
        state["group"].run(case["steps"])
        return [_samples(case, p) for _, p in state["pairs"]]
    p = state["p"]
    p.run(case["steps"])
    out = [_samples(case, p)]
    if case["snapshot"]:
        u = p.get_field("u")
        out.append(u if case["fp64"] else u.astype(np.float32))
    return out


# ---------------------------------------------------------------- work
def _points(case):
    return {"tri": 12, "tet": 50}.get(case["shape"], (case["order"] + 1) ** DIM[case["shape"]])


def _counts(case, nel):
    """Elements and nodes of a mesh."""
    N = case["order"]
    if case["shape"] == "hex":
        return nel ** 3, (nel * N + 1) ** 3
    if case["shape"] == "quad":
        return nel ** 2, (nel * N + 1) ** 2
    if case["shape"] == "tri":
        e, edges = 2 * nel ** 2, 3 * nel ** 2 + 2 * nel
        return e, 3 * e + 2 * edges + (nel + 1) ** 2
    e = 6 * nel ** 3
    faces = 12 * nel ** 3 + 6 * nel ** 2
    edges = 7 * nel ** 3 + 9 * nel ** 2 + 3 * nel
    return e, 10 * e + 6 * faces + 2 * edges + (nel + 1) ** 3


def work(case):
    """Per step: displacement and velocity read and written once, the mass,
    the material (and, where it varies over the elements, the geometry) read
    once per element point; the gradient and divergence sums of every point."""
    real = 8 if case["fp64"] or case["kind"] == "dt" else 4
    P, dim = _points(case), DIM[case["shape"]]
    c = 1 if case["physics"] == "acoustic" else dim
    mat = {"acoustic": 1, "ti": 5, "coupled": 3}.get(case["physics"], 2 if dim == 3 else 4)
    simplex = case["shape"] in ("tri", "tet")
    geom = dim * dim if case["jitter"] and not simplex else 0
    line = P if simplex else case["order"] + 1
    edges = _member_edges(case) if case["kind"] == "group" else [case["nel"]]
    shots = case["shots"] if case["kind"] == "shots" else 1
    B = F = 0
    for nel in edges:
        E, G = _counts(case, nel)
        state = (2 if case["kind"] == "dt" else 4) * c * G * shots
        model = G + E * P * (mat + geom) + E * (dim * dim if not geom else 0)
        B += case["steps"] * (state + model) * real
        F += case["steps"] * E * P * shots * c * (4 * dim * line + 4 * dim * dim)
    return {"bytes": float(B), "flops": float(F)}


# ---------------------------------------------------------------- 64-bit answer
def _gll(N):
    leg = np.polynomial.legendre.Legendre.basis(N)
    x = np.concatenate([[-1.0], np.sort(leg.deriv().roots().real), [1.0]])
    return x, 2.0 / (N * (N + 1) * leg(x) ** 2)


def _lagrange(x, t):
    """Values and derivatives of the Lagrange polynomials on x at points t: [len(t)][len(x)]."""
    P = [np.polynomial.Polynomial.fromroots(np.delete(x, i)) for i in range(len(x))]
    P = [p / p(x[i]) for i, p in enumerate(P)]
    return np.stack([p(t) for p in P], axis=1), np.stack([p.deriv()(t) for p in P], axis=1)


class _Element:
    """Reference element: nodes [P][dim], weights [P], phi / dphi at points."""

    def __init__(self, shape, order):
        self.shape, self.dim = shape, DIM[shape]
        if shape in ("hex", "quad"):
            self.x1, w1 = _gll(order)
            n, d = order + 1, self.dim
            idx = np.stack([(np.arange(n ** d) // n ** a) % n for a in range(d)], axis=1)
            self.idx, self.nodes, self.w = idx, self.x1[idx], np.prod(w1[idx], axis=1)
        else:
            self._simplex()

    def _simplex(self):
        d = self.dim
        pts, w = [], []

        def orbit(bary, weight):
            seen = {tuple(b) for b in _permutations(bary)}
            for b in sorted(seen):
                pts.append(b)
                w.append(weight)

        if d == 2:
            r7 = math.sqrt(7.0)
            # the 12-point rule's 4-digit nodes on (-1,-1), (1,-1), (-1,1)
            orbit(((1 + 0.1706) / 2, (1 - 0.5853) / 2, (1 - 0.5853) / 2), (84 * r7 + 294) / (400 * r7 + 1280))
            orbit(((1 + 0.413) / 2, (1 - 0.413) / 2, 0.0), 2 * r7 * (2 + r7) ** 4 / (9520 * r7 + 25280))
            orbit((1.0, 0.0, 0.0), (1838 * r7 + 4942) / (124080 * r7 + 330960))
            corner = np.array([[-1.0, -1.0], [1.0, -1.0], [-1.0, 1.0]])
        else:
            ga, de, al = 0.9503775858394107e-01, 0.1252462362578136, 0.2928294047674109
            orbit((1 - 3 * ga, ga, ga, ga), 6 * 0.7542468904648131e-02)
            orbit((0.5 - de, 0.5 - de, de, de), 6 * 0.1360991755970793e-01)
            for b, wt in ((0.1972862280257976, 0.1840177904191860e-02), (0.4256461243139345, 0.1831324329245650e-02)):
                orbit((1 - 2 * b, b, b, 0.0), 6 * wt)
            orbit((1 - al, al, 0.0, 0.0), 6 * 0.8268179517797114e-03)
            orbit((1.0, 0.0, 0.0, 0.0), 6 * 0.2143608668049743e-03)
            corner = np.array([[0.0, 0, 0], [0, 1.0, 0], [1.0, 0, 0], [0, 0, 1.0]])
        self.nodes, self.w = np.array(pts) @ corner, np.array(w)
        self.corner_inv = np.linalg.inv(np.concatenate([corner, np.ones((d + 1, 1))], axis=1))
        if d == 2:  # P3 and two of the bubble's linear multiples
            powers = [(3 - b - c, b, c) for b in range(4) for c in range(4 - b)] + [(2, 1, 1), (1, 2, 1)]
        else:  # P3, face bubbles x P2, interior bubble x P2
            powers = [(3 - b - c - e, b, c, e) for b in range(4) for c in range(4 - b) for e in range(4 - b - c)]
            for opp in range(4):
                f = [v for v in range(4) if v != opp]
                for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2)):
                    q = [0 if v == opp else 1 for v in range(4)]
                    q[f[a]] += 1
                    q[f[b]] += 1
                    powers.append(tuple(q))
            for a in range(4):
                for b in range(a, 4):
                    q = [1] * 4
                    q[a] += 1
                    q[b] += 1
                    powers.append(tuple(q))
        self.powers = np.array(powers)
        self.coef = np.linalg.inv(self._generators(self.nodes)[0])

    def _generators(self, x):
        lam = np.concatenate([x, np.ones((len(x), 1))], axis=1) @ self.corner_inv
        e = self.powers
        val = np.prod(lam[:, None, :] ** e, axis=2)
        der = np.zeros((self.dim, len(x), len(e)))
        for v in range(self.dim + 1):
            low = np.maximum(e - (np.arange(self.dim + 1) == v), 0)
            dv = e[:, v] * np.prod(lam[:, None, :] ** low, axis=2)
            der += self.corner_inv[:self.dim, v][:, None, None] * dv
        return val, der

    def basis(self, x):
        """phi [m][P] and its reference gradient [dim][m][P] at points x [m][dim]."""
        if self.shape in ("tri", "tet"):
            val, der = self._generators(x)
            return val @ self.coef, der @ self.coef
        L = [_lagrange(self.x1, x[:, a]) for a in range(self.dim)]
        pick = lambda k: np.prod([L[a][1 if a == k else 0][:, self.idx[:, a]]  # noqa: E731
                                  for a in range(self.dim)], axis=0)
        return pick(-1), np.stack([pick(k) for k in range(self.dim)])

    def vertex(self, x):
        """P1 shape functions [m][nv] and gradients [dim][m][nv] (the geometry map)."""
        if self.shape in ("tri", "tet"):
            lam = np.concatenate([x, np.ones((len(x), 1))], axis=1) @ self.corner_inv
            g = np.repeat(self.corner_inv[:self.dim, None, :], len(x), axis=1)
            return lam, g
        s = np.array([(-1, -1), (1, -1), (1, 1), (-1, 1)] if self.dim == 2 else
                     [(-1, -1, -1), (-1, 1, -1), (1, 1, -1), (1, -1, -1),
                      (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1)], dtype=float)
        f = (1 + x[:, None, :] * s) / 2
        val = np.prod(f, axis=2)
        g = [np.prod(np.delete(f, a, axis=2), axis=2) * s[:, a] / 2 for a in range(self.dim)]
        return val, np.stack(g)


def _permutations(b):
    if len(b) == 1:
        return [tuple(b)]
    return [(b[i],) + r for i in range(len(b)) for r in _permutations(b[:i] + b[i + 1:])]


def _locate(el, V, C, x):
    """First element that holds x, and its reference coordinates."""
    vx = V[C]
    box = np.all((vx.min(axis=1) <= x + 1e-6) & (vx.max(axis=1) >= x - 1e-6), axis=1)
    for e in np.nonzero(box)[0]:
        r = np.zeros((1, el.dim)) if el.shape in ("hex", "quad") else el.nodes.mean(axis=0)[None]
        for _ in range(30):
            N, g = el.vertex(r)
            r = r + np.linalg.solve((g[:, 0] @ vx[e]).T, x - (N @ vx[e])[0])
        ok = np.all(np.abs(r) <= 1 + 1e-9) if el.shape in ("hex", "quad") else np.all(el.vertex(r)[0] >= -1e-9)
        if ok:
            return e, r
    raise ValueError("point outside the mesh")


def _integrate(case, md):
    """(seismograms [shots][receivers][c][steps]) of one problem in 64 bits."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    el = _Element(case["shape"], case["order"])
    T = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
    dim, phys, c = el.dim, case["physics"], md["comps"]
    _, dphi = el.basis(el.nodes)
    D = T(dphi)  # [k][q][j]
    N, g = el.vertex(el.nodes)
    vx = T(md["V"][md["C"]])  # [e][v][x]
    J = torch.einsum("kqv,evx->eqkx", T(g), vx)
    det = torch.linalg.det(J)
    iJ = torch.linalg.inv(J)  # [e][q][x][k]: d xi_k / d x_x
    del J
    mat = torch.einsum("qv,mev->meq", T(N), T(md["par"]))
    wd = T(el.w) * det
    # node numbers: points at the same place are one node
    X = torch.einsum("qv,evx->eqx", T(N), vx)
    key = torch.zeros(X.shape[:2], dtype=torch.int64, device=dev)
    for a in range(dim):
        key = key * (1 << 21) + torch.round(X[..., a] / LENGTH * (1 << 20) + 0.2345).to(torch.int64)
    _, conn = torch.unique(key, return_inverse=True)
    G = int(conn.max()) + 1
    flat = conn.reshape(-1)
    xyz = torch.zeros((G, dim), dtype=torch.float64, device=dev)
    xyz[flat] = X.reshape(-1, dim)
    del key, X
    rho = mat[0] if phys != "acoustic" else torch.ones_like(det)
    mass = torch.zeros(G, dtype=torch.float64, device=dev).index_add_(0, flat, (wd * rho).reshape(-1))
    # material constants with the weight and detJ folded in
    if phys == "acoustic":
        k = [mat[0] ** 2 * wd]
    elif phys == "ti":  # A C F L N
        r, vpv, vph, vsv, vsh, eta = mat
        k = [r * vph ** 2, r * vpv ** 2, eta * r * (vph ** 2 - 2 * vsv ** 2), r * vsv ** 2, r * vsh ** 2]
        k = [x * wd for x in k]
    elif dim == 3:  # lambda, mu
        k = [mat[0] * (mat[1] ** 2 - 2 * mat[2] ** 2) * wd, mat[0] * mat[2] ** 2 * wd]
    else:  # C11 C13 C33 C55
        k = [mat[i] * wd for i in (1, 2, 3, 4)]

    def stress(H, k):  # H[e][q][c][x] = d u_c / d x_x
        if phys == "acoustic":
            return H * k[0][..., None, None]
        s = torch.empty_like(H)
        if phys == "ti":
            A, Cc, F, L, Nn = k
            xx, yy, zz = H[..., 0, 0], H[..., 1, 1], H[..., 2, 2]
            s[..., 0, 0] = A * xx + (A - 2 * Nn) * yy + F * zz
            s[..., 1, 1] = (A - 2 * Nn) * xx + A * yy + F * zz
            s[..., 2, 2] = F * (xx + yy) + Cc * zz
            for a, b, m in ((1, 2, L), (0, 2, L), (0, 1, Nn)):
                s[..., a, b] = s[..., b, a] = m * (H[..., a, b] + H[..., b, a])
        elif dim == 3:
            s = k[1][..., None, None] * (H + H.transpose(-1, -2))
            tr = k[0] * (H[..., 0, 0] + H[..., 1, 1] + H[..., 2, 2])
            for a in range(3):
                s[..., a, a] += tr
        else:
            c11, c13, c33, c55 = k
            s[..., 0, 0] = c11 * H[..., 0, 0] + c13 * H[..., 1, 1]
            s[..., 1, 1] = c13 * H[..., 0, 0] + c33 * H[..., 1, 1]
            s[..., 0, 1] = s[..., 1, 0] = c55 * (H[..., 0, 1] + H[..., 1, 0])
        return s

    # columns: the components of one shot, or the shots of a scalar field
    S = case["shots"] if case["kind"] == "shots" else 1
    cols = c * S
    E = det.shape[0]
    block = max(1, int(2e8) // (el.nodes.shape[0] * cols * dim))

    def stiffness(u):  # sum over elements of -K_e u_e, [G][cols]
        out = torch.zeros_like(u)
        for b in range(0, E, block):
            s = slice(b, min(E, b + block))
            ue = u[conn[s]]  # [e][j][cols]
            d = torch.einsum("kqj,ejc->eqkc", D, ue)
            H = torch.einsum("eqxk,eqkc->eqcx", iJ[s], d)
            H = stress(H, [x[s] for x in k])
            f = torch.einsum("eqxk,eqcx->ekqc", iJ[s], H)
            r = torch.einsum("kqj,ekqc->ejc", D, f)
            out.index_add_(0, conn[s].reshape(-1), r.reshape(-1, cols), alpha=-1.0)
        return out

    src = []
    for s in md["sources"]:
        e, r = _locate(el, md["V"], md["C"], s["location"])
        phi, dp = el.basis(r)
        if "moment_tensor" in s:
            m = s["moment_tensor"]
            M = np.array([[m[0], m[5], m[4]], [m[5], m[1], m[3]], [m[4], m[3], m[2]]]) if dim == 3 \
                else np.array([[m[0], m[2]], [m[2], m[1]]])
            Jr = el.vertex(r)[1][:, 0] @ md["V"][md["C"][e]]  # [k][x]
            f = np.linalg.solve(Jr, dp[:, 0]).T @ M
        else:
            f = phi[0][:, None] * np.asarray(s["direction"])
        src.append((conn[e], T(f), s))
    rec = [(conn[e], T(el.basis(r)[0][0])) for e, r in
           (_locate(el, md["V"], md["C"], x) for x in md["receivers"])]
    rec_n, rec_w = torch.stack([n for n, _ in rec]), torch.stack([w for _, w in rec])

    u = _initial(md, xyz, 0)
    if S > 1:
        u = u * T(np.cos(md["shot_phase"]))
        v = torch.zeros_like(u)
    else:
        v = _initial(md, xyz, 1)
    a_old, dt, out = torch.zeros_like(u), md["dt"], []
    for n in range(case["steps"]):
        a = stiffness(u)
        for nodes, f, s in src:
            x = (math.pi * s["center_freq"] * (n * dt - s["time_delay"])) ** 2
            stf = s["amplitude"] * (1 - 2 * x) * math.exp(-x)
            if S > 1:
                a[:, s["shot"]].index_add_(0, nodes, f[:, 0] * stf)
            else:
                a.index_add_(0, nodes, f * stf)
        a /= mass[:, None]
        v += 0.5 * dt * (a + a_old)
        u += dt * v + 0.5 * dt * dt * a
        a_old = a
        out.append(torch.einsum("rp,rpc->rc", rec_w, u[rec_n]))
    seis = torch.stack(out, dim=-1)  # [r][cols][steps]
    return (seis.transpose(0, 1)[:, :, None] if S > 1 else seis).cpu().numpy()


def exact(case, seed):
    if case["kind"] == "dt" or case["physics"] == "coupled":
        return None
    if case["kind"] == "group":
        return [_integrate(case, _model(case, seed * 100 + k, nel))
                for k, nel in enumerate(_member_edges(case))]
    out = [_integrate(case, _model(case, seed))]
    return out + [None] if case["snapshot"] else out
