"""The step keeps the half-step velocity w = v + dt/2 a_ between steps; what a
caller sees is the reference's state (u, v, a_) whatever it does in between.

One problem is advanced by every kind of call (graph run, host-launched run,
single step, three-call sequence), its v and a_ read back, and v, a_ and the
time step changed on the way; a literal v += dt/2 (a + a_), u += dt v + dt^2/2
a, a_ = a on the FP64 oracle's accelerations is the reference
(Order2Newmark.cpp:85-114).  Tolerances: operation order only in FP64
(1e-10), the repository's FP32 target (1e-4).
"""
import numpy as np
import pytest

from salvus_b200 import configs, core
from test_gpu_parity import build_pair, oracle_dt, rel_l2

pytestmark = pytest.mark.gpu

CFGS = {"quad": lambda: configs.standing_wave_2d(nel=6, order=4),
        "hex": lambda: configs.elastic_hex(nel=2, order=3, n_receivers=0),
        "tet": lambda: configs.simplex_tet(n=2, mesh="kuhn", n_receivers=0),
        "coupled": lambda: configs.coupled_2d(nel=6, order=3, n_receivers=0)}


@pytest.mark.parametrize("precision,tol", [(core.FP64, 1e-10), (core.FP32, 1e-4)])
@pytest.mark.parametrize("kind", sorted(CFGS))
def test_state_between_calls(kind, precision, tol):
    cfg = dict(CFGS[kind](), sources=[], receivers=[])
    dt = oracle_dt(cfg)
    mesh, p, orc, idx = build_pair(cfg, precision, dt)
    back = np.argsort(idx)
    rng = np.random.default_rng(3)
    k = rng.uniform(1, 3, (mesh.n_components, mesh.dim)) * 2 * np.pi / cfg["L"]
    X = mesh.node_coords()
    u = np.sin(X @ k.T)
    v = np.cos(X @ k.T) * 3.0
    ap = np.zeros_like(u)
    p.set_field("u", u)
    p.set_field("v", v)

    def literal(n):
        nonlocal u, v, ap
        for _ in range(n):
            orc.set_field("u", u[back])
            orc.set_field("v", v[back])
            a = orc.acceleration(0.0)[idx]
            v = v + 0.5 * dt * (a + ap)
            u = u + dt * v + 0.5 * dt * dt * a
            ap = a

    def check():
        for name, want in (("u", u), ("v", v), ("a_", ap)):
            assert rel_l2(p.get_field(name), want) <= tol, name

    assert np.array_equal(p.get_field("v"), v.astype(np.float32 if precision == core.FP32 else float))
    p.run(41)  # one graph, a remainder graph
    literal(41)
    check()
    check()  # reading changes nothing
    dt *= 0.8
    p.set_dt(dt)
    check()  # nor does a new time step
    p.step()
    p.run(3, core.RUN_PLAIN)
    literal(4)
    check()
    v = 0.5 * v
    p.set_field("v", v)
    p.run(8)
    literal(8)
    ap = 0.25 * ap
    p.set_field("a_", ap)
    check()
    for _ in range(2):
        p.assembleIntoGlobalDof()
        p.applyInverseMassMatrix()
        p.takeTimeStep()
    literal(2)
    check()
