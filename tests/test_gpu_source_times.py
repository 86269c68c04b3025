"""The source-time functions of the coming step are evaluated ahead of it: a new
time step, a source added between runs and single-launch group runs each make
them stale.  Against the FP64 oracle's accelerations stepped literally (v +=
dt/2 (a + a_), u += dt v + dt^2/2 a, sources at t = n dt), and bitwise against a
problem that ran alone.  Tolerances: operation order only in FP64 (1e-10), the
repository's FP32 target (1e-4)."""
import numpy as np
import pytest

from salvus_b200 import configs, core
from test_gpu_group import make
from test_gpu_parity import build_pair, oracle_dt, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(core.FP64, 1e-10), (core.FP32, 1e-4)])
@pytest.mark.parametrize("kind", ["quad", "hex"])
def test_time_step_and_sources_change(kind, precision, tol):
    cfg = (configs.ricker_2d(nel=5, order=4, n_receivers=0) if kind == "quad"
           else configs.elastic_hex(nel=3, order=4, n_receivers=0))
    dt = oracle_dt(cfg)
    f0 = 0.02 / dt
    centres = cfg["vertices"][cfg["cells"]].mean(axis=1)
    c = 1 if kind == "quad" else 3
    first, second = (dict(location=tuple(centres[e]), center_freq=f0, time_delay=0.3 / f0,
                          amplitude=1e3, direction=[1.0, -0.5, 0.3][:c])
                     for e in (len(centres) // 2, 1))
    cfg["sources"], cfg["receivers"] = [first], []
    mesh, p, orc, idx = build_pair(cfg, precision, dt)
    back = np.argsort(idx)
    u = np.zeros((mesh.n_nodes, mesh.n_components))
    v, ap, n = u.copy(), u.copy(), 0

    def literal(steps):
        nonlocal u, v, ap, n
        for _ in range(steps):
            orc.set_field("u", u[back])
            a = orc.acceleration(n * dt)[idx]
            v = v + 0.5 * dt * (a + ap)
            u = u + dt * v + 0.5 * dt * dt * a
            ap = a
            n += 1

    def advance(steps):
        p.run(steps)
        literal(steps)
        assert rel_l2(p.get_field("u"), u) <= tol
        assert rel_l2(p.get_field("a_"), ap) <= tol

    advance(20)
    dt *= 0.7
    p.set_dt(dt)
    advance(1)
    advance(20)
    s = second
    p.add_source(s["location"], s["center_freq"], s["time_delay"], s["amplitude"], direction=s["direction"])
    orc.add_source(s["location"], s["center_freq"], s["time_delay"], s["amplitude"], s["direction"])
    advance(1)
    advance(33)
    p.step()
    literal(1)
    p.assembleIntoGlobalDof()
    p.applyInverseMassMatrix()
    p.takeTimeStep()
    literal(1)
    advance(9)


@pytest.mark.parametrize("form", ["persistent", "partitioned", "stages"])
@pytest.mark.parametrize("kind,edges", [("quad", (9, 14)), ("hex", (3, 4))])
def test_member_alone_between_group_runs(kind, edges, form, monkeypatch):
    monkeypatch.setenv("SALVUS_GROUP_STEP", form)
    keep = [make(kind, edge, 40 + k) for k, edge in enumerate(edges)]
    group = core.Group([p for _, p in keep])
    group.run(40)
    keep[0][1].run(9)
    keep[1][1].step()
    group.run(33)
    group.synchronize()
    for k, edge in enumerate(edges):
        m, q = make(kind, edge, 40 + k)
        q.run(73 + (9, 1)[k])
        p = keep[k][1]
        assert p.step_index == q.step_index
        for f in ("u", "v", "a_"):
            assert np.array_equal(p.get_field(f), q.get_field(f)), (k, f)
        assert np.array_equal(p.seismograms(), q.seismograms())
        assert np.abs(q.seismograms()).max() > 0
    group.close()
