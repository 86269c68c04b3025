"""Acoustic quadrilaterals that are all parallelograms store a scalar per point
and one metric per element; the records of SALVUS_MESH_PER_POINT_GEOMETRY give
the same bits (solo and grouped), and a mesh with one moved vertex keeps the
records and matches the oracle."""
import numpy as np
import pytest

from salvus_b200 import configs, core, meshgen
from test_gpu_parity import build_pair, oracle_dt, rel_l2

pytestmark = pytest.mark.gpu


def model(nx, ny, order, shear):
    V, C = meshgen.structured_quad(nx, ny, 8e3, 6e3)
    V = V @ np.array([[1.0, 0.3 * shear], [-0.2 * shear, 1.0]])
    rng = np.random.default_rng(order)
    par = meshgen.per_element_vertex(rng.uniform(3000, 4500, len(V)), C)[None]
    return dict(shape=core.QUAD, order=order, physics=core.ACOUSTIC, vertices=V, cells=C, params=par)


def problem(cfg, flags, dt):
    mesh = core.Mesh(cfg["shape"], cfg["order"], cfg["physics"], cfg["vertices"], cfg["cells"],
                     cfg["params"], flags=flags)
    p = core.Problem(mesh, core.FP32, dt=dt)
    v = cfg["vertices"][cfg["cells"]].mean(axis=1)
    p.add_source(v[len(v) // 3], 0.02 / dt, 10 * dt, 1e3, direction=[1.0])
    p.add_receiver(v[len(v) // 2])
    p.set_field("u", np.sin(1e-3 * mesh.node_coords()[:, :1]))
    return p


def state(p):
    return [p.get_field(f) for f in ("u", "v", "a_")] + [p.seismograms()]


@pytest.mark.parametrize("order", range(1, 11))
@pytest.mark.parametrize("shear", [0, 1])
def test_factors_equal_records(order, shear):
    cfg = model(7, 5, order, shear)
    dt = oracle_dt(cfg)
    a, b = problem(cfg, 0, dt), problem(cfg, core.MESH_PER_POINT_GEOMETRY, dt)
    a.run(40)
    b.run(40)
    for x, y in zip(state(a), state(b)):
        assert np.array_equal(x, y)
    assert np.abs(a.seismograms()).max() > 0


def test_groups_of_both_layouts():
    cfgs = [model(7, 5, 4, 1), model(13, 9, 4, 0)]
    dt = min(oracle_dt(c) for c in cfgs)
    solo = [problem(c, 0, dt) for c in cfgs]
    flags = [0, core.MESH_PER_POINT_GEOMETRY]
    keep = [problem(c, f, dt) for c, f in zip(cfgs, flags)]
    group = core.Group(keep)
    group.run(40)
    group.synchronize()
    for p, q in zip(solo, keep):
        p.run(40)
        for x, y in zip(state(p), state(q)):
            assert np.array_equal(x, y)
    group.close()


@pytest.mark.parametrize("moved", [0.0, 1e-7, 0.1])
def test_nearly_parallelograms_against_oracle(moved):
    cfg = model(6, 6, 4, 1)
    h = 1e3
    cfg["vertices"] = cfg["vertices"].copy()
    cfg["vertices"][24] += moved * h
    cfg["receivers"] = cfg["vertices"][cfg["cells"]].mean(axis=1)[[3, 20, 33]]
    dt = oracle_dt(cfg)
    mesh, p, orc, idx = build_pair(cfg, core.FP32, dt)
    X = mesh.node_coords()
    u0 = np.sin(1e-3 * X[:, :1]) * np.cos(7e-4 * X[:, 1:])
    p.set_field("u", u0)
    orc.set_field("u", u0[np.argsort(idx)])
    p.run(200)
    assert rel_l2(p.seismograms(), orc.run(200, dt)) <= 1e-4
