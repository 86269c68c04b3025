"""Metric of acoustic quadrilaterals in FP32: every product w detJ vp^2 times a
metric entry is rounded once, also where a mesh of squares keeps one number per
point.

The element metric of a uniform mesh is one number, so an error in its rounding
is an error of the modulus at every point; spacings are used whose metric lies
almost half a unit in the last place from the nearest FP32 number (a relative
error above 5e-8).  The strain energy 1/2 u^T K u of one FP32 field, in FP32 and
in FP64, shows it: on orders 1 and 2 the derivative matrix is exact in FP32, and
the roundings of the points' own products and sums are independent of each other
and average out, 2^-24 / sqrt(points) times the few by which K u cancels, below
3e-9 on the 10^4 points here.  The bound is 1e-8.
"""
import numpy as np
import pytest

from salvus_b200 import configs, core, meshgen
from test_gpu_parity import build_pair, oracle_dt, rel_l2

pytestmark = pytest.mark.gpu


def spacing(seed):
    """h whose metric (2 / h)^2 is badly rounded in FP32, always upwards."""
    rng = np.random.default_rng(seed)
    h = rng.uniform(100.0, 180.0, 200000)
    m = (2.0 / h) ** 2
    return float(h[np.argmax(m.astype(np.float32) / m)])


def model(nx, ny, order, hx, hy, turn=0.0):
    V, C = meshgen.structured_quad(nx, ny, nx * hx, ny * hy)
    c, s = np.cos(turn), np.sin(turn)
    V = V @ np.array([[c, s], [-s, c]])
    rng = np.random.default_rng(order)
    par = meshgen.per_element_vertex(rng.uniform(3000, 4500, len(V)), C)[None]
    return dict(shape=core.QUAD, order=order, physics=core.ACOUSTIC, vertices=V, cells=C, params=par)


def mesh(cfg, flags=0):
    return core.Mesh(cfg["shape"], cfg["order"], cfg["physics"], cfg["vertices"], cfg["cells"],
                     cfg["params"], flags=flags)


@pytest.mark.parametrize("flags", [0, core.MESH_PER_POINT_GEOMETRY])
@pytest.mark.parametrize("square", [True, False])
@pytest.mark.parametrize("order", [1, 2])
def test_metric_is_rounded_once(order, square, flags):
    hx = spacing(1)
    hy = hx if square else spacing(2)
    for h in (hx, hy):
        assert float(np.float32((2 / h) ** 2)) / (2 / h) ** 2 > 1 + 5e-8
    m = mesh(model(70, 60, order, hx, hy), flags)
    X = m.node_coords()
    k = 2 * np.pi / (9 * hx)
    u = (np.sin(k * X[:, :1] + 0.3) * np.cos(0.8 * k * X[:, 1:])).astype(np.float32)
    e = []
    for precision in (core.FP32, core.FP64):
        p = core.Problem(m, precision, dt=1e-3)
        p.set_field("u", u)
        e.append(p.energy()[1])
    assert abs(e[0] / e[1] - 1) <= 1e-8


@pytest.mark.parametrize("turn", [0.0, 0.4])
@pytest.mark.parametrize("order", range(1, 11))
def test_squares_against_oracle(order, turn):
    """Squares (and squares turned by an angle) through the one-number layout,
    alone and in a group with a mesh of rectangles, which keeps records."""
    # CTAs hold 128 / (N+1) elements: several and a remainder
    cfg = dict(model(7, 13, order, 150.0, 150.0, turn), L=2e3)
    v = cfg["vertices"][cfg["cells"]].mean(axis=1)
    cfg["receivers"] = v[[2, 40, 77]]
    cfg["sources"] = []
    dt = oracle_dt(cfg)
    pairs = [build_pair(cfg, core.FP32, dt) for _ in range(2)]
    (m, p, orc, idx), q = pairs[0], pairs[1][1]
    X = m.node_coords()
    u0 = np.sin(2e-3 * X[:, :1]) * np.cos(3e-3 * X[:, 1:])
    p.set_field("u", u0)
    q.set_field("u", u0)
    orc.set_field("u", u0[np.argsort(idx)])
    p.run(60)
    assert rel_l2(p.seismograms(), orc.run(60, dt)) <= 1e-4
    other = core.Problem(mesh(model(5, 6, order, 150.0, 90.0)), core.FP32, dt=0.5 * dt)
    g = core.Group([other, q])
    g.run(60)
    g.synchronize()
    assert np.array_equal(q.get_field("u"), p.get_field("u"))
    g.close()


@pytest.mark.parametrize("turn", [0.0, 0.4])
def test_layouts_agree(turn):
    """One number per point and the records of a mesh of squares hold the same
    rounded products."""
    cfg = model(24, 24, 4, 150.0, 150.0, turn)
    ps = []
    for flags in (0, core.MESH_PER_POINT_GEOMETRY):
        p = core.Problem(mesh(cfg, flags), core.FP32, dt=1.2e-3)
        X = p.mesh.node_coords()
        p.set_field("u", np.sin(2e-3 * X[:, :1]) * np.cos(3e-3 * X[:, 1:]))
        p.run(40)
        ps.append(p.get_field("u"))
    assert np.array_equal(*ps)
