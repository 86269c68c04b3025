"""The two-nodes-per-thread gather of acoustic quadrilateral meshes (227 k
nodes and more): odd and even node counts, distorted cells and sources on
shared nodes, bitwise against the three-call sequence, whose assembly gathers
one node per thread; and the same through a group of problems."""
import numpy as np
import pytest

from salvus_b200 import configs, core, meshgen

pytestmark = pytest.mark.gpu


def make(nx, ny, order, precision):
    V, C = meshgen.structured_quad(nx, ny, 1e4, 1e4 * ny / nx)
    rng = np.random.default_rng(nx)
    h = 1e4 / nx
    inner = np.all((V > 0.5 * h) & (V < V.max(axis=0) - 0.5 * h), axis=1)
    V[inner] += rng.uniform(-0.1 * h, 0.1 * h, (inner.sum(), 2))
    par = meshgen.per_element_vertex(rng.uniform(3000, 4000, len(V)), C)[None]
    mesh = core.Mesh(core.QUAD, order, core.ACOUSTIC, V, C, par)
    p = core.Problem(mesh, precision, dt=0.02 * h / 4000 / order)
    e = len(C) // 2 + nx // 2
    for x in (V[C[e]].mean(axis=0), V[C[e]][2], V[C[e + 1]].mean(axis=0)):
        p.add_source(x, 0.01 / p.dt, 0.5 * p.dt, 1e3, direction=[1.0])
    p.add_receiver(V[C[e]].mean(axis=0) + 0.1 * h)
    X = mesh.node_coords()
    p.set_field("u", np.sin(2e-3 * X[:, :1]) * np.cos(3e-3 * X[:, 1:]))
    return p


def state(p):
    return [p.get_field(f) for f in ("u", "v", "a_")] + [p.seismograms()]


@pytest.mark.parametrize("precision", [core.FP32, core.FP64])
@pytest.mark.parametrize("nx,ny,order", [(125, 125, 4), (160, 159, 3), (67, 71, 7)])
def test_pairs_equal_three_call(nx, ny, order, precision):
    a, b = (make(nx, ny, order, precision) for _ in range(2))
    assert a.mesh.n_nodes >= 6 * 256 * 148
    n = 41
    a.run(n)
    for _ in range(n):
        b.assembleIntoGlobalDof()
        b.applyInverseMassMatrix()
        b.takeTimeStep()
    for x, y in zip(state(a), state(b)):
        assert np.array_equal(x, y)
    assert np.abs(a.seismograms()).max() > 0


def test_pairs_in_a_group():
    sizes = [(90, 90, 4), (71, 80, 4), (33, 35, 4)]
    solo = [make(*s, core.FP32) for s in sizes]
    keep = [make(*s, core.FP32) for s in sizes]
    assert sum(p.mesh.n_nodes for p in keep) >= 6 * 256 * 148
    group = core.Group(keep)
    group.run(35)
    group.synchronize()
    for p, q in zip(solo, keep):
        p.run(35)
        for x, y in zip(state(p), state(q)):
            assert np.array_equal(x, y)
    group.close()
