"""The two-nodes-per-thread gather with fixed boundary nodes, and in groups of
orders other than four, bitwise against the three-call sequence and the members
alone."""
import numpy as np
import pytest

from salvus_b200 import core
from test_gpu_gather_pairs import make, state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [core.FP32, core.FP64])
def test_pairs_with_fixed_nodes(precision):
    a, b = (make(159, 160, 3, precision) for _ in range(2))
    assert a.mesh.n_nodes >= 6 * 256 * 148
    fixed = a.mesh.boundary_nodes()
    u0 = a.get_field("u")
    u0[fixed] = 0.0
    for p in (a, b):
        p.set_field("u", u0)
        p.set_dirichlet(fixed)
    a.run(33)
    for _ in range(33):
        b.assembleIntoGlobalDof()
        b.applyInverseMassMatrix()
        b.takeTimeStep()
    for x, y in zip(state(a), state(b)):
        assert np.array_equal(x, y)
    assert not a.get_field("u")[fixed].any() and np.abs(a.get_field("u")).max() > 0


@pytest.mark.parametrize("sizes", [[(115, 115, 3), (111, 109, 3)], [(45, 41, 8), (50, 34, 8), (2, 3, 8)],
                                   [(50, 51, 10)]])
def test_pairs_in_groups(sizes):
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
