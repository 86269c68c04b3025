"""Sources added by the node gather: several in one element, in neighbouring
elements (nodes of two and more source elements) and on shared vertices,
against the FP64 oracle, and the three-call sequence bitwise against the run.
Tolerances: operation order only in FP64 (1e-10), the repository's FP32
target (1e-4)."""
import numpy as np
import pytest

from salvus_b200 import configs, core
from test_gpu_parity import build_pair, oracle_dt, rel_l2

pytestmark = pytest.mark.gpu

CFGS = {"quad": lambda: configs.ricker_2d(nel=5, order=4, n_receivers=4, radius=1.5e3),
        "hex": lambda: configs.elastic_hex(nel=3, order=3, n_receivers=4),
        "tet": lambda: configs.simplex_tet(n=2, mesh="kuhn", n_receivers=4)}


@pytest.mark.parametrize("precision,tol", [(core.FP64, 1e-10), (core.FP32, 1e-4)])
@pytest.mark.parametrize("kind", sorted(CFGS))
def test_sources_sharing_nodes(kind, precision, tol):
    cfg = CFGS[kind]()
    dt = oracle_dt(cfg)
    f0 = 0.02 / dt
    v = cfg["vertices"][cfg["cells"]]
    e = len(cfg["cells"]) // 2
    centre, near = v[e].mean(axis=0), v[e + 1].mean(axis=0)
    spots = [centre, 0.9 * centre + 0.1 * v[e][0], near, v[e][1], v[0].mean(axis=0)]
    c = 1 if cfg["physics"] == core.ACOUSTIC else 3
    cfg["sources"] = [dict(location=tuple(x), center_freq=f0 * (1 + 0.1 * k), time_delay=0.8 / f0,
                           amplitude=1e3 * (k + 1), direction=[1.0, -0.5, 0.3][:c])
                      for k, x in enumerate(spots)]
    pairs = [build_pair(cfg, precision, dt) for _ in range(2)]
    (mesh, p, orc, idx), q = pairs[0], pairs[1][1]
    n = 60
    p.run(n)
    assert rel_l2(p.seismograms(), orc.run(n, dt)) <= tol
    assert rel_l2(p.get_field("u"), orc.get_field("u")[idx]) <= tol
    for _ in range(n):
        q.assembleIntoGlobalDof()
        q.applyInverseMassMatrix()
        q.takeTimeStep()
    for f in ("u", "v", "a_"):
        assert np.array_equal(p.get_field(f), q.get_field(f)), f
    assert np.array_equal(p.seismograms(), q.seismograms())
