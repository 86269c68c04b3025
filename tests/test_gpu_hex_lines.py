"""Line-exchange hexahedron kernels at the edges of their CTAs (one element,
counts that leave a CTA part full): one assembled acceleration of a random
field against the FP64 oracle, for every order, both precisions, acoustic,
isotropic and transversely isotropic material, parallelepipeds and general
hexahedra.  Tolerances: the repository's for one assembly (FP64 1e-12 from the
operation order, on general hexahedra too; FP32 4e-6)."""
import numpy as np
import pytest

from salvus_b200 import configs, core, meshgen
from test_gpu_parity import build_pair, rel_l2

pytestmark = pytest.mark.gpu


def model(counts, order, kind, jitter):
    nx, ny, nz = counts
    V, C = meshgen.structured_hex(nx, ny, nz, 1e3 * nx, 1.2e3 * ny, 0.9e3 * nz)
    rng = np.random.default_rng(10 * order + nx)
    V = V + jitter * rng.uniform(-100, 100, V.shape)
    vary = lambda x: x * rng.uniform(0.9, 1.1, len(V))  # noqa: E731
    pe = lambda x: meshgen.per_element_vertex(x, C)  # noqa: E731
    rho, vp, vs = vary(2700.0), vary(6000.0), vary(3400.0)
    if kind == "acoustic":
        par = pe(vp)[None]
    elif kind == "ti":
        par = configs.ti_params(rho, vp, vs, C, configs.VTI)
    else:
        par = np.stack([pe(rho), pe(vp), pe(vs)])
    return dict(shape=core.HEX, order=order, vertices=V, cells=C, params=par, L=1e3,
                physics=core.ACOUSTIC if kind == "acoustic" else core.ELASTIC3D)


@pytest.mark.parametrize("precision,tol", [(core.FP64, 1e-12), (core.FP32, 4e-6)])
@pytest.mark.parametrize("kind", ["acoustic", "iso", "ti"])
@pytest.mark.parametrize("order", range(1, 7))
def test_one_assembly(order, kind, precision, tol):
    for counts in ((1, 1, 1), (2, 1, 3), (3, 3, 1), (5, 7, 1)):
        for jitter in (0.0, 1.0):
            mesh, p, orc, idx = build_pair(model(counts, order, kind, jitter), precision, 1e-4)
            u = np.random.default_rng(1).standard_normal((mesh.n_nodes, mesh.n_components))
            u = u.astype(np.float32).astype(np.float64)
            p.set_field("u", u)
            p.assembleIntoGlobalDof()
            p.applyInverseMassMatrix()
            orc.set_field("u", u[np.argsort(idx)])
            assert rel_l2(p.get_field("a"), orc.acceleration(0.0)[idx]) <= tol, (counts, jitter)
