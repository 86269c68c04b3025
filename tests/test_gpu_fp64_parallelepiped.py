"""FP64 elastic hexahedra: one Jacobian per element is taken only where it is as
accurate as the Jacobians of the points.

Sheared cubes far from the origin, their vertices moved by up to a few units in
the last place of the coordinates, against the stiffness action with geometry in
extended precision (numpy longdouble) on the same coordinates.  The default
layout and SALVUS_MESH_PER_POINT_GEOMETRY each have an error of the order of
eps |x| / h from the sums that form their Jacobians; the default must not be
further off (10 % for what the two share: the points' determinants).
"""
import numpy as np
import pytest

from salvus_b200 import core, meshgen

pytestmark = pytest.mark.gpu

RHO, VP, VS = 2500.0, 4000.0, 2300.0


def sheared(n, offset, ulps, seed):
    V, C = meshgen.structured_hex(n, n, n, 1e3, 1e3, 1e3)
    A = np.array([[1.0, 0.3, 0.1], [0.0, 1.0, 0.2], [0.0, 0.0, 1.0]])
    V = V @ A.T + offset
    rng = np.random.default_rng(seed)
    return V + rng.integers(-ulps, ulps + 1, V.shape) * np.spacing(V), C


def exact_action(mesh, V, C, order, u):
    """-K u on longdouble geometry, nodes in the mesh's numbering."""
    T = np.longdouble
    x, w, dphi = core.element_tables(core.HEX, order)
    # the library's vertex order
    sg = np.array([(-1, -1, -1), (-1, 1, -1), (1, 1, -1), (1, -1, -1),
                   (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1)], dtype=T)
    f = (1 + x.astype(T)[:, None, :] * sg) / 2
    g = np.stack([np.prod(np.delete(f, a, axis=2), axis=2) * sg[:, a] / 2 for a in range(3)])
    J = np.einsum("kqv,evx->eqkx", g, V[C].astype(T))  # d x_x / d xi_k
    det = np.einsum("eqx,eqx->eq", J[:, :, 0], np.cross(J[:, :, 1], J[:, :, 2]))
    iJ = np.stack([np.cross(J[:, :, 1], J[:, :, 2]), np.cross(J[:, :, 2], J[:, :, 0]),
                   np.cross(J[:, :, 0], J[:, :, 1])], axis=-1) / det[..., None, None]  # [x][k]
    conn = mesh.connectivity()
    D = dphi.astype(T)  # [k][i][q]
    H = np.einsum("eqxk,eqkc->eqcx", iJ, np.einsum("kiq,eic->eqkc", D, u.astype(T)[conn]))
    lam, mu = T(RHO * (VP ** 2 - 2 * VS ** 2)), T(RHO * VS ** 2)
    s = mu * (H + H.transpose(0, 1, 3, 2))
    tr = lam * np.einsum("eqcc->eq", H)
    for a in range(3):
        s[..., a, a] += tr
    wd = w.astype(T) * det
    r = np.einsum("kiq,eqkc->eic", D, np.einsum("eqxk,eqcx->eqkc", iJ, s * wd[..., None, None]))
    out = np.zeros(u.shape, dtype=T)
    np.subtract.at(out, conn.ravel(), r.reshape(-1, 3))
    return out


@pytest.mark.parametrize("ulps", [0, 2, 4])
@pytest.mark.parametrize("order", [2, 4])
def test_default_layout_is_as_accurate_as_per_point(order, ulps):
    errors = {0: [], core.MESH_PER_POINT_GEOMETRY: []}
    for seed in range(3):
        V, C = sheared(2, 2.0e5, ulps, seed)
        par = np.stack([np.full(C.shape, c) for c in (RHO, VP, VS)])
        for flags in errors:
            m = core.Mesh(core.HEX, order, core.ELASTIC3D, V, C, par, flags=flags)
            p = core.Problem(m, core.FP64, dt=1e-3)
            # constant strain: every element's residual is the derivative of a
            # linear field, so the Jacobians' errors are all that shows
            rng = np.random.default_rng(seed)
            X = m.node_coords() - 2.0e5
            u = 1e-3 * X @ rng.uniform(-1, 1, (3, 3)) + np.sin(X @ rng.uniform(-5e-3, 5e-3, (3, 3)))
            p.set_field("u", u)
            p.assembleIntoGlobalDof()
            want = exact_action(m, V, C, order, u)
            errors[flags].append(float(np.linalg.norm(p.get_field("a") - want) / np.linalg.norm(want)))
    rms = {f: np.sqrt(np.mean(np.square(e))) for f, e in errors.items()}
    print(rms)
    assert rms[0] <= 1.1 * rms[core.MESH_PER_POINT_GEOMETRY]
