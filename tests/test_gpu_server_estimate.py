"""The server's estimate of a job's device memory covers every array that the
mesh and the problem of an acoustic quadrilateral job hold, counted with the
estimate's own allowance of nodes (read from the error of a job that exceeds
its budget)."""
import re

import numpy as np
import pytest

from salvus_b200 import core, meshgen, serving

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [1, 4, 10])
def test_estimate_counts_every_array(order):
    n = 450
    V, C = meshgen.structured_quad(n, n, 1e4, 1e4)
    par = np.full((1, len(C), 4), 4000.0)
    srv = serving.Server(budget_bytes=1 << 20)
    with pytest.raises(core.SalvusError) as err:
        srv.submit(dict(shape=core.QUAD, order=order, physics=core.ACOUSTIC, vertices=V, cells=C,
                        params=par, sources=[], receivers=[]), 1e-3, 10)
    srv.close()
    estimate = int(re.search(r"about (\d+) bytes", str(err.value)).group(1))
    E, P = len(C), (order + 1) ** 2
    G = E * order ** 2 * 5 // 4 + 4 * E
    per_point = 4 + 4 + 16 + 4 + 8  # connectivity, incidence, records, one-number layout, set-up mass
    per_node = 4 + 8 + 8 + 4  # offsets, incidence pairs, inverse mass in both precisions
    vertices = 4 * (2 + 1) * 8  # coordinates and speed
    fields = 4 * 4 * G + 4 * E * P + 8 * G  # u w a a_, residual, staging
    assert estimate >= E * (P * per_point + vertices) + G * per_node + fields
