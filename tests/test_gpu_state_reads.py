"""Reading and preparing a problem's state leaves the rest of it alone: no device memory
is taken to read v of an FP64 problem; a seismogram read that fails leaves the caller's
array."""
import numpy as np
import pytest
import torch

from salvus_b200 import configs, core

pytestmark = pytest.mark.gpu


def problem(cfg, precision=core.FP32, dt=1.5e-3):
    m = core.Mesh(cfg["shape"], cfg["order"], cfg["physics"], cfg["vertices"], cfg["cells"],
                  cfg["params"])
    p = core.Problem(m, precision, dt=dt)
    for r in cfg.get("receivers", []):
        p.add_receiver(r)
    return p


def test_reading_v_takes_no_device_memory():
    p = problem(configs.elastic_hex(nel=22, order=4, n_receivers=0), core.FP64, dt=1e-4)
    n = 8 * p.mesh.n_nodes * p.c
    assert n >= 16 << 20
    p.set_field("u", np.random.default_rng(1).standard_normal((p.mesh.n_nodes, p.c)))
    p.run(2)
    p.get_field("u")
    before = torch.cuda.mem_get_info()[0]
    v = p.get_field("v")
    assert before - torch.cuda.mem_get_info()[0] < n // 2
    assert np.abs(v).max() > 0
    # the staging area is the steps' own: they go on as if nothing had been read
    q = problem(configs.elastic_hex(nel=22, order=4, n_receivers=0), core.FP64, dt=1e-4)
    q.set_field("u", np.random.default_rng(1).standard_normal((p.mesh.n_nodes, p.c)))
    p.run(3)
    q.run(5)
    assert np.array_equal(p.get_field("v"), q.get_field("v"))
    assert np.array_equal(p.get_field("u"), q.get_field("u"))


@pytest.mark.parametrize("steps", [32, 3000])
def test_failed_seismogram_read_leaves_the_array(steps):
    cfg = configs.ricker_2d(nel=6, order=4, n_receivers=16)
    p = problem(cfg)
    p.run(steps)
    want = p.seismograms()
    bad = np.zeros((p.mesh.n_nodes, 1))
    bad[p.mesh.n_nodes // 3] = np.nan
    p.set_field("u", bad)
    p.run(64)
    out = np.full(want.shape, 7.0)
    rc = core.lib().salvus_get_seismograms(p.h, 0, steps, core._dp(out))
    assert rc == core.E_NONFINITE
    assert np.all(out == 7.0)
