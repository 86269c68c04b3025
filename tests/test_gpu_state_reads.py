"""Reading and preparing a problem's state leaves the rest of it alone: fields read back
as they were set; no device memory is taken to read v of an FP64 problem; a seismogram
read that fails leaves the caller's array; a host allocation that fails in set_field is
an error code."""
import os
import subprocess
import sys
import textwrap

import numpy as np
import pytest
import torch

from salvus_b200 import configs, core

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def problem(cfg, precision=core.FP32, dt=1.5e-3):
    m = core.Mesh(cfg["shape"], cfg["order"], cfg["physics"], cfg["vertices"], cfg["cells"],
                  cfg["params"])
    p = core.Problem(m, precision, dt=dt)
    for r in cfg.get("receivers", []):
        p.add_receiver(r)
    return p


@pytest.mark.parametrize("precision", [core.FP32, core.FP64])
@pytest.mark.parametrize("kind", ["quad", "coupled"])
def test_assembly_and_empty_runs_keep_the_fields(kind, precision):
    cfg = (configs.standing_wave_2d(nel=6, order=4) if kind == "quad"
           else configs.coupled_2d(nel=6, order=3, n_receivers=0))
    p = problem(cfg, precision)
    rng = np.random.default_rng(5)
    shape = (p.mesh.n_nodes, p.c)
    # a_ far above v / dt: v + dt/2 a_ keeps few digits of v
    want = {"u": rng.standard_normal(shape), "v": rng.standard_normal(shape),
            "a_": 1e9 * rng.standard_normal(shape)}
    if precision == core.FP32:
        want = {f: x.astype(np.float32).astype(float) for f, x in want.items()}
    for f, x in want.items():
        p.set_field(f, x)

    def check():
        for f, x in want.items():
            assert np.array_equal(p.get_field(f), x), f

    p.run(0)
    check()
    p.assembleIntoGlobalDof()
    check()
    p.applyInverseMassMatrix()
    check()
    if kind == "quad" and precision == core.FP32:
        g = core.Group([p])
        g.run(0)
        g.synchronize()
        check()
        g.close()

@pytest.mark.parametrize("precision", [core.FP32, core.FP64])
@pytest.mark.parametrize("kind", ["quad", "coupled"])
def test_graphs_captured_before_the_velocity_is_converted(kind, precision):
    """prepare_run captures while v is as it was set; the run converts it first."""
    cfg = (configs.standing_wave_2d(nel=6, order=4) if kind == "quad"
           else configs.coupled_2d(nel=6, order=3, n_receivers=0))
    got = []
    for prepare in (False, True):
        p = problem(cfg, precision)
        x = np.random.default_rng(6).standard_normal((3, p.mesh.n_nodes, p.c))
        p.set_field("u", x[0])
        p.set_field("v", 100.0 * x[1])
        p.set_field("a_", 1e5 * x[2])
        if prepare:
            p.prepare_run(41)
        p.run(41)
        got.append([p.get_field(f) for f in ("u", "v", "a_")])
    for a, b in zip(*got):
        assert np.array_equal(a, b) and np.isfinite(a).all()


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


def test_set_field_reports_a_failed_host_allocation():
    """The address space is limited around the call in a process of its own: an
    error code, not the end of the process; the field is as it was, and the next
    call works."""
    code = textwrap.dedent("""
        import resource
        import numpy as np
        from salvus_b200 import configs, core
        cfg = configs.elastic_hex(nel=34, order=4, n_receivers=0)
        m = core.Mesh(cfg["shape"], cfg["order"], cfg["physics"], cfg["vertices"], cfg["cells"],
                      cfg["params"], flags=core.MESH_FP32_ONLY)
        p = core.Problem(m, core.FP32, dt=1e-4)
        u = np.random.default_rng(1).standard_normal((m.n_nodes, 3))
        assert 24 << 20 < 4 * u.size < 64 << 20
        p.set_field("u", u)
        p.run(3)
        v = p.get_field("v")
        size = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
        hard = resource.getrlimit(resource.RLIMIT_AS)[1]
        resource.setrlimit(resource.RLIMIT_AS, (size + (8 << 20), hard))
        try:
            p.set_field("v", u)
            raise SystemExit("not refused")
        except core.SalvusError as e:
            code = e.code
        finally:
            resource.setrlimit(resource.RLIMIT_AS, (hard, hard))
        assert code == core.E_OOM, code
        assert np.abs(v).max() > 0 and np.array_equal(p.get_field("v"), v)
        p.set_field("v", u)
        assert np.array_equal(p.get_field("v"), u.astype(np.float32))
        print("refused and went on")
    """)
    # every large allocation is a mapping of its own, none served from freed memory
    env = dict(os.environ, MALLOC_MMAP_THRESHOLD_=str(1 << 20))
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=env, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "refused and went on" in r.stdout, r.stdout + r.stderr
