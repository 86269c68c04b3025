"""SALVUS_BATCH_CONFIG="i,j": the CTA shapes that the indices stand for, read
back from salvus_problem_autotune, their results, which are the same
bits, and that a pin holds after other problems of the same size have been
tuned."""
import numpy as np
import pytest

from salvus_b200 import configs, core

pytestmark = pytest.mark.gpu

# (shots, elements) per CTA of the stiffness kernel; the last: one element and
# the most shots that fit, two per thread
STIFFNESS = [(32, 1), (32, 2), (32, 4), (64, 1), (64, 2), (128, 1), (128, 2), (256, 1), (256, 1)]
# (shots, nodes) per CTA of the gather
GATHER = [(32, 4), (32, 8), (64, 2), (64, 4), (128, 1), (128, 2), (256, 1), (32, 8),
          (64, 4), (128, 2), (128, 4), (256, 2),
          (32, 16), (32, 32), (64, 8), (64, 16), (128, 4), (128, 8), (256, 2), (256, 4),
          (32, 32), (64, 16), (128, 8), (256, 4)]


def problem(mesh, cfg, n_shots):
    p = core.Problem(mesh, core.FP32, dt=4e-3, n_shots=n_shots)
    for s in cfg["sources"]:
        p.add_source(s["location"], s["center_freq"], 0.0, 1.0, shot=s["shot"])
    for r in cfg["receivers"]:
        p.add_receiver(r)
    p.set_field("u", configs.standing_wave_initial(mesh.node_coords(), cfg["L"]), shot=n_shots - 1)
    return p


@pytest.mark.parametrize("step", ["", "unfused"])
@pytest.mark.parametrize("order", [1, 4])
def test_indices_pin_their_shapes(order, step, monkeypatch):
    if step:
        monkeypatch.setenv("SALVUS_BATCH_STEP", step)
    n_shots = 256
    cfg = configs.batched_quad(nel=5, order=order, n_shots=n_shots, n_receivers=3)
    mesh = core.Mesh(cfg["shape"], cfg["order"], cfg["physics"], cfg["vertices"], cfg["cells"],
                     cfg["params"])
    want = None
    pins = [(i, 0) for i in range(len(STIFFNESS))] + [(0, j) for j in range(len(GATHER))]
    for i, j in pins:
        monkeypatch.setenv("SALVUS_BATCH_CONFIG", f"{i},{j}")
        p = problem(mesh, cfg, n_shots)
        assert p.autotune() == (*STIFFNESS[i], *GATHER[j]), (i, j)
        p.run(12)
        got = [p.get_field(f, shot=s) for f in ("u", "v") for s in (0, n_shots - 1)]
        got.append(p.seismograms())
        want = want or got
        assert np.abs(want[1]).max() > 0
        for a, b in zip(got, want):
            assert np.array_equal(a, b), (i, j)


def test_pin_after_tuning(monkeypatch):
    """Tuning results are shared by problems of one size; a pin is not lost to them."""
    cfg = configs.batched_quad(nel=7, order=3, n_shots=64, n_receivers=1)
    mesh = core.Mesh(cfg["shape"], cfg["order"], cfg["physics"], cfg["vertices"], cfg["cells"],
                     cfg["params"])
    monkeypatch.delenv("SALVUS_BATCH_CONFIG", raising=False)
    tuned = problem(mesh, cfg, 64).autotune()
    for i, j in ((0, 0), (1, 3), (2, 1)):
        monkeypatch.setenv("SALVUS_BATCH_CONFIG", f"{i},{j}")
        assert problem(mesh, cfg, 64).autotune() == (*STIFFNESS[i], *GATHER[j])
    monkeypatch.setenv("SALVUS_BATCH_CONFIG", "5,0")  # 128 shots per CTA: not at 64 shots
    assert problem(mesh, cfg, 64).autotune() == tuned
