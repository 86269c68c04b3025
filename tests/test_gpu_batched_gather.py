"""Every split of the batched node gather (shots per CTA x nodes per CTA x nodes
per thread, pinned through SALVUS_BATCH_CONFIG) gives the same bits, at shot
counts that fill one and several 32-shot groups and at an odd node count."""
import numpy as np
import pytest

from salvus_b200 import configs, core

pytestmark = pytest.mark.gpu

LANES = (32, 32, 64, 64, 128, 128, 256, 256, 32, 64, 128, 256)  # shots per CTA of each split


@pytest.mark.parametrize("n_shots", [20, 65, 256])
@pytest.mark.parametrize("step", ["", "unfused"])
def test_gather_splits_agree(n_shots, step, monkeypatch):
    if step:
        monkeypatch.setenv("SALVUS_BATCH_STEP", step)
    cfg = configs.batched_quad(nel=6, order=4, n_shots=n_shots, n_receivers=3)
    mesh = core.Mesh(cfg["shape"], cfg["order"], cfg["physics"], cfg["vertices"], cfg["cells"],
                     cfg["params"])
    X = mesh.node_coords()
    u0 = configs.standing_wave_initial(X, cfg["L"])
    padded = (n_shots + 31) // 32 * 32
    want = None
    for k, lanes in enumerate(LANES):
        if padded % lanes:
            continue
        monkeypatch.setenv("SALVUS_BATCH_CONFIG", f"0,{k}")
        p = core.Problem(mesh, core.FP32, dt=4e-3, n_shots=n_shots)
        for s in cfg["sources"]:
            p.add_source(s["location"], s["center_freq"], 0.0, 1.0, shot=s["shot"])
        for r in cfg["receivers"]:
            p.add_receiver(r)
        for s in (0, n_shots // 2, n_shots - 1):
            p.set_field("u", (s + 1) * u0, shot=s)
        p.run(20)
        got = [p.get_field(f, shot=s) for f in ("u", "v") for s in (0, n_shots - 1)]
        got.append(p.seismograms())
        if want is None:
            want = got
            assert np.abs(want[0]).max() > 0
        for a, b in zip(got, want):
            assert np.array_equal(a, b), (k, lanes)


@pytest.mark.parametrize("n_shots", [20, 65, 96, 224, 256])
@pytest.mark.parametrize("order", [1, 2, 4, 5, 6])
def test_stiffness_splits_agree(n_shots, order, monkeypatch):
    """The same for the stiffness kernel's splits (0-5), one and two shots per
    thread; two neighbouring shots with a source in one element and elsewhere
    take the mixed path of the paired kernel."""
    cfg = configs.batched_quad(nel=5, order=order, n_shots=n_shots, n_receivers=3)
    mesh = core.Mesh(cfg["shape"], cfg["order"], cfg["physics"], cfg["vertices"], cfg["cells"],
                     cfg["params"])
    u0 = configs.standing_wave_initial(mesh.node_coords(), cfg["L"])
    padded = (n_shots + 31) // 32 * 32
    want = None
    for k, lanes in enumerate((32, 32, 32, 64, 128, None)):
        if padded % (lanes or 32) or (lanes is None and padded < 64):
            continue
        monkeypatch.setenv("SALVUS_BATCH_CONFIG", f"{k},0")
        p = core.Problem(mesh, core.FP32, dt=4e-3, n_shots=n_shots)
        for s in cfg["sources"]:
            p.add_source(s["location"], s["center_freq"], 0.0, 1.0, shot=s["shot"])
        for r in cfg["receivers"]:
            p.add_receiver(r)
        p.set_field("u", u0, shot=n_shots // 2)
        p.run(20)
        got = [p.get_field(f, shot=s) for f in ("u", "v") for s in (0, n_shots // 2, n_shots - 1)]
        got.append(p.seismograms())
        if want is None:
            want = got
            assert np.abs(want[1]).max() > 0 and np.abs(want[-1]).max() > 0
        for a, b in zip(got, want):
            assert np.array_equal(a, b), (k, lanes)
