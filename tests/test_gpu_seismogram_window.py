"""Reading seismograms back: any window of the ring, across its wrap, equals
the samples read one step at a time; fields of odd sizes come back as they
were set."""
import numpy as np
import pytest

from salvus_b200 import configs, core

pytestmark = pytest.mark.gpu


def make(nel, order, n_shots, n_receivers, capacity):
    cfg = configs.batched_quad(nel=nel, order=order, n_shots=n_shots, n_receivers=n_receivers)
    mesh = core.Mesh(cfg["shape"], cfg["order"], cfg["physics"], cfg["vertices"], cfg["cells"],
                     cfg["params"])
    p = core.Problem(mesh, core.FP32, dt=2e-3, n_shots=n_shots)
    for s in cfg["sources"]:
        p.add_source(s["location"], s["center_freq"], 0.0, 1.0, shot=s["shot"])
    for r in cfg["receivers"]:
        p.add_receiver(r)
    p.set_seismogram_capacity(capacity)
    x = mesh.node_coords()
    for s in range(n_shots):
        p.set_field("u", np.cos(np.pi * x.sum(axis=1) / cfg["L"] + s), shot=s)
    return p


@pytest.mark.parametrize("n_shots", [1, 3])
@pytest.mark.parametrize("capacity", [1, 7, 50])
def test_windows_of_the_ring(n_shots, capacity):
    p = make(4, 3, n_shots, 5, capacity)
    one = []
    for n in range(63):
        p.step()
        one.append(p.seismograms(n, 1))
    all_ = np.concatenate(one, axis=-1)
    assert np.abs(all_).max() > 0
    for count in {1, capacity // 2, capacity}:
        for first in {63 - capacity, 63 - count}:
            if count > 0:
                assert np.array_equal(p.seismograms(first, count), all_[..., first:first + count])
    with pytest.raises(core.SalvusError):
        p.seismograms(62 - capacity, 1)


@pytest.mark.parametrize("precision", [core.FP32, core.FP64])
@pytest.mark.parametrize("nel,order", [(1, 1), (85, 3), (180, 2), (91, 8)])
def test_field_round_trip(precision, nel, order):
    cfg = configs.standing_wave_2d(nel=nel, order=order)
    mesh = core.Mesh(cfg["shape"], cfg["order"], cfg["physics"], cfg["vertices"], cfg["cells"],
                     cfg["params"])
    p = core.Problem(mesh, precision, dt=1e-3)
    rng = np.random.default_rng(2)
    for name in ("u", "v", "a_"):
        x = rng.standard_normal((mesh.n_nodes, 1))
        p.set_field(name, x)
        want = x if precision == core.FP64 else x.astype(np.float32).astype(np.float64)
        assert np.array_equal(p.get_field(name), want)
