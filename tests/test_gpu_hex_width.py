"""A CTA width pinned for one problem does not stay with the mesh: later
problems of orders 4 to 6 take the narrow CTAs and the plain step again."""
import pytest

from salvus_b200 import configs, core

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [4, 5, 6])
def test_unpinned_after_pinned(order, monkeypatch):
    monkeypatch.delenv("SALVUS_HEX_STEP", raising=False)
    monkeypatch.delenv("SALVUS_HEX_CONFIG", raising=False)
    cfg = configs.elastic_hex(nel=3, order=order, n_receivers=0)
    m = core.Mesh(cfg["shape"], cfg["order"], cfg["physics"], cfg["vertices"], cfg["cells"],
                  cfg["params"])
    narrow = 128 // (order + 1) ** 2
    assert core.Problem(m, core.FP32, dt=1e-4).step_config() == (core.STEP_PLAIN, narrow)
    monkeypatch.setenv("SALVUS_HEX_CONFIG", "0,1")
    assert core.Problem(m, core.FP32, dt=1e-4).step_config() == (core.STEP_PLAIN, 2 * narrow)
    monkeypatch.delenv("SALVUS_HEX_CONFIG")
    assert core.Problem(m, core.FP32, dt=1e-4).step_config() == (core.STEP_PLAIN, narrow)
