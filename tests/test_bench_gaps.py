"""bench.py's launch gaps of the shot-batched step count every kernel, the
receivers too: they run on the problem's stream, in series with the others."""
import pytest

import bench


def test_every_kernel_counts():
    kernels = {"stiffness": 0.44, "sources": 0.011, "gather_update": 0.29, "receivers": 0.017}
    assert bench.launch_gaps(0.763, kernels) == pytest.approx(0.763 - 0.758)
