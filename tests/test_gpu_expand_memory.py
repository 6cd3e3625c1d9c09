"""A large expansion gives its work memory back when it returns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_work_memory_is_given_back(gpu):
    """150,000 atoms at L = 30 need 2.2 GB for their Y_lm; what stays with the
    process is less than the bound of 256 MB that smaller calls may keep."""
    rng = np.random.default_rng(1)
    n, L, q = 150000, 30, np.array([0.1])
    xyz, f = rng.normal(size=(n, 3)) * 30, np.ones(n)
    small = gpu.expand(xyz[:50], f[:50], f[:50], f[:50], 1.0, q, L)          # tables of L, module
    free = gpu.device_memory()[0]
    out = gpu.expand(xyz, f, f, f, 1.0, q, L)
    assert np.isfinite(out).all() and np.isfinite(small).all()
    assert gpu.device_memory()[0] >= free - (256 << 20)
