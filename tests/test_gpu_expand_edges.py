"""The expansion at the end of the number range: weights near the smallest
normal numbers give the scaled coefficients, not zeros."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("e", [-960, -990, -1010])
def test_tiny_weights(gpu, e):
    """2^e times the weights, 2^e times the coefficients: to 2^-45 of the
    channel's largest, and the spacing of subnormal numbers, 2^-1074, for each
    of the 700 atoms' terms times 4 pi."""
    rng = np.random.default_rng(-e)
    xyz, q = rng.normal(size=(700, 3)) * 9, np.linspace(0.0, 0.4, 4)
    f = [rng.uniform(1, 9, 700) for _ in range(3)]
    one = gpu.expand(xyz, f[0], f[1], f[2], 1.0, q, 5).reshape(3, -1)
    f[1] = np.ldexp(f[1], e)
    got = gpu.expand(xyz, f[0], f[1], f[2], 1.0, q, 5).reshape(3, -1)
    assert np.array_equal(got[[0, 2]], one[[0, 2]])
    want, up = np.ldexp(one[1], 100), np.ldexp(got[1], 100 - e)
    assert np.all(np.abs(up - want) <= 2.0 ** -45 * np.abs(want).max() + 700 * 4 * np.pi * 2.0 ** (100 - e - 1074))
