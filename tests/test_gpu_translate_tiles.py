"""The FP32 translation's block forms: columns (n = L + 1 - m up to 28) and row
tiles (n = 29 to 32).  How many slices a block runs (one, a window of eight,
more than a window) only moves work between blocks, so the cross terms are
the same bits; against the FP64 path they are within 1e-5 of each channel
(the mixed path's tolerance).  L across the edge of the two forms and of the
classes of n, lists whose last slices hold 1 to 16 combos, a padded q tile."""
import numpy as np
import pytest

from test_gpu_fixed import SC, case

pytestmark = pytest.mark.gpu


def cross(gpu, L, Q, n, cells, slices, prec=1):
    rng = np.random.default_rng(L + n)
    q, A, B, z, idx = case(L, Q, n, cells, SC, rng)
    flat = [np.ascontiguousarray(x).view(np.float64).reshape(-1) for x in (A, B)]
    a, mult, peak = gpu.bin_experiment(q, 1e3 * np.exp(-9 * q * q), np.full(len(q), 10.0), q, 1.75)
    p = gpu.Plan(flat[0], flat[1], q, z, L, a, mult, peak, np.array([1.0]), np.array([1.0]), precision=prec)
    if slices:
        p.set_tiles(slices, 0)
    p.set_poses(idx)
    p.run(gpu.FIT_NONE)
    out = p.results(cross=True)["cross"]
    p.close()
    return out


@pytest.mark.parametrize("L,Q,n,cells", [(1, 3, 7, 5), (7, 9, 700, 420), (12, 8, 300, 200), (27, 9, 60, 45),
                                         (28, 2, 437, 300), (29, 9, 17, 9), (30, 3, 900, 700), (31, 8, 33, 17)])
def test_slices_per_block_keep_the_bits(gpu, L, Q, n, cells):
    got = cross(gpu, L, Q, n, cells, 0)
    for slices in (1, 8, 9, 40):
        assert np.array_equal(got, cross(gpu, L, Q, n, cells, slices))
    want = cross(gpu, L, Q, n, cells, 0, prec=0)
    scale = np.abs(want).max(axis=-1, keepdims=True)
    assert np.max(np.abs(got - want) / scale) <= 1e-5
