"""The two-beta FP32 rotation (8 or more gamma pairs per thread) against the
one-beta form: the same sums in the same order, so the cross terms of a plan
are the same bits whatever the tile choice.  L + 1 even and odd (a last block
of one beta), more and fewer gamma pairs than the four groups hold, q tiles
with one and seven padded q; above L = 31 against the FP64 path (1e-5 of each
channel, the mixed path's tolerance)."""
import numpy as np
import pytest

from test_gpu_fixed import SC, case

pytestmark = pytest.mark.gpu


def cross(gpu, L, Q, gamma, prec=1):
    rng = np.random.default_rng(L)
    q, A, B, z, idx = case(L, Q, 40, 23, SC, rng)
    flat = [np.ascontiguousarray(x).view(np.float64).reshape(-1) for x in (A, B)]
    a, mult, peak = gpu.bin_experiment(q, 1e3 * np.exp(-9 * q * q), np.full(len(q), 10.0), q, 1.75)
    p = gpu.Plan(flat[0], flat[1], q, z, L, a, mult, peak, np.array([1.0]), np.array([1.0]), precision=prec)
    if gamma:
        p.set_tiles(0, gamma)
    p.set_poses(idx)
    p.run(gpu.FIT_NONE)
    out = p.results(cross=True)["cross"]
    p.close()
    return out


@pytest.mark.parametrize("L,Q,gamma", [(1, 1, 8), (6, 15, 8), (11, 8, 12), (20, 9, 8), (23, 9, 16)])
def test_tile_choice_keeps_the_bits(gpu, L, Q, gamma):
    assert np.array_equal(cross(gpu, L, Q, 2), cross(gpu, L, Q, gamma))


@pytest.mark.parametrize("L,Q", [(24, 9), (31, 2), (36, 3), (48, 2)])
def test_large_l_against_fp64(gpu, L, Q):
    got, want = cross(gpu, L, Q, 0), cross(gpu, L, Q, 0, prec=0)
    scale = np.abs(want).max(axis=-1, keepdims=True)
    assert np.max(np.abs(got - want) / scale) <= 1e-5
