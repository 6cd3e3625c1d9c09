"""The FP32 per-pose kernel has two forms with the same arithmetic, chosen by
poses per combo, L and the size of the launch: a pose's cross terms are the
same bits whatever list it is in.  Lists from one pose per combo to many,
launches of one block, of less than a wave and of several, a ragged last
block, q tiles with one and with all q; the same poses as parts of a batch,
whose pieces are chained."""
import numpy as np
import pytest

from test_gpu_fixed import SC, coefficients

pytestmark = pytest.mark.gpu


def dimer(gpu, L, Q):
    rng = np.random.default_rng(L)
    q, A = coefficients(L, Q, 12.0, SC[0], rng)
    _, B = coefficients(L, Q, 9.0, SC[1], rng)
    flat = [np.ascontiguousarray(x).view(np.float64).reshape(-1) for x in (A, B)]
    a, mult, peak = gpu.bin_experiment(q, 1e3 * np.exp(-9 * q * q), np.full(len(q), 10.0), q, 1.75)
    return gpu.Plan(flat[0], flat[1], q, np.array([8.0, 9.0, 10.0]), L, a, mult, peak, np.array([1.0]),
                    np.array([1.0]), precision=1)


def lists(L, few, many):
    """`few` poses of distinct combos, and those with `many` more of few combos."""
    rng = np.random.default_rng(7 * L)
    K, N = L + 1, 2 * L + 1
    zbg = rng.permutation(3 * K * N)[:few]
    z, b2, g2 = zbg // (K * N), zbg // N % K, zbg % N
    b1, a2, g1 = rng.integers(K, size=few), rng.integers(N, size=few), rng.integers(N, size=few)
    sparse = ((((z * K + b1) * K + b2) * N + a2) * N + g1) * N + g2
    k = rng.integers(3, size=many)
    dense = ((((z[k] * K + rng.integers(K, size=many)) * K + b2[k]) * N + rng.integers(N, size=many)) * N
             + rng.integers(N, size=many)) * N + g2[k]
    return sparse.astype(np.int64), np.concatenate([sparse, dense]).astype(np.int64)


def cross(gpu, p, idx):
    p.set_poses(idx)
    p.run(gpu.FIT_NONE)
    return p.results(cross=True)["cross"]


@pytest.mark.parametrize("L,Q,few,many", [(1, 1, 3, 9), (6, 9, 33, 300), (12, 8, 900, 9000), (17, 65, 1800, 30000),
                                          (29, 9, 64, 640)])
def test_same_bits_in_sparse_and_dense_lists(gpu, L, Q, few, many):
    p = dimer(gpu, L, Q)
    sparse, dense = lists(L, few, many)
    a, b = cross(gpu, p, sparse), cross(gpu, p, dense)
    assert np.array_equal(a, b[:few])
    p.close()


def test_pieces_of_a_batch(gpu):
    plans, want = [], []
    for L, Q, few, many in ((6, 9, 33, 0), (12, 8, 500, 4000), (9, 17, 300, 0), (4, 3, 1, 0)):
        p = dimer(gpu, L, Q)
        idx = lists(L, few, many)[1]
        p.set_poses(idx)
        p.run(gpu.FIT_GRID)
        want.append(p.results()["chi"].copy())
        plans.append(p)
    b = gpu.Batch(plans)
    for _ in range(2):
        b.run()
        for p, w in zip(plans, want):
            assert np.array_equal(p.results()["chi"], w)
    b.close()
    for p in plans:
        p.close()
