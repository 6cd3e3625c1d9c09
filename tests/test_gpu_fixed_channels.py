"""Each channel pair of the fixed-point cross terms under its own norms: a
channel far weaker than the others (hydration beside vacuum and dummy, by a
factor of ten to 1e6, in one molecule or both, or absent) keeps its
significant bits.  Unit of a pair: |A_a| |B_b| + |A_b| |B_a| + |A_a| |A_b| +
|B_a| |B_b| (2-norms at that q; the last two are the self terms' rounding).
Each pair's rms error against long double may not exceed that of the FP64
kernels, up to the noise of the tables that both share (1.25)."""
import numpy as np
import pytest

from test_gpu_fixed import case, reference, scores

pytestmark = pytest.mark.gpu
PAIRS = ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))


def norms(X):
    """[3][Q]; the largest entry taken out, for squares that would overflow"""
    top = np.abs(X).max((1, 2))
    return top[:, None] * np.sqrt((np.abs(X / np.where(top > 0, top, 1)[:, None, None]) ** 2).sum(-1))


def units(A, B):
    a, b = norms(A), norms(B)
    with np.errstate(over="ignore"):
        return (np.stack([a[x] * b[y] + a[y] * b[x] for x, y in PAIRS]),
                np.stack([a[x] * a[y] + b[x] * b[y] for x, y in PAIRS]))


@pytest.mark.parametrize("L,Q,skip,scales", [
    (8, 5, 1, ((100.0, 90.0, 9.0), (70.0, 60.0, 6.0))), (8, 5, 0, ((100.0, 90.0, 0.1), (70.0, 60.0, 0.07))),
    (12, 3, 1, ((100.0, 90.0, 0.1), (70.0, 60.0, 50.0))), (5, 9, 1, ((1e-3, 90.0, 5.0), (70.0, 1e-4, 0.0))),
    (20, 2, 1, ((100.0, 90.0, 1e-4), (7.0, 6.0, 0.01)))])
def test_weak_channels_against_long_double(gpu, oracle, L, Q, skip, scales):
    rng = np.random.default_rng(1000 * L + Q)
    q, A, B, z, idx = case(L, Q, 40, 11, scales, rng)
    want = reference(oracle, A, B, q, z, L, idx, skip)
    got = scores(gpu, A, B, q, z, L, idx, skip, gpu.FIT_NONE)
    fp64 = scores(gpu, A, B, q, z, L, idx, skip, gpu.FIT_LBFGSB)
    unit, own = units(A, B)
    u = (unit + own).astype(np.longdouble)
    worse = []
    for c in range(6):
        if not u[c].all():
            assert not got[:, c].any()
            continue
        rms = [np.sqrt(float(((np.abs(x[:, c].astype(np.longdouble) - want[:, c]) / u[c]) ** 2).mean()))
               for x in (got, fp64)]
        print("pair %s: fixed %.3g, FP64 %.3g" % ((PAIRS[c],) + tuple(rms)))
        worse += [PAIRS[c]] if rms[0] > 1.25 * rms[1] + 2.0 ** -55 else []
    assert not worse
