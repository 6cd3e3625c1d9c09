"""The fixed-point accumulation of the expansion and its integer series ratios
against the oracle, at the edges of the kernel's chunks (512 atoms), of Y_lm's
scales (l = 0, 5, 6, 24, 25) and beyond L = 31, and at arguments whose
cancelling series would amplify one wrongly rounded ratio a million-fold.

Tolerance: 1e-13 of sum_a |f_a j_l(q r_a)| times the largest |Y_lm|, for each
channel, q and l: the sums' own rounding is about 2^-53 of that (times the
square root of the number of atoms for the oracle), the angles' functions and
x^l differ by a few units of the last place."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("natoms,L,Q,qmax,radius", [
    (1, 1, 3, 0.5, 20.0), (3, 6, 4, 0.5, 48.0), (127, 5, 3, 0.5, 20.0), (511, 3, 2, 0.4, 15.0), (512, 24, 2, 0.5, 30.0),
    (513, 25, 3, 0.6, 40.0), (1025, 12, 4, 1e-3, 20.0), (40, 31, 3, 0.5, 45.0), (30, 40, 3, 0.6, 45.0)])
def test_expansion_against_oracle(gpu, oracle, natoms, L, Q, qmax, radius):
    rng = np.random.default_rng(natoms + 17 * L)
    d = rng.normal(size=(natoms, 3))
    xyz = d / np.linalg.norm(d, axis=1, keepdims=True) * radius * rng.uniform(0.01, 1.0, (natoms, 1)) ** 0.4
    vac, dum, sasa = rng.uniform(1, 16, natoms), rng.uniform(0.8, 6, natoms), rng.uniform(0, 0.5, natoms)
    q = oracle.mkarray(0.0, qmax, Q)
    got = gpu.expand(xyz, vac, dum, sasa, 3.5, q, L).reshape(3, Q, (L + 1) ** 2, 2)
    want = oracle.expand(xyz, vac, dum, sasa, 3.5, q, L).reshape(3, Q, (L + 1) ** 2, 2)
    r = np.sqrt((xyz * xyz).sum(1))
    for l in range(L + 1):
        j = np.array([[abs(oracle.sbessel(l, x * y)) for y in r] for x in q])
        for c, f in enumerate((vac, dum, 3.5 * sasa)):
            unit = 4 * np.pi * np.sqrt((2 * l + 1) / (4 * np.pi)) * (j @ f)
            e = np.abs(got - want)[c, :, l * l:(l + 1) ** 2].max((1, 2))
            assert np.all(e <= 1e-13 * unit + 1e-300), (l, c, e / unit)


def test_not_finite_weight_stays_in_its_channel(gpu):
    rng = np.random.default_rng(2)
    xyz, q = rng.normal(size=(40, 3)) * 8, np.linspace(0, 0.4, 5)
    f = [rng.uniform(1, 9, 40) for _ in range(3)]
    good = gpu.expand(xyz, f[0], f[1], f[2], 1.0, q, 6).reshape(3, -1)
    f[1][11] = np.nan
    bad = gpu.expand(xyz, f[0], f[1], f[2], 1.0, q, 6).reshape(3, -1)
    assert np.array_equal(bad[[0, 2]], good[[0, 2]])
    assert np.isnan(bad[1]).all()
