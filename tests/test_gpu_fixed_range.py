"""Coefficients as large and as small as FP64 products allow keep their terms
in the fixed-point contractions: finite where the FP64 kernels' terms are, and
within 2^-47 of |A_a| |B_b| + |A_b| |B_a| (and the self terms' rounding) of
them."""
import numpy as np
import pytest

from test_gpu_fixed import case, scores
from test_gpu_fixed_channels import units

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scales", [((1e-200, 1e-201, 1e-199), (1e150, 0.0, 0.0)),
                                    ((1e-290, 0.0, 1e-280), (0.0, 1e150, 1e140)),
                                    ((1e160, 1e100, 1e90), (1e20, 1e21, 1e22))])
def test_large_and_small_coefficients(gpu, scales):
    q, A, B, z, idx = case(6, 5, 20, 6, scales, np.random.default_rng(3))
    got = scores(gpu, A, B, q, z, 6, idx, 1, gpu.FIT_NONE)
    fp64 = scores(gpu, A, B, q, z, 6, idx, 1, gpu.FIT_LBFGSB)
    unit, own = units(A, B)
    assert np.array_equal(np.isfinite(got), np.isfinite(fp64))
    ok = np.isfinite(fp64)
    assert ok.any() and np.abs(fp64[ok]).max() > 0
    with np.errstate(invalid="ignore", over="ignore"):
        e, tol = np.abs(got - fp64), 2.0 ** -47 * unit + 2.0 ** -50 * own
    assert np.all((e <= tol[None])[ok])
