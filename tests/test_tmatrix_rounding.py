"""The translation matrices' floats come from a fused sum only where an
interval around it rounds to one float (kernels_faithful.cu, tm_value): the
same statement compiled for the host against the sum with every operation
rounded.  Alternating terms over many binades, from no cancellation to sums
far below their terms, one term and as many as L = 48 has, zeros; the interval
must also be narrow enough to be of use."""
import ctypes as C
import subprocess

import numpy as np
import pytest

SRC = r'''
#include <math.h>
#include <stdint.h>
#include <string.h>
/* 1: the fused sum decides, 0: it does not; *same: it gives the plain sum's float */
int decide(const double *d, const double *b, int n, int *same)
{
	double v = 0, r = 0, m;
	uint32_t top = 0;
	for (int k = 0; k < n; k++) {
		double w = d[k] * b[k];
		r = k % 2 ? r - w : r + w;
		v = fma(k % 2 ? -d[k] : d[k], b[k], v);
		uint64_t u;
		memcpy(&u, &v, 8);
		uint32_t h = (uint32_t)(u >> 32) & 0x7fffffff;
		if (h > top) top = h;
	}
	uint64_t u = (uint64_t)(top + 1) << 32;
	memcpy(&m, &u, 8);
	m *= 4.0 * n * 0x1p-53;
	*same = (float)v == (float)r;
	return (float)(v - m) == (float)(v + m);
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("tm")
    (d / "t.c").write_text(SRC)
    subprocess.run(["gcc", "-O2", "-std=c11", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(d / "t.so"),
                    str(d / "t.c"), "-lm"], check=True)
    return C.CDLL(str(d / "t.so"))


@pytest.mark.parametrize("n,spread,cancel", [(1, 0, 0), (2, 3, 0), (2, 0, 1), (11, 20, 0), (21, 4, 1), (31, 40, 0),
                                             (49, 8, 1), (49, 0, 0)])
def test_decided_floats_are_the_plain_sums(lib, n, spread, cancel):
    rng = np.random.default_rng(n + spread)
    dp, same, used = C.POINTER(C.c_double), C.c_int(0), 0
    for _ in range(4000):
        d = rng.normal(size=n) * 2.0 ** rng.uniform(-spread, spread, n)
        b = rng.normal(size=n)
        if cancel:
            b[-1] = -np.sum(d[:-1] * b[:-1] * (-1.0) ** np.arange(n - 1)) / (d[-1] * (-1.0) ** (n - 1))
            b[-1] *= 1.0 + rng.choice([0.0, 1e-12, 1e-6])
        if rng.random() < 0.1:
            d[rng.integers(n)] = 0.0
        if lib.decide(d.ctypes.data_as(dp), b.ctypes.data_as(dp), n, C.byref(same)):
            used += 1
            assert same.value
    assert cancel or used > 3900
