"""The float translation matrices, taken from a fused sum where an interval
around it rounds to one float (kernels_faithful.cu, tm_value), against the
kernel's own FP64 form, which rounds every operation: (float) of its doubles,
bit for bit.  Real Bessel values from far below to far above the cancelling
range, and random ones over 30 binades; one pair to all of L = 48; odd q."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,Q,kind", [(1, 1, "series"), (4, 9, "random"), (12, 13, "series"), (20, 24, "random"),
                                      (30, 9, "series"), (30, 9, "random"), (48, 3, "series")])
def test_floats_are_the_rounded_doubles(gpu, oracle, L, Q, kind):
    torch = pytest.importorskip("torch")
    lib, K, N, nz = gpu.load(), L + 1, 2 * L + 1, 3
    rng = np.random.default_rng(10 * L + Q)
    NT = (Q + 7) // 8
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    ll1 = np.array([(l, l1) for l in range(K) for l1 in range(l, K)], dtype=np.int32)
    ds, pairs = dev(np.asarray(oracle.dsymb(L), dtype=np.float64).reshape(-1)), dev(ll1)
    if kind == "series":
        bes = torch.zeros(nz * N * Q, dtype=torch.float64, device="cuda")
        z, q = dev(np.array([0.02, 8.0, 60.0])), dev(np.linspace(0.0, 0.5, Q) if Q > 1 else np.array([0.3]))
        torch.cuda.synchronize()
        assert lib.sxsk_bessel_z(ptr(z), nz, ptr(q), Q, L, ptr(bes), C.c_void_p(0)) == 0
    else:
        bes = dev(rng.normal(size=nz * N * Q) * 2.0 ** rng.uniform(-15, 15, nz * N * Q))
    out = [torch.zeros(NT * nz * K * K * K * 8, dtype=t, device="cuda") for t in (torch.float64, torch.float32)]
    torch.cuda.synchronize()
    for form in (0, 1):
        assert lib.sxsk_tmatrix(ptr(bes), ptr(ds), nz, Q, L, ptr(pairs), len(ll1), C.c_void_p(0), ptr(out[form]), form,
                                C.c_void_p(0)) == 0
    torch.cuda.synchronize()
    d, f = (x.cpu().numpy() for x in out)
    assert np.abs(d).max() > 0
    np.testing.assert_array_equal(f, d.astype(np.float32))
