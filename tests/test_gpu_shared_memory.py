"""A kernel's dynamic shared memory limit belongs to the function, not to a
launch: threads that launch one kernel with different sizes at the same time
must not refuse one another's launches.  The kernels whose size depends on the
call: the L-BFGS-B fit (q points, poses) and the two-beta FP32 rotation (L),
launched from two threads on streams of their own; and server jobs of
different q grids and pose counts, which fit on several workers at once, with
the results of the same jobs alone."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _both(calls, reps):
    """Each call `reps` times from a thread of its own; the statuses."""
    rc, gate = [[] for _ in calls], threading.Barrier(len(calls))

    def loop(k):
        gate.wait()
        for _ in range(reps):
            rc[k].append(calls[k]())

    th = [threading.Thread(target=loop, args=(k,)) for k in range(len(calls))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    return rc


@pytest.fixture
def torch(gpu):
    t = pytest.importorskip("torch")
    yield t
    t.cuda.synchronize()


def test_fits_of_two_threads(gpu, torch):
    """One pose: 15 doubles a q point, so 78 and 120 KB.  A model without
    (c1, c2): one evaluation."""
    lib = gpu.load()

    def call(Q):
        f = lambda n: torch.rand(n, dtype=torch.float64, device="cuda")  # noqa: E731
        q, x, a = torch.linspace(0, 0.5, Q, dtype=torch.float64, device="cuda"), f(6 * Q), f(6 * Q)
        x[Q:] = 0.0
        out, st = f(4), torch.cuda.Stream()
        torch.cuda.synchronize()
        p = [C.c_void_p(v.data_ptr()) for v in (x, q, a)]
        o = [C.c_void_p(out.data_ptr() + 8 * i) for i in range(4)]
        return lambda k=(q, x, a, out, st): lib.sxs_fit_lbfgsb_launch(
            p[0], C.c_int(0), C.c_int(1), C.c_int(Q), p[1], p[2], C.c_double(0.5), C.c_double(1.0), C.c_int(0), *o,
            C.c_void_p(0), C.c_void_p(k[4].cuda_stream))

    assert not any(map(any, _both([call(Q) for Q in (660, 1024)], 300)))


def test_rotations_of_two_threads(gpu, torch):
    """50 and 53 KB of shared memory; one q tile of tables."""
    lib = gpu.load()

    def call(L):
        K, N, Q = L + 1, 2 * L + 1, 2
        f = lambda n: torch.zeros(n, dtype=torch.float32, device="cuda")  # noqa: E731
        spf, dtab, out = f(3 * K * K * Q * 2), f(K * K * N * N), f(K * N * K * (K + 1) // 2 * 3 * 8 * 2)
        tw, st = torch.zeros(2 * N, dtype=torch.float64, device="cuda"), torch.cuda.Stream()
        torch.cuda.synchronize()
        p = [C.c_void_p(v.data_ptr()) for v in (spf, dtab, tw, out)]
        return lambda k=(spf, dtab, tw, out, st): lib.sxsk_rotate(
            p[0], p[1], p[2], C.c_int(Q), C.c_int(L), C.c_int(0), p[3], C.c_int(1), C.c_int(16),
            C.c_void_p(k[4].cuda_stream))

    assert not any(map(any, _both([call(L) for L in (56, 60)], 400)))


def test_server_fits_side_by_side(gpu):
    from test_gpu_fixed import SC, case
    jobs = []
    for k, (Q, n) in enumerate(((201, 5000), (101, 700), (77, 1300), (201, 40), (333, 9), (51, 2600))):
        q, A, B, z, idx = case(3, Q, n, 40, SC, np.random.default_rng(Q + n))
        a, mult, peak = gpu.bin_experiment(q, 1e3 * np.exp(-9 * q * q), np.full(len(q), 10.0), q, 1.75)
        jobs.append(dict(A=A.view(np.float64).reshape(-1), B=B.view(np.float64).reshape(-1), qvals=q, zvals=z, L=3, a=a,
                         mult=mult, peak=peak, index=idx, fit=gpu.FIT_LBFGSB, precision=k % 2))
    want = []
    for j in jobs:
        p = gpu.Plan(j["A"], j["B"], j["qvals"], j["zvals"], j["L"], j["a"], j["mult"], j["peak"],
                     precision=j["precision"])
        p.set_poses(j["index"])
        p.run(gpu.FIT_LBFGSB)
        want.append(p.results())
        p.close()
    srv = gpu.Server(max_active=4)
    t = [srv.submit(**j) for _ in range(12) for j in jobs]
    got = [srv.wait(k) for k in t]
    srv.close()
    for i, g in enumerate(got):
        for k in ("chi", "c1", "c2"):
            np.testing.assert_array_equal(g[k], want[i % len(jobs)][k])
