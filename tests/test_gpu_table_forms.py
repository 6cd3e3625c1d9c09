"""FP64 runs keep their rotation, translation and matrix tables in one of two
forms by the fit that follows (limbs for the grid, doubles for L-BFGS-B).  The
two fits in turn on one plan, and mixed in one server under the same molecule
keys and with other partners, give the bits of each alone."""
import numpy as np
import pytest

from test_gpu_fixed import SC, case

pytestmark = pytest.mark.gpu
GRID = (np.array([0.98, 1.0, 1.02]), np.array([0.0, 1.0, 2.0, 3.0]))


def job(gpu, L, Q, n, seed):
    q, A, B, z, idx = case(L, Q, n, 17, SC, np.random.default_rng(seed))
    a, mult, peak = gpu.bin_experiment(q, 1e3 * np.exp(-9 * q * q), np.full(len(q), 10.0), q, 1.75)
    return dict(A=A.view(np.float64).reshape(-1), B=B.view(np.float64).reshape(-1), qvals=q, zvals=z, L=L, a=a,
                mult=mult, peak=peak, index=idx, c1grid=GRID[0], c2grid=GRID[1])


def plan(gpu, j, precision=0):
    p = gpu.Plan(j["A"], j["B"], j["qvals"], j["zvals"], j["L"], j["a"], j["mult"], j["peak"], *GRID,
                 precision=precision)
    p.set_poses(j["index"])
    return p


def results(p, fit):
    p.run(fit)
    return p.results(cross=True)


def alone(gpu, j, fit):
    p = plan(gpu, j)
    r = results(p, fit)
    p.close()
    return r


def same(a, b, keys):
    for k in keys:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


def test_fits_in_turn_on_one_plan(gpu):
    j = job(gpu, 7, 19, 120, 1)
    want = {f: alone(gpu, j, f) for f in (gpu.FIT_GRID, gpu.FIT_LBFGSB)}
    p = plan(gpu, j)
    for f in (gpu.FIT_GRID, gpu.FIT_LBFGSB, gpu.FIT_GRID, gpu.FIT_GRID, gpu.FIT_LBFGSB):
        same(results(p, f), want[f], ("chi", "c1", "c2", "cross"))
    p.close()


def test_fits_mixed_in_one_server(gpu):
    js = [job(gpu, 7, 19, 120, 1), job(gpu, 7, 19, 90, 1)]
    js.append(dict(js[0], B=js[0]["B"].reshape(3, -1) * np.array([[1.0], [1e-3], [40.0]])))   # a partner unlike the first
    js[2]["B"] = js[2]["B"].reshape(-1)
    kinds = [(k, f) for f in (gpu.FIT_GRID, gpu.FIT_LBFGSB) for k in (0, 1, 2)]
    want = {(k, f): alone(gpu, js[k], f) for k, f in kinds}
    srv = gpu.Server(max_active=3)
    todo = [kinds[i] for i in np.random.default_rng(2).integers(len(kinds), size=60)]
    t = [srv.submit(fit=f, precision=0, keyA=11, keyB=12 + k // 2, **js[k]) for k, f in todo]
    for i, kf in zip(t, todo):
        same(srv.wait(i), want[kf], ("chi", "c1", "c2"))
    srv.close()
