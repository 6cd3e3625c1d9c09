"""The block-cooperative L-BFGS-B kernel at the edges of its shapes (fewer
poses than a block's slots, one more than a multiple, long and short q
grids, each threads-per-block choice) against the same solver on the host,
on the plan's own cross terms.  Tolerances as for the other fits (only exp
differs between the two): chi 1e-8 relative, (c1, c2) 1e-6."""
import numpy as np
import pytest

from test_gpu_exact import host_fit  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Q,n,prec", [(2, 1, 0), (5, 17, 1), (51, 16, 0), (64, 700, 0), (65, 33, 1), (203, 300, 0),
                                      (1024, 9, 0)])
def test_block_fit_matches_host_solver(gpu, host_fit, Q, n, prec):  # noqa: F811
    from libfmftsaxs_gb300 import synth
    rng = np.random.default_rng(1000 * Q + n)
    L = 3
    q = gpu.mkarray(0.0, 0.4, Q)
    rec = synth.make_molecule(50, 6.0, 5)
    lig = synth.make_molecule(30, 5.0, 6)
    f = [np.array([gpu.ff_type(e) for e in m.elements]) for m in (rec, lig)]
    A, B = (gpu.expand(m.xyz, v[:, 0], v[:, 1], rng.uniform(0, 0.4, m.natoms), gpu.ff_water(), q, L)
            for m, v in zip((rec, lig), f))
    inten = 1e5 * np.exp(-12.0 * q * q) * (1.0 + 0.02 * rng.normal(size=Q))
    a, mult, peak = gpu.bin_experiment(q, inten, 0.01 * inten, q, 1.75)
    z = np.arange(9.0, 14.0)
    index, _ = gpu.poses_to_indices(synth.random_rotations(2 * n, rng), synth.random_translations(2 * n, 9, 13, rng), z, L)
    index = index[:n]
    p = gpu.Plan(A, B, q, z, L, a, mult, peak, precision=prec)
    p.set_poses(index)
    p.run(gpu.FIT_LBFGSB)
    r = p.results(cross=True)
    p.close()
    c = r["cross"]
    s = peak / (c[:, 0, 0] + c[:, 3, 0] + c[:, 5, 0] + c[:, 2, 0] - c[:, 1, 0] - c[:, 4, 0])
    want = np.array([host_fit((c[i] * s[i]).reshape(-1), q, a, mult) for i in range(len(index))])
    np.testing.assert_allclose(r["chi"], want[:, 0], rtol=1e-8, atol=0)
    np.testing.assert_allclose(r["c1"], want[:, 1], rtol=0, atol=1e-6)
    np.testing.assert_allclose(r["c2"], want[:, 2], rtol=0, atol=1e-6)
