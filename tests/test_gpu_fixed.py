"""The fixed-point contractions of the plain path (kernels_fixed.cu) against
the same sums in long double (binary128 on aarch64) from the oracle's
Wigner-d, translation and twiddle tables, at the edges of their tiles: column
classes and gamma groups by L, q tiles by Q, slices and pose blocks by the
number of poses.

Tolerance: the tables that both sides take in FP64 (the device's Bessel
values differ from the oracle's by a few units of the last place) move a
cross term by about 2^-50 |A| |B| (2-norms of the channels at that q, the
largest), the limbs by 2^-54; 2^-47 |A| |B| is allowed.  The FP64 kernels (an
L-BFGS-B run has them) are held to the same reference: the fixed-point error
may not be the larger one, up to the noise of the tables they share (1.25)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def coefficients(L, Q, radius, scales, rng):
    """A_lm(q) of a real density with the size profile of a molecule."""
    q = np.arange(Q) * 0.3 / max(1, Q - 1)
    out = np.zeros((3, Q, (L + 1) ** 2), dtype=np.complex128)
    for c, s in enumerate(scales):
        for l in range(L + 1):
            amp = s * np.exp(-((q * radius - l) / 4.0) ** 2)
            for m in range(l + 1):
                v = rng.normal() + 1j * rng.normal()
                if m == 0:
                    v = v.real * 1j ** (l % 2)
                out[c, :, l * l + l + m] = v * amp
                out[c, :, l * l + l - m] = (-1) ** (l + m) * np.conj(v * amp)
    return q, out


def reference(oracle, A, B, q, z, L, index, skip):
    """[n][6][Q] in long double"""
    K, N, Q = L + 1, 2 * L + 1, len(q)
    ld, lc = np.longdouble, np.clongdouble
    v, dig = np.asarray(index, dtype=np.int64).copy(), []
    for base in (N, N, N, K, K):
        dig.append(v % base)
        v //= base
    g2, g1, a2, b2, b1 = dig
    step = 2 * (3.14159265358 if skip else np.pi) / N
    tw = np.array([np.cos(i * step) - 1j * np.sin(i * step) for i in range(N)]).astype(lc)
    beta = 3.14159265358 / L
    wig = {b: oracle.wigner_d(L, b * beta).astype(ld) for b in set(b1) | set(b2)}
    ds = oracle.dsymb(L)
    m_ = np.arange(K)

    def rotated(C, b, g):
        out = np.zeros((K, K, 3, Q), dtype=lc)
        for l in range(K):
            m1 = np.arange(-l, l + 1)
            M = wig[b][l, L:L + l + 1, L - l:L + l + 1] * tw[(m1 * g) % N]
            out[:l + 1, l] = (M[:, :, None, None] * C[:, :, l * l:(l + 1) ** 2].transpose(2, 0, 1)[None]).sum(1)
        return out

    A, B = A.astype(lc), B.astype(lc)
    P = {k: rotated(A, *k) for k in set(zip(b1, g1))}
    U = {k: rotated(np.conj(B), *k) for k in set(zip(b2, g2))}
    T = {}
    for zi in set(v):
        re, im = oracle.t_matrix(L, oracle.besselj_n(float(z[zi]), q, L), ds, Q)
        T[zi] = (re - 1j * im).reshape(Q, K, K, K).astype(lc)          # conj(T)[q][m][l][l1]
    R = {k: np.stack([np.einsum("qlk,kcq->lcq", T[k[0]][:, m], U[k[1:]][m]) for m in range(K)])
         for k in set(zip(v, b2, g2))}
    pairs = ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))
    mul = (1, 2, 2, 1, 2, 1)
    out = np.zeros((len(index), 6, Q), dtype=ld)
    for i in range(len(index)):
        w = tw[(m_ * a2[i]) % N] * np.where(m_ > 0, 2, 1)
        p, r = P[b1[i], g1[i]], R[v[i], b2[i], g2[i]] * w[:, None, None, None]
        for c, (x, y) in enumerate(pairs):
            f = (p[:, :, x] * r[:, :, y]).real.sum((0, 1))
            if x != y:
                f = f + (p[:, :, y] * r[:, :, x]).real.sum((0, 1))
            out[i, c] = 2 * f
            for C in (A, B):
                out[i, c] += mul[c] * (C[x] * np.conj(C[y])).real.sum(-1)
    return out


def case(L, Q, n, cells, scales, rng):
    q, A = coefficients(L, Q, 12.0, scales[0], rng)
    _, B = coefficients(L, Q, 9.0, scales[1], rng)
    z = np.array([8.0, 9.0, 10.0])
    K, N = L + 1, 2 * L + 1
    combos = [(rng.integers(3), rng.integers(K), rng.integers(N)) for _ in range(cells)]
    recs = [(rng.integers(K), rng.integers(N)) for _ in range(4)]
    idx = np.zeros(n, dtype=np.int64)
    for i in range(n):
        zi, b2, g2 = combos[i % cells]
        b1, g1 = recs[rng.integers(4)]
        idx[i] = ((((zi * K + b1) * K + b2) * N + rng.integers(N)) * N + g1) * N + g2
    return q, A, B, z, idx


def scores(gpu, A, B, q, z, L, index, skip, fit):
    flat = [np.ascontiguousarray(x).view(np.float64).reshape(-1) for x in (A, B)]
    a, mult, peak = gpu.bin_experiment(q, 1e3 * np.exp(-9 * q * q), np.full(len(q), 10.0), q, 1.75)
    p = gpu.Plan(flat[0], flat[1], q, z, L, a, mult, peak, np.array([1.0]), np.array([1.0]))
    p.set_poses(index, skip=skip)
    p.run(fit)
    out = p.results(cross=True)["cross"]
    p.close()
    return out


SC = ((100.0, 90.0, 9.0), (70.0, 60.0, 5.0))


@pytest.mark.parametrize("L,Q,n,cells,skip,scales", [
    (1, 1, 1, 1, 1, SC), (2, 9, 40, 33, 0, SC), (3, 8, 17, 9, 1, SC), (7, 3, 20, 5, 1, SC), (8, 2, 16, 8, 0, SC),
    (11, 4, 15, 3, 1, SC), (15, 3, 24, 17, 1, SC), (16, 2, 12, 4, 0, SC), (19, 2, 10, 3, 1, SC), (20, 3, 12, 3, 1, SC),
    (23, 1, 8, 2, 1, SC), (27, 1, 8, 2, 0, SC), (30, 1, 8, 2, 1, SC), (31, 2, 6, 2, 1, SC),
    (6, 5, 20, 6, 1, ((1e-130, 1e-131, 0.0), (3e140, 1e140, 0.0)))])
def test_fixed_point_against_long_double(gpu, oracle, L, Q, n, cells, skip, scales):
    rng = np.random.default_rng(100 * L + Q)
    q, A, B, z, idx = case(L, Q, n, cells, scales, rng)
    want = reference(oracle, A, B, q, z, L, idx, skip)
    got = scores(gpu, A, B, q, z, L, idx, skip, gpu.FIT_NONE)
    fp64 = scores(gpu, A, B, q, z, L, idx, skip, gpu.FIT_LBFGSB)
    norm = [np.sqrt((np.abs(X / max(s)) ** 2).sum(-1).max(0)) * max(s) for X, s in zip((A, B), scales)]
    unit = (norm[0] * norm[1]).astype(np.longdouble)
    # the self terms are common FP64 sums of both sides: compare what is added to them
    e_fix, e_ref = (np.abs(x.astype(np.longdouble) - want) for x in (got, fp64))
    own = norm[0] ** 2 + norm[1] ** 2                     # their rounding
    assert np.all(e_fix <= 2.0 ** -47 * unit + 2.0 ** -50 * own)
    rms = [np.sqrt(float(((e / (unit + own)) ** 2).mean())) for e in (e_fix, e_ref)]
    print("rms error / (|A||B| + |A|^2 + |B|^2): fixed %.3g, FP64 %.3g" % tuple(rms))
    assert rms[0] <= 1.25 * rms[1] + 2.0 ** -55


def test_not_finite_stays_at_its_q(gpu):
    rng = np.random.default_rng(5)
    L, Q = 5, 11
    q, A, B, z, idx = case(L, Q, 30, 7, SC, rng)
    good = scores(gpu, A, B, q, z, L, idx, 1, gpu.FIT_NONE)
    A[1, 4, 7] = np.nan
    B[0, 9, 3] = np.inf
    bad = scores(gpu, A, B, q, z, L, idx, 1, gpu.FIT_NONE)
    keep = [i for i in range(Q) if i not in (4, 9)]
    assert np.array_equal(bad[:, :, keep], good[:, :, keep])
    assert not np.isfinite(bad[:, :, [4, 9]]).any()
