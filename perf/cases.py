"""Measured cases of the scoring library: what its users have it do, through
the public Python entry points (a ctypes mirror of the C API).

A case is a dict of plain values; its "kind" says which call it is:

  oneshot  score_flat: everything from host buffers in one call (with
           "ingest" the poses start as rotation matrices and translations
           and go through poses_to_indices_gpu first, as correlate does)
  plan     a resident Plan of one dimer scored again: run + results; with
           "relist" a pass sets and scores two new pose lists, with "topk"
           the best poses are selected on the device too
  expand   expand: the A_lm(q) coefficients of one molecule from its atoms
  serve    a Server: several ligands against one receptor, submitted
           together and collected
  batch    a Batch: uneven dimers scored by one graph replay

Sizes follow the repository's configurations: L in 10-30, 51-201 q, 1,000 to
210,000 poses, molecules of a few hundred to 8,000 atoms, the 11 x 41 grid of
(c1, c2).  Molecules are seeded uniform balls of atoms, poses uniform
rotations with |t| uniform in the grid's range, the experiment a noisy
profile of one native pose.  Coefficients, grid indices and the binned
experiment are made here in 64 bits, so `exact` can start from the same
inputs without the library.
"""
import math

import numpy as np
import torch

import libfmftsaxs_gb300 as lib

PI = 3.14159265358        # the value the library's grids and series use
C1_GRID = np.array([0.95 + 0.01 * k for k in range(11)])
C2_GRID = np.array([0.1 * k for k in range(41)])
QMAX = 0.5
# vacuum and excluded-volume form factors and radii of C, N, O, S; water
FF_VAC = np.array([5.9992, 6.9946, 7.9994, 15.9998])
FF_DUM = np.array([5.49096, 0.83166, 3.04942, 6.63324])
RADIUS = np.array([1.87, 1.83, 1.55, 1.97])
FF_WATER = 3.50968
# several plans share the card: each may hold this much of translated rows
BUDGET = 24 << 30


def listed():
    """The calls that stand for the library's use, smallest first."""
    return [
        # a few refined poses of a small dimer through the drop-in call: plain
        # FP64 and the reference's own L-BFGS-B fit; latency and launches count
        dict(name="oneshot_fp64_lbfgs_1k", kind="oneshot", L=10, Q=51, rec=500, lig=300, poses=1000, fp64=True,
             lbfgs=True, skip=1, cross=True, ingest=False, tmin=25, tmax=40),
        # a docking run's output scored once, from its rotations and translations
        dict(name="oneshot_mixed_10k", kind="oneshot", L=15, Q=51, rec=1500, lig=1000, poses=10000, fp64=False,
             lbfgs=False, skip=1, cross=False, ingest=True, tmin=25, tmax=40),
        # the smallest benchmark configuration, plain FP64: the grid fit, then
        # the drop-in's L-BFGS-B
        dict(name="plan_fp64_10k", kind="plan", L=15, Q=51, rec=1500, lig=1000, poses=10000, fp64=True, lbfgs=False,
             skip=1, relist=False, topk=0, tmin=25, tmax=40),
        dict(name="plan_fp64_lbfgs_10k", kind="plan", L=15, Q=51, rec=1500, lig=1000, poses=10000, fp64=True,
             lbfgs=True, skip=1, relist=False, topk=0, tmin=25, tmax=40),
        # odd sizes, the exact-twiddle variant, a new list per pass (iterated docking)
        dict(name="relist_fp64_ragged", kind="plan", L=17, Q=77, rec=2111, lig=907, poses=23457, fp64=True,
             lbfgs=False, skip=0, relist=True, topk=0, tmin=28, tmax=47),
        # one list of the production complex on the plain FP64 path
        dict(name="plan_fp64_70k", kind="plan", L=20, Q=101, rec=3500, lig=2000, poses=70000, fp64=True, lbfgs=False,
             skip=1, relist=False, topk=0, tmin=30, tmax=50),
        # the production complex, mixed precision: the headline configuration
        dict(name="plan_mixed_210k", kind="plan", L=20, Q=101, rec=3500, lig=2000, poses=210000, fp64=False,
             lbfgs=False, skip=1, relist=False, topk=100, tmin=30, tmax=50),
        # the large expansion with a list sparse in translated rows
        dict(name="plan_mixed_l30_40k", kind="plan", L=30, Q=201, rec=8000, lig=4000, poses=40000, fp64=False,
             lbfgs=False, skip=1, relist=False, topk=1000, tmin=40, tmax=65),
        # A_lm of the production receptor, and of the largest molecule
        dict(name="expand_3500", kind="expand", atoms=3500, L=20, Q=101),
        dict(name="expand_8000_l30", kind="expand", atoms=8000, L=30, Q=201),
        # ligands screened against one receptor through the serving loop
        dict(name="serve_6", kind="serve", jobs=6, L=20, Q=101, rec=3500, lig=1000, poses=12000, tmin=25, tmax=45),
        # many uneven dimers in one launch
        dict(name="batch_8", kind="batch", jobs=8, lmin=10, lmax=25, qmax_points=101, poses=3000, tmin=25, tmax=45),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(("oneshot", "plan", "plan", "plan", "expand", "expand", "serve", "batch"))
    if kind == "expand":
        L, Q = rng.randint(8, 30), rng.randint(33, 201)
        return dict(kind=kind, atoms=_log(rng, 300, 8000), L=L, Q=Q)
    tmin = rng.randint(24, 36)
    tmax = tmin + rng.randint(8, 20)
    if kind == "serve":
        return dict(kind=kind, jobs=rng.randint(2, 6), L=rng.randint(10, 20), Q=rng.randint(41, 101),
                    rec=_log(rng, 500, 3500), lig=_log(rng, 300, 1000), poses=_log(rng, 2000, 12000), tmin=tmin,
                    tmax=tmax)
    if kind == "batch":
        return dict(kind=kind, jobs=rng.randint(3, 8), lmin=rng.randint(8, 12), lmax=rng.randint(16, 25),
                    qmax_points=rng.randint(51, 101), poses=_log(rng, 1000, 6000), tmin=tmin, tmax=tmax)
    L, Q = rng.randint(10, 30), rng.randint(41, 201)
    fp64 = rng.random() < 0.5
    c = dict(kind=kind, L=L, Q=Q, rec=_log(rng, 500, 8000), lig=_log(rng, 300, 4000), fp64=fp64,
             lbfgs=rng.random() < 0.25, skip=rng.randint(0, 1), tmin=tmin, tmax=tmax)
    pairs = Q * (L + 1) * (L + 2) // 2
    # poses log-uniform, up to the work of the largest listed case of the path
    top = min(210000 if kind == "plan" else 20000, (1600000000 if fp64 else 4000000000) // pairs,
              20000 if c["lbfgs"] else 210000)
    c["poses"] = _log(rng, 1000, top)
    if kind == "oneshot":
        return dict(c, cross=c["poses"] < 3000, ingest=rng.random() < 0.5)
    return dict(c, relist=rng.random() < 0.3, topk=rng.choice((0, 100)))


# ------------------------------------------------------------------ inputs
def _dev():
    return torch.device("cuda")


def _rng(*seed):
    return np.random.default_rng([int(s) for s in seed])


def _qvals(Q, qmax=QMAX):
    """lib.mkarray's grid: the step added up."""
    step, q = qmax / (Q - 1), np.zeros(Q)
    for i in range(1, Q):
        q[i] = q[i - 1] + step
    return q


def _molecule(n, rng):
    """n atoms in a ball at protein density: coordinates centred at the
    origin, (vacuum, dummy, accessible fraction), the mean radius."""
    R = (n / 0.06 * 3.0 / (4.0 * math.pi)) ** (1.0 / 3.0)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    r = R * rng.uniform(size=n) ** (1.0 / 3.0)
    x = d * r[:, None]
    el = rng.choice(4, size=n, p=(0.63, 0.17, 0.19, 0.01))
    # buried inside, up to half of the sphere free at the surface
    sasa = np.clip((r - (R - 4.0)) / 4.0, 0.0, 1.0) * rng.uniform(0.0, 0.5, size=n)
    return x - x.mean(axis=0), FF_VAC[el], FF_DUM[el], sasa, float(RADIUS[el].mean())


def _legendre(L, x):
    """Orthonormal Legendre functions [m][l][x] (zero for l < m), with the
    Condon-Shortley phase: Y_lm = out e^{i m phi}."""
    s = torch.sqrt(torch.clamp(1.0 - x * x, min=0.0))
    out = torch.zeros((L + 1, L + 1) + x.shape, dtype=torch.float64, device=x.device)
    pmm = torch.full_like(x, math.sqrt(1.0 / (4.0 * math.pi)))
    for m in range(L + 1):
        if m:
            pmm = -math.sqrt((2 * m + 1) / (2.0 * m)) * s * pmm
        out[m, m] = pmm
        if m < L:
            out[m, m + 1] = math.sqrt(2 * m + 3) * x * pmm
        for l in range(m + 2, L + 1):
            a = math.sqrt((4.0 * l * l - 1) / (l * l - m * m))
            b = math.sqrt(((l - 1.0) ** 2 - m * m) / (4.0 * (l - 1) ** 2 - 1))
            out[m, l] = a * (x * out[m, l - 1] - b * out[m, l - 2])
    return out


def _legendre_p(n, x):
    """P_p(x), p = 0..n."""
    out = [torch.ones_like(x), x.clone()]
    for p in range(1, n):
        out.append(((2 * p + 1) * x * out[p] - p * out[p - 1]) / (p + 1))
    return torch.stack(out[:n + 1])


def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return torch.tensor(x, device=_dev()), torch.tensor(w, device=_dev())


def _bessel(L, x):
    """j_l(x), l = 0..L, by Gauss quadrature of its Legendre integral."""
    t, w = _gauss(96)
    P = _legendre_p(max(L, 1), t)[:L + 1] * w
    c, s = torch.cos(x[..., None] * t), torch.sin(x[..., None] * t)
    return [((-1) ** (l // 2)) * 0.5 * ((c if l % 2 == 0 else s) @ P[l]) for l in range(L + 1)]


def _bessel_series(l, x):
    """j_l(x) as the library defines it: the power series from 1/(2l+1)!!,
    stopped where |term / sum| <= 1e-5, times x^l."""
    tl1, f = 2.0 * l + 1.0, 1.0
    for i in range(1, 2 * l + 2, 2):
        f *= float(i)
    term = torch.full_like(x, 1.0 / f)
    total, num, live = term.clone(), (-1.0) * x * x, x > 0
    for k in range(1, 100000):
        live = live & ((term / total).abs() > 0.00001)
        if not bool(live.any()):
            break
        t2 = term * (num / ((2.0 * k) * (2.0 * k + tl1)))
        term = torch.where(live, t2, term)
        total = torch.where(live, total + t2, total)
    return torch.where(x > 0, total * x ** float(l), torch.full_like(x, 1.0 if l == 0 else 0.0))


def _coefficients(xyz, f, q, L, bessel=None):
    """A_lm(q) = 4 pi i^l sum_a f_a j_l(q r_a) conj(Y_lm(a)) of weights f
    [channels][atoms]: complex [channels][Q][(L+1)^2]."""
    d = _dev()
    x = torch.tensor(xyz, device=d)
    f = torch.tensor(np.asarray(f), device=d)
    q = torch.tensor(q, device=d)
    r = torch.sqrt((x * x).sum(1))
    th = _legendre(L, x[:, 2] / r)                                   # [m][l][atom]
    ph = torch.atan2(x[:, 1], x[:, 0])
    e = torch.exp(-1j * ph * torch.arange(L + 1, device=d)[:, None])  # [m][atom]
    qr = q[:, None] * r[None, :]
    js = bessel(qr) if bessel else _bessel(L, qr)
    out = torch.zeros((f.shape[0], len(q), (L + 1) ** 2), dtype=torch.complex128, device=d)
    for l in range(L + 1):
        yp = th[:l + 1, l] * e[:l + 1]                               # conj(Y_lm), m = 0..l
        sg = torch.tensor([(-1.0) ** m for m in range(l, 0, -1)], dtype=torch.float64, device=d)
        y = torch.cat([(sg[:, None] * yp[1:].conj().flip(0)), yp]) if l else yp
        w = (f[:, None, :] * js[l]).reshape(-1, len(r))
        a = torch.complex(w @ y.real.T, w @ y.imag.T) * (4.0 * PI * 1j ** l)
        out[:, :, l * l:(l + 1) ** 2] = a.reshape(f.shape[0], len(q), 2 * l + 1)
    return out


def _poses(n, tmin, tmax, rng):
    """Uniform ligand rotations [n][9] and translations [n][3]."""
    v = rng.normal(size=(n, 4))
    w, x, y, z = (v / np.linalg.norm(v, axis=1, keepdims=True)).T
    R = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w), 2 * (x * y + z * w),
                  1 - 2 * (x * x + z * z), 2 * (y * z - x * w), 2 * (x * z - y * w), 2 * (y * z + x * w),
                  1 - 2 * (x * x + y * y)], axis=1)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return R, d * rng.uniform(tmin, tmax, size=n)[:, None]


def _indices(R, T, zvals, L):
    """The packed grid index of each pose whose z is on the grid: the Euler
    angles, rounded to three decimals, rounded to the grid without wrap."""
    z = np.round(np.sqrt((T * T).sum(1)))
    c1 = lambda v: np.clip(v, -1.0, 1.0)  # noqa: E731
    b1 = np.arccos(c1(T[:, 2] / z))
    sb = z * np.sin(b1)
    g1 = np.arccos(c1(-T[:, 0] / sb))
    g1 = np.where(T[:, 1] / sb < 0.0, 2 * PI - g1, g1)
    cb, s, cg, sg = np.cos(b1), np.sin(b1), np.cos(g1), np.sin(g1)
    M = R.reshape(-1, 3, 3)
    rec = np.stack([np.stack([cg * cb, -sg * cb, s], 1), np.stack([sg, cg, np.zeros_like(s)], 1),
                    np.stack([-cg * s, sg * s, cb], 1)], 1)
    m = rec @ M
    b2 = np.arccos(c1(m[:, 2, 2]))
    s2 = np.sin(b2)
    a2 = np.arccos(c1(m[:, 0, 2] / s2))
    a2 = np.where(m[:, 1, 2] / s2 < 0.0, 2 * PI - a2, a2)
    g2 = np.arccos(c1(-m[:, 2, 0] / s2))
    g2 = np.where(m[:, 2, 1] / s2 < 0.0, 2 * PI - g2, g2)
    z, b1, g1, a2, b2, g2 = (np.round(v * 1000.0) / 1000.0 for v in (z, b1, g1, a2, b2, g2))
    slot = np.round(z - zvals[0]).astype(np.int64)
    keep = (slot >= 0) & (slot < len(zvals))
    N, nb = 2 * L + 1, L + 1
    half = lambda v: np.floor(v + 0.5).astype(np.int64)  # noqa: E731
    i = slot * nb + half(b1 / (PI / L))
    i = i * nb + half(b2 / (PI / L))
    for a in (2 * PI - a2, g1, 2 * PI - g2):
        i = i * N + half(a / (2.0 * PI / N))
    # the reference's angles are not wrapped: a pose at the end of the last
    # slot can carry past the grid, which the library refuses
    keep &= i < len(zvals) * nb * nb * N ** 3
    return i[keep]


def _binned(eq, ei, ee, q, rm):
    """The six weighted moments of the experiment per q bin, the exponent
    of the excluded-volume correction and the first intensity."""
    a, j = np.zeros((len(q), 6)), 0
    for i in range(len(q)):
        lo = q[max(i - 1, 0)]
        while j < len(eq) and lo <= eq[j] <= q[i]:
            w = 1.0 / (ee[j] * ee[j])
            a[i] += np.array([ei[j] * ei[j], ei[j], eq[j] * ei[j], 1.0, eq[j], eq[j] * eq[j]]) * w
            j += 1
    return (a / j).reshape(-1), (4.0 * PI / 3.0) ** 1.5 * rm * rm / (16.0 * PI), float(ei[0])


class Dimer:
    """One dimer's inputs as host arrays, from the seed alone."""

    def __init__(self, L, Q, rec, lig, poses, tmin, tmax, seed, lists=1, receptor=None):
        rng = _rng(seed, L, Q, poses)
        self.L, self.Q = L, Q
        self.q = _qvals(Q)
        self.z = np.arange(float(tmin), tmax + 1.0)
        if receptor is None:
            m = _molecule(rec, rng)
            f = np.stack([m[1], m[2], FF_WATER * m[3]])
            receptor = (m, f, _flat(_coefficients(m[0], f, self.q, L)))
        self.receptor = receptor
        (xa, _, _, _, ra), fa, self.A = receptor
        xb, vb, db, sb, rb = _molecule(lig, rng)
        fb = np.stack([vb, db, FF_WATER * sb])
        self.B = _flat(_coefficients(xb, fb, self.q, L))
        self.rm = (ra * len(xa) + rb * len(xb)) / (len(xa) + len(xb))
        # the experiment: the joined native pose, 1 % noise
        R, T = _poses(1, tmin, tmax, rng)
        xn = np.concatenate([xa, xb @ R[0].reshape(3, 3).T + T[0]])
        fn = np.concatenate([fa, fb], axis=1)
        amp = _coefficients(xn - xn.mean(axis=0), (fn[0] - fn[1] + fn[2])[None], self.q, min(L, 12))
        inten = (amp.abs() ** 2).sum(-1)[0].cpu().numpy()
        self.ei = inten * (1.0 + 0.01 * rng.normal(size=Q))
        self.ee = 0.01 * inten
        self.RT = [_poses(poses, tmin, tmax, rng) for _ in range(lists)]
        self.index = [_indices(r, t, self.z, L) for r, t in self.RT]
        self.a, self.mult, self.peak = _binned(self.q, self.ei, self.ee, self.q, self.rm)


def _flat(c):
    return torch.view_as_real(c).cpu().numpy().reshape(-1)


def _dimer(case, seed):
    return Dimer(case["L"], case["Q"], case["rec"], case["lig"], case["poses"], case["tmin"], case["tmax"], seed,
                 lists=2 if case.get("relist") else 1)


def _batch_dimers(case, seed):
    """Uneven dimers: L and Q spread over the case's range, pose counts over
    a factor of sixteen."""
    out, n = [], case["jobs"]
    for k in range(n):
        f = k / max(1, n - 1)
        L = int(round(case["lmin"] + (case["lmax"] - case["lmin"]) * ((k * 3) % n) / max(1, n - 1)))
        Q = 51 if k % 2 else case["qmax_points"]
        out.append(Dimer(L, Q, 500 + 250 * k, 300 + 150 * k, int(case["poses"] * 16 ** f / 4), case["tmin"],
                         case["tmax"], seed * 64 + k))
    return out


def _serve_dimers(case, seed):
    first = Dimer(case["L"], case["Q"], case["rec"], case["lig"], case["poses"], case["tmin"], case["tmax"], seed * 64)
    return [first] + [Dimer(case["L"], case["Q"], case["rec"], case["lig"] + 37 * k, case["poses"] - 211 * k,
                            case["tmin"], case["tmax"], seed * 64 + k, receptor=first.receptor)
                      for k in range(1, case["jobs"])]


def _plan(d, fp64):
    p = lib.Plan(d.A, d.B, d.q, d.z, d.L, d.a, d.mult, d.peak, C1_GRID, C2_GRID,
                 precision=lib.FP64 if fp64 else lib.MIXED)
    p.set_budget(BUDGET)
    return p


# ------------------------------------------------------------- the protocol
def prepare(case, seed):
    """What a program holds before the call: host inputs, and the plan,
    server or batch that it keeps."""
    lib.init(0)
    kind = case["kind"]
    if kind == "expand":
        m = _molecule(case["atoms"], _rng(seed, case["atoms"], case["L"]))
        return dict(case=case, mol=m, q=_qvals(case["Q"]))
    if kind == "batch":
        ds = _batch_dimers(case, seed)
        plans = []
        for d in ds:
            plans.append(_plan(d, False))
            plans[-1].set_poses(d.index[0], skip=1)
        return dict(case=case, plans=plans, batch=lib.Batch(plans, arena_bytes=BUDGET))
    if kind == "serve":
        return dict(case=case, dimers=_serve_dimers(case, seed), server=lib.Server(hbm_cap=2 * BUDGET, max_active=4))
    d = _dimer(case, seed)
    s = dict(case=case, d=d, at=0)
    if kind == "plan":
        s["plan"] = _plan(d, case["fp64"])
        if not case["relist"]:
            s["plan"].set_poses(d.index[0], skip=case["skip"])
    return s


def run(s):
    """One pass through the public entry points; its results."""
    case = s["case"]
    kind = case["kind"]
    if kind == "expand":
        x, vac, dum, sasa, _ = s["mol"]
        return lib.expand(x, vac, dum, sasa, FF_WATER, s["q"], case["L"])
    if kind == "batch":
        s["batch"].run()
        return [p.results() for p in s["plans"]]
    if kind == "serve":
        t = [s["server"].submit(d.A, d.B, d.q, d.z, d.L, d.a, d.mult, d.peak, d.index[0], C1_GRID, C2_GRID, keyA=1)
             for d in s["dimers"]]
        got = [s["server"].wait(k) for k in t]
        return [dict(chi=g["chi"], c1=g["c1"], c2=g["c2"]) for g in got]
    d = s["d"]
    fit = lib.FIT_LBFGSB if case["lbfgs"] else lib.FIT_GRID
    if kind == "oneshot":
        index = d.index[0]
        if case["ingest"]:
            index = lib.poses_to_indices_gpu(d.RT[0][0], d.RT[0][1], d.z, d.L)[0]
        r = lib.score_flat(d.A, d.B, d.q, d.z, d.L, index, d.a, d.mult, d.peak, skip=case["skip"], fit=fit,
                           c1grid=C1_GRID, c2grid=C2_GRID, cross=case["cross"],
                           precision=lib.FP64 if case["fp64"] else lib.MIXED)
        return dict(r, index=index) if case["ingest"] else r
    p = s["plan"]
    if case["relist"]:
        for index in d.index:                 # the lists of two docking rounds
            p.set_poses(index, skip=case["skip"])
            p.run(fit)
        return p.results()
    p.run(fit)
    r = p.results()
    if case["topk"]:
        r["best"] = p.topk(case["topk"])
    return r


# --------------------------------------------------------------- work, exact
def _score_work(L, Q, n, rows, nz, cells):
    """Multiply-adds of the factorized correlation: both rotation tables'
    touched rows, the translation of `rows` rows, the per-pose sums and the
    grid's cells; bytes: coefficients and pose list in, scores out."""
    K, NP = L + 1, (L + 1) * (L + 2) // 2
    tri = sum((K - m) ** 2 for m in range(K))
    rot = sum((l + 1) * (2 * l + 1) for l in range(K))
    flops = n * Q * NP * 54.0 + rows * Q * tri * 12.0 + 2 * min(n, K * (2 * L + 1)) * Q * rot * 24.0
    flops += n * Q * 11 * 40.0 + n * cells * 10.0
    return {"bytes": 2 * 3.0 * Q * K * K * 16 + n * (8 + 28.0), "flops": flops}


def _touched(L, n, nz):
    cells = nz * (L + 1) * (2 * L + 1)
    return cells * (1.0 - math.exp(-n / cells))


def work(case):
    kind = case["kind"]
    if kind == "expand":
        K2, n, Q = (case["L"] + 1) ** 2, case["atoms"], case["Q"]
        return {"bytes": n * 48.0 + 3.0 * Q * K2 * 16, "flops": 12.0 * n * Q * K2 + 60.0 * n * Q * (case["L"] + 1)}
    if kind in ("batch", "serve"):
        tot = {"bytes": 0.0, "flops": 0.0}
        n = case["jobs"]
        for k in range(n):
            if kind == "serve":
                L, Q, m = case["L"], case["Q"], case["poses"] - 211 * k
            else:
                L = int(round(case["lmin"] + (case["lmax"] - case["lmin"]) * ((k * 3) % n) / max(1, n - 1)))
                Q, m = 51 if k % 2 else case["qmax_points"], int(case["poses"] * 16 ** (k / max(1, n - 1)) / 4)
            nz = case["tmax"] - case["tmin"] + 1
            w = _score_work(L, Q, m, _touched(L, m, nz), nz, 451)
            tot = {key: tot[key] + w[key] for key in tot}
        return tot
    nz = case["tmax"] - case["tmin"] + 1
    w = _score_work(case["L"], case["Q"], case["poses"], _touched(case["L"], case["poses"], nz), nz,
                    0 if case["lbfgs"] else 451)
    times = 2 if case.get("relist") else 1
    if case.get("cross"):
        w["bytes"] += case["poses"] * 48.0 * case["Q"]
    return {key: v * times for key, v in w.items()}


def _wigner(L, nb):
    """d^l_{m m1}(b PI / L) as [b][l][m + L][m1 + L], from the eigenvectors of
    J_y: d = V exp(-i beta M) V^H with the sign convention of the expansion."""
    out = np.zeros((nb, L + 1, 2 * L + 1, 2 * L + 1))
    for l in range(L + 1):
        m = np.arange(-l, l)
        c = np.sqrt(l * (l + 1.0) - m * (m + 1.0))
        jy = np.zeros((2 * l + 1, 2 * l + 1), dtype=np.complex128)
        jy[np.arange(1, 2 * l + 1), np.arange(2 * l)] = c / 2j
        jy[np.arange(2 * l), np.arange(1, 2 * l + 1)] = -c / 2j
        w, v = np.linalg.eigh(jy)
        w = np.round(w)
        for b in range(nb):
            d = (v * np.exp(-1j * w * (b * (PI / (nb - 1))))) @ v.conj().T
            out[b, l, L - l:L + l + 1, L - l:L + l + 1] = d.real
    return out


def _rotated(flat, L, Q, rows, tw, wig, conj):
    """Rotation table of the touched rows (b N + g): complex [rows][m][l][3][Q],
    sum over m1 of tw[(m1 g) mod N] d^l_{m m1}(b) A_{l m1}."""
    N, K = 2 * L + 1, L + 1
    dev = _dev()
    A = torch.view_as_complex(torch.tensor(flat, device=dev).reshape(3, Q, K * K, 2))
    if conj:
        A = A.conj()
    out = torch.zeros((len(rows), K, K, 3 * Q), dtype=torch.complex128, device=dev)
    b, g = torch.tensor(rows // N, device=dev), torch.tensor(rows % N, device=dev)
    W = torch.tensor(wig, device=dev)
    for l in range(K):
        m1 = torch.arange(-l, l + 1, device=dev)
        ph = tw[(m1[None, :] * g[:, None]) % N]                       # [rows][m1]
        M = ph[:, None, :] * W[b, l, L:L + l + 1, L - l:L + l + 1]    # [rows][m][m1]
        C = A[:, :, l * l:(l + 1) ** 2].permute(2, 0, 1).reshape(2 * l + 1, 3 * Q)
        out[:, :l + 1, l] = (M.reshape(-1, 2 * l + 1) @ C).reshape(len(rows), l + 1, 3 * Q)
    return out.reshape(len(rows), K, K, 3, Q)


def _translation(L, q, z):
    """<l m| exp(i q z cos theta) |l1 m> with the library's Bessel series:
    complex [Q][m][l][l1]."""
    t, w = _gauss(2 * L + 2)
    Y = _legendre(L, t)
    x = torch.tensor(q * z, device=_dev())
    P = _legendre_p(2 * L, t)
    N = 2 * L + 1
    rad = torch.stack([_bessel_series(p, x) * (2 * p + 1) for p in range(N)])          # [p][Q]
    out = torch.zeros((len(q), L + 1, L + 1, L + 1), dtype=torch.complex128, device=_dev())
    for par in (0, 1):                        # even p are real, odd p imaginary
        ps = torch.arange(par, N, 2, device=_dev())
        sg = torch.tensor([(1.0 if (p // 2) % 2 == 0 else -1.0) for p in range(par, N, 2)], dtype=torch.float64,
                          device=_dev())
        # sum over |l - l1| <= p <= l + l1 is the full sum: other p integrate to zero
        f = (rad[ps] * sg[:, None]).T @ P[ps]                                           # [Q][t]
        for m in range(L + 1):
            Yw = Y[m] * (2 * math.pi * w)
            T = torch.einsum("lt,qt,kt->qlk", Yw, f, Y[m])
            l = torch.arange(L + 1, device=_dev())
            T = T * (((l[:, None] + l[None, :]) % 2) == par)
            out[:, m] += T * (1.0 if par == 0 else 1j)
    return out


def _self_terms(A, B, L, Q):
    out = 0.0
    for c in (A, B):
        v = torch.view_as_complex(torch.tensor(c, device=_dev()).reshape(3, Q, (L + 1) ** 2, 2))
        out = out + torch.stack([mul * (v[i] * v[j].conj()).real.sum(-1)
                                 for i, j, mul in ((0, 0, 1), (0, 1, 2), (0, 2, 2), (1, 1, 1), (1, 2, 2), (2, 2, 1))])
    return out


def _cross_terms(d, index, skip):
    """The six cross terms of every pose, [n][6][Q]."""
    L, Q = d.L, d.Q
    K, N, dev = L + 1, 2 * L + 1, _dev()
    v, dig = index.copy(), []
    for base in (N, N, N, K, K):
        dig.append(v % base)
        v //= base
    g2, g1, a2, b2, b1 = dig
    step = 2 * (PI if skip else math.pi) / N
    tw = torch.tensor([complex(math.cos(i * step), -math.sin(i * step)) for i in range(N)], dtype=torch.complex128,
                      device=dev)
    wig = _wigner(L, K)
    ur, ri = np.unique(b1 * N + g1, return_inverse=True)
    P = _rotated(d.A, L, Q, ur, tw, wig, False)
    ul, li = np.unique(b2 * N + g2, return_inverse=True)
    U = _rotated(d.B, L, Q, ul, tw, wig, True)
    cst = _self_terms(d.A, d.B, L, Q)
    out = torch.zeros((len(index), 6, Q), dtype=torch.float64, device=dev)
    mm = np.arange(K)
    for z in np.unique(v):
        sel = np.nonzero(v == z)[0]
        T = _translation(L, d.q, float(d.z[z])).conj()
        for c0 in range(0, len(sel), 256):
            s = sel[c0:c0 + 256]
            lu, lj = np.unique(li[s], return_inverse=True)
            Ru = torch.zeros((len(lu), K, K, 3, Q), dtype=torch.complex128, device=dev)
            Us = U[torch.tensor(lu, device=dev)]
            for m in range(K):
                Ru[:, m] = torch.einsum("qlk,rkcq->rlcq", T[:, m], Us[:, m])
            w = tw[torch.tensor((mm[None, :] * a2[s][:, None]) % N, device=dev)]
            w[:, 1:] *= 2.0
            R = Ru[torch.tensor(lj, device=dev)] * w[:, :, None, None, None]
            p = P[torch.tensor(ri[s], device=dev)]
            f = [(p[:, :, :, i] * R[:, :, :, j]).real.sum((1, 2)) for i in range(3) for j in range(3)]
            F = torch.stack([f[0], f[1] + f[3], f[2] + f[6], f[4], f[5] + f[7], f[8]], 1)
            out[torch.tensor(s, device=dev)] = cst + 2.0 * F
    return out


def _grid_fit(cross, d):
    """The best cell of the (c1, c2) grid per pose: the peak rescale, the
    piecewise-linear model, the best scale."""
    dev = _dev()
    q = torch.tensor(d.q, device=dev)
    a = torch.tensor(d.a, device=dev).reshape(-1, 6)
    c1, c2 = torch.tensor(C1_GRID, device=dev), torch.tensor(C2_GRID, device=dev)
    G = c1[:, None] ** 3 * torch.exp(-d.mult * (c1[:, None] ** 2 - 1.0) * q * q)      # [c1][q]
    h = torch.cat([torch.tensor([q[0] + 1.0], device=dev, dtype=torch.float64), q[1:] - q[:-1]])
    chi, best = [], []
    for k in range(0, cross.shape[0], 1024):
        x = cross[k:k + 1024]
        s = x[:, 0, 0] + x[:, 3, 0] + x[:, 5, 0] + x[:, 2, 0] - x[:, 1, 0] - x[:, 4, 0]
        x = x * (d.peak / s)[:, None, None]
        VV, VD, VW, DD, DW, WW = (x[:, c, None, :] for c in range(6))
        al, be = VV - G * VD + G * G * DD, VW - G * DW
        scores = []
        for v in c2:
            y = al + v * be + v * v * WW
            tan = torch.cat([torch.zeros_like(y[..., :1]), y[..., 1:] - y[..., :-1]], -1) / h
            buf = y - tan * q
            up = (buf * a[:, 1] + tan * a[:, 2]).sum(-1)
            down = (buf * buf * a[:, 3] + 2.0 * tan * buf * a[:, 4] + tan * tan * a[:, 5]).sum(-1)
            scores.append(a[:, 0].sum() - up * up / down)
        sc = torch.stack(scores, -1).reshape(len(x), -1)
        m, i = sc.min(-1)
        chi.append(torch.sqrt(m))
        best.append(i)
    chi, best = torch.cat(chi).cpu().numpy(), torch.cat(best).cpu().numpy()
    return dict(chi=chi, c1=C1_GRID[best // len(C2_GRID)], c2=C2_GRID[best % len(C2_GRID)],
                cell=best.astype(np.int32))


def exact(case, seed):
    """What run returns, from the formulas in 64 bits.  The L-BFGS-B fit's
    stopping point has no value of its own: only its cross terms have one."""
    kind = case["kind"]
    if kind == "expand":
        x, vac, dum, sasa, _ = _molecule(case["atoms"], _rng(seed, case["atoms"], case["L"]))
        L = case["L"]
        return _flat(_coefficients(x, np.stack([vac, dum, FF_WATER * sasa]), _qvals(case["Q"]), L,
                                   bessel=lambda qr: [_bessel_series(l, qr) for l in range(L + 1)]))
    if kind in ("batch", "serve"):
        ds = _batch_dimers(case, seed) if kind == "batch" else _serve_dimers(case, seed)
        out = [_grid_fit(_cross_terms(d, d.index[0], 1), d) for d in ds]
        return out if kind == "batch" else [{k: o[k] for k in ("chi", "c1", "c2")} for o in out]
    if case["lbfgs"] and not case.get("cross"):
        return None
    # the sums over all q of the large lists take longer than they tell
    if case["poses"] * case["Q"] * (case["L"] + 1) ** 2 > 4e9:
        return None
    d = _dimer(case, seed)
    index = d.index[-1]
    cross = _cross_terms(d, index, case["skip"])
    r = dict(chi=None, c1=None, c2=None) if case["lbfgs"] else _grid_fit(cross, d)
    if kind == "plan":
        if case["topk"]:
            r["best"] = None
        return r
    r.pop("cell", None)                       # score_flat returns no cells
    if case["cross"]:
        r["cross"] = cross.cpu().numpy()
    if case["ingest"]:
        r["index"] = None
    return r
