"""Performance cases of the cluster and periodic-array solvers.

A case is one unit of work as a program with the treams_b200 package does it, through its public
entry points: `prepare` makes the inputs (host arrays, which is what the package takes) and what a
program keeps between calls, `run` makes one pass, `exact` states the same result in plain numpy
and torch with 64-bit numbers, independent of the package.

Geometry follows the package's workloads: spheres packed by random sequential addition at 15-20%
fill, radii 0.15..0.3, k0 0.5..3, permittivities 2..6 with a small loss, lmax 3..6.
"""
import functools
import math
import pathlib
import sys
from fractions import Fraction

import numpy as np
import torch

sys.path.insert(0, str(pathlib.Path(__file__).resolve().parent.parent / "treams-rs_b200"))

import treams_b200 as t  # noqa: E402
from treams_b200 import lattice as tl  # noqa: E402

LISTED = [
    # The smallest whole calculation: eight spheres, one plane wave, cross sections (latency).
    dict(name="dense_8_lmax3", kind="dense", count=8, lmax=3, waves=1, precision="fp64", k0=1.3, eps=4.0, loss=0.1),
    # The default precision at a middle size with an odd number of spheres.
    dict(name="dense_61_lmax5_fp64", kind="dense", count=61, lmax=5, waves=3, precision="fp64", k0=2.0, eps=2.25,
         loss=0.01),
    # The largest: the benchmark's precision cluster, three plane waves, mixed precision.
    dict(name="dense_512_lmax4_mixed", kind="dense", count=512, lmax=4, waves=3, precision="mixed", k0=2.0, eps=2.25,
         loss=0.01),
    # Mixed precision at the sweep's highest degree, a ragged size (131 * 96 = 12576 modes).
    dict(name="dense_131_lmax6_mixed", kind="dense", count=131, lmax=6, waves=2, precision="mixed", k0=1.7, eps=3.0,
         loss=0.05),
    # T-matrix of a whole particle cluster in one global basis: 96 right-hand sides at once.
    dict(name="global_tmatrix_40_lmax4", kind="tmatrix", count=40, lmax=4, lmax_global=6, precision="fp64", k0=1.2,
         eps=4.0, loss=0.02),
    # One factor kept, an angle sweep of 17 incidences solved forward and pulled back (gradients).
    dict(name="sweep_200_lmax4_17", kind="sweep", count=200, lmax=4, waves=17, precision="mixed", k0=2.0, eps=2.25,
         loss=0.01),
    # The matrix-free solver on the benchmark's largest cluster with its best preconditioner.
    dict(name="gmres_4096_lmax3_two_level", kind="gmres", count=4096, lmax=3, waves=1, pre="two_level", k0=1.5,
         eps=4.0, loss=0.05),
    # The matrix-free solver as the reference has it (no preconditioner), at the highest degree.
    dict(name="gmres_300_lmax6_none", kind="gmres", count=300, lmax=6, waves=1, pre="none", k0=1.5, eps=2.5,
         loss=0.02),
    # Lattice sums over a Brillouin-zone grid: 4096 Bloch vectors, every degree an lmax-6 array needs.
    dict(name="lattice_4096_l12", kind="lattice", nk=4096, lsum=12, period=0.74, k0=4.0, im=0.0, z=0.0),
    # Lattice sums between two sheets of a stack in a lossy embedding (complex k, shift off the plane).
    dict(name="lattice_1000_l8_lossy_shift", kind="lattice", nk=1000, lsum=8, period=0.74, k0=4.0, im=0.05, z=0.3),
    # Array T-matrices over a k-space grid (1021: no multiple of the number of SMs).
    dict(name="array_1021_lmax6", kind="array", nk=1021, lmax=6, period=0.74, k0=4.0, radius=0.2, eps=9.0, loss=0.0),
    # A parameter sweep: 24 different clusters in one call, precision chosen per cluster.
    dict(name="batch_24", kind="batch", count=24, most=96, k0=2.0, precision="auto"),
]


def listed():
    return [dict(c) for c in LISTED]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dense", "dense", "dense", "tmatrix", "sweep", "gmres", "gmres", "lattice", "lattice", "array",
                       "batch"])
    optics = dict(k0=round(rng.uniform(0.8, 2.2), 3), eps=round(rng.uniform(2.0, 4.0), 3),
                  loss=round(rng.uniform(0.005, 0.1), 4))
    lmax = rng.randint(3, 6)
    modes = 2 * lmax * (lmax + 2)
    if kind == "dense":
        precision = rng.choice(["fp64", "mixed"])
        top = 5000 if precision == "fp64" else 20000
        return dict(kind=kind, count=_log_int(rng, 8, top // modes), lmax=lmax, waves=rng.randint(1, 3),
                    precision=precision, **optics)
    if kind == "tmatrix":
        return dict(kind=kind, count=_log_int(rng, 4, 2500 // modes), lmax=lmax, lmax_global=rng.randint(4, 7),
                    precision=rng.choice(["fp64", "mixed"]), **optics)
    if kind == "sweep":
        return dict(kind=kind, count=_log_int(rng, 20, 10000 // modes), lmax=lmax, waves=rng.randint(2, 20),
                    precision=rng.choice(["fp64", "mixed"]), **optics)
    if kind == "gmres":
        pre = rng.choice(["none", "block_jacobi", "two_level"])
        top = {3: 3000, 4: 1200, 5: 500, 6: 300}[lmax]
        optics["eps"] = min(optics["eps"], 3.0)
        return dict(kind=kind, count=_log_int(rng, 30, top), lmax=lmax, waves=1, pre=pre, **optics)
    if kind == "lattice":
        lossy = rng.random() < 0.4
        return dict(kind=kind, nk=_log_int(rng, 64, 1500 if lossy else 4096), lsum=rng.randint(6, 10 if lossy else 12),
                    period=round(rng.uniform(0.5, 1.0), 3), k0=round(rng.uniform(3.0, 5.0), 3),
                    im=round(rng.uniform(0.05, 0.2), 3) if lossy else 0.0,
                    z=round(rng.uniform(0.1, 0.35), 3) if lossy else 0.0)
    if kind == "array":
        return dict(kind=kind, nk=_log_int(rng, 32, 1021), lmax=lmax, period=round(rng.uniform(0.5, 1.0), 3),
                    k0=round(rng.uniform(3.0, 5.0), 3), radius=0.2, eps=round(rng.uniform(2.0, 9.0), 2), loss=0.0)
    return dict(kind=kind, count=rng.randint(5, 20), most=_log_int(rng, 24, 96), k0=optics["k0"], precision="auto")


# ---- inputs ---------------------------------------------------------------------------------


def _pack(rng, radii, fill):
    """Random sequential addition of spheres in a cubic box."""
    side = (np.sum(4.0 / 3.0 * np.pi * radii**3) / fill) ** (1.0 / 3.0)
    pos = np.empty((len(radii), 3))
    for i, r in enumerate(radii):
        while True:
            c = rng.uniform(0.0, side, 3)
            gap2 = ((pos[:i] - c) ** 2).sum(axis=1) - (radii[:i] + r + 0.005) ** 2
            if i == 0 or gap2.min() > 0.0:
                break
        pos[i] = c
    return pos


def _directions(rng, count):
    v = rng.standard_normal((count, 3))
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def _cluster(case, rng):
    n = case["count"]
    large = case["kind"] == "gmres" and case["lmax"] == 3
    radii = np.full(n, 0.2) if large else rng.uniform(0.15, 0.3, n)
    pos = _pack(rng, radii, 0.2 if large else 0.15)
    return dict(lmax=case["lmax"], k0=case["k0"], radii=radii, eps=np.full(n, complex(case["eps"], case["loss"])),
                positions=pos)


def _inputs(case, seed):
    """Every input of a case, from the seed alone (shared by prepare and exact)."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("lattice", "array"):
        a = case["period"]
        # Bloch vectors over the first Brillouin zone; the lattice slightly off square
        d = rng.uniform(-0.03, 0.03, 2) * a
        lat = np.array([[a, d[0]], [d[1], a]])
        out = dict(lattice=lat, kpars=rng.uniform(-np.pi / a, np.pi / a, (case["nk"], 2)))
        if kind == "lattice":
            out["k"] = complex(case["k0"], case["k0"] * case["im"]) if case["im"] else case["k0"]
            out["shift"] = np.array([0.1 * a, 0.2 * a, case["z"] * a]) if case["z"] else None
        return out
    if kind == "batch":
        out = []
        sizes = np.random.default_rng([case["count"], case["most"]])  # sizes belong to the case, values to the seed
        for _ in range(case["count"]):
            n, lmax = int(sizes.integers(case["most"] // 6, case["most"] + 1)), int(sizes.integers(3, 7))
            radii = rng.uniform(0.1, 0.3, n)
            eps = rng.uniform(2, 4, n) + 1j * rng.uniform(0.01, 0.2, n)
            k0 = case["k0"] * rng.uniform(0.6, 1.2)
            pos = _pack(rng, radii, 0.15)
            b = plane_waves(lmax, pos, k0 * np.array([[0.0, 0.0, 1.0]]), [1])
            out.append(dict(lmax=lmax, k0=k0, radii=radii, eps=eps, positions=pos, B=b))
        return out
    c = _cluster(case, rng)
    if kind in ("dense", "sweep", "gmres"):
        c["kvecs"] = case["k0"] * _directions(rng, case["waves"])
        c["pols"] = rng.integers(0, 2, case["waves"])
    if kind in ("sweep", "gmres"):
        c["B"] = plane_waves(c["lmax"], c["positions"], c["kvecs"], c["pols"])
    if kind == "sweep":
        c["G"] = np.asfortranarray(rng.standard_normal(c["B"].shape) + 1j * rng.standard_normal(c["B"].shape))
    return c


def _geometry(c):
    return c["lmax"], c["k0"], c["radii"], c["eps"], c["positions"]


def prepare(case, seed):
    state = dict(case=case, inputs=_inputs(case, seed))
    if case["kind"] == "sweep":  # the factor is what a program keeps between incidences
        state["factor"] = t.sphere_cluster_factor(*_geometry(state["inputs"]), case["precision"])
    return state


def run(state):
    case, c = state["case"], state["inputs"]
    kind = case["kind"]
    if kind == "dense":
        b = t.plane_wave_expansion(c["lmax"], c["positions"], c["kvecs"], c["pols"])
        f = t.sphere_cluster_factor(*_geometry(c), case["precision"])
        x, _ = f.solve(b)
        f.close()
        sca, ext = t.cross_sections(c["lmax"], c["k0"], c["positions"], x, b)
        return dict(x=x, sca=sca, ext=ext)
    if kind == "tmatrix":
        f = t.sphere_cluster_factor(*_geometry(c), case["precision"])
        out = f.global_tmatrix(case["lmax_global"], c["positions"].mean(axis=0))
        f.close()
        return out
    if kind == "sweep":
        x, _ = state["factor"].solve(c["B"])
        g, _ = state["factor"].pullback_incident(c["G"])
        return dict(x=x, g=g)
    if kind == "gmres":
        return t.SphereCluster(*_geometry(c)).solve(c["B"], preconditioner=case["pre"]).value
    if kind == "lattice":
        return tl.lsumsw2d_batch(case["lsum"], c["k"], c["lattice"], c["kpars"], shift=c["shift"])
    if kind == "array":
        return tl.array_solve_batch(case["lmax"], case["k0"], case["radius"], complex(case["eps"], case["loss"]),
                                    c["lattice"], c["kpars"])
    clusters = [(d["lmax"], d["k0"], d["radii"], d["eps"], d["positions"], d["B"]) for d in c]
    return t.batch_solve(clusters, case["precision"])[0]


def work(case):
    """Bytes in and out and the floating-point operations of the algorithm (complex multiply-add: 8)."""
    kind = case["kind"]
    if kind == "lattice":
        terms = (case["lsum"] + 1) ** 2
        points = 150  # lattice points within the cutoff of either part at the automatic split
        return dict(bytes=case["nk"] * 16 * (1 + terms), flops=case["nk"] * terms * points * 2 * 8)
    if kind == "array":
        m = 2 * case["lmax"] * (case["lmax"] + 2)
        return dict(bytes=case["nk"] * 16 * (1 + m * m),
                    flops=case["nk"] * (8 * m**3 + (2 * case["lmax"] + 1) ** 2 * 150 * 16))
    if kind == "batch":
        n = case["count"] * 0.58 * case["most"] * 58  # mean spheres and modes per sphere
        return dict(bytes=32 * n, flops=case["count"] * 8 / 3 * (n / case["count"]) ** 3 * 2)
    lmax, count = case["lmax"], case["count"]
    n = count * 2 * lmax * (lmax + 2)
    table = (2 * lmax + 1) ** 2
    if kind == "gmres":
        applications = 6 if case["pre"] == "two_level" else 25
        return dict(bytes=count * 48 + 32 * n, flops=applications * 8.0 * count * n * table)
    if kind == "sweep":
        return dict(bytes=8.0 * n * n + 64 * n * case["waves"], flops=16.0 * n * n * case["waves"])
    columns = case["waves"] if kind == "dense" else 2 * case["lmax_global"] * (case["lmax_global"] + 2)
    out = 16 * (n * columns if kind == "dense" else columns**2)
    return dict(bytes=count * 48 + out, flops=8 / 3 * n**3 + 8.0 * n * n * columns)


# ---- the same results in plain numpy and torch, 64 bits ----------------------------------------


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _lm(lmax):
    return [(l, m) for l in range(1, lmax + 1) for m in range(-l, l + 1)]


@functools.lru_cache(maxsize=None)
def _wigner3j(j1, j2, j3, m1, m2, m3):
    """Racah's formula in rational numbers."""
    if m1 + m2 + m3 or not abs(j1 - j2) <= j3 <= j1 + j2 or abs(m1) > j1 or abs(m2) > j2 or abs(m3) > j3:
        return 0.0
    f = math.factorial
    total = Fraction(0)
    for k in range(max(0, j2 - j3 - m1, j1 - j3 + m2), min(j1 + j2 - j3, j1 - m1, j2 + m2) + 1):
        den = (f(k) * f(j1 + j2 - j3 - k) * f(j1 - m1 - k) * f(j2 + m2 - k) * f(j3 - j2 + m1 + k)
               * f(j3 - j1 - m2 + k))
        total += Fraction((-1) ** k, den)
    tri = Fraction(f(j1 + j2 - j3) * f(j1 - j2 + j3) * f(-j1 + j2 + j3), f(j1 + j2 + j3 + 1))
    rest = f(j1 + m1) * f(j1 - m1) * f(j2 + m2) * f(j2 - m2) * f(j3 + m3) * f(j3 - m3)
    return (-1) ** (j1 - j2 - m3) * math.copysign(math.sqrt(total * total * tri * rest), total)


@functools.lru_cache(maxsize=None)
def _translation_weights(ldst, lsrc):
    """(2, destinations, sources, harmonics): A and B of the vector translation coefficients as sums over
    the products of radial function and solid harmonic of degree p, order m - mu (index p p + p + m - mu)."""
    order = ldst + lsrc
    w = np.zeros((2, len(_lm(ldst)), len(_lm(lsrc)), (order + 1) ** 2), complex)
    for s, (l, m) in enumerate(_lm(lsrc)):
        for d, (lam, mu) in enumerate(_lm(ldst)):
            pref = 0.5 * (-1) ** m * math.sqrt((2 * l + 1) * (2 * lam + 1) / (l * (l + 1) * lam * (lam + 1)))
            for p in range(max(abs(l - lam), abs(m - mu)), l + lam + 1):
                cross = (l + lam - p) % 2
                if cross:
                    factor = math.sqrt((l + lam + 1 + p) * (l + lam + 1 - p) * (p + lam - l) * (p - lam + l))
                else:
                    factor = l * (l + 1) + lam * (lam + 1) - p * (p + 1)
                ratio = math.sqrt(math.factorial(p - m + mu) / math.factorial(p + m - mu))
                w[cross, d, s, p * p + p + m - mu] += (
                    pref * factor * (2 * p + 1) * 1j ** ((lam - l + p) % 4) * ratio
                    * _wigner3j(l, lam, p, m, -mu, mu - m) * _wigner3j(l, lam, p - cross, 0, 0, 0))
    return w


def _solid(order, u):
    """r^p P_p^m(z/r) e^(i m phi) for every p <= order at the vectors u (..., 3), index p p + p + m."""
    x, y, z = u[..., 0], u[..., 1], u[..., 2]
    r2, xy = (u * u).sum(-1), torch.complex(x, y)
    out = torch.zeros(u.shape[:-1] + ((order + 1) ** 2,), dtype=torch.complex128, device=u.device)
    diagonal = torch.ones_like(xy)
    for m in range(order + 1):
        if m:
            diagonal = -(2 * m - 1) * xy * diagonal
        p, prev = diagonal, torch.zeros_like(diagonal)
        for deg in range(m, order + 1):
            if deg > m:
                p, prev = ((2 * deg - 1) * z * p - (deg + m - 1) * r2 * prev) / (deg - m), p
            out[..., deg * deg + deg + m] = p
            if m:
                ratio = math.factorial(deg - m) / math.factorial(deg + m)
                out[..., deg * deg + deg - m] = (-1) ** m * ratio * p.conj()
    return out


def _hankel(last, z):
    """Outgoing spherical Hankel functions h_0 .. h_last by the upward recurrence."""
    z = z.to(torch.complex128)
    e = torch.exp(1j * z) / z
    prev, cur, out = e, -1j * e, []
    for p in range(last + 1):
        out.append(cur)
        prev, cur = cur, (2 * p + 1) / z * cur - prev
    return torch.stack(out, -1)


def _bessel(last, z):
    """Spherical Bessel functions j_0 .. j_last by the downward recurrence, normalised by
    sum (2p + 1) j_p^2 = 1 for real z and by the larger of j_0 and j_1 else."""
    z = z.to(torch.complex128)
    small = z.abs() < 1e-8
    zz = torch.where(small, torch.ones_like(z), z)
    start = last + 30 + int(2 * float(zz.abs().max()))
    nxt, cur = torch.zeros_like(zz), torch.full_like(zz, 1e-300)
    f = [None] * (start + 1)
    for p in range(start, -1, -1):
        f[p] = cur
        nxt, cur = cur, (2 * p + 1) / zz * cur - nxt
        big = cur.abs() > 1e100
        if bool(big.any()):
            scale = torch.where(big, torch.full_like(zz, 1e-100), torch.ones_like(zz))
            nxt, cur = nxt * scale, cur * scale
            for q in range(p, start + 1):
                f[q] = f[q] * scale
    j0, j1 = torch.sin(zz) / zz, torch.sin(zz) / zz**2 - torch.cos(zz) / zz
    scale = torch.where(j0.abs() >= j1.abs(), j0 / f[0], j1 / f[1])
    out = torch.stack([f[p] * scale for p in range(last + 1)], -1)
    zero = torch.zeros_like(out)
    zero[..., 0] = 1.0
    return torch.where(small[..., None], zero, out)


def _table(order, k, d, singular=True):
    """Radial function times solid harmonic at the displacements d (..., 3)."""
    r = d.norm(dim=-1)
    u = d / torch.where(r == 0, torch.ones_like(r), r)[..., None]
    radial = (_hankel if singular else _bessel)(order, k * r)
    degree = torch.tensor([p for p in range(order + 1) for _ in range(2 * p + 1)], device=d.device)
    return radial[..., degree] * _solid(order, u)


def _mie(lmax, k0, radii, eps):
    """(N, lmax, 2, 2) T blocks of spheres in helicity modes from the Mie coefficients a, b."""
    x = torch.tensor(k0 * np.asarray(radii), dtype=torch.complex128)
    m = torch.sqrt(torch.tensor(np.asarray(eps, complex)))
    l = torch.arange(1, lmax + 1)
    jx, jm, hx = _bessel(lmax, x), _bessel(lmax, m * x), _hankel(lmax, x)

    def riccati(f, z):  # z f_l and its derivative
        z = z[:, None]
        return z * f[:, 1:], z * f[:, :-1] - l * f[:, 1:]

    (px, dpx), (pm, dpm), (xx, dxx) = riccati(jx, x), riccati(jm, m * x), riccati(hx, x)
    m = m[:, None]
    a = (m * pm * dpx - px * dpm) / (m * pm * dxx - xx * dpm)
    b = (pm * dpx - m * px * dpm) / (pm * dxx - m * xx * dpm)
    same, cross = -0.5 * (a + b), -0.5 * (a - b)
    return torch.stack([torch.stack([same, cross], -1), torch.stack([cross, same], -1)], -2)


def plane_waves(lmax, positions, kvecs, pols):
    """Regular expansion coefficients of helicity plane waves (real wavevectors) at the positions, (n, p)."""
    out = np.zeros((len(positions), len(_lm(lmax)), 2, len(pols)), complex)
    for c, (kv, pol) in enumerate(zip(np.asarray(kvecs, float), pols)):
        k, kt = np.linalg.norm(kv), np.hypot(kv[0], kv[1])
        cos, sin = kv[2] / k, kt / k
        e = (kv[0] - 1j * kv[1]) / kt if kt else 1.0
        # P_l^m / sin^m for m >= 0, every l <= lmax (+1 degree of freedom below the diagonal)
        leg = {}
        for m in range(lmax + 2):
            p, prev = float((-1) ** m * math.prod(range(2 * m - 1, 0, -2))), 0.0
            for deg in range(m, lmax + 1):
                if deg > m:
                    p, prev = ((2 * deg - 1) * cos * p - (deg + m - 1) * prev) / (deg - m), p
                leg[deg, m] = p
        phase = np.exp(1j * positions @ kv)
        for q, (l, m) in enumerate(_lm(lmax)):
            pref = 2.0 * math.sqrt(math.pi * (2 * l + 1) / (l * (l + 1))) * 1j ** l
            am = abs(m)
            norm = math.sqrt(math.factorial(l - am) / math.factorial(l + am))
            sign = (-1) ** am if m < 0 else 1
            if m == 0:
                tau, pi = sin * leg[l, 1], 0.0
            else:
                power = sin ** (am - 1)
                pi = am * power * leg[l, am]
                tau = power * (l * cos * leg[l, am] - (l + am) * leg.get((l - 1, am), 0.0))
            angular = tau + (2 * pol - 1) * (pi if m >= 0 else -pi)
            out[:, q, 1 - pol, c] = pref * sign * norm * e**m * angular * phase
    return np.asfortranarray(out.reshape(-1, len(pols)))


class _Coupling:
    """The coupling C between all spheres (i != j), applied from the stored pair tables."""

    def __init__(self, lmax, k0, positions, singular=True):
        dev = _dev()
        pos = torch.as_tensor(positions, device=dev)
        self.n, self.q = len(pos), len(_lm(lmax))
        self.order = 2 * lmax
        w = torch.as_tensor(_translation_weights(lmax, lmax), device=dev)
        self.w = torch.stack([w[0] + w[1], w[0] - w[1]])  # (helicity, destinations, sources, harmonics)
        self.z = torch.empty((self.n, (self.order + 1) ** 2, self.n), dtype=torch.complex128, device=dev)
        step = max(1, 400_000 // self.n)
        eye = torch.eye(self.n, dtype=torch.bool, device=dev)
        for i in range(0, self.n, step):
            d = pos[i:i + step, None] - pos[None]
            own = eye[i:i + step]
            d = torch.where(own[..., None], torch.ones_like(d), d)
            z = _table(self.order, k0, d, singular)
            self.z[i:i + step] = torch.where(own[..., None], torch.zeros_like(z), z).transpose(1, 2)

    def apply(self, x):
        """C x for one column, x (n modes)."""
        xs = x.reshape(self.n, 2 * self.q)
        g = torch.empty((self.n, self.z.shape[1], 2 * self.q), dtype=x.dtype, device=x.device)
        for i in range(0, self.n, 256):
            g[i:i + 256] = torch.matmul(self.z[i:i + 256], xs)
        g = g.reshape(self.n, -1, self.q, 2)
        return torch.einsum("bdst,itsb->idb", self.w, g).reshape(-1)

    def dense(self):
        """C as (N, modes, N, modes) blocks, helicity pairs interleaved."""
        out = torch.zeros((self.n, self.q, 2, self.n, self.q, 2), dtype=self.z.dtype, device=self.z.device)
        for i in range(self.n):
            for b in range(2):
                blk = torch.einsum("dst,tj->djs", self.w[b], self.z[i])
                out[i, :, b, :, :, b] = blk
        return out


def _apply_t(lmax, blocks, x):
    """Block-diagonal T on x (n, p)."""
    q = len(_lm(lmax))
    degree = torch.tensor([l - 1 for l, _ in _lm(lmax)], device=x.device)
    full = blocks.to(x.device)[:, degree]  # (N, q, 2, 2)
    return torch.einsum("iqab,iqbp->iqap", full, x.reshape(-1, q, 2, x.shape[1])).reshape(x.shape)


def _system(c):
    """A = I - T C and the T blocks."""
    lmax, k0, radii, eps, pos = _geometry(c)
    blocks = _mie(lmax, k0, radii, eps)
    cpl = _Coupling(lmax, k0, pos)
    n = cpl.n * 2 * cpl.q
    a = cpl.dense().reshape(n, n)
    del cpl
    for j in range(0, n, 4096):
        a[:, j:j + 4096] = -_apply_t(lmax, blocks, a[:, j:j + 4096])
    a.diagonal().add_(1.0)
    return a, blocks


def _solve_cluster(c, b):
    a, blocks = _system(c)
    return torch.linalg.solve(a, _apply_t(c["lmax"], blocks, torch.as_tensor(b, device=a.device)))


def _gmres(apply, b, rtol=1e-14, restart=60, most=600):
    """Restarted GMRES with twice orthogonalised Arnoldi vectors."""
    x = torch.zeros_like(b)
    for _ in range(most // restart):
        r = b - apply(x)
        beta = r.norm()
        if beta <= rtol * b.norm():
            break
        v = torch.zeros((restart + 1, b.numel()), dtype=b.dtype, device=b.device)
        h = torch.zeros((restart + 1, restart), dtype=b.dtype, device=b.device)
        v[0] = r / beta
        used = restart
        for j in range(restart):
            w = apply(v[j])
            for _ in range(2):
                p = v[: j + 1].conj() @ w
                w = w - v[: j + 1].T @ p
                h[: j + 1, j] += p
            h[j + 1, j] = w.norm()
            v[j + 1] = w / h[j + 1, j]
            e = torch.zeros(j + 2, dtype=b.dtype, device=b.device)
            e[0] = beta
            y = torch.linalg.lstsq(h[: j + 2, : j + 1], e[:, None]).solution[:, 0]
            if (h[: j + 2, : j + 1] @ y - e).norm() <= 0.3 * rtol * b.norm():
                used = j + 1
                break
        x = x + v[:used].T @ y
    return x


_GL = np.polynomial.legendre.leggauss(240)


def _lattice_points(lat, radius):
    inv = np.linalg.inv(lat)
    span = [int(np.ceil(radius * np.linalg.norm(inv[:, i]))) + 1 for i in range(2)]
    g = np.stack(np.meshgrid(*(np.arange(-s, s + 1) for s in span), indexing="ij"), -1).reshape(-1, 2)
    p = g @ lat
    return p[np.linalg.norm(p, axis=1) <= radius]


def _harmonic_norm(lsum):
    return np.array([math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - m) / math.factorial(l + m))
                     for l in range(lsum + 1) for m in range(-l, l + 1)])


def _direct_sums(lsum, k, lat, kpars, shift):
    """D_lm = sum_R h_l(k |r + R|) Y_lm(-r - R) e^(i kpar.R), summed term by term (complex k)."""
    dev = _dev()
    points = _lattice_points(lat, 38.0 / k.imag)
    out = torch.zeros((len(kpars), (lsum + 1) ** 2), dtype=torch.complex128, device=dev)
    kp = torch.as_tensor(kpars, device=dev)
    norm = torch.as_tensor(_harmonic_norm(lsum), device=dev)
    for i in range(0, len(points), 50_000):
        p = torch.as_tensor(points[i:i + 50_000], device=dev)
        d = -torch.cat([p, torch.zeros_like(p[:, :1])], 1) - torch.as_tensor(shift, device=dev)
        table = _table(lsum, k, d) * norm
        out += torch.exp(1j * (kp @ p.T)) @ table
    return out


def _ewald_sums(lsum, k, lat, kpars):
    """The same at r = 0 and real k by Ewald's split, every integral by Gauss-Legendre quadrature."""
    dev = _dev()
    area = abs(np.linalg.det(lat))
    kl = k * math.sqrt(area)
    eta = math.sqrt(2 * math.pi) / kl * max(kl / 8.0, 1.0)
    c = 0.5 / eta**2
    ls = torch.arange(lsum + 1, dtype=torch.float64, device=dev)
    degree = torch.tensor([l for l in range(lsum + 1) for _ in range(2 * l + 1)], device=dev)
    nodes, weights = (torch.as_tensor(v, device=dev) for v in _GL)
    # real space: I_2l(z) = int_eta^inf t^2l exp(-z^2 t^2 / 2 + 1 / (2 t^2)) dt, t = eta e^s
    pts = _lattice_points(lat, math.sqrt(2 * (80.0 + c)) / (k * eta))
    pts = torch.as_tensor(pts[np.linalg.norm(pts, axis=1) > 0], device=dev)
    z = k * pts.norm(dim=1)
    top = 0.5 * torch.log(1.0 + 140.0 / (0.5 * (z * eta) ** 2))
    s = 0.5 * top[:, None] * (nodes + 1.0)
    base = -0.5 * (z[:, None] * eta) ** 2 * torch.exp(2 * s) + c * torch.exp(-2 * s)
    integral = torch.stack([(torch.exp((2 * l + 1) * s + base) * weights).sum(1) for l in range(lsum + 1)], 1)
    integral = integral * 0.5 * top[:, None] * eta ** (2 * ls + 1)
    d = -torch.cat([pts, torch.zeros_like(pts[:, :1])], 1)
    norm = torch.as_tensor(_harmonic_norm(lsum), device=dev)
    harmonic = _solid(lsum, d / d.norm(dim=1, keepdim=True)) * norm
    radial = -1j * math.sqrt(2 / math.pi) * z[:, None] ** ls * integral
    kp = torch.as_tensor(kpars, device=dev)
    out = torch.exp(1j * (kp @ pts.T)) @ (radial[:, degree] * harmonic)
    # reciprocal space: F_n(v) = Gamma(1/2 - n, v) / (-v)^(1/2 - n) on the lower side of the cut
    rec = 2 * math.pi * np.linalg.inv(lat).T
    kmax = np.linalg.norm(kpars, axis=1).max()
    g = torch.as_tensor(_lattice_points(rec, k * math.sqrt(1 + 2 * eta**2 * 80.0) + kmax), device=dev)
    terms = {}  # (l, m): [(n, beta power, coefficient)]
    for l in range(lsum + 1):
        for m in range(-l, l + 1):
            am = abs(m)
            if (l - am) % 2:
                continue
            front = math.sqrt((2 * l + 1) * math.factorial(l + m) * math.factorial(l - m)) / (area * k * k * (-2.0) ** l)
            terms[l, m] = [((l - am) // 2 - p, p, front * (-1j) ** (m % 4)
                            / (math.factorial(n) * math.factorial(p + am) * math.factorial(p)))
                           for p in range((l - am) // 2 + 1) for n in [(l - am) // 2 - p]]
    for i in range(0, len(kpars), 512):
        q = kp[i:i + 512, None] + g[None]
        b2 = (q * q).sum(-1) / k**2
        v = (b2 - 1.0) / (2 * eta**2)
        a = v.abs()
        flat = a.reshape(-1)
        evan = torch.empty((lsum // 2 + 1, flat.numel()), dtype=torch.float64, device=dev)
        for j in range(0, flat.numel(), 100_000):  # int_1^inf t^(-1/2 - n) e^(-a t) dt, t = e^s
            aj = flat[j:j + 100_000, None]
            top = torch.log(1.0 + 60.0 / aj)
            s = 0.5 * top * (nodes + 1.0)
            base = -aj * torch.exp(s)
            for n in range(lsum // 2 + 1):
                evan[n, j:j + 100_000] = (torch.exp((0.5 - n) * s + base) * weights).sum(1) * 0.5 * top[:, 0]
        f = []
        for n in range(lsum // 2 + 1):
            b = 0.5 - n
            series, term = torch.full_like(a, 1.0 / b), torch.ones_like(a)
            for kk in range(1, 60):
                term = term * torch.where(v < 0, a, torch.zeros_like(a)) / kk
                series = series + term / (b + kk)
            prop = torch.complex(math.gamma(b) * a ** -b, (-1) ** n * series)
            ev = torch.complex(torch.zeros_like(a), -((-1) ** n) * evan[n].reshape(a.shape))
            f.append(torch.where(v < 0, prop, ev) * (2 * eta**2) ** n / (math.sqrt(2) * eta))
        for (l, m), parts in terms.items():
            az = torch.complex(q[..., 0], q[..., 1] if m >= 0 else -q[..., 1]) / k
            poly = sum(w * f[n] * b2**p for n, p, w in parts)
            out[i:i + 512, l * l + l + m] += (az ** abs(m) * poly).sum(1)
    # self term: sqrt(1 / 4 pi) / (2 sqrt pi) Gamma(-1/2, -c) / (-c)^(-1/2) of the split
    total, term = 0.0, 1.0
    for kk in range(200):
        term = term * c / kk if kk else 1.0
        total += term / (kk - 0.5)
    out[:, 0] += _harmonic_norm(0)[0] * 0.5 / math.sqrt(math.pi) * complex(-2 * math.sqrt(math.pi), -total / math.sqrt(c))
    return out


def exact(case, seed):
    kind, c = case["kind"], _inputs(case, seed)
    if kind == "dense":
        b = plane_waves(c["lmax"], c["positions"], c["kvecs"], c["pols"])
        x = _solve_cluster(c, b)
        bt = torch.as_tensor(b, device=x.device)
        cpl = _Coupling(c["lmax"], c["k0"], c["positions"], singular=False)
        sca = [torch.vdot(x[:, p], x[:, p] + cpl.apply(x[:, p])).real.item() / c["k0"] ** 2 for p in range(b.shape[1])]
        ext = [-torch.vdot(bt[:, p], x[:, p]).real.item() / c["k0"] ** 2 for p in range(b.shape[1])]
        return dict(x=x.cpu().numpy(), sca=np.array(sca), ext=np.array(ext))
    if kind == "tmatrix":
        a, blocks = _system(c)
        lg, lmax = case["lmax_global"], c["lmax"]
        d = torch.as_tensor(c["positions"] - c["positions"].mean(axis=0), device=a.device)

        def expansion(ldst, lsrc, disp):  # regular translation blocks (N, modes, modes)
            z = _table(ldst + lsrc, c["k0"], disp, singular=False)
            w = torch.as_tensor(_translation_weights(ldst, lsrc), device=a.device)
            out = torch.zeros((len(disp), w.shape[1], 2, w.shape[2], 2), dtype=z.dtype, device=z.device)
            for b, sign in ((0, 1.0), (1, -1.0)):
                out[:, :, b, :, b] = torch.einsum("dst,it->ids", w[0] + sign * w[1], z)
            return out.reshape(len(disp), 2 * w.shape[1], 2 * w.shape[2])

        ein = expansion(lmax, lg, d).reshape(a.shape[0], -1)
        eout = expansion(lg, lmax, -d)
        x = torch.linalg.solve(a, _apply_t(lmax, blocks, ein)).reshape(len(d), -1, ein.shape[1])
        return torch.einsum("iab,ibc->ac", eout, x).cpu().numpy()
    if kind == "sweep":
        a, blocks = _system(c)
        x = torch.linalg.solve(a, _apply_t(c["lmax"], blocks, torch.as_tensor(c["B"], device=a.device)))
        y = torch.linalg.solve(a.mH, torch.as_tensor(c["G"], device=a.device))
        g = _apply_t(c["lmax"], blocks.mH, y)
        return dict(x=x.cpu().numpy(), g=g.cpu().numpy())
    if kind == "gmres":
        blocks = _mie(c["lmax"], c["k0"], c["radii"], c["eps"])
        cpl = _Coupling(c["lmax"], c["k0"], c["positions"])
        b = torch.as_tensor(c["B"], device=cpl.z.device)

        def a(v):
            return v - _apply_t(c["lmax"], blocks, cpl.apply(v)[:, None])[:, 0]

        cols = [_gmres(a, _apply_t(c["lmax"], blocks, b[:, p:p + 1])[:, 0]) for p in range(b.shape[1])]
        return torch.stack(cols, 1).cpu().numpy()
    if kind == "lattice":
        if case["im"]:
            return _direct_sums(case["lsum"], c["k"], c["lattice"], c["kpars"], c["shift"]).cpu().numpy()
        return _ewald_sums(case["lsum"], c["k"], c["lattice"], c["kpars"]).cpu().numpy()
    if kind == "array":
        lmax = case["lmax"]
        z = _ewald_sums(2 * lmax, case["k0"], c["lattice"], c["kpars"])
        z = z / torch.as_tensor(_harmonic_norm(2 * lmax), device=z.device)
        w = torch.as_tensor(_translation_weights(lmax, lmax), device=z.device)
        q, m = w.shape[1], 2 * w.shape[1]
        s = torch.zeros((len(z), q, 2, q, 2), dtype=z.dtype, device=z.device)
        for b, sign in ((0, 1.0), (1, -1.0)):
            s[:, :, b, :, b] = (z @ (w[0] + sign * w[1]).reshape(q * q, -1).T).reshape(-1, q, q)
        blocks = _mie(lmax, case["k0"], [case["radius"]], [complex(case["eps"], case["loss"])])
        tm = _apply_t(lmax, blocks, torch.eye(m, dtype=z.dtype, device=z.device))
        a = torch.eye(m, dtype=z.dtype, device=z.device) - tm @ s.reshape(-1, m, m)
        return torch.linalg.solve(a, tm.expand(len(z), m, m)).cpu().numpy()
    return [_solve_cluster(d, d["B"]).cpu().numpy() for d in c]
