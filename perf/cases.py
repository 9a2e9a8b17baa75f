"""The work a user has this framework do, as cases that can be timed.

A case is a dict of plain values; its "path" names the entry point:

  translations  trans_calculator.get_AB_arrays_device: VSWF translation arrays
  scatter       ScatteringSystem.planewave_scatter_batch: assembly, LU, solve,
                cross sections of a finite cluster at several frequencies
  scan          ScatteringSystem.dispersion_scan: a 2D lattice over (omega, k)
  field         ScatteringSystem.scattered_E_device: a field map
  modes         beyn.scatsys_quadrature: the contour sums of the eigensolver
  serving       serving.Server: a mix of independent solves, all at once

Particles, media and frequencies are those of the benchmark's configurations:
spheres of eps -12 + 1.2i in eps 2.25, 1.6-2.6 eV, 400 nm pitch, 580 nm
lattices.  ``exact`` computes the same quantities in plain 64-bit torch from
the defining formulas (Bessel recurrences, 3j symbols by Racah's sum, the
lattice sums by Ewald's method with quadrature, dense LU).
"""
import math
from fractions import Fraction
from functools import lru_cache

import numpy as np
import torch

EV = 1.602176634e-19
HBAR = 1.054571817e-34
C0 = 299792458.0
EPS_IN, EPS_OUT = -12 + 1.2j, 2.25
R_FINITE, R_LATTICE, R_FIELD = 50e-9, 80e-9, 60e-9
PITCH, LATTICE = 400e-9, 580e-9
E_LO, E_HI = 1.6, 2.6
LAYER_Z = 150e-9          # height of a bilayer's second plane
CONTOUR = (2.10, 0.05, 0.02)  # ellipse in eV: centre, half axes


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # one call of the translation kernel at the size of a coupling study; the largest multipole order in use
        {"name": "translations_many", "path": "translations", "n": 150001, "lMax": 6, "J": 3, "lossy": True},
        # a single small cluster at one frequency: the smallest solve, all latency
        {"name": "scatter_few", "path": "scatter", "spheres": 5, "lMax": 2, "nw": 1, "mode": 1, "scat": False},
        # a spectrum of a 4 x 4 array (the benchmark's mode-problem configuration)
        {"name": "scatter_spectrum", "path": "scatter", "spheres": 16, "lMax": 2, "nw": 32, "mode": 1, "scat": False},
        # a spectrum in plain complex128 with the scattering cross section too
        {"name": "scatter_fp64", "path": "scatter", "spheres": 13, "lMax": 3, "nw": 9, "mode": 0, "scat": True},
        # clusters between the batched and the large solver: the middle of the serving mix
        {"name": "scatter_mid", "path": "scatter", "spheres": 101, "lMax": 3, "nw": 3, "mode": 1, "scat": False},
        # the 30 x 30 array of the eigenmode benchmark, one frequency
        {"name": "scatter_large", "path": "scatter", "spheres": 900, "lMax": 2, "nw": 1, "mode": 1, "scat": False},
        # band structures of the benchmark's two lattices, and of a bilayer
        {"name": "scan_square", "path": "scan", "lattice": "square", "lMax": 3, "nw": 16, "nk": 256, "mode": 1},
        {"name": "scan_honeycomb", "path": "scan", "lattice": "honeycomb", "lMax": 3, "nw": 5, "nk": 201, "mode": 1},
        {"name": "scan_bilayer", "path": "scan", "lattice": "bilayer", "lMax": 2, "nw": 3, "nk": 33, "mode": 1},
        # a field map above a solved array
        {"name": "field_map", "path": "field", "spheres": 400, "lMax": 3, "points": 40001},
        # eigenmodes of an array: several contour nodes with many right-hand sides each
        {"name": "modes", "path": "modes", "spheres": 361, "lMax": 2, "nodes": 6, "columns": 64},
        # a burst of requests to the server: finite clusters and lattice points mixed
        {"name": "serving", "path": "serving", "requests": 24, "max_spheres": 250, "mix": 7, "workers": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["translations", "scatter", "scatter", "scatter", "scan", "scan", "field", "modes", "serving"])
    if path == "translations":
        lMax = rng.randint(1, 6)
        ne = lMax * (lMax + 2)
        return {"path": path, "n": _log_int(rng, 64, min(1_000_000, 150001 * 2304 // ne ** 2)), "lMax": lMax,
                "J": rng.choice([1, 3]), "lossy": rng.random() < 0.5}
    if path == "scatter":
        lMax = rng.randint(1, 4)
        n = 2 * lMax * (lMax + 2)
        spheres = _log_int(rng, 2, 14400 // n)
        N = spheres * n
        nw = rng.randint(1, 32) if N <= 512 else rng.randint(1, max(1, min(4, 14400 // N)))
        return {"path": path, "spheres": spheres, "lMax": lMax, "nw": nw, "mode": 0 if N <= 512 and rng.random() < 0.3 else 1,
                "scat": rng.random() < 0.3}
    if path == "scan":
        lattice = rng.choice(["square", "honeycomb", "bilayer"])
        lMax = rng.randint(1, 3 if lattice != "bilayer" else 2)
        most = {"square": 4096, "honeycomb": 1005, "bilayer": 99}[lattice]
        nw = rng.randint(1, 8)
        return {"path": path, "lattice": lattice, "lMax": lMax, "nw": nw,
                "nk": _log_int(rng, 1, min(256, most // nw)), "mode": rng.choice([0, 1])}
    if path == "field":
        spheres = _log_int(rng, 1, 400)
        return {"path": path, "spheres": spheres, "lMax": rng.randint(1, 3), "points": _log_int(rng, 100, 40001)}
    if path == "modes":
        lMax = rng.randint(1, 3)
        n = 2 * lMax * (lMax + 2)
        return {"path": path, "spheres": _log_int(rng, 8, 5776 // n), "lMax": lMax, "nodes": rng.randint(2, 6),
                "columns": _log_int(rng, 8, 64)}
    return {"path": path, "requests": rng.randint(4, 24), "max_spheres": rng.randint(30, 250),
            "mix": rng.randint(0, 10 ** 6), "workers": rng.choice([4, 8])}


# ---------------------------------------------------------------- inputs, from the seed alone

def _omegas(rng, n):
    return np.sort(rng.uniform(E_LO, E_HI, n)) * EV / HBAR


def _cluster(n, rng):
    """n positions on a square grid of 400 nm pitch, each displaced by up to a tenth of it."""
    side = math.ceil(math.sqrt(n))
    i = np.arange(n)
    xy = np.stack([i % side, i // side], 1) * PITCH + rng.uniform(-0.1, 0.1, (n, 2)) * PITCH
    return np.concatenate([xy - xy.mean(0), np.zeros((n, 1))], 1)


def _lattice(kind):
    """Basis vectors, positions in the cell, corners of the Bloch-vector path."""
    a = LATTICE
    if kind == "honeycomb":
        d = a / math.sqrt(3) / 2
        return ((a, 0.0), (a / 2, a * math.sqrt(3) / 2), np.array([[-d, 0, 0], [d, 0, 0]]),
                [(0, 0), (4 * math.pi / (3 * a), 0), (math.pi / a, math.pi / (math.sqrt(3) * a)), (0, 0)])
    pos = [[0, 0, 0]] if kind == "square" else [[0, 0, 0], [a / 2, a / 2, LAYER_Z]]
    return (a, 0.0), (0.0, a), np.array(pos, dtype=float), [(0, 0), (math.pi / a, 0), (math.pi / a, math.pi / a), (0, 0)]


def _bloch(kind, n, rng):
    """n Bloch vectors along the path, off its corners by a seeded shift."""
    P = np.array(_lattice(kind)[3], dtype=float)
    s = np.concatenate([[0], np.cumsum(np.linalg.norm(np.diff(P, axis=0), axis=1))])
    t = (np.arange(n) + rng.uniform(0.1, 0.9)) / n * s[-1]
    return np.stack([np.interp(t, s, P[:, c]) for c in (0, 1)], 1)


def _translations_in(case, seed):
    rng = np.random.default_rng(seed)
    n = case["n"]
    r = np.exp(rng.uniform(math.log(50e-9), math.log(10e-6), n))
    ke = math.sqrt(EPS_OUT) * rng.uniform(E_LO, E_HI, n) * EV / HBAR / C0
    kr = ke * (1 + 1j * (rng.uniform(0, 1e-3, n) if case["lossy"] else 0.0)) * r
    return kr.astype(np.complex128), np.arccos(rng.uniform(-1, 1, n)), rng.uniform(0, 2 * math.pi, n)


def _scatter_in(case, seed):
    rng = np.random.default_rng(seed)
    return _cluster(case["spheres"], rng), _omegas(rng, case["nw"])


def _scan_in(case, seed):
    rng = np.random.default_rng(seed)
    return _omegas(rng, case["nw"]), _bloch(case["lattice"], case["nk"], rng)


def _field_in(case, seed):
    rng = np.random.default_rng(seed)
    pos = _cluster(case["spheres"], rng)
    l = np.concatenate([np.full(2 * i + 1, i) for i in range(1, case["lMax"] + 1)] * 2)
    size = (case["spheres"], l.size)
    f = (rng.normal(size=size) + 1j * rng.normal(size=size)) * 0.1 ** l  # amplitudes fall with the order
    side = math.ceil(math.sqrt(case["points"]))
    half = 0.5 * PITCH * math.ceil(math.sqrt(case["spheres"]))
    i = np.arange(case["points"])
    step = 2 * half / max(1, side - 1)
    pts = np.stack([(i % side) * step - half, (i // side) * step - half, np.full(i.size, 100e-9)], 1)
    return pos, f.reshape(-1), pts, math.sqrt(EPS_OUT) * rng.uniform(E_LO, E_HI) * EV / HBAR / C0


def _modes_in(case, seed):
    rng = np.random.default_rng(seed)
    pos = _cluster(case["spheres"], rng)
    size = (case["spheres"] * 2 * case["lMax"] * (case["lMax"] + 2), case["columns"])
    return pos, (rng.normal(size=size) + 1j * rng.normal(size=size)) / math.sqrt(2)


def _serving_in(case, seed):
    """The mix (kinds and sizes) belongs to the case, positions and frequencies to the seed."""
    mix, rng = np.random.default_rng(case["mix"]), np.random.default_rng(seed)
    out = []
    for _ in range(case["requests"]):
        if mix.uniform() < 0.7:
            ns, lMax = int(mix.integers(min(16, case["max_spheres"]), case["max_spheres"] + 1)), int(mix.integers(2, 5))
            out.append({"pos": _cluster(ns, rng), "lMax": lMax, "omega": _omegas(rng, 1)[0], "lattice": None})
        else:
            lat = "square" if mix.uniform() < 0.5 else "honeycomb"
            out.append({"lattice": lat, "lMax": 3, "omega": _omegas(rng, 1)[0], "k": _bloch(lat, 1, rng)[0]})
    return out


# ---------------------------------------------------------------- the calls

def prepare(case, seed):
    import qpms_gb300 as qpms
    path = case["path"]
    if path == "translations":
        ne = case["lMax"] * (case["lMax"] + 2)
        A = torch.empty((case["n"], ne, ne), dtype=torch.complex128, device="cuda")
        return {"path": path, "J": case["J"], "calc": qpms.trans_calculator(case["lMax"]),
                "in": [torch.from_numpy(x).cuda() for x in _translations_in(case, seed)], "A": A, "B": torch.empty_like(A)}
    if path == "scatter":
        pos, om = _scatter_in(case, seed)
        return {"path": path, "ss": qpms.ScatteringSystem(pos, R_FINITE, EPS_IN, EPS_OUT, case["lMax"]), "omegas": om,
                "mode": case["mode"], "scat": case["scat"]}
    if path == "scan":
        b1, b2, pos, _ = _lattice(case["lattice"])
        om, kv = _scan_in(case, seed)
        return {"path": path, "omegas": om, "k": kv, "mode": case["mode"],
                "ss": qpms.ScatteringSystem(pos, R_LATTICE, EPS_IN, EPS_OUT, case["lMax"], lattice=(b1, b2))}
    if path == "field":
        pos, f, pts, k = _field_in(case, seed)
        return {"path": path, "ss": qpms.ScatteringSystem(pos, R_FIELD, EPS_IN, EPS_OUT, case["lMax"]), "k": k,
                "f": torch.from_numpy(f).cuda(), "points": torch.from_numpy(pts).cuda()}
    if path == "modes":
        pos, V = _modes_in(case, seed)
        return {"path": path, "ss": qpms.ScatteringSystem(pos, R_FINITE, EPS_IN, EPS_OUT, case["lMax"]), "V": V,
                "nodes": case["nodes"]}
    from qpms_gb300 import serving
    reqs = []
    lattices = {}
    for q in _serving_in(case, seed):
        if q["lattice"] is None:
            reqs.append({"system": qpms.ScatteringSystem(q["pos"], R_FINITE, EPS_IN, EPS_OUT, q["lMax"]),
                         "omega": q["omega"]})
            continue
        if q["lattice"] not in lattices:
            b1, b2, pos, _ = _lattice(q["lattice"])
            lattices[q["lattice"]] = qpms.ScatteringSystem(pos, R_LATTICE, EPS_IN, EPS_OUT, 3, lattice=(b1, b2))
        reqs.append({"system": lattices[q["lattice"]], "omega": q["omega"], "k": q["k"]})
    return {"path": path, "server": serving.Server(hbm_budget=40 << 30, mode=1, workers=case["workers"]), "requests": reqs}


def run(s):
    path = s["path"]
    if path == "translations":
        s["calc"].get_AB_arrays_device(*s["in"], s["J"], s["A"], s["B"],
                                       stream=torch.cuda.current_stream().cuda_stream)
        return [s["A"], s["B"]]
    if path == "scatter":
        r = s["ss"].planewave_scatter_batch(s["omegas"], mode=s["mode"], want_f=True, want_scat=s["scat"])
        return [r["f"], r["sigma_ext"]] + ([r["sigma_scat"]] if s["scat"] else [])
    if path == "scan":
        r = s["ss"].dispersion_scan(s["omegas"], s["k"], want_f=True, mode=s["mode"])
        return [r["logdet"], r["f"], r["sigma_ext"]]
    if path == "field":
        return s["ss"].scattered_E_device(s["k"], s["f"], s["points"])
    if path == "modes":
        from qpms_gb300 import beyn
        c, rr, ri = (x * EV / HBAR for x in CONTOUR)
        return list(beyn.scatsys_quadrature(s["ss"].s, s["ss"].fecv_size, c, rr, ri, s["nodes"], 0, s["nodes"],
                                            s["V"].shape[1], Vhat=s["V"]))
    tickets = [s["server"].submit(q["system"], q["omega"], k=q.get("k", (0.0, 0.0))) for q in s["requests"]]
    results = [s["server"].wait(t) for t in tickets]
    return [r["f"] for r in results] + [np.array([r["sigma_ext"] for r in results])]


def work(case):
    """Bytes: inputs and outputs once.  Operations: the real multiply-adds of the dense products, factorisations
    and solves (a complex product counts 8), and of the sums over orders."""
    path = case["path"]
    if path == "serving":
        size = [len(q["pos"]) * 2 * q["lMax"] * (q["lMax"] + 2) if q["lattice"] is None else
                (30 if q["lattice"] == "square" else 60) for q in _serving_in(case, 0)]
        return {"bytes": float(sum(16 * N + 64 for N in size)), "flops": float(sum(_solve_flops(N, 1) for N in size))}
    lMax = case["lMax"]
    ne = lMax * (lMax + 2)
    if path == "translations":
        terms = sum(c.size for c in _multipliers(lMax)[0] + _multipliers(lMax)[1])
        return {"bytes": case["n"] * (32.0 * ne * ne + 32), "flops": 4.0 * case["n"] * terms}
    if path == "scan":
        N = 2 * ne * len(_lattice(case["lattice"])[2])
        return {"bytes": case["nw"] * (8.0 + case["nk"] * (16 * N + 16)) + 16 * case["nk"],
                "flops": case["nw"] * case["nk"] * _solve_flops(N, 1)}
    N = case["spheres"] * 2 * ne
    if path == "scatter":
        return {"bytes": case["nw"] * (16.0 * N + 24) + 24 * case["spheres"], "flops": case["nw"] * _solve_flops(N, 1)}
    if path == "field":
        return {"bytes": 24.0 * case["spheres"] + 16 * N + 72 * case["points"],
                "flops": 1.0 * case["points"] * case["spheres"] * 60 * ne}
    return {"bytes": 80.0 * N * case["columns"], "flops": case["nodes"] * _solve_flops(N, case["columns"])}


def _solve_flops(N, nrhs):
    return 8.0 / 3 * N ** 3 + 8.0 * N * N * nrhs


# ---------------------------------------------------------------- the same in plain 64-bit torch

def exact(case, seed):
    path = case["path"]
    with torch.no_grad():
        if path == "translations":
            kr, th, ph = (torch.from_numpy(x).to(_dev()) for x in _translations_in(case, seed))
            return list(_ab(case["lMax"], case["J"], kr, torch.cos(th), torch.sin(th), ph))
        if path == "scatter":
            pos, om = _scatter_in(case, seed)
            got = [_scatter(pos, w, case["lMax"], case["scat"]) for w in om]
            return [np.stack([g[0] for g in got])] + [np.array([g[i] for g in got]) for i in range(1, 3 if case["scat"] else 2)]
        if path == "scan":
            om, kv = _scan_in(case, seed)
            got = [_lattice_solve(case["lattice"], case["lMax"], w, kv) for w in om]
            return [np.stack([g[i] for g in got]) for i in range(3)]
        if path == "field":
            return _field(*_field_in(case, seed), case["lMax"])
        if path == "modes":
            return _contour_sums(*_modes_in(case, seed), case["lMax"], case["nodes"])
        f, sig = [], []
        for q in _serving_in(case, seed):
            if q["lattice"] is None:
                a, b = _scatter(q["pos"], q["omega"], q["lMax"], False)
            else:
                _, a, b = (x[0] for x in _lattice_solve(q["lattice"], q["lMax"], q["omega"], q["k"][None]))
            f.append(a)
            sig.append(b)
        return f + [np.array(sig)]


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _orders(lMax):
    return [(l, m) for l in range(1, lMax + 1) for m in range(-l, l + 1)]


@lru_cache(maxsize=None)
def _three_j(j1, j2, j3, m1, m2, m3):
    """Wigner 3j symbol by Racah's sum, in rational numbers up to the last square root."""
    if m1 + m2 + m3 or j3 < abs(j1 - j2) or j3 > j1 + j2 or abs(m1) > j1 or abs(m2) > j2 or abs(m3) > j3:
        return 0.0
    F = math.factorial
    pre = Fraction(F(j1 + j2 - j3) * F(j1 - j2 + j3) * F(-j1 + j2 + j3), F(j1 + j2 + j3 + 1))
    pre *= F(j1 + m1) * F(j1 - m1) * F(j2 + m2) * F(j2 - m2) * F(j3 + m3) * F(j3 - m3)
    s = Fraction(0)
    for k in range(max(0, j2 - j3 - m1, j1 - j3 + m2), min(j1 + j2 - j3, j1 - m1, j2 + m2) + 1):
        s += Fraction((-1) ** k, F(k) * F(j3 - j2 + k + m1) * F(j3 - j1 + k - m2) * F(j1 + j2 - j3 - k) *
                      F(j1 - k - m1) * F(j2 - k + m2))
    if s == 0:
        return 0.0
    return (-1) ** (j1 - j2 - m3) * (1 if s > 0 else -1) * math.sqrt(pre * s * s)


def _legendre_norm(p, m):
    """P_p^m -> fully normalised, without the 4 pi: sqrt((2p + 1) (p - m)! / (p + m)!)."""
    return math.sqrt(Fraction((2 * p + 1) * math.factorial(p - m), math.factorial(p + m)))


@lru_cache(maxsize=None)
def _multipliers(lMax):
    """Per element (y, y') the coefficients over p of A (real) and B (imaginary) in the functions
    z_p P_p^|d| e^{i d phi}, d = m' - m (Cruzan's expressions; power-normalised waves, Condon-Shortley phase)."""
    A, B = [], []
    for n, m in _orders(lMax):
        for v, u in _orders(lMax):
            d = u - m
            pre = (-1) ** u * math.sqrt((2 * n + 1) * (2 * v + 1) / (n * (n + 1) * v * (v + 1)))
            a, b = [], []
            for q in range(min(n, v, (n + v - abs(d)) // 2) + 1):
                p = n + v - 2 * q
                a.append(pre * (-1) ** (d < 0 and d % 2) * 0.5 * (n * (n + 1) + v * (v + 1) - p * (p + 1)) *
                         math.sqrt(2 * p + 1) * _three_j(n, v, p, -m, u, m - u) * _three_j(n, v, p, 0, 0, 0) *
                         _legendre_norm(p, abs(d)) * (-1) ** ((n - v + p) // 2))
            for q in range(min(n, v, (n + v + 1 - abs(d)) // 2) + 1):
                p = n + v - 2 * q
                t = math.sqrt(((p + 1) ** 2 - (n - v) ** 2) * ((n + v + 1) ** 2 - (p + 1) ** 2))
                b.append(pre * (-1) ** (d < 0 and d % 2) * 0.5 * t * math.sqrt(2 * p + 3) *
                         _three_j(n, v, p + 1, -m, u, m - u) * _three_j(n, v, p, 0, 0, 0) *
                         _legendre_norm(p + 1, abs(d)) * (-1) ** ((n - v + p) // 2 + 1))
            A.append(np.array(a))
            B.append(np.array(b))
    return A, B


@lru_cache(maxsize=None)
def _contraction(lMax, lattice):
    """The multipliers as dense (slots p^2 + p + d) x (elements) matrices; a lattice sum's B stops at A's last term."""
    A, B = _multipliers(lMax)
    out = [np.zeros(((2 * lMax + 2) ** 2, len(A))) for _ in (0, 1)]
    e = 0
    for n, m in _orders(lMax):
        for v, u in _orders(lMax):
            for q in range(len(A[e])):
                p = n + v - 2 * q
                out[0][p * p + p + u - m, e] = A[e][q]
            for q in range(min(len(B[e]), len(A[e])) if lattice else len(B[e])):
                p = n + v - 2 * q + 1
                out[1][p * p + p + u - m, e] = B[e][q]
            e += 1
    return out


def _bessel(J, L, x):
    """z_0 .. z_L of kind 1 (regular) or 3 (outgoing) at the complex tensor x, stacked first."""
    if J == 3:
        e = torch.exp(1j * x)
        z = [-1j * e / x, -e * (x + 1j) / x ** 2]
        for l in range(1, L):
            z.append((2 * l + 1) / x * z[l] - z[l - 1])
        return torch.stack(z[:L + 1])
    top = int(float(x.abs().max())) + L + 40  # downward recurrence, normalised to j_0 or j_1
    hi, lo, keep = torch.zeros_like(x), torch.full_like(x, 1e-100), {}
    for l in range(top, 0, -1):
        hi, lo = lo, (2 * l + 1) / x * lo - hi
        if l - 1 <= L:
            keep[l - 1] = lo
        big = lo.abs() > 1e100
        if bool(big.any()):
            s = torch.where(big, torch.full_like(x, 1e-100), torch.ones_like(x))
            hi, lo, keep = hi * s, lo * s, {k: v * s for k, v in keep.items()}
    j0, j1 = torch.sin(x) / x, torch.sin(x) / x ** 2 - torch.cos(x) / x
    small = x.abs() < 0.5  # j_1 by its series there
    j1 = torch.where(small, sum((-1) ** k * x ** (2 * k + 1) / (2 ** k * math.factorial(k) * math.prod(range(1, 2 * k + 4, 2)))
                                for k in range(9)), j1)
    scale = torch.where(j0.abs() >= j1.abs(), j0 / keep[0], j1 / keep[1])
    return torch.stack([keep[l] * scale for l in range(L + 1)])


def _legendre(L, ct, st):
    """{(l, m): P_l^m}, m >= 0, with the Condon-Shortley phase."""
    P = {(0, 0): torch.ones_like(ct)}
    for m in range(L + 1):
        if m:
            P[m, m] = -(2 * m - 1) * st * P[m - 1, m - 1]
        for l in range(m + 1, L + 1):
            P[l, m] = ((2 * l - 1) * ct * P[l - 1, m] - ((l + m - 1) * P[l - 2, m] if l > m + 1 else 0)) / (l - m)
    return P


def _ab(lMax, J, kr, ct, st, phi):
    """Translation arrays A, B (n x nelem x nelem)."""
    L, ne = 2 * lMax + 1, lMax * (lMax + 2)
    CA, CB = (torch.from_numpy(c).to(kr.device).to(kr.dtype) for c in _contraction(lMax, False))
    A = torch.empty((kr.numel(), ne * ne), dtype=kr.dtype, device=kr.device)
    B = torch.empty_like(A)
    for i in range(0, kr.numel(), 50000):
        at = slice(i, i + 50000)
        z, P, ph = _bessel(J, L, kr[at]), _legendre(L, ct[at], st[at]), phi[at]
        w = torch.stack([z[p] * P[p, abs(d)] * torch.exp(1j * d * ph) for p in range(L + 1) for d in range(-p, p + 1)], 1)
        A[at], B[at] = w @ CA, 1j * (w @ CB)
    return A.view(-1, ne, ne), B.view(-1, ne, ne)


def _translation_matrix(pos, k, lMax, J):
    """S with zero self blocks: the (electric, magnetic) waves of every particle, A for like and B for unlike types."""
    ne, p = lMax * (lMax + 2), torch.from_numpy(pos).to(_dev())
    np_ = p.shape[0]
    S = torch.zeros((np_, 2, ne, np_, 2, ne), dtype=torch.complex128, device=p.device)
    step = max(1, 20000 // np_)
    for i in range(0, np_, step):
        d = p[i:i + step, None] - p[None]
        r = d.norm(dim=2)
        own = r == 0
        r = torch.where(own, PITCH, r)
        st = torch.hypot(d[..., 0], d[..., 1]) / r
        A, B = _ab(lMax, J, (k * r).to(torch.complex128).reshape(-1), (d[..., 2] / r).reshape(-1), st.reshape(-1),
                   torch.atan2(d[..., 1], d[..., 0]).reshape(-1))
        A, B = (x * (~own).reshape(-1, 1, 1) for x in (A, B))
        A, B = (x.view(-1, np_, ne, ne).permute(0, 2, 1, 3) for x in (A, B))
        for a in (0, 1):
            for b in (0, 1):
                S[i:i + step, a, :, :, b, :] = A if a == b else B
    return S.view(np_ * 2 * ne, np_ * 2 * ne)


def _mie(lMax, radius, omega):
    """Diagonal of a sphere's T-matrix, electric then magnetic waves."""
    ki, ke = (np.sqrt(complex(e)) * omega / C0 for e in (EPS_IN, EPS_OUT))

    def waves(J, x):
        z = _bessel(J, lMax + 1, torch.tensor([x], dtype=torch.complex128)).numpy()[:, 0]
        return z, [z[l] / x - z[l + 1] + l / x * z[l] for l in range(lMax + 1)]

    (zi, fi), (ze, fe), (zs, fs) = waves(1, ki * radius), waves(1, ke * radius), waves(3, ke * radius)
    el = [(-ki * fe[l] * zi[l] + ke * ze[l] * fi[l]) / (-ke * fi[l] * zs[l] + ki * zi[l] * fs[l]) for l in range(lMax + 1)]
    mg = [(-ke * fe[l] * zi[l] + ki * ze[l] * fi[l]) / (-ki * fi[l] * zs[l] + ke * zi[l] * fs[l]) for l in range(lMax + 1)]
    return np.array([t[l] for t in (el, mg) for l, _ in _orders(lMax)])


def _angular(lMax, ct, st):
    """{(l, m): (P, m P / sin, dP / dtheta)} of the power-normalised harmonics; regular on the axis."""
    P = _legendre(lMax + 1, ct, st)
    R = _legendre_over_sine(lMax + 1, ct, st)
    out = {}
    for l in range(1, lMax + 1):
        for m in range(l + 1):
            nf = _legendre_norm(l, m) / math.sqrt(4 * math.pi * l * (l + 1))
            low = (l + m) * (l - m + 1) * P[l, m - 1] if m else -P[l, 1]
            der = -0.5 * (low - (P[l, m + 1] if m < l else 0))
            v = (nf * P[l, m], nf * m * R[l, m] if m else torch.zeros_like(ct), nf * der)
            out[l, m] = v
            if m:
                out[l, -m] = tuple((-1) ** (m + s) * x for s, x in zip((0, 1, 0), v))
    return out


def _legendre_over_sine(L, ct, st):
    """P_l^m / sin theta for m >= 1."""
    R = {}
    for m in range(1, L + 1):
        R[m, m] = -torch.ones_like(ct) if m == 1 else -(2 * m - 1) * st * R[m - 1, m - 1]
        for l in range(m + 1, L + 1):
            R[l, m] = ((2 * l - 1) * ct * R[l - 1, m] - ((l + m - 1) * R[l - 2, m] if l > m + 1 else 0)) / (l - m)
    return R


def _incidence(lMax, kd, E):
    """Regular-wave coefficients of a plane wave of direction kd, amplitude E, electric then magnetic."""
    x, y, z = kd / np.linalg.norm(kd)
    s, phi = math.hypot(x, y), math.atan2(y, x)
    Et = E[0] * z * math.cos(phi) + E[1] * z * math.sin(phi) - E[2] * s
    Ep = -E[0] * math.sin(phi) + E[1] * math.cos(phi)
    ang = _angular(lMax, torch.tensor([z], dtype=torch.float64), torch.tensor([s], dtype=torch.float64))
    el, mg = [], []
    for l, m in _orders(lMax):
        _, pi, tau = (float(v) for v in ang[l, m])
        e = np.exp(-1j * m * phi)
        mg.append(4 * math.pi * 1j ** l * (-1j * pi * Et - tau * Ep) * e)
        el.append(-4 * math.pi * 1j ** (l + 1) * (tau * Et - 1j * pi * Ep) * e)
    return np.array(el + mg)


def _scatter(pos, omega, lMax, scat):
    """f, sigma_ext and, if asked for, sigma_scat of a cluster under normal incidence, E along x."""
    k = math.sqrt(EPS_OUT) * omega / C0
    T = torch.from_numpy(np.tile(_mie(lMax, R_FINITE, omega), len(pos))).to(_dev())
    inc = _incidence(lMax, np.array([0.0, 0.0, 1.0]), (1.0, 0.0, 0.0))
    a = torch.from_numpy((np.exp(1j * k * pos[:, 2])[:, None] * inc[None]).reshape(-1)).to(_dev())
    M = _translation_matrix(pos, k, lMax, 3).mul_(-T[:, None])
    M.diagonal().add_(1)
    f = torch.linalg.solve(M, T * a)
    del M
    out = [f.cpu().numpy(), -float(torch.vdot(a, f).real) / k ** 2]
    if scat:
        out.append(float(torch.vdot(f, f + _translation_matrix(pos, k, lMax, 1) @ f).real) / k ** 2)
    return out


def _contour_sums(pos, V, lMax, nodes):
    """A0, A1 and their every-second-node versions over the ellipse."""
    c, rr, ri = (x * EV / HBAR for x in CONTOUR)
    Vd = torch.from_numpy(V).to(_dev())
    out = [torch.zeros_like(Vd) for _ in range(4)]
    for i in range(nodes):
        t = 2 * math.pi * i / nodes
        dz = complex(-rr * math.sin(t), ri * math.cos(t)) * (2 * math.pi / nodes)
        rel = complex(rr * math.cos(t), ri * math.sin(t))
        z = complex(c) + rel
        M = _translation_matrix(pos, np.sqrt(complex(EPS_OUT)) * z / C0, lMax, 3)
        M.mul_(-torch.from_numpy(np.tile(_mie(lMax, R_FINITE, z), len(pos))).to(_dev())[:, None])
        M.diagonal().add_(1)
        X = torch.linalg.solve(M, Vd)
        del M
        for j, w in enumerate((dz, dz * rel)):
            out[j] += w * X
            if i % 2 == 0:
                out[j + 2] += 2 * w * X
    return [x.cpu().numpy() for x in out]


def _field(pos, f, pts, k, lMax):
    """E of outgoing waves of all particles at the points."""
    p, w = torch.from_numpy(pos).to(_dev()), torch.from_numpy(pts).to(_dev())
    f = f.reshape(len(pos), 2, -1)
    E = torch.zeros((len(pts), 3), dtype=torch.complex128, device=w.device)
    for i in range(len(pos)):
        d = w - p[i]
        r = d.norm(dim=1)
        rho = torch.hypot(d[:, 0], d[:, 1])
        ct, st, phi = d[:, 2] / r, rho / r, torch.atan2(d[:, 1], d[:, 0])
        x = (k * r).to(torch.complex128)
        h, ang = _bessel(3, lMax, x), _angular(lMax, ct, st)
        Er, Et, Ep = (torch.zeros_like(x) for _ in range(3))
        for y, (l, m) in enumerate(_orders(lMax)):
            leg, pi, tau = ang[l, m]
            e = torch.exp(1j * m * phi)
            rad, der = h[l] / x, h[l - 1] - l * h[l] / x
            N, M = complex(f[i, 0, y]), complex(f[i, 1, y])
            Er += N * l * (l + 1) * leg * rad * e
            Et += (N * tau * der + M * 1j * pi * h[l]) * e
            Ep += (N * 1j * pi * der - M * tau * h[l]) * e
        sf, cf = torch.sin(phi), torch.cos(phi)
        E += torch.stack([st * cf * Er + ct * cf * Et - sf * Ep, st * sf * Er + ct * sf * Et + cf * Ep, ct * Er - st * Et], 1)
    return E


# ---- lattices

@lru_cache(maxsize=None)
def _solid(n, m):
    """|q|^n P_n^m(q_z / |q|) = q_par^m sum_ab c[a, b] q_par^{2a} q_z^b."""
    poly = np.polynomial.legendre.leg2poly([0] * n + [1])
    if m:
        poly = np.polynomial.polynomial.polyder(poly, m)
    c = {}
    for j, a in enumerate(poly):
        if (n - m - j) % 2 == 0 and a:
            h = (n - m - j) // 2
            for t in range(h + 1):
                c[h - t, j + 2 * t] = c.get((h - t, j + 2 * t), 0.0) + (-1) ** m * a * math.comb(h, t)
    return c


def _erfc_scaled(kappa, eta):
    """pi / kappa erfc(kappa / 2 eta) for kappa > 0 or on the negative imaginary axis."""
    x = kappa / (2 * eta)
    re = torch.erfc(x.real).to(kappa.dtype)
    t, wt = np.polynomial.legendre.leggauss(64)
    y = -x.imag
    erfi = sum(wi * 0.5 * torch.exp((0.5 * y * (ti + 1)) ** 2) for ti, wi in zip(t, wt)) * y * 2 / math.sqrt(math.pi)
    return math.pi / kappa * torch.where(x.imag == 0, re, 1 + 1j * erfi)


def _lattice_sums(b1, b2, s, k, beta, L):
    """sigma_nm = sum_R h_n(k |d|) P_n^|m| e^{i m phi_d} e^{i beta.d}, d = R - s, n <= L, for each row of beta (with
    the reference's sign (-1)^m where m < 0): Ewald's split for s in the plane, the plane-wave expansion for s off
    it.  The term d = 0 is left out."""
    dev = beta.device
    B = np.array([b1, b2], dtype=float)
    area = abs(np.linalg.det(B))
    G = 2 * math.pi * np.linalg.inv(B).T
    off = s[2] != 0
    eta = math.sqrt(math.pi / area) * 1.3
    n_out = 40 if off else 9
    ij = np.stack(np.meshgrid(*[np.arange(-n_out, n_out + 1)] * 2), -1).reshape(-1, 2)
    g = torch.from_numpy(ij @ G).to(dev)
    q = g[None] - beta[:, None]
    q2 = (q ** 2).sum(2)
    phase = torch.exp(-1j * (g @ torch.from_numpy(s[:2]).to(dev)))[None]
    kap2 = q2 - k * k
    kappa = torch.where(kap2 > 0, torch.sqrt(kap2.abs()).to(torch.complex128), -1j * torch.sqrt(kap2.abs()))
    e1 = torch.complex(q[..., 0], q[..., 1])
    if off:
        ez = torch.exp(-kappa * abs(s[2])) / (2 * kappa)
        qz = 1j * kappa * math.copysign(1.0, -s[2])
    else:
        gauss = torch.where(kap2 / (4 * eta * eta) < 700, torch.exp(-(kap2 / (4 * eta * eta)).clamp(max=700)), 0.0)
        mom = [_erfc_scaled(kappa, eta)]
        for j in range(L // 2 + 1):
            mom.append(gauss * math.gamma(j + 0.5) * (2 * eta) ** (2 * j + 1) - kap2 * mom[j])
        d = torch.from_numpy(np.array([r for r in (ij @ B - s[:2]) if 0 < r @ r < (7.0 / eta) ** 2])).to(dev)
        d2 = (d ** 2).sum(1)
        t, wt = (torch.from_numpy(v).to(dev) for v in np.polynomial.legendre.leggauss(80))
        top = torch.sqrt(eta * eta + 46 / d2)
        xi = eta + 0.5 * (top - eta)[:, None] * (t + 1)
        ker = torch.exp(-d2[:, None] * xi ** 2 + k * k / (4 * xi ** 2)) * 0.5 * (top - eta)[:, None] * wt
        bloch = torch.exp(1j * (beta @ d.T))
        ed = torch.complex(d[:, 0], d[:, 1])
    sig = {}
    for n in range(L + 1):
        c = -1j * 2 ** (n + 1) / (math.sqrt(math.pi) * k ** (n + 1))
        long = c * (-1j) ** n * math.pi ** 1.5 * 2 ** (1 - n) / area
        for m in range(-n, n + 1):
            co, am = _solid(n, abs(m)), abs(m)
            pw = e1 ** am if m >= 0 else e1.conj() ** am
            if off:
                y = sum(a * q2 ** i * qz ** j for (i, j), a in co.items())
                sig[n, m] = long * (pw * y * ez * phase).sum(1)
                continue
            if (n - am) % 2:
                sig[n, m] = torch.zeros(beta.shape[0], dtype=torch.complex128, device=dev)
                continue
            v = long / (2 * math.pi) * (pw * phase * sum(a * q2 ** i * mom[j // 2] for (i, j), a in co.items())).sum(1)
            at0 = sum(a * d2 ** i for (i, j), a in co.items() if j == 0)
            pd = ed ** am if m >= 0 else ed.conj() ** am
            v = v + c * (bloch * (at0 * pd * (ker * xi ** (2 * n)).sum(1))[None]).sum(1)
            if n == 0 and not s.any():
                x = (k / (2 * eta)) ** 2
                J = eta * sum(x ** j / math.factorial(j) / (2 * j - 1) for j in range(1, 40))
                v = v - (1 - c * (J - eta))
            sig[n, m] = v
    return torch.stack([sig[n, m] * (-1) ** max(0, -m) for n in range(L + 1) for m in range(-n, n + 1)], 1)


def _lattice_solve(kind, lMax, omega, kv):
    """log|det M|, f and sigma_ext for each Bloch vector (E along x, made transverse; evanescent incidence: zero)."""
    b1, b2, pos, _ = _lattice(kind)
    k = math.sqrt(EPS_OUT) * omega / C0
    ne, nk, dev = lMax * (lMax + 2), len(kv), _dev()
    CA, CB = (torch.from_numpy(c).to(dev).to(torch.complex128) for c in _contraction(lMax, True))
    beta = torch.from_numpy(np.ascontiguousarray(kv)).to(dev)
    W = torch.zeros((nk, len(pos), 2, ne, len(pos), 2, ne), dtype=torch.complex128, device=dev)
    for r in range(len(pos)):
        for c in range(len(pos)):
            w = _lattice_sums(b1, b2, pos[r] - pos[c], k, beta, 2 * lMax + 1)
            A, B = (w @ CA).view(nk, ne, ne), 1j * (w @ CB).view(nk, ne, ne)
            for a in (0, 1):
                for b in (0, 1):
                    W[:, r, a, :, c, b, :] = A if a == b else B
    N = len(pos) * 2 * ne
    T = torch.from_numpy(np.tile(_mie(lMax, R_LATTICE, omega), len(pos))).to(dev)
    M = torch.eye(N, dtype=torch.complex128, device=dev) - T[:, None] * W.view(nk, N, N)
    a = np.zeros((nk, N), dtype=np.complex128)
    for i, (x, y) in enumerate(kv):
        if x * x + y * y >= k * k:
            continue
        kd = np.array([x, y, math.sqrt(k * k - x * x - y * y)])
        E = np.array([1.0, 0, 0]) - kd * kd[0] / (kd @ kd)
        a[i] = (np.exp(1j * pos @ kd)[:, None] * _incidence(lMax, kd, E / np.linalg.norm(E))[None]).reshape(-1)
    a = torch.from_numpy(a).to(dev)
    f = torch.linalg.solve(M, (T * a)[..., None])[..., 0]
    sig = -(a.conj() * f).sum(1).real / k ** 2
    return [x.cpu().numpy() for x in (torch.linalg.slogdet(M)[1], f, sig)]
