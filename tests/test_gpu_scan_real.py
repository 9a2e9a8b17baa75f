"""The scan kernel for real wavenumbers against the general lattice assembly
(one matrix at a time, its own Ewald parameter and no tables) for every lMax,
self and cross pairs, oblique cells, layers, one to a few hundred Bloch vectors,
Bloch vectors at Gamma, on and next to reciprocal-lattice points and close to
Rayleigh anomalies from both sides; and lossy media, which keep the general
kernel.

Both agree with the oracle to 1e-10 (Frobenius, the matrices' parity
tolerance); the quantities of the scan are compared at that times the factors
they carry: f to 1e-10 times the matrices' condition number, log|det| to
1e-10 sqrt(N) times it.
"""
import numpy as np
import pytest

from qpms_gb300.workloads import C0, EV, HBAR

pytestmark = pytest.mark.gpu
A = 580e-9
CELLS = {
    "square": ((A, 0), (0, A), [[0, 0, 0]]),
    "honeycomb": ((A, 0), (A / 2, A * np.sqrt(3) / 2), [[-A / np.sqrt(12), 0, 0], [A / np.sqrt(12), 0, 0]]),
    "oblique": ((A, 0.1 * A), (0.3 * A, 0.9 * A), [[0, 0, 0], [0.4 * A, 0.3 * A, 0], [0.1 * A, 0.6 * A, 0]]),
    "bilayer": ((A, 0), (0, A), [[0, 0, 0], [0.5 * A, 0.4 * A, 0.3 * A]]),
}


@pytest.fixture(scope="module")
def gpu():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qpms_gb300
    return qpms_gb300


def _check(gpu, cell, lMax, eps, om, kv, pick):
    b1, b2, pos = CELLS[cell]
    ss = gpu.ScatteringSystem(np.array(pos, dtype=float), 60e-9, -12 + 1.2j, eps, lMax, lattice=(b1, b2))
    r = ss.dispersion_scan(om, kv, want_f=True, mode=0)
    for i, w in enumerate(om):
        kap = (np.sqrt(eps + 0j) * w / C0).real
        for j in pick:
            M = ss(w).modeproblem_matrix_full(k=kv[j])
            cond = np.linalg.cond(M)
            ld = np.linalg.slogdet(M)[1]
            assert abs(r["logdet"][i, j] - ld) <= 1e-10 * np.sqrt(len(M)) * cond
            kz2 = kap ** 2 - kv[j] @ kv[j]
            if kz2 <= 0:
                assert not r["f"][i, j].any()
                continue
            kd = np.array([*kv[j], np.sqrt(kz2)])
            E = np.array([1.0, 0, 0]) - kd * kd[0] / (kd @ kd)
            b = ss(w).apply_Tmatrices_full(ss.planewave_full(kd, E / np.linalg.norm(E)))
            f = np.linalg.solve(M, b)
            assert np.linalg.norm(r["f"][i, j] - f) <= 1e-10 * cond * np.linalg.norm(f)


@pytest.mark.parametrize("cell", list(CELLS))
@pytest.mark.parametrize("lMax", [1, 2, 3, 4])
@pytest.mark.parametrize("eps", [2.25, 2.25 + 0.05j])
def test_scan_against_single_matrices(gpu, cell, lMax, eps):
    om = np.array([1.7, 2.3]) * EV / HBAR
    k0 = 1.5 * om[0] / C0
    b = np.linalg.inv(np.array(CELLS[cell][:2])).T * 2 * np.pi
    kv = np.array([[0, 0], b[0] / 2, 0.3 * b[0] + 0.2 * b[1], b[0], b[0] * (1 + 1e-7), [k0 * (1 + 1e-6), 0],
                   [k0 * (1 - 1e-6), 0], [0, 0.999 * k0]])
    _check(gpu, cell, lMax, eps, om, kv, range(len(kv)))


@pytest.mark.parametrize("nk", [1, 3, 301])
def test_counts_of_bloch_vectors(gpu, nk):
    rng = np.random.default_rng(nk)
    kv = rng.uniform(-1, 1, (nk, 2)) * np.pi / A
    _check(gpu, "honeycomb", 2, 2.25, np.array([1.8, 2.0, 2.2]) * EV / HBAR, kv, sorted({0, nk // 2, nk - 1}))
