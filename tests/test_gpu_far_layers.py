"""Lattice sums between planes far apart, |k dz| from 5 to 150.

An order of the reciprocal-lattice sum decays as e^{-sqrt(q^2 - k^2) |dz|}, q = |beta + K|, and the propagating ones
(q < k) not at all, so the sum's range has to grow with k: checked against the oracle for lMax 1 to 4, both signs of
dz, real and lossy media, and a Bloch vector that puts an order just inside or just outside q = k; then as the mode
problem and the scan of a bilayer 4 um apart.  Tolerances: 1e-11 of the arrays' norms, that of the layers' sums
elsewhere (the phases, up to 150, carry that times 2^-53); the mode problem 1e-10, the parity tolerance of the
layered lattices; log|det| 1e-10 sqrt(N) times the condition number.
"""
import ctypes as C

import numpy as np
import pytest

from qpms_gb300.workloads import C0, EV, HBAR

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qpms_gb300
    return qpms_gb300


class _Cplx(C.Structure):
    _fields_ = [("re", C.c_double), ("im", C.c_double)]


class _Cart2(C.Structure):
    _fields_ = [("x", C.c_double), ("y", C.c_double)]


class _Cart3(C.Structure):
    _fields_ = [("x", C.c_double), ("y", C.c_double), ("z", C.c_double)]


def _check(gpu, orc, lMax, k, beta, shift):
    f = C.CDLL(gpu.lib()._name).qpms_trans_calculator_get_AB_arrays_e32
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_ssize_t, C.c_ssize_t, C.c_double,
                  _Cplx, _Cart2, _Cart2, _Cart2, _Cart3, C.c_double, C.c_double]
    norm, b1, b2, kc = 65536 | 8, (1.0, 0.0), (0.3, 1.1), complex(k)
    calc = gpu.trans_calculator(lMax, norm)
    ne = lMax * (lMax + 2)
    A, B = (np.zeros((ne, ne), dtype=np.complex128) for _ in range(2))
    rc = f(calc.c, A.ctypes.data, None, B.ctypes.data, None, ne, 1, 1.6, _Cplx(kc.real, kc.imag), _Cart2(*b1),
           _Cart2(*b2), _Cart2(*beta), _Cart3(*shift), 60.0, 500.0)
    assert rc == 0, gpu.last_error()
    Ao, Bo = orc.get_AB_arrays_e32(orc.TransCalculator(lMax, norm), 1.6, kc, b1, b2, beta, shift, 60, 500)
    assert np.linalg.norm(A - Ao) <= 1e-11 * np.linalg.norm(Ao)
    assert np.linalg.norm(B - Bo) <= 1e-11 * np.linalg.norm(Bo)


@pytest.mark.parametrize("lMax", [1, 2, 3, 4])
@pytest.mark.parametrize("k,sign", [(9.0, 1), (9.0, -1), (9.0 + 0.02j, -1)])
@pytest.mark.parametrize("kz", [5, 10, 20, 45, 57, 60, 65, 72, 80, 90, 150])
def test_far_planes(gpu, orc, lMax, k, sign, kz):
    _check(gpu, orc, lMax, k, (0.7, -0.4), (0.2, 0.45, sign * kz / abs(k)))


@pytest.mark.parametrize("lMax", [1, 4])
@pytest.mark.parametrize("kz", [40, 65, 100])
@pytest.mark.parametrize("side", [1 - 1e-3, 1 + 1e-3])
def test_an_order_next_to_k(gpu, orc, lMax, kz, side):
    """The order of K = (0, 2 pi / 1.1) lies next to k."""
    _check(gpu, orc, lMax, 9.0, (0.0, 9.0 * side - 2 * np.pi / 1.1), (0.2, 0.45, kz / 9.0))


@pytest.mark.parametrize("lMax", [1, 2])
@pytest.mark.parametrize("eps", [2.25, 2.25 + 0.001j])
def test_bilayer_four_micrometres_apart(gpu, orc, lMax, eps):
    a, kv = 580e-9, np.array([[0.0, 0.0], [2e6, -1e6]])
    b1, b2 = (a, 0.0), (0.0, a)
    pos = np.array([[0, 0, 0], [0.5 * a, 0.4 * a, 4e-6]])
    om = np.array([2.1]) * EV / HBAR  # k dz = 64
    ss = gpu.ScatteringSystem(pos, 60e-9, -12 + 1.2j, eps, lMax, lattice=(b1, b2))
    n = 2 * lMax * (lMax + 2)
    k = np.sqrt(eps + 0j) * om[0] / C0
    r = ss.dispersion_scan(om, kv, want_f=True, mode=0)
    for j in range(2):
        T = np.stack([ss(om[0]).apply_Tmatrices_full(np.eye(2 * n)[i].astype(complex)) for i in range(n)], 1)[:n]
        O = orc.periodic_modeproblem(orc.TransCalculator(lMax), pos, np.stack([T, T]), k, b1, b2, (*kv[j], 0.0),
                                     ss.adjusted_eta(k, kv[j]))
        M = ss(om[0]).modeproblem_matrix_full(k=kv[j])
        assert np.linalg.norm(M - O) <= 1e-10 * np.linalg.norm(O)
        far = np.s_[:n, n:]  # the block of the two planes
        assert np.linalg.norm(M[far] - O[far]) <= 1e-9 * np.linalg.norm(O[far])
        assert abs(r["logdet"][0, j] - np.linalg.slogdet(O)[1]) <= 1e-10 * np.sqrt(2 * n) * np.linalg.cond(O)
