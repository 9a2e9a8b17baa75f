"""The batched LU's kernels at the edges of their ranges: the shared-memory
kernel up to 64 unknowns, the cluster kernel above (whole and ragged panels of 8
columns, up to the largest order, clusters of several sizes), the substitutions
by warps and by blocks of 32 unknowns.

General matrices with row exchanges go through the drop-in factorisation
(qpms_scatsysw_modeproblem_matrix_full_factorise, scatsystem.c:2202-2244), whose
factors must be those of P M = L U with LAPACK's pivots.  Tolerance: the
backward error of Gaussian elimination, |P M - L U| <= gamma |L| |U| elementwise
(Higham, Accuracy and Stability of Numerical Algorithms, theorem 9.3) with
gamma = 4 N u for complex products, u = 2^-53; the solutions' residuals
within 3 gamma |L| |U| |x| (theorem 9.4).
"""
import numpy as np
import pytest

from qpms_gb300.workloads import EV, HBAR, jittered_square_cluster

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qpms_gb300
    return qpms_gb300


def _factorise(gpu, np_, M):
    """Factors, 0-based pivots and the solver of a caller's matrix of 6 np_ unknowns."""
    ss = gpu.ScatteringSystem(jittered_square_cluster(np_, np.random.default_rng(0)), 50e-9, -12 + 1.2j, 2.25, 1)
    ssw = ss(2.0 * EV / HBAR)
    N = M.shape[0]
    a, piv = np.array(M, dtype=np.complex128, order="C"), np.zeros(N, dtype=np.int32)
    lu = gpu.lib().qpms_scatsysw_modeproblem_matrix_full_factorise(a.ctypes.data, piv.ctypes.data, ssw.ssw, None)
    assert lu.a, gpu.last_error()

    def solve(b):
        x, b = np.empty_like(b), np.ascontiguousarray(b)
        assert gpu.lib().qpms_scatsys_scatter_solve(x.ctypes.data, b.ctypes.data, lu), gpu.last_error()
        return x
    return a, piv - 1, solve, (ssw, piv)  # the factors refer to both


@pytest.mark.parametrize("np_", [1, 5, 6, 10, 11, 12, 21, 22, 32, 43, 64, 85])
def test_factors_and_solutions(gpu, np_):
    scipy_linalg = pytest.importorskip("scipy.linalg")
    N = 6 * np_
    rng = np.random.default_rng(N)
    M = rng.normal(size=(N, N)) + 1j * rng.normal(size=(N, N))
    a, piv, solve, _keep = _factorise(gpu, np_, M)
    assert np.array_equal(piv, scipy_linalg.lu_factor(M)[1])
    PM = M.copy()
    for i, p in enumerate(piv):
        PM[[i, p]] = PM[[p, i]]
    L, U = np.tril(a, -1) + np.eye(N), np.triu(a)
    gamma = 4 * N * 2.0 ** -53
    LU = np.abs(L) @ np.abs(U)
    assert np.all(np.abs(PM - L @ U) <= 2 * gamma * LU)  # twice: the product formed here rounds too
    b = rng.normal(size=N) + 1j * rng.normal(size=N)
    x = solve(b)
    r = np.abs(M @ x - b)
    for i, p in enumerate(piv):
        r[[i, p]] = r[[p, i]]
    assert np.all(r <= 2 * 3 * gamma * (LU @ np.abs(x)))


@pytest.mark.parametrize("np_", [4, 20])
def test_a_zero_column_is_reported(gpu, np_):
    N = 6 * np_
    rng = np.random.default_rng(1)
    M = rng.normal(size=(N, N)) + 1j * rng.normal(size=(N, N))
    M[:, N - 3] = 0
    a, _, _, _keep = _factorise(gpu, np_, M)
    assert a[N - 3, N - 3] == 0
    assert "U(%d,%d) is exactly zero" % (N - 2, N - 2) in gpu.last_error()


@pytest.mark.parametrize("np_,nw", [(10, 3), (11, 1), (22, 70), (43, 9), (43, 40), (85, 2), (85, 20)])
def test_batches_complex64_and_complex128(gpu, np_, nw):
    """Batches that fill clusters of 16, 8, 4 and 1 CTAs: the complex64 factors with refinement (to a residual of
    1e-13 |b|) and the complex128 factors give the same solutions, to 1e-13 times the matrices' condition (below
    1e3 for these clusters) in each."""
    ss = gpu.ScatteringSystem(jittered_square_cluster(np_, np.random.default_rng(np_)), 50e-9, -12 + 1.2j, 2.25, 1)
    om = np.linspace(1.7, 2.5, nw) * EV / HBAR
    f1 = ss.planewave_scatter_batch(om, mode=1, want_f=True)["f"]
    f0 = ss.planewave_scatter_batch(om, mode=0, want_f=True)["f"]
    assert np.all(np.linalg.norm(f1 - f0, axis=1) <= 2e-10 * np.linalg.norm(f0, axis=1))
    i = nw // 2
    M = ss(om[i]).modeproblem_matrix_full()
    k = ss(om[i]).wavenumber().real
    b = ss(om[i]).apply_Tmatrices_full(ss.planewave_full(np.array([0, 0, k]), np.array([1.0, 0, 0])))
    assert np.linalg.norm(M @ f0[i] - b) <= 1e-13 * np.linalg.norm(b)
