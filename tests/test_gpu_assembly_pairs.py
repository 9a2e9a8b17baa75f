"""The finite assembly over unordered pairs: single particles, odd counts, chunks
that a batch of frequencies cuts in the middle, mixed particle kinds (the row
scaling of (R, C) and (C, R) differs), out-of-plane positions (both parities of
the harmonics) and particles above one another (the polar axis), for every lMax,
against the oracle (1e-10 Frobenius, the matrices' parity tolerance; and
elementwise to 1e-9 where an element is above 1e-9 of the largest)."""
import numpy as np
import pytest

from qpms_gb300.workloads import C0, EV, HBAR

pytestmark = pytest.mark.gpu
EPS = (-12 + 1.2j, 3.0 + 0.1j)
RAD = (50e-9, 40e-9)


@pytest.fixture(scope="module")
def gpu():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qpms_gb300
    return qpms_gb300


@pytest.mark.parametrize("lMax", range(1, 7))
@pytest.mark.parametrize("np_", [1, 2, 3, 8, 13])
def test_matrix(gpu, lMax, np_):
    from oracle import orc
    rng = np.random.default_rng(10 * lMax + np_)
    pos = np.stack([np.arange(np_) * 3e-7, rng.uniform(-1, 1, np_) * 2e-7, rng.uniform(-1, 1, np_) * 2e-7], 1)
    if np_ > 2:
        pos[2] = pos[0] + [0, 0, 3.5e-7]  # on the polar axis of particle 0
    kinds = (np.arange(np_) % 2).astype(np.int32)
    ss = gpu.ScatteringSystem(pos, list(RAD), list(EPS), 2.25, lMax, kinds=kinds)
    om = 2.05 * EV / HBAR * (1 + 0.01j)
    M = ss(om).modeproblem_matrix_full()
    T = np.stack([np.diag(orc.tmatrix_sphere_diag(lMax, RAD[k], om, EPS[k], 2.25)) for k in kinds])
    O = orc.finite_modeproblem(orc.TransCalculator(lMax), pos, T, np.sqrt(2.25 + 0j) * om / C0)
    assert np.linalg.norm(M - O) <= 1e-10 * np.linalg.norm(O)
    big = np.abs(O) > 1e-9 * np.abs(O).max()
    assert np.all(np.abs(M - O)[big] <= 1e-9 * np.abs(O)[big] + 1e-13 * np.abs(O).max())


@pytest.mark.parametrize("nw", [1, 7])
def test_batch_equals_single_matrices(gpu, nw):
    """Frequencies of one batch through the scatter: its residual is formed with the batch's matrices, sigma_scat with
    the regular-wave matrix (Bessel kind 1, T = -1) of the same kernel; each matrix by itself must give the same."""
    rng = np.random.default_rng(3)
    pos = rng.uniform(-1, 1, (5, 3)) * 6e-7
    ss = gpu.ScatteringSystem(pos, list(RAD), list(EPS), 2.25, 2, kinds=np.array([0, 1, 1, 0, 1], dtype=np.int32))
    om = np.linspace(1.7, 2.4, nw) * EV / HBAR
    r = ss.planewave_scatter_batch(om, mode=0, want_f=True, want_scat=True)
    for i, w in enumerate(om):
        k = 1.5 * w / C0
        M = ss(w).modeproblem_matrix_full()
        a = ss.planewave_full(np.array([0, 0, k]), np.array([1.0, 0, 0]))
        b = ss(w).apply_Tmatrices_full(a)
        f = r["f"][i]
        assert np.linalg.norm(M @ f - b) <= 1e-12 * np.linalg.norm(b)
        R = ss.translation_matrix_full(k, J=1)
        sc = np.vdot(f, f + R @ f).real / k ** 2
        assert abs(r["sigma_scat"][i] - sc) <= 1e-11 * abs(sc)
