"""The translation kernel at the edges of its chunks: batches of one translation,
of a few more than the resident CTAs, and ragged ones, for every lMax.  The
elements that reciprocity pairs are each compared with the oracle, which forms
them one by one (1e-11 of the matrix norm, the arrays' parity tolerance), for
normalisations that break the pairs' symmetry too."""
import numpy as np
import pytest

from qpms_gb300.workloads import translation_vectors

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qpms_gb300
    return qpms_gb300


def _compare(gpu, lMax, norm, n, J):
    from oracle import orc
    kr, th, ph = translation_vectors(n, seed=n + lMax)
    A, B = gpu.trans_calculator(lMax, norm).get_AB_arrays(kr, th, ph, False, J)
    pick = np.unique(np.concatenate([np.arange(min(n, 12)), np.arange(max(0, n - 12), n), np.arange(0, n, 97)]))
    oA, oB = orc.TransCalculator(lMax, norm).get_AB_batch(kr[pick], th[pick], ph[pick], J)
    for G, O in ((A[pick], oA), (B[pick], oB)):
        err = np.linalg.norm((G - O).reshape(len(pick), -1), axis=1)
        assert np.all(err <= 1e-11 * np.linalg.norm(O.reshape(len(pick), -1), axis=1))
        assert np.all(np.abs(G - O) <= 1e-11 * np.abs(O) + 1e-13 * np.abs(O).max(axis=(1, 2), keepdims=True))


@pytest.mark.parametrize("lMax", range(1, 11))
@pytest.mark.parametrize("n", [1, 457, 1000])
def test_chunks(gpu, lMax, n):
    _compare(gpu, lMax, 65536 | 8, n, 3)


@pytest.mark.parametrize("norm", [65536, 32768 | 65536 | 8, 65536 | 8 | 16, 65536 | 8 | 32, 65536 | 8 | 128])
@pytest.mark.parametrize("J", [1, 2, 4])
def test_normalisations(gpu, norm, J):
    _compare(gpu, 4, norm, 65, J)


@pytest.mark.parametrize("lMax", [1, 3, 6, 7])
def test_nan_everywhere_at_zero_distance(gpu, lMax):
    kr = np.array([1.0, 0.0, 2.0 + 0.1j])
    A, B = gpu.trans_calculator(lMax).get_AB_arrays(kr, 0.3, 0.4, False, 3)
    assert np.isnan(A[1]).all() and np.isnan(B[1]).all()
    assert np.isfinite(A[[0, 2]]).all() and np.isfinite(B[[0, 2]]).all()
