"""A matrix so small that the dense solver's diagonal blocks cannot be inverted in the factors' type (the square of a
pivot is zero) is refused as one with a zero pivot, not answered with numbers that are none; one scaled within the
type's range is solved.  (Matrices far above 1 are not: a block and its inverse share a slot as I - D^-1.)  Residuals:
1e-10, a hundred times the solver's stagnation level for these matrices."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(N, exp, mode):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qpms_gb300
    rng = np.random.default_rng(N)
    A = (rng.normal(size=(N, N)) + 1j * rng.normal(size=(N, N))) * 2.0 ** exp
    M = torch.tensor(A.T.copy(), device="cuda")  # column-major
    b = torch.ones(N, dtype=torch.complex128, device="cuda")
    x = torch.empty_like(b)
    res, it = np.zeros(1), np.zeros(1, dtype=np.int32)
    rc = qpms_gb300.lib().qpms_gpu_dense_solve(N, 1, M.data_ptr(), b.data_ptr(), x.data_ptr(), mode, res.ctypes.data,
                                               it.ctypes.data)
    return rc, qpms_gb300.last_error(), np.linalg.norm(A @ x.cpu().numpy() - 1) / np.sqrt(N) if rc == 0 else None


@pytest.mark.parametrize("N", [64, 128, 132, 300])
@pytest.mark.parametrize("mode,exp", [(1, -83), (1, -300), (0, -600)])
def test_too_small_is_refused(N, mode, exp):
    rc, message, _ = _solve(N, exp, mode)
    assert rc != 0 and "zero pivot" in message


@pytest.mark.parametrize("N", [64, 128, 132, 300])
@pytest.mark.parametrize("mode,exp", [(1, 0), (1, -40), (0, 0), (0, -400)])
def test_within_range_is_solved(N, mode, exp):
    rc, message, res = _solve(N, exp, mode)
    assert rc == 0, message
    assert res <= 1e-10
