"""The batched LU over its types' range: a matrix scaled by a power of two has the same multipliers and pivots, pivots
scaled by it and solutions scaled by its inverse, bit for bit, as long as no number leaves the normal range; at 2^+-N
where the square of a pivot leaves it too (FP32: past 2^+-63, FP64: past 2^+-511)."""
import numpy as np
import pytest

from test_gpu_batchlu_rounding import batch_lu, gpu  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 6, 40, 64, 65, 200, 512])
@pytest.mark.parametrize("dtype,exps", [(np.complex64, [-70, -62, -50, 50, 62, 75]),
                                        (np.complex128, [-900, -560, -515, -400, 400, 515, 560, 900])])
def test_powers_of_two(gpu, N, dtype, exps):  # noqa: F811
    rng = np.random.default_rng(N)
    M = (rng.normal(size=(1, N, N)) + 1j * rng.normal(size=(1, N, N))).astype(dtype)
    b = (rng.normal(size=(1, N)) + 1j * rng.normal(size=(1, N))).astype(dtype)
    real = M.real.dtype.type
    A, piv, x = batch_lu(gpu, M, b)
    L = np.tril(A[0], -1)
    for e in exps:
        f = real(2) ** real(e)
        A2, piv2, x2 = batch_lu(gpu, M * f, b)
        assert np.array_equal(piv, piv2)
        assert np.array_equal(np.tril(A2[0], -1), L)
        assert np.array_equal(np.triu(A2[0]), np.triu(A[0]) * f)
        assert np.array_equal(x2 * f, x)
