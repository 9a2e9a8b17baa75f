"""The roundings of the batched substitutions (qg_batchlu.cu): an unknown's many small products are summed before they
are taken off its right-hand side.

A row of a unit triangle with up to 63 products of half a unit roundoff each, on a right-hand side of 1: subtracted
one by one every product is rounded away (1 - u/2 is 1), summed first none is.  Tolerance: one unit in the last place
below 1, for the rounding of the sum and of the difference.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qpms_gb300
    return qpms_gb300


def batch_lu(gpu, A, b):
    A, b = A.copy(), b.copy()
    nm, N = b.shape
    piv = np.zeros((nm, N), dtype=np.int32)
    f = C.CDLL(gpu.lib()._name).qpms_gpu_debug_batch_lu
    f.argtypes = [C.c_int, C.c_int, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p]
    rc = f(int(A.dtype == np.complex128), nm, N, A.ctypes.data, piv.ctypes.data, b.ctypes.data)
    assert rc == 0, gpu.last_error()
    return A, piv, b


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("upper", [False, True])
@pytest.mark.parametrize("N", [2, 17, 31, 32, 33, 64, 65, 96, 97, 130, 512])
def test_small_products_are_summed_first(gpu, N, upper, dtype):
    half = 12 if dtype == np.complex64 else 27
    l, y, u = 2.0 ** -half, 2.0 ** -(25 - 12 if dtype == np.complex64 else 27), 2.0 ** -(25 if dtype == np.complex64 else 54)
    width = N if N <= 64 else 32
    rows = [min(r + width, N) - 1 for r in range(0, N, width)]  # the last row of each triangle
    if upper:
        rows = [r for r in range(0, N, width)]
    M = np.eye(N, dtype=dtype)
    b = np.full((2, N), y, dtype=dtype)
    b[1] *= 1j
    want = b.copy()
    for r in rows:
        others = range(r + 1, min(r + width, N)) if upper else range(r - r % width, r)
        M[r, list(others)] = l
        b[:, r] = want[:, r] = (1, 1j)
        want[:, r] *= 1 - len(others) * u
    A, piv, x = batch_lu(gpu, np.stack([M, M]), b)
    assert np.array_equal(A, np.stack([M, M])) and np.array_equal(piv, np.tile(np.arange(N, dtype=np.int32), (2, 1)))
    assert np.abs(x - want).max() <= 2 * u
