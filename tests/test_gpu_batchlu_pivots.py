"""Pivots of the batched LU: the largest |Re| + |Im| of a column, compared as exactly as in FP64, the first of equals;
complex64 numbers whose FP32 sums are equal or overflow included.  Columns are built so that the choice decides the
whole sequence: candidates sit in one column of an otherwise diagonal matrix."""
import numpy as np
import pytest

from test_gpu_batchlu_rounding import batch_lu, gpu  # noqa: F401

pytestmark = pytest.mark.gpu

F = np.float32
TINY, BIG = F(2.0 ** -149), F(3e38)
COLUMNS = [  # candidates in rows, the best one
    ([1 + 1e-8j, 1 + 5e-8j, 1 + 4e-8j], 1),                 # all sums round to 1
    ([1 - 5e-8j, -1 - 4e-8j, 4e-8 + 1j], 0),
    ([F(1.5) + F(2.0 ** -24) * 1j, F(1.5) + F(2.0 ** -24) * 1j], 0),   # equal: the first
    ([F(1.0) + F(2.0 ** -23) * 1j, F(1.0) + F(2.9e-7) * 1j, F(1.0) + F(2.6e-7) * 1j], 1),
    ([0.75 + 0.25j, 0.5 + 0.5j, 0.25 + 0.75j], 0),
    ([BIG + F(2e38) * 1j, BIG + F(2.5e38) * 1j, BIG + F(2.2e38) * 1j], 1),  # past FP32's range
    ([TINY * F(3) + TINY * 1j, TINY * F(2) + TINY * F(3) * 1j], 1),
    ([0.0, 1e-30, 0.5e-30j], 1),
]


@pytest.mark.parametrize("N", [8, 40, 64, 70, 200, 512])
@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
def test_best_of_close_candidates(gpu, N, dtype):  # noqa: F811
    Ms, want = [], []
    for col, best in COLUMNS:
        for c in sorted({0, N // 2, N - len(col)}):
            for step in sorted({1, max(1, (N - c) // len(col))}):  # next to each other, and over other threads' rows
                rows = [c + i * step for i in range(len(col))]
                M = np.zeros((N, N), dtype=dtype)
                M[np.arange(N), np.arange(N)] = 1
                M[c:, c] = 0
                M[rows, c] = np.array(col, dtype=np.complex64)
                Ms.append(M)
                want.append((c, rows[best]))
    Ms = np.stack(Ms)
    A, piv, _ = batch_lu(gpu, Ms, np.ones((len(Ms), N), dtype=dtype))
    for i, (c, r) in enumerate(want):
        assert piv[i, c] == r, (i, c, r, piv[i, c])
