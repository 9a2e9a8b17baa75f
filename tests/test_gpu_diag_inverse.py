"""The LU's diagonal-block inversion at the edges of its steps and blocks.

A block is inverted eight columns a step, a cluster of CTAs holding a quarter of
its columns each: last blocks of 4, 8, 12 ... columns end in a partial step or in
any of the four CTAs, 64- and 128-wide blocks (128 for many right-hand sides) and
complex128 ones take different instances.

Tolerances: the systems are 2 I plus a random matrix of norm about 2 / sqrt(2),
condition below 100 or so at these sizes, and the solution comes out of an FP64
refinement to a residual of 1e-13: within 1e-10 of numpy's.  A complex64 inverse
that is right contracts the error by 2^-10 or better per pass, so 1e-13 takes at
most 5 passes; a wrong one stalls and needs the complex128 factors.
"""
import numpy as np
import pytest

import qpms_gb300

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("N", [4, 8, 12, 31, 36, 60, 64, 68, 72, 96, 100, 124, 128, 132, 140, 160, 196, 260])
def test_partial_blocks(N, mode):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(N)
    M = (rng.normal(size=(N, N)) + 1j * rng.normal(size=(N, N))) / (2 * np.sqrt(N)) + 2 * np.eye(N)
    for nrhs in (1, 48):
        B = rng.normal(size=(N, nrhs)) + 1j * rng.normal(size=(N, nrhs))
        tM, tB = (torch.from_numpy(a.reshape(-1, order="F").copy()).cuda() for a in (M, B))
        tX = torch.empty_like(tB)
        res, it = np.zeros(1), np.zeros(1, dtype=np.int32)
        rc = qpms_gb300.lib().qpms_gpu_dense_solve(N, nrhs, tM.data_ptr(), tB.data_ptr(), tX.data_ptr(), mode,
                                                   res.ctypes.data, it.ctypes.data)
        assert rc == 0, qpms_gb300.last_error()
        ref = np.linalg.solve(M, B)
        X = tX.cpu().numpy().reshape((N, nrhs), order="F")
        assert np.linalg.norm(X - ref) <= 1e-10 * np.linalg.norm(ref)
        assert res[0] <= 1e-12 and it[0] <= 5
