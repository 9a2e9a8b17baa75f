"""The one-launch substitution sweeps at the edges of their tiles and blocks:
last tiles of fewer than 16 rows, one block, last blocks of a few rows, one and
several right-hand sides (instances for 1, 2, 4 and 8), more of them by chunks of
eight with a short last one, both sides of the line to the tensor-core products
(32 columns, or 200,000 divided by the unknowns up to 128), complex64 and complex128
factors.

Tolerances: the systems are 2 I plus a random matrix of norm about 2 / sqrt(2),
and an FP64 refinement takes the residual to 1e-13: within 1e-10 of numpy's.
Right substitutions with complex64 factors contract the error by 2^-10 or better
per pass (5 passes at most), with complex128 ones the first pass ends at rounding
(2 at most); an entry of a wrong block stalls the refinement.
"""
import numpy as np
import pytest

import qpms_gb300

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("N", [16, 20, 63, 65, 129, 144, 257, 516, 1000, 2500])
def test_sweep_tiles(N, mode):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(N)
    M = (rng.normal(size=(N, N)) + 1j * rng.normal(size=(N, N))) / (2 * np.sqrt(N)) + 2 * np.eye(N)
    tM = torch.from_numpy(M.reshape(-1, order="F").copy()).cuda()
    Ball = rng.normal(size=(N, 131)) + 1j * rng.normal(size=(N, 131))
    ref = np.linalg.solve(M, Ball)
    for nrhs in (1, 2, 3, 4, 7, 8, 9, 32, 33, 77, 81, 128, 131):
        tB = torch.from_numpy(Ball[:, :nrhs].reshape(-1, order="F").copy()).cuda()
        tX = torch.empty_like(tB)
        res, it = np.zeros(1), np.zeros(1, dtype=np.int32)
        rc = qpms_gb300.lib().qpms_gpu_dense_solve(N, nrhs, tM.data_ptr(), tB.data_ptr(), tX.data_ptr(), mode,
                                                   res.ctypes.data, it.ctypes.data)
        assert rc == 0, qpms_gb300.last_error()
        X = tX.cpu().numpy().reshape((N, nrhs), order="F")
        assert np.linalg.norm(X - ref[:, :nrhs]) <= 1e-10 * np.linalg.norm(ref[:, :nrhs])
        assert res[0] <= 1e-12 and it[0] <= (5 if mode else 2)


_CHILD = r"""
import sys, numpy as np, torch
sys.path.insert(0, sys.argv[1])
import qpms_gb300
N, nrhs = 1500, 136
rng = np.random.default_rng(7)
M = (rng.normal(size=(N, N)) + 1j * rng.normal(size=(N, N))) / (2 * np.sqrt(N)) + 2 * np.eye(N)
B = rng.normal(size=(N, nrhs)) + 1j * rng.normal(size=(N, nrhs))
tM, tB = (torch.from_numpy(a.reshape(-1, order="F").copy()).cuda() for a in (M, B))
tX = torch.empty_like(tB)
res, it = np.zeros(1), np.zeros(1, dtype=np.int32)
rc = qpms_gb300.lib().qpms_gpu_dense_solve(N, nrhs, tM.data_ptr(), tB.data_ptr(), tX.data_ptr(), 1,
                                           res.ctypes.data, it.ctypes.data)
assert rc == 0, qpms_gb300.last_error()
X = tX.cpu().numpy().reshape((N, nrhs), order="F")
ref = np.linalg.solve(M, B)
assert np.linalg.norm(X - ref) <= 1e-10 * np.linalg.norm(ref) and it[0] <= 5
np.save(sys.argv[2], X)
"""


def test_products_past_the_line(tmp_path):
    """136 columns at 1,500 unknowns take the tensor-core products: the factors'
    digit planes cut once give bit for bit the result of cutting each step's panel."""
    import os
    import subprocess
    import sys
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = []
    for flag in ("1", "0"):
        f = str(tmp_path / ("x%s.npy" % flag))
        subprocess.run([sys.executable, "-c", _CHILD, root, f], env=dict(os.environ, QPMS_GB300_FACTOR_PLANES=flag),
                       check=True, timeout=600)
        out.append(np.load(f))
    assert np.array_equal(out[0], out[1])
