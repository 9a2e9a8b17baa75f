"""Contours of one lane, whose solver captures its launches, beside other threads' work on the legacy default stream:
neither disturbs the other (a blocking stream under capture makes every call on the legacy stream fail), and the
results are those of the calls by themselves, bit for bit."""
import threading

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


def test_contours_beside_scatters(gpu):
    a = (np.arange(8) - 3.5) * 400e-9
    X, Y = np.meshgrid(a, a, indexing="ij")
    pos = np.stack([X.ravel(), Y.ravel(), 0 * X.ravel()], 1)
    sym = gpu.ScatteringSystem(pos, 50e-9, -12 + 1.2j, 2.25, 2, sym="D4h")
    ss = gpu.ScatteringSystem(jittered_square_cluster(40, np.random.default_rng(0)), 50e-9, -12 + 1.2j, 2.25, 2)
    c, rr, ri = (x * EV / HBAR for x in (2.1, 0.05, 0.02))
    iri = int(np.argmax(sym.saecv_sizes))

    def contour():
        r = sym.find_modes(c, rr, ri, iri=iri, contour_points=8, l=12, seed=7, mode=1, rank_tol=0.0)
        return np.asarray(r["ranktest_SV"])

    def scatter():  # one frequency: no lanes, the legacy default stream
        return ss.planewave_scatter_batch([2.0 * EV / HBAR], mode=1, want_f=True)["f"]
    want = contour(), scatter()
    errors, stop = [], threading.Event()

    def beside():
        try:
            while not stop.is_set():
                assert np.array_equal(scatter(), want[1])
        except Exception as e:
            errors.append(e)
    th = threading.Thread(target=beside)
    th.start()
    try:
        for _ in range(6):
            assert np.array_equal(contour(), want[0])
    finally:
        stop.set()
        th.join()
    assert not errors, errors
