"""Frequencies of a large finite scatter and nodes of a contour on several lanes
(threads, streams, solvers): every frequency and node is solved exactly as it is
by itself, whatever the count (one lane, fewer units than lanes, a ragged last
round), and calls from several threads at once do not disturb one another."""
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


def _system(gpu, n, lMax):
    return gpu.ScatteringSystem(jittered_square_cluster(n, np.random.default_rng(n)), 50e-9, -12 + 1.2j, 2.25, lMax)


@pytest.mark.parametrize("nw", [1, 2, 3, 4, 5, 9])
def test_scatter_frequencies(gpu, nw):
    ss = _system(gpu, 40, 2)  # 640 unknowns: the dense solver
    om = np.linspace(1.7, 2.5, nw) * EV / HBAR
    r = ss.planewave_scatter_batch(om, mode=1, want_f=True, want_scat=True)
    assert np.all(r["residual"] <= 1e-12)
    for i, w in enumerate(om):
        one = ss.planewave_scatter_batch([w], mode=1, want_f=True, want_scat=True)
        # the same launches in the same order, on one lane
        assert np.array_equal(r["f"][i], one["f"][0])
        assert r["sigma_ext"][i] == one["sigma_ext"][0] and r["sigma_scat"][i] == one["sigma_scat"][0]


@pytest.mark.parametrize("nodes", [1, 2, 5])
def test_contour_nodes(gpu, nodes):
    """The sums of a node range equal the nodes' own sums (the lanes add in another order: 1e-14 of the sums' scale)."""
    from qpms_gb300 import beyn
    ss = _system(gpu, 36, 2)
    c, rr, ri = (x * EV / HBAR for x in (2.1, 0.05, 0.02))
    args = (ss.s, ss.fecv_size, c, rr, ri, 7)
    whole = beyn.scatsys_quadrature(*args, 1, 1 + nodes, 12)
    parts = [beyn.scatsys_quadrature(*args, i, i + 1, 12) for i in range(1, 1 + nodes)]
    for j in range(4):
        s = sum(p[j] for p in parts)
        scale = max(np.linalg.norm(p[j]) for p in parts)
        assert np.linalg.norm(whole[j] - s) <= 1e-14 * scale


def test_calls_from_several_threads(gpu):
    om = np.linspace(1.8, 2.4, 3) * EV / HBAR
    systems = [_system(gpu, n, 2) for n in (34, 40, 46)]
    want = [s.planewave_scatter_batch(om, mode=1, want_f=True)["f"] for s in systems]
    got = [None] * 3

    def work(i):
        for _ in range(3):
            got[i] = systems[i].planewave_scatter_batch(om, mode=1, want_f=True)["f"]
    th = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


def test_an_error_reaches_the_caller(gpu):
    with pytest.raises(Exception, match="mode"):
        _system(gpu, 40, 2).planewave_scatter_batch(np.array([2.0, 2.1]) * EV / HBAR, mode=3)
