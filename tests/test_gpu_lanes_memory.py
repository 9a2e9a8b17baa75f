"""Contour sums and scatters have the same bits on however many lanes the free memory allows: with nearly all memory
free (two lanes of nodes, four of frequencies), and with 1.2 and 2 GB left of it (3,000 unknowns take 0.4 GB a lane;
a call's lanes share half of what is free)."""
import numpy as np
import pytest

from qpms_gb300.workloads import EV, HBAR, jittered_square_cluster

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def system():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import qpms_gb300
    pos = jittered_square_cluster(100, np.random.default_rng(3))
    return torch, qpms_gb300.ScatteringSystem(pos, 50e-9, -12 + 1.2j, 2.25, 3)


def _with_left(torch, left, f):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    block = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
    try:
        return f()
    finally:
        torch.cuda.synchronize()
        del block
        torch.cuda.empty_cache()


def test_contour_sums(system):
    from qpms_gb300 import beyn
    torch, ss = system
    c, rr, ri = (x * EV / HBAR for x in (2.1, 0.05, 0.02))

    def sums():
        return beyn.scatsys_quadrature(ss.s, ss.fecv_size, c, rr, ri, 7, 0, 5, 12)[:4]
    want = sums()
    for left in (1200 << 20, 2 << 30):
        for a, b in zip(_with_left(torch, left, sums), want):
            assert np.array_equal(a, b)


def test_scatters(system):
    torch, ss = system
    om = np.linspace(1.8, 2.4, 5) * EV / HBAR

    def f():
        return ss.planewave_scatter_batch(om, mode=1, want_f=True)["f"]
    want = f()
    for left in (1200 << 20, 2 << 30):
        assert np.array_equal(_with_left(torch, left, f), want)
