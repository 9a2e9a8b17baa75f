"""The field kernel at the edges of its tiles (8 particles, 128 points) for every
lMax and Bessel kind, real and complex wavenumbers, with points on the particles'
polar axes, against the oracle.

Tolerance: the kernel and the oracle sum the same waves in different bases, each
term's rounding error a few ulp of the largest wave of its particle; 1e-12 of
the field's norm covers up to 17 particles of 96 waves (17 * 96 * 2^-53 * 5 =
9e-13).
"""
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


@pytest.mark.parametrize("lMax", range(1, 7))
@pytest.mark.parametrize("J,k", [(3, 1.7e7), (3, 1.7e7 + 2e5j), (1, 1.3e7), (1, 1.3e7 + 3e5j), (2, 1.1e7), (4, 1.2e7)])
def test_edges_of_tiles(gpu, lMax, J, k):
    from oracle import orc
    rng = np.random.default_rng(lMax)
    for np_, npts in ((1, 1), (8, 129), (9, 3), (17, 127)):
        pos = np.stack([np.arange(np_) * 300e-9, rng.uniform(-1e-7, 1e-7, np_), rng.uniform(-1e-7, 1e-7, np_)], 1)
        pts = rng.uniform(-6e-7, 6e-7, (npts, 3)) + [0, 8e-7, 0]
        pts[0] = pos[0] + [0, 0, 4e-7]           # polar axes, both ends
        if npts > 2:
            pts[1] = pos[0] - [0, 0, 3e-7]
            pts[2] = pos[np_ // 2] + [2e-7, 0, 0]
        f = rng.normal(size=(np_, 2 * lMax * (lMax + 2), 2)).reshape(-1, 2) @ [1, 1j]
        ss = gpu.ScatteringSystem(pos, 50e-9, -12 + 1.2j, 2.25, lMax)
        E = ss.scattered_E(k, f, pts, btyp=J)
        O = orc.scattered_E(lMax, pos, J, k, f, pts)
        assert np.linalg.norm(E - O) <= 1e-12 * np.linalg.norm(O), (np_, npts)


@pytest.mark.parametrize("lMax", [1, 3, 6])
def test_regular_waves_at_their_origin(gpu, lMax):
    from oracle import orc
    rng = np.random.default_rng(lMax)
    pos = np.array([[1e-7, 2e-7, 3e-7]])
    f = rng.normal(size=(2 * lMax * (lMax + 2), 2)) @ [1, 1j]
    ss = gpu.ScatteringSystem(pos, 50e-9, -12 + 1.2j, 2.25, lMax)
    E = ss.scattered_E(1.3e7, f, pos, btyp=1)
    O = orc.scattered_E(lMax, pos, 1, 1.3e7, f, pos)
    assert np.linalg.norm(E - O) <= 1e-13 * np.linalg.norm(O)
    assert np.isnan(ss.scattered_E(1.3e7, f, pos, btyp=3)).any()
