"""The field kernel rounds once per particle at the size of the sum.

A particle of field E and n others of equal small fields, each the sum of two waves (l = 0 and 2 of the cartesian
form) of 0.4 units in the last place of E: added wave by wave they vanish, added as particles each is rounded once.
Tolerance: half a unit per particle, and 8 units for the fields themselves.
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


def _axis(x):
    """Re E_z of the electric wave (1, 0) on its axis: sqrt(6 / 4 pi) j_1(x) / x."""
    x = np.longdouble(x)
    return np.sqrt(6 / (4 * np.longdouble(np.pi))) * (np.sin(x) / x ** 2 - np.cos(x) / x) / x


def test_a_particle_is_rounded_once(gpu):
    import torch
    n, k, npts = 100, 1.3e7, 5_000_000  # enough points that no list of particles is split
    ra, rb = 1.1 / k, 2.42 / k          # j_0 = j_2 at kr = 2.46
    pos = np.array([[0, 0, -ra]] + [[0, 0, -rb]] * n)
    ss = gpu.ScatteringSystem(pos, 50e-9, -12 + 1.2j, 2.25, 1)
    f = np.zeros((n + 1, 6), dtype=complex)
    Ea, Eb = _axis(k * np.longdouble(ra)), _axis(k * np.longdouble(rb))
    f[0, 1] = float(1.5 / Ea)
    f[1:, 1] = 0.8 * 2.0 ** -52 / float(Eb)
    want = float(f[0, 1].real * Ea - np.longdouble(1.5)) + n * 0.8 * 2.0 ** -52
    cvf = torch.tensor(f.ravel(), device="cuda")
    E = ss.scattered_E_device(k, cvf, torch.zeros((npts, 3), dtype=torch.float64, device="cuda"))
    got = E[:, 2].real - 1.5
    assert (got == got[0]).all()
    assert abs(float(got[0]) - want) <= (0.5 * n + 8) * 2.0 ** -52
