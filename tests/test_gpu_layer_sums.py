"""Lattice sums between planes on both sides of the rule that picks their form.

Pairs of planes at |k dz| >= 2.5, and nearer ones whose reciprocal sum has at most
4,000 points, take the reciprocal-lattice sum; the others take Ewald's split sum.
Checked against the oracle at |k dz| and at the number of points just below and
above the line, lMax 1 to 4 (58, 63, 68, 72 over |dz| is the largest |beta + K|), both
signs of dz, lossy media, and a lattice whose index rows are too long for the phase
tables.  Tolerance: 1e-11 of the arrays' norms, that of the shifted sums elsewhere
(the split sums cancel by up to e^2, eta is chosen so).
"""
import ctypes as C
import math

import numpy as np
import pytest

import qpms_gb300

pytestmark = pytest.mark.gpu
CUT = {1: 58, 2: 63, 3: 68, 4: 72}


class _Cplx(C.Structure):
    _fields_ = [("re", C.c_double), ("im", C.c_double)]


class _Cart2(C.Structure):
    _fields_ = [("x", C.c_double), ("y", C.c_double)]


class _Cart3(C.Structure):
    _fields_ = [("x", C.c_double), ("y", C.c_double), ("z", C.c_double)]


def _line(lMax, area):
    return CUT[lMax] * math.sqrt(area / (4000 * 4 * math.pi))


CASES = [(lMax, 2.3 + im * 1j, 1.6, (1.0, 0.0), f * _line(lMax, 1.0) * s)
         for lMax in (1, 2, 3, 4) for f, s, im in ((0.98, 1, 0.0), (1.02, -1, 0.0), (1.02, 1, 0.1))]
CASES += [(2, 2.45 / 0.2, 5.0, (1.0, 0.0), 0.2), (2, 2.55 / 0.2, 5.0, (1.0, 0.0), -0.2),
          (3, 2.55 / 0.2 + 0.2j, 5.0, (1.0, 0.0), 0.2), (2, 9.0, 1.6, (10.0, 0.0), 0.3),
          (1, 9.0 + 0.1j, 1.6, (10.0, 0.0), -0.3)]


@pytest.mark.parametrize("lMax,k,eta,b1,dz", CASES)
def test_layer_sums(orc, lMax, k, eta, b1, dz):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    L = C.CDLL(qpms_gb300.lib()._name)
    f = L.qpms_trans_calculator_get_AB_arrays_e32
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_ssize_t, C.c_ssize_t, C.c_double,
                  _Cplx, _Cart2, _Cart2, _Cart2, _Cart3, C.c_double, C.c_double]
    norm, beta, b2 = 65536 | 8, (0.7, -0.4), (0.0, 1.0)
    kc, shift = complex(k), (0.2, 0.45, dz)
    calc = qpms_gb300.trans_calculator(lMax, norm)
    ne = lMax * (lMax + 2)
    A, B = (np.zeros((ne, ne), dtype=np.complex128) for _ in range(2))
    rc = f(calc.c, A.ctypes.data, None, B.ctypes.data, None, ne, 1, eta, _Cplx(kc.real, kc.imag), _Cart2(*b1),
           _Cart2(*b2), _Cart2(*beta), _Cart3(*shift), 60.0, 500.0)
    assert rc == 0, qpms_gb300.last_error()
    Ao, Bo = orc.get_AB_arrays_e32(orc.TransCalculator(lMax, norm), eta, kc, b1, b2, beta, shift, 60, 500)
    assert np.linalg.norm(A - Ao) <= 1e-11 * np.linalg.norm(Ao)
    assert np.linalg.norm(B - Bo) <= 1e-11 * np.linalg.norm(Bo)
