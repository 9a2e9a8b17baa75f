"""The oracle's lattice sums between planes far apart, against a plane-wave sum written out here.

With w = -shift.z, q = beta + K, gamma = sqrt(q^2 / k^2 - 1) on the outgoing branch (-i sqrt(1 - q^2 / k^2) for
propagating orders), the sum of h_n P_n^|m| e^{i m phi} e^{i beta.(R - s)} over the plane's lattice is
  (-i)^(n+1) 2 pi / (k^2 A) sum_K e^{i K.s} e^{-gamma k |w|} / gamma P_n^|m|(i sgn(w) gamma) (-1)^m e^{i m alpha}
(alpha the angle of q; times (-1)^m for m < 0; the Condon-Shortley phase of P cancels the first (-1)^m).  An order decays as e^{-sqrt(q^2 - k^2) |w|}: the orders left out here, past
q^2 = k^2 + (160 / w)^2, are below 1e-60.  Tolerance 1e-12 of the largest value of each
degree n: the phases, up to k |w| = 150, carry that times 2^-53 each.
"""
import cmath
import math

import numpy as np
import pytest


def far_sum(lMax_e, k, b1, b2, beta, shift):
    k = complex(k)
    area = b1[0] * b2[1] - b1[1] * b2[0]
    r1 = np.array([b2[1], -b2[0]]) * 2 * math.pi / area
    r2 = np.array([-b1[1], b1[0]]) * 2 * math.pi / area
    w = -shift[2]
    pmax = math.sqrt(k.real ** 2 + (160 / abs(w)) ** 2)
    lim = pmax + math.hypot(*beta)
    I1, I2 = (int(lim * math.hypot(*b) / (2 * math.pi)) + 2 for b in (b1, b2))
    i, j = np.meshgrid(np.arange(-I1, I1 + 1), np.arange(-I2, I2 + 1), indexing="ij")
    K = i[..., None] * r1 + j[..., None] * r2
    q = K + np.array(beta)
    keep = np.hypot(q[..., 0], q[..., 1]) <= pmax
    K, q = K[keep], q[keep]
    st = np.hypot(q[:, 0], q[:, 1]) / k  # sin(theta)
    gam = np.sqrt(st - 1 + 0j) * np.sqrt(st + 1)
    if k.imag == 0:
        gam = np.where(st.real < 1, -1j * np.abs(gam), gam)
    else:
        gam = np.where((gam * k).real < 0, -gam, gam)
    x, alpha = 1j * math.copysign(1, w) * gam, np.arctan2(q[:, 1], q[:, 0])
    f = np.exp(1j * (K @ np.array(shift[:2]))) * np.exp(-gam * k * abs(w)) / gam
    out = np.zeros((lMax_e + 1) ** 2, dtype=complex)
    for m in range(lMax_e + 1):
        P = math.prod(range(1, 2 * m, 2)) * st ** m
        Pm = np.zeros_like(P)
        for n in range(m, lMax_e + 1):
            if n > m:
                P, Pm = ((2 * n - 1) * x * P - (n + m - 1) * Pm) / (n - m), P
            c = cmath.exp(-1j * cmath.pi / 2 * (n + 1)) * 2 * math.pi / (k * k * area)
            out[n * (n + 1) + m] = c * np.sum(f * P * np.exp(1j * m * alpha))
            out[n * (n + 1) - m] = (-1) ** m * c * np.sum(f * P * np.exp(-1j * m * alpha)) if m else out[n * (n + 1)]
    return out


OBLIQUE = ((1.0, 0.0), (0.3, 1.1))


@pytest.mark.parametrize("kz", [5, 20, 45, 57, 60, 65, 72, 80, 90, 150])
@pytest.mark.parametrize("k,sign", [(9.0, 1), (9.0, -1), (9.0 + 0.02j, -1)])
def test_oracle_keeps_the_slow_orders(orc, k, sign, kz):
    dz = sign * kz / abs(k)
    shift = (0.31, -0.2, dz)
    want = far_sum(9, k, *OBLIQUE, (0.7, -0.4), shift)
    got = orc.ewald_sigma_xy(9, np.inf, k, *OBLIQUE, (0.7, -0.4), shift, 20, 160)[0]
    for n in range(10):
        w = want[n * n:(n + 1) ** 2]
        assert np.abs(got[n * n:(n + 1) ** 2] - w).max() <= 1e-12 * np.abs(w).max()
