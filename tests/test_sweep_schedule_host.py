"""The schedule of the one-launch substitution sweeps (sweep_tiles in qg_dense.cu), restated in numpy.

A CTA takes tiles of 16 rows by an atomic ticket, ascending rows forward, descending backward; with more right-hand
sides than a tile holds, consecutive tickets are the chunks of one row tile.  An entry of the result is its own flag
(not a number until it is stored), looked at once ahead and then until it has arrived.  Checked under arbitrary
interleavings of few or many CTAs: the sweeps solve the system; an awaited entry always belongs to a tile of the same
chunk with an earlier ticket, so every wait ends whatever number of CTAs is resident; every entry is stored once; and
the result does not depend on the interleaving, bit for bit.
"""
import random

import numpy as np
import pytest

ROWS = 16


def _schur_lu(M, nb):
    """Schur-form block LU without pivoting: D -> I - D^-1 in its slot, its column block times D^-1."""
    A = M.copy()
    N = len(A)
    for k in range(0, N, nb):
        e = min(k + nb, N)
        Di = np.linalg.inv(A[k:e, k:e])
        A[:, k:e] = A[:, k:e] @ Di
        A[k:e, k:e] = np.eye(e - k) - Di
        A[e:, e:] -= A[e:, k:e] @ A[k:e, e:]
    return A


def _sweep(A, nb, B, NR, backward, ctas, rnd):
    N, nrhs = B.shape
    ntiles, nblk, nch = -(-N // ROWS), -(-N // nb), -(-nrhs // NR)
    Y = np.full(B.shape, np.nan, dtype=complex)
    ticket = [-1]
    owner = {}  # (row tile, chunk) -> ticket

    def cta():
        while True:
            ticket[0] += 1
            tk = ticket[0]
            if tk >= ntiles * nch:
                return
            tr, ch = divmod(tk, nch)
            tile = ntiles - 1 - tr if backward else tr
            owner[tile, ch] = tk
            row0, r1 = tile * ROWS, min((tile + 1) * ROWS, N)
            cols = slice(NR * ch, min(NR * (ch + 1), nrhs))
            j = row0 // nb
            acc = np.zeros((r1 - row0, cols.stop - cols.start), dtype=complex)
            for k in (range(nblk - 1, j, -1) if backward else range(j)):
                k0, k1 = k * nb, min((k + 1) * nb, N)
                for t in range(k0 // ROWS, -(-k1 // ROWS)):
                    assert owner[t, ch] < tk  # the awaited entries' tile
                first = Y[k0:k1, cols].copy()  # a look ahead of the wait
                yield
                while np.isnan(first).any():
                    yield
                    first = np.where(np.isnan(first), Y[k0:k1, cols], first)
                acc += A[row0:r1, k0:k1] @ first
            assert np.isnan(Y[row0:r1, cols]).all()
            value = B[row0:r1, cols] - acc
            for r in rnd.sample(range(r1 - row0), r1 - row0):  # entries arrive one by one, in any order
                Y[row0 + r, cols] = value[r]
                yield

    running = [cta() for _ in range(ctas)]
    for _ in range(2_000_000):
        if not running:
            break
        c = rnd.choice(running)
        try:
            next(c)
        except StopIteration:
            running.remove(c)
    assert not running, "a wait did not end"
    return Y


@pytest.mark.parametrize("N,nb,nrhs,NR", [(4, 64, 1, 1), (100, 64, 1, 1), (260, 128, 1, 1), (196, 64, 2, 2),
                                          (132, 64, 3, 4), (260, 128, 8, 8), (132, 64, 9, 8), (200, 128, 20, 8)])
def test_sweeps_solve(N, nb, nrhs, NR):
    rng = np.random.default_rng(N + nrhs)
    M = rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N)) + 3 * np.sqrt(N) * np.eye(N)
    b = rng.standard_normal((N, nrhs)) + 1j * rng.standard_normal((N, nrhs))
    A = _schur_lu(M, nb)
    ref = np.linalg.solve(M, b)
    results = []
    for seed, ctas in enumerate((1, 2, 7, 40)):
        rnd = random.Random(seed)
        z = _sweep(A, nb, _sweep(A, nb, b, NR, False, ctas, rnd), NR, True, ctas, rnd)
        x = np.concatenate([z[k:k + nb] - A[k:k + nb, k:k + nb] @ z[k:k + nb] for k in range(0, N, nb)])
        assert np.abs(x - ref).max() <= 1e-10 * np.abs(ref).max()
        results.append(x)
    assert all(np.array_equal(r, results[0]) for r in results)
