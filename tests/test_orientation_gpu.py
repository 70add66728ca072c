"""The orientation-average kernel (k_orient) against a plain numpy contraction
of the downloaded T-matrices with Clebsch-Gordan rows from the eigenvectors of
J^2, at orders around its tiles and launch ranges (8, 15/16, 31/32, 63/64) and
with 1, 2, 4, 5, 8 and 9 grains (chunks of 2, 4 and 8 per warp), averaged and
copied grains mixed."""
import numpy as np
import pytest

from costuum_b200 import CosTuuM
from costuum_b200.tmatrix import block

pytestmark = pytest.mark.gpu

LAM = 1e-6


def _rows(n1, n2):
    """<n1 m n2 -m | N 0>, N = |n1 - n2| .. n1 + n2 (up to a sign), m = 0 .. M."""
    M = min(n1, n2)
    m = np.arange(-M, M + 1)
    diag = n1 * (n1 + 1) + n2 * (n2 + 1) - 2.0 * m * m
    off = np.sqrt((n1 * (n1 + 1) - m[:-1] * m[1:]) * (n2 * (n2 + 1.0) - m[:-1] * m[1:]))
    _, v = np.linalg.eigh(np.diag(diag) + np.diag(off, 1) + np.diag(off, -1))
    return v.T[:, M:]


def _average(T, N, p, pairs):
    """{(i1, n1, i2, n2): averaged elements m = 0 .. M} of the given pairs."""
    out = {}
    for n1, n2 in pairs:
        M, par = min(n1, n2), (n1 + n2) % 2
        C = _rows(n1, n2)[par::2]
        pN = p[abs(n1 - n2):n1 + n2 + 1][par::2]
        m = np.arange(M + 1)
        sg, f = (-1.0) ** m, np.where(m == 0, 1.0, 2.0)
        for i1 in (0, 1):
            i2 = i1 ^ par
            t = np.array([block(T, N, k)[i1 * (N + 1 - max(k, 1)) + n1 - max(k, 1),
                                         i2 * (N + 1 - max(k, 1)) + n2 - max(k, 1)]
                          for k in m])
            out[i1, n1, i2, n2] = sg * (C.T @ (pN * (C @ (f * sg * t))))
    return out


@pytest.mark.parametrize("orders", [
    [1], [7, 8], [9, 15, 16, 17], [31, 32, 33, 8, 1], [10] * 8, [12, 24, 40] * 3,
    [63, 64, 65]])
def test_average_of_downloaded_tmatrices(ctx, orders):
    N = np.array(orders)
    r = np.maximum(0.5, 0.5 * N) * LAM / (2 * np.pi)
    d = np.where(np.arange(N.size) % 2, 0.9, 1.2)
    res = ctx.tmatrix_batch_fixed(r, LAM, 1.4 + 0.02j, d, N, 2 * N)
    assert np.all(res.status == 0)
    T = [res.tmatrix(i) for i in range(N.size)]
    sets = np.stack([CosTuuM.MishchenkoOrientationDistribution(c, 2 * N.max()).coefficients
                     for c in (0.6, 0.2)])
    which = np.where(np.arange(N.size) % 3 == 2, -1, np.arange(N.size) % 2)
    ctx.orientation_average(sets, which)
    rng = np.random.default_rng(5)
    for i, n in enumerate(orders):
        Ta = res.tmatrix(i)
        if which[i] < 0:
            assert np.array_equal(Ta, T[i])
            continue
        pairs = {(1, 1), (1, n), (n, 1), (n, n), (max(1, n - 1), n), (n, max(1, n - 1))}
        pairs |= {tuple(v) for v in rng.integers(1, n + 1, (12, 2))}
        for (i1, n1, i2, n2), want in _average(T[i], n, sets[which[i]], pairs).items():
            got = np.array([block(Ta, n, k)[i1 * (n + 1 - max(k, 1)) + n1 - max(k, 1),
                                            i2 * (n + 1 - max(k, 1)) + n2 - max(k, 1)]
                            for k in range(min(n1, n2) + 1)])
            # rows of unit norm: two products of M + 1 terms, weights p <= 1, and
            # table entries from recurrences of n1 + n2 steps
            scale = 2 * np.max(np.abs(T[i]))
            assert np.all(np.abs(got - want) <= 64 * (n1 + n2) * 2.0 ** -53 * scale)
