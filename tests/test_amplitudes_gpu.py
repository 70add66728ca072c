"""The amplitude kernels (k_amp, k_azimuth) against a plain numpy contraction
of the downloaded T-matrices, at orders around the tile and launch edges
(8, 16, 32, 64 rows; four- and sixteen-angle groups)."""
import numpy as np
import pytest

from costuum_b200.tmatrix import Context, block

pytestmark = pytest.mark.gpu

LAM = 1e-6
EPS = 2.0 ** -53


def _angular(cost, N, m):
    """(m d / sin, d') of d^n_{0m} for n = max(m, 1) .. N, [angles, n]."""
    s = np.sqrt((1 - cost) * (1 + cost))
    prev, cur = np.zeros_like(cost), np.ones_like(cost)
    for i in range(1, m + 1):
        cur = cur * np.sqrt((2 * i - 1) / (2 * i)) * s
    p, t = [], []
    for n in range(m, N + 1):
        a, b = np.sqrt(n * n - m * m), np.sqrt((n + 1) ** 2 - m * m)
        nxt = ((2 * n + 1) * cost * cur - a * prev) / b
        if n > 0:
            p.append(m * cur / s)
            t.append((n * b * nxt - (n + 1) * a * prev) / ((2 * n + 1) * s))
        prev, cur = cur, nxt
    return np.array(p).T, np.array(t).T


def _amplitudes(T, N, k, cin, cout, phi):
    """S[4, pairs] and the sums of the terms' magnitudes (the scale of the
    rounding errors) for pairs (cin[i], cout[i], phi[i])."""
    S, scale = np.zeros((4, len(cin)), complex), np.zeros(len(cin))
    for m in range(N + 1):
        n = np.arange(max(m, 1), N + 1)
        a = np.sqrt((2.0 * n + 1) / (n * (n + 1.0)))
        c = np.tile(1j ** ((n[None, :] - n[:, None] - 1) % 4) * np.outer(a, a), (2, 2))
        B = block(T, N, m) * c
        (pi, ti), (po, to) = _angular(cin, N, m), _angular(cout, N, m)
        v = [np.hstack([pi, ti]), np.hstack([ti, pi])]
        u = [np.hstack([po, to]), np.hstack([to, po])]
        f = (2.0 if m else 1.0) * np.cos(m * phi)
        g = (2.0 if m else 0.0) * np.sin(m * phi)
        w = (f, g, -g, f)
        for q in range(4):
            y = v[q % 2] @ B.T
            S[q] += w[q] * np.sum(u[q // 2] * y, axis=1)
            scale += 2 * np.sum(np.abs(u[q // 2]) * (np.abs(v[q % 2]) @ np.abs(B).T), axis=1)
    return S / k, scale / k


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("orders,ntheta", [
    ([1, 2, 7, 8, 9], 1), ([10, 15, 16, 17], 4), ([31, 32, 33, 5], 5),
    ([12, 24], 16), ([12, 40, 3], 17), ([63, 64, 65], 33), ([100, 128], 9)])
def test_extinction_of_downloaded_tmatrices(ctx, orders, ntheta):
    N = np.array(orders)
    x = np.maximum(0.5, 0.55 * N)
    r, k = x * LAM / (2 * np.pi), 2 * np.pi / LAM
    res = ctx.tmatrix_batch_fixed(r, LAM, 1.4 + 0.02j, 1.1, N, 2 * N)
    assert np.all(res.status == 0)
    theta = np.linspace(0.21, 2.9, ntheta)
    q = ctx.observables(theta)
    for i, n in enumerate(orders):
        S, scale = _amplitudes(res.tmatrix(i), n, k, np.cos(theta), np.cos(theta),
                               np.zeros(ntheta))
        f = 2 * np.pi / k / (np.pi * r[i] ** 2)
        ref = f * np.stack([(S[0] + S[3]).imag, (S[0] - S[3]).imag, (S[3] - S[0]).real], 1)
        # sums of 2 (2 n + 2) n products whose factors carry the rounding of
        # recurrences of n steps
        tol = f * scale * EPS * 16 * (n + 4)
        assert np.all(np.abs(q[i] - ref) <= tol[:, None])


@pytest.mark.parametrize("nin,nout", [(1, 181), (3, 5), (17, 2)])
def test_angle_pairs_of_one_grain(ctx, nin, nout):
    n, x = 20, 9.0
    r, k = x * LAM / (2 * np.pi), 2 * np.pi / LAM
    res = ctx.tmatrix_batch_fixed([r], LAM, 1.5 + 0.01j, 0.8, n, 2 * n)
    ti, to = np.linspace(0.3, 2.8, nin), np.linspace(0.25, 2.7, nout)
    ti, to = (v.ravel() for v in np.meshgrid(ti, to, indexing="ij"))
    phi = np.linspace(-2.0, 3.0, ti.size)
    Z = ctx.scattering_matrix(0, ti, 0.0, to, phi)
    S, scale = _amplitudes(res.tmatrix(0), n, k, np.cos(ti), np.cos(to), phi)
    # Z00 = (|S11|^2 + |S12|^2 + |S21|^2 + |S22|^2) / 2 and Z33, of amplitudes
    # with errors d: 4 |S| d each; e^{i m phi} adds m roundings
    d = scale * EPS * 16 * (2 * n + 4)
    tol = 4 * np.max(np.abs(S), axis=0) * d + 4 * d * d
    assert np.all(np.abs(Z[:, 0, 0] - 0.5 * np.sum(np.abs(S) ** 2, axis=0)) <= tol)
    z33 = (S[3] * S[0].conj() - S[1] * S[2].conj()).real
    assert np.all(np.abs(Z[:, 3, 3] - z33) <= tol)
