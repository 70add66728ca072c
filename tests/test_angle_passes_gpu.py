"""More distinct angles than one pass of the amplitude kernels holds (512 MB of
pi and tau columns: 2032 angles at order 128, 13107 at order 50): every pass
gives what calls of fewer angles give, bit for bit where those have the same
groups of 16 angles, and the memory is bounded."""
import numpy as np
import pytest

import oracle as O  # noqa: F401 (the helpers' path)
from test_amplitudes_gpu import _amplitudes
from costuum_b200.tmatrix import Context

pytestmark = pytest.mark.gpu

LAM = 1e-6
K = 2 * np.pi / LAM
ORDERS = [128, 17, 64]


@pytest.fixture(scope="module")
def batch():
    c = Context(0)
    N = np.array(ORDERS)
    r = 0.55 * N * LAM / (2 * np.pi)
    res = c.tmatrix_batch_fixed(r, LAM, 1.4 + 0.02j, 1.1, N, 2 * N)
    assert np.all(res.status == 0)
    yield c, res, r
    c.close()


def test_observables_of_many_angles(batch):
    c, res, r = batch
    theta = np.linspace(0.2, 2.9, 2032 * 2 + 7)
    q = c.observables(theta).copy()
    for i0 in range(0, theta.size, 94 * 16):
        part = slice(i0, i0 + 94 * 16)
        assert np.array_equal(q[:, part], c.observables(theta[part]))
    # values around the passes' edges (groups of 16 angles)
    pick = np.array([0, 2015, 2016, 2031, 2032, 2033, 4031, 4032, 4063, 4064, 4070])
    for i, n in enumerate(ORDERS):
        S, scale = _amplitudes(res.tmatrix(i), n, K, np.cos(theta[pick]),
                               np.cos(theta[pick]), np.zeros(pick.size))
        f = 2 * np.pi / K / (np.pi * r[i] ** 2)
        ref = f * np.stack([(S[0] + S[3]).imag, (S[0] - S[3]).imag, (S[3] - S[0]).real], 1)
        # (as in the test of fewer angles)
        tol = f * scale * 2.0 ** -53 * 16 * (n + 4)
        assert np.all(np.abs(q[i, pick] - ref) <= tol[:, None])


def test_gradients_of_many_angles():
    c = Context(0)
    N = np.array([100, 17])
    c.tmatrix_batch_fixed(0.55 * N * LAM / (2 * np.pi), LAM, 1.4 + 0.02j, 1.1, N, 2 * N)
    theta = np.linspace(0.2, 2.9, 3322 + 40)
    q, dq = (a.copy() for a in c.gradients(theta))
    for part in (slice(0, 1600), slice(1600, None)):
        q1, dq1 = c.gradients(theta[part])
        assert np.array_equal(q[:, part], q1) and np.array_equal(dq[:, part], dq1)
    c.close()


def test_memory_of_many_angles():
    import torch
    c = Context(0)
    n = 128
    c.tmatrix_batch_fixed([0.55 * n * LAM / (2 * np.pi)], LAM, 1.4 + 0.02j, 1.1, n, 2 * n)
    before = torch.cuda.mem_get_info()[0]
    c.observables(np.linspace(0.2, 2.9, 8000))
    grown = before - torch.cuda.mem_get_info()[0]
    c.close()
    # 512 MB of columns, 264 MB of m sums (8000 x 129 x 4), each with the quarter
    # that buffers grow by; 100 MB for all else
    assert grown <= 1.25 * (512 * 2 ** 20 + 8000 * 129 * 4 * 16) + 100e6


def _directions(nj):
    return np.random.default_rng(4).uniform(0.1, 3.0, (6, nj))


def test_directions_of_many_jobs(batch):
    # two angles of their own per job, the grains' jobs mixed: several passes
    c, res, _ = batch
    nj = 6000
    ti, pi, to, po = _directions(nj)[:4]
    g = np.arange(nj) % len(ORDERS)
    Z = c.scattering_matrix(g, ti, pi, to, po)
    for i, n in enumerate(ORDERS):
        # the same pairs alone, in groups of the same 16
        own = np.flatnonzero(g == i)
        for i0 in range(0, own.size, 800):
            p = own[i0:i0 + 800]
            assert np.array_equal(Z[p], c.scattering_matrix(i, ti[p], pi[p], to[p], po[p]))
        pick = own[[0, 1, 15, 16, 503, 504, 505, 1007, 1008, 1009, 1999]]
        S, scale = _amplitudes(res.tmatrix(i), n, K, np.cos(ti[pick]), np.cos(to[pick]),
                               po[pick] - pi[pick])
        # (as in the test of one grain's angle pairs)
        d = scale * 2.0 ** -53 * 16 * (2 * n + 4)
        tol = 4 * np.max(np.abs(S), axis=0) * d + 4 * d * d
        assert np.all(np.abs(Z[pick, 0, 0] - 0.5 * np.sum(np.abs(S) ** 2, axis=0)) <= tol)


def test_a_pass_costs_its_own_launches(batch):
    # at order 128 a pass holds 1016 such jobs; another one adds its columns,
    # four sizes of blocks and the azimuths, and the T-matrices are not copied
    # again
    c, _, _ = batch

    def launches(nj):
        a = _directions(nj)
        before = c.kernel_launches
        c.scattering_matrix(0, *a[:4])
        return c.kernel_launches - before
    assert launches(2000) - launches(1000) <= 6
    assert launches(3000) - launches(2000) <= 6
