"""Scratch of the tangents: classes of at most 32 members keep their matrices
in shared memory, so only larger ones take device memory."""
import numpy as np
import pytest

from costuum_b200.tmatrix import Context, tmatrix_size

pytestmark = pytest.mark.gpu

LAM = 1e-6


def _fixed(c, orders):
    N = np.array(orders)
    r = 0.5 * N * LAM / (2 * np.pi)
    c.tmatrix_batch_fixed(r, LAM, 1.4 + 0.02j, 1.2, N, 2 * N)


def test_gradients_of_mixed_orders():
    orders = [40, 9, 33, 70, 32, 34, 12]
    th = [0.4, 1.1]
    c = Context(0)
    _fixed(c, orders)
    q, dq = (a.copy() for a in c.gradients(th))
    for i, n in enumerate(orders):
        _fixed(c, [n])
        q1, dq1 = c.gradients(th)
        assert np.array_equal(q1[0], q[i]) and np.array_equal(dq1[0], dq[i])
    c.close()


def test_no_scratch_for_small_classes():
    import torch
    n, order = 512, 24
    c = Context(0)
    _fixed(c, [order] * n)
    before = torch.cuda.mem_get_info()[0]
    c.gradients([0.4])
    grown = before - torch.cuda.mem_get_info()[0]
    c.close()
    # the three tangents, and T and its tangents averaged in half the size, each
    # with the quarter that buffers grow by; 100 MB for all else
    assert grown <= 1.25 * (3 + 4 / 2) * n * tmatrix_size(order) * 16 + 100e6
