"""Bessel tables in every layout of their launch: small orders with a CTA per
kind, others with a warp per kind, slots of one node count packed, ratios in
shared memory or in the output by the launch's share of orders up to 64. A
grain's T-matrix is the same, bit for bit, whichever it was."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LAM = 1e-6


def _run(ctx, orders):
    N = np.array(orders)
    r = 0.5 * N * LAM / (2 * np.pi)
    res = ctx.tmatrix_batch_fixed(r, LAM, 1.5 + 0.03j, 0.8, N, 2 * N)
    assert np.all(res.status == 0)
    return [res.tmatrix(i) for i in range(len(orders))], res.q


@pytest.mark.parametrize("orders", [
    [7, 9, 16], [5, 24, 17, 9],    # a CTA per kind, 32 and 64 nodes
    [1, 25, 31, 32, 33, 64],       # a warp per kind, all in shared memory
    [10] * 7, [17] * 5, [16] * 2, [70] * 3,  # one node count
    [64] * 3 + [65],               # more than a quarter of the work is
    [12, 64, 100, 100, 66],        # less than a quarter
    [65, 128]])                    # none
def test_mixed_orders(ctx, orders):
    T, q = _run(ctx, orders)
    for i, n in enumerate(orders):
        if i > 2 and n == orders[0]:
            assert np.array_equal(T[i], T[0])  # (equal grains)
            continue
        # beside a small grain and beside a large one
        for other in (2, 90):
            T1, q1 = _run(ctx, [n, other])
            assert np.array_equal(T[i], T1[0]), (n, other)
            assert np.array_equal(q[i, 2:4], q1[0, 2:4]), (n, other)
