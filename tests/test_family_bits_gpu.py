"""The block-kernel families for at most 64 members round alike: a grain has the
same T-matrix, bit for bit, whichever of them runs a size bucket. (The family
for at most 128 members applies the row and column factors in another place, so
it is left out.)"""
import numpy as np
import pytest

from costuum_b200.tmatrix import Context

pytestmark = pytest.mark.gpu

LAM = 1e-6


@pytest.mark.parametrize("bucket,orders,families", [
    (0, [6, 7, 8], [0, 1, 2, 3]), (1, [9, 15, 16], [1, 2, 3]), (2, [17, 31, 32], [2, 3])])
def test_same_bits(bucket, orders, families):
    N = np.array(orders * 4)
    rng = np.random.default_rng(bucket)
    x = rng.uniform(0.3, 0.7, N.size) * N
    d = np.exp(rng.uniform(-0.7, 0.7, N.size))
    m = rng.uniform(1.3, 2.0, N.size) + 1j * 10 ** rng.uniform(-3, 0, N.size)
    c = Context(0)
    first = None
    for f in families:
        table = [0, 1, 2, 3, 4]
        table[bucket] = f
        c.set_dispatch(table)
        res = c.tmatrix_batch_fixed(x * LAM / (2 * np.pi), LAM, m, d, N, 2 * N)
        assert np.all(res.status == 0)
        T = [res.tmatrix(i) for i in range(N.size)]
        first = first or T
        for a, b in zip(first, T):
            assert np.array_equal(a, b), f
    c.close()
