"""The convergence test of a group of orders (1, 4 or 8 per launch, 128 threads
per CTA) at the list lengths where the group or the CTA changes: a grain's
orders, status and m = 0 sums do not depend on the grains beside it, so every
batch equals the first grains of the largest one bit for bit."""
import numpy as np
import pytest

import _helpers as H

pytestmark = pytest.mark.gpu

GRAINS = H.config2_sample(300, 11)


@pytest.fixture(scope="module")
def whole(ctx):
    r, lam, m, d = GRAINS
    return ctx.tmatrix_batch(r, lam, m, d)


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 32, 33, 65, 127, 128, 129])
def test_batch_equals_prefix_of_a_larger_one(ctx, whole, n):
    r, lam, m, d = GRAINS
    res = ctx.tmatrix_batch(r[:n], lam, m[:n], d[:n])
    assert np.array_equal(res.nmax, whole.nmax[:n])
    assert np.array_equal(res.status, whole.status[:n])
    assert np.array_equal(res.q[:, [0, 1, 4, 5]], whole.q[:n, [0, 1, 4, 5]])
