"""Block rounds on the two round streams after a change of the batch size: the
Q sums of grains above order 24 are shared by several CTAs, whose counters are
laid out and cleared for each batch size. Every batch equals the same grains in a
fresh context bit for bit."""
import numpy as np
import pytest

import _helpers as H
from costuum_b200.tmatrix import Context

pytestmark = pytest.mark.gpu


def _run(c, n):
    r, lam, m, d = H.config2_sample(1600, 17, xmin=14.0, xmax=28.0)
    return c.tmatrix_batch(r[:n], lam, m[:n], d[:n], min_order=25)


def test_q_sums_after_a_smaller_batch():
    sizes = (1600, 1100, 1600, 700)
    want = {}
    for n in set(sizes):
        c = Context(0)
        want[n] = _run(c, n)
        c.close()
    c = Context(0)
    c.profile(True)
    _run(c, min(sizes))
    # (the batches have rounds on both round streams)
    assert {1, 2} <= set(c.timeline()["stream"])
    c.profile(False)
    for n in sizes:
        got = _run(c, n)
        assert np.all(got.nmax > 24)
        for a, b in ((got.nmax, want[n].nmax), (got.status, want[n].status),
                     (got.q, want[n].q)):
            assert np.array_equal(a, b)
    c.close()
