"""Context.kernel_launches counts the kernels of a block launch: one up to 32
members, three (assembly, factors, solves) in the families above. The family
of a size bucket is chosen by the dispatch table, so two tables differ by two
kernels per block launch."""
import pytest

from costuum_b200.tmatrix import Context

pytestmark = pytest.mark.gpu

ONE, THREE = [0, 1, 2, 3, 4], [3, 3, 3, 3, 4]


def _launches(c, table, call):
    c.set_dispatch(table)
    call()  # (tables of the orders are made once)
    before = c.kernel_launches
    call()
    return c.kernel_launches - before


def test_fixed_batch():
    c = Context(0)
    # order 12: classes of at most 8 and of 9..12 members, two block launches
    call = lambda: c.tmatrix_batch_fixed([2e-7], 1e-6, 1.5 + 0.1j, 0.8, 12, 24)
    assert _launches(c, THREE, call) - _launches(c, ONE, call) == 2 * 2
    c.close()


def test_order_loops():
    c = Context(0)
    call = lambda: c.tmatrix_batch([1e-7], 1e-6, 1.5 + 0.1j, 0.8)
    host = _launches(c, THREE, call) - _launches(c, ONE, call)
    assert host > 0 and host % 2 == 0
    c.set_batch_mode(Context.BATCH_GRAPH)
    graph = _launches(c, THREE, call) - _launches(c, ONE, call)
    assert c.last_batch_mode == Context.BATCH_GRAPH
    assert graph > 0 and graph % 2 == 0
    c.close()
