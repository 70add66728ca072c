"""Contexts made after others were closed take over their streams and memory
pool: results, memory and concurrent use are those of fresh contexts."""
import threading

import numpy as np
import pytest

import _helpers as H
from costuum_b200.tmatrix import Context

pytestmark = pytest.mark.gpu

GRAINS = H.config2_sample(40, 3)


def _run(graph=False, grad=False):
    c = Context(0)
    try:
        if graph:
            c.set_batch_mode(Context.BATCH_GRAPH)
        r, lam, m, d = GRAINS
        res = c.tmatrix_batch(r, lam, m, d)
        obs = c.observables([0.3, 1.2])
        out = [res.nmax, res.q, np.array(obs)]
        if grad:
            out.append(np.array(c.gradients([0.3, 1.2])[1]))
        return out
    finally:
        c.close()


@pytest.mark.parametrize("graph", [False, True])
def test_results_of_reused_contexts(graph):
    first = _run(graph, True)
    for _ in range(3):
        for a, b in zip(first, _run(graph, True)):
            assert np.array_equal(a, b)


def test_memory_goes_back():
    import torch
    _run(True, True)
    free0 = torch.cuda.mem_get_info()[0]
    for _ in range(6):
        _run(True, True)
    # at most four idle contexts with 32 MB each, and what the driver rounds to
    assert free0 - torch.cuda.mem_get_info()[0] <= 4 * (32 << 20) + (64 << 20)


def test_threads_with_contexts_of_their_own():
    want = _run()
    got, errors = {}, []

    def work(k):
        try:
            for j in range(4):
                got[k, j] = _run()
        except Exception as e:  # noqa: BLE001 (reported below)
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert len(got) == 24
    for out in got.values():
        for a, b in zip(want, out):
            assert np.array_equal(a, b)
