"""One object per particle: what an object takes from the device fits what the
idle context before it kept, so that no memory is mapped or returned from one
object to the next (each time up to tens of ms)."""
import gc

import numpy as np
import pytest

from costuum_b200 import CosTuuM

pytestmark = pytest.mark.gpu

LAM = 1e-6


def _particle(x):
    t = CosTuuM.TMatrix(x * LAM / (2 * np.pi), 0.6, LAM, 1.5 + 0.02j)
    t.get_scattering_matrix(0.3, 0.0, np.linspace(0.0, np.pi, 181), 0.5)
    t.get_absorption_cross_sections(np.linspace(0.2, 1.4, 5), 20)
    return t


@pytest.mark.parametrize("x", [1.0, 5.0, 11.0])
def test_objects_take_over_memory(x):
    import torch
    for _ in range(2):
        t = _particle(x)
        del t
        gc.collect()
    idle = torch.cuda.mem_get_info()[0]
    t = _particle(x)
    assert abs(torch.cuda.mem_get_info()[0] - idle) <= 2 << 20
    del t
