"""The assembly, factor and solve kernels of the classes above 32 members at
the edges of their tiles (32 rows and columns, 64 rows per solve) and around
the largest class whose factors fit shared memory (118 members): blocks
m = 0, 1, 2 against the oracle, within the T tolerance of the parity tests or
four times the oracle's own change under a 1e-15 change of r_ev."""
import numpy as np
import pytest

import _helpers as H
import oracle as O
from costuum_b200 import tmatrix as TM

pytestmark = pytest.mark.gpu

LAM, M, D = 1e-6, 1.4 + 0.02j, 1.1


def _blocks(r, N):
    T0, _, _ = O.tmatrix_m0(r, LAM, M, D, N, 2 * N)
    return [T0.ravel()] + [O.tmatrix_mblock(r, LAM, M, D, N, 2 * N, m).ravel()
                           for m in (1, 2)]


@pytest.mark.parametrize("N", [33, 63, 64, 65, 66, 97, 118, 119, 128])
def test_blocks_at_tile_edges(ctx, N):
    r = 0.6 * N * LAM / (2 * np.pi)
    ref = _blocks(r, N)
    near = [_blocks(r * (1 + e), N) for e in (1e-15, -1e-15)]
    res = ctx.tmatrix_batch_fixed([r], LAM, M, D, N, 2 * N)
    assert res.status[0] == 0
    T = res.tmatrix(0)
    for m, b in enumerate(ref):
        norm = np.linalg.norm(b)
        own = max(np.linalg.norm(c[m] - b) for c in near) / norm
        err = np.linalg.norm(TM.block(T, N, m).ravel() - b) / norm
        assert err <= max(H.T_TOL, 4 * own), (m, err, own)
