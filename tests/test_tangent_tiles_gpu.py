"""Tangents at the edges of the tile kernels: fixed orders around 8, 16 and 32
(a class of m = 0 or 1 has as many members as the order) and node counts with
every remainder of a chunk of four, against central differences of the GPU
forward. The tolerance of test_gradients_gpu applies: 1e-6 up to order 16,
1e-5 above, where the difference quotient resolves no more."""
import numpy as np
import pytest

import oracle as O
import test_gradients_gpu as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nmax,extra", [
    (2, 1), (3, 2), (7, 3), (8, 0), (9, 1), (15, 2), (16, 3), (17, 0),
    (24, 1), (31, 2), (32, 3), (33, 0)])
def test_tangents_at_class_sizes(ctx, nmax, extra):
    lam = 1e-6
    # size parameters whose series end near this order
    x = {2: 0.05, 3: 0.2, 7: 2.0, 8: 2.5, 9: 3.0, 15: 7.0, 16: 8.0, 17: 8.5,
         24: 14.0, 31: 19.5, 32: 20.0, 33: 21.0}[nmax]
    r = np.array([x, 0.9 * x]) * lam / (2 * np.pi)
    m = np.array([1.5 + 0.05j, 1.35 + 0.2j])
    d = np.array([1.3, 0.8])
    n = np.full(2, nmax)
    ng = np.full(2, 2 * nmax + 4 + extra)
    coeffs = O.orientation_coefficients(2, 0.5, 2 * nmax + 2)
    ctx.tmatrix_batch_fixed(r, lam, m, d, n, ng)
    q, dq = ctx.gradients(G.THETAS, coeffs)
    params = np.stack([m.real, m.imag, r, d], axis=1)
    fds = [G._fd_gpu(ctx, params, lam, n, ng, coeffs, rel)
           for rel in (1e-6, 1e-5, 3e-5)]
    G._compare(dq, fds, q, tol=1e-6 if nmax <= 16 else 1e-5)
