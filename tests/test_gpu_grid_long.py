"""Grids whose tiles' sums do not fit in shared memory (above 1 638 400 points)
against the oracle: rows and dots, below and above the limit.  1e-13 of the
largest value, or of the magnitudes that a dot adds up.
"""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [1_638_400, 1_638_401, 1_700_003])
def test_long_grid(n):
    from atomx_b200.quadrature import yk_on_grid, yk_pair_dot_batch_on_grid
    r = np.geomspace(1e-6, 60.0, n)
    f = [np.cos(c * np.log(r)) * np.exp(-r / 9) for c in (1.0, 2.5, 4.0)]
    P = np.stack(f)
    Q = 0.1 * P[::-1].copy()
    W = np.stack([f[0], f[2]])
    a, b, ks = np.array([0, 1, 2]), np.array([1, 1, 0]), np.array([0, 2, 1])
    ptr, cons = np.array([0, 2, 3, 5]), np.array([0, 1, 1, 0, 1])
    got = yk_pair_dot_batch_on_grid(P, Q, P, Q, a, b, ks, np.ones(3, dtype=bool), W, ptr, cons, r)
    for m in range(3):
        rho = P[a[m]] * P[b[m]] + Q[a[m]] * Q[b[m]]
        y = oracle.yk_on_grid(rho, r, int(ks[m]))
        if m == 0:
            assert np.max(np.abs(yk_on_grid(rho, r, int(ks[m])) - y)) <= 1e-13 * np.abs(y).max()
        for s in range(ptr[m], ptr[m + 1]):
            assert abs(got[s] - W[cons[s]] @ y) <= 1e-13 * (np.abs(W[cons[s]]) @ np.abs(y))
