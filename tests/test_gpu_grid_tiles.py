"""Tiles, frames and consumers of the arbitrary-grid kernel at their edges.

Grid lengths around the warp chunks (32) and tiles (128), ranks that give
many frames (a frame spans a factor e^(128/(k+1)), so frame starts fall at
tile edges and inside chunks), rows with more consumers than one pass takes,
and cuts of the output, against the oracle's serial scans.  Tolerance as for
every result of this kernel: 1e-13 of the largest value of a result, here of
the sum of the magnitudes that a dot adds up (|W| . |Y|).
"""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [1, 2, 31, 33, 127, 128, 129, 256, 385, 1000])
@pytest.mark.parametrize("k_max,span", [(3, 1e4), (64, 1e12), (200, 1e9)])
def test_rows_and_dots(n, k_max, span):
    from atomx_b200.quadrature import coulomb_tables, yk_on_grid, yk_pair_dot_batch_on_grid
    rng = np.random.default_rng(n + k_max)
    r = np.geomspace(1e-6, 1e-6 * span, n) if n > 1 else np.array([0.3])
    rows, waves = 9, 4
    PA, QA, PB, QB = (rng.normal(size=(waves, n)) for _ in range(4))
    W = rng.normal(size=(3, n))
    a, b = rng.integers(0, waves, rows), rng.integers(0, waves, rows)
    ks = rng.integers(0, k_max + 1, rows)
    ks[0] = k_max
    if n > 300 and k_max > 3:
        assert coulomb_tables(r, k_max)[2].shape[0] > 3  # several frames
    ok = np.ones(rows, dtype=bool)
    ok[4] = False
    ptr = np.concatenate([[0], np.cumsum([1, 2, 3, 4, 5, 0, 8, 9, 1])])
    cons = rng.integers(0, 3, ptr[-1])
    for cut in (None, 0, n // 2, n - 1):
        args = (PA, QA, PB, QB, a, b, ks, ok, W, ptr, cons, r)
        got = yk_pair_dot_batch_on_grid(*args, i_cut=cut)
        ref = oracle.yk_pair_dot_batch_on_grid(*args, i_cut=cut)
        ic = n - 1 if cut is None else cut
        for m in range(rows):
            rho = PA[a[m]] * PB[b[m]] + QA[a[m]] * QB[b[m]]
            y = oracle.yk_on_grid(rho, r, int(ks[m]), i_cut=cut)
            if cut != 0 and m < 3:
                mine = yk_on_grid(rho, r, int(ks[m]), i_cut=cut)
                assert np.max(np.abs(mine - y[:ic + 1])) <= 1e-13 * max(np.max(np.abs(y[:ic + 1])), 1e-300)
            for s in range(ptr[m], ptr[m + 1]):
                size = np.abs(W[cons[s], :ic + 1]) @ np.abs(y[:ic + 1])
                assert abs(got[s] - ref[s]) <= 1e-13 * size + 1e-300, (m, s)
