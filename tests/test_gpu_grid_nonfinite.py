"""Non-finite samples on arbitrary grids, against the oracle's serial scans.

An infinite or NaN sample of the density at the ends, beside them, inside and
at tile edges: the same points of Y^k are infinite (with the same sign) or NaN
as in the serial scans, on grids of one frame and of many, and the finite
points agree (1e-13 of the largest).  Dots with such rows likewise.
"""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _same(got, ref):
    fin = np.isfinite(ref)
    assert np.array_equal(np.isfinite(got), fin)
    assert np.array_equal(got[~fin], ref[~fin], equal_nan=True)
    assert np.all(np.abs(got[fin] - ref[fin]) <= 1e-13 * max(np.abs(ref[fin]).max(initial=0.0), 1e-300))


@pytest.mark.parametrize("n,k,span", [(1, 2, 1.0), (2, 0, 10.0), (150, 3, 1e3), (1000, 2, 1e4), (1000, 64, 1e12)])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_same_points(n, k, span, bad):
    from atomx_b200.quadrature import yk_on_grid, yk_pair_dot_batch_on_grid
    rng = np.random.default_rng(n + k)
    r = np.geomspace(1e-6, 1e-6 * span, n) if n > 1 else np.array([0.3])
    rho = np.abs(rng.normal(size=n)) + 0.1
    w = np.ones((1, n))
    one, zero = np.ones((1, n)), np.zeros((1, n))
    for p in sorted({0, 1, 31, 127, 128, n // 2, n - 2, n - 1} & set(range(n))):
        x = rho.copy()
        x[p] = bad
        for cut in (None, n // 2):
            ref = oracle.yk_on_grid(x, r, k, i_cut=cut)
            ic = n - 1 if cut is None else cut
            _same(yk_on_grid(x, r, k, i_cut=cut), ref[:ic + 1])
            args = (x[None], zero, one, zero, np.array([0]), np.array([0]), np.array([k]), np.array([True]), w,
                    np.array([0, 1]), np.array([0]), r)
            with np.errstate(invalid="ignore"):
                _same(yk_pair_dot_batch_on_grid(*args, i_cut=cut), oracle.yk_pair_dot_batch_on_grid(*args, i_cut=cut))
