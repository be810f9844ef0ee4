"""Rows with many consumers, and short rows, on arbitrary grids.

More than four consumers are dotted from y in shared memory, in segments of 64
tiles of 128 points: lengths and cuts around a segment and around the one to
eight tiles that give a block its warps, consumers around four and around the
warps of a block, rows of both kinds in one call, against the oracle (1e-13 of
the magnitudes that a dot adds up).  The entry point that is not told the
number of consumers gives the same to rounding.
"""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [1, 100, 128, 129, 257, 1024, 1025, 8191, 8192, 8193, 17000])
@pytest.mark.parametrize("counts", [(1, 0, 4), (4, 5, 0, 1), (7, 8, 9, 2), (33, 1, 64)])
def test_dots(n, counts):
    from atomx_b200 import _native
    from atomx_b200.quadrature import GridTables, yk_pair_dot_batch_on_grid
    rng = np.random.default_rng(n)
    r = np.geomspace(1e-6, 60.0, n) if n > 1 else np.array([0.3])
    rows, k_max = len(counts), 40
    P, Q, W = rng.normal(size=(5, n)), rng.normal(size=(5, n)), rng.normal(size=(6, n))
    a, b = rng.integers(0, 5, (2, rows))
    ks = rng.integers(0, k_max + 1, rows)
    ptr = np.concatenate([[0], np.cumsum(counts)])
    cons = rng.integers(0, 6, ptr[-1])
    ok = np.ones(rows, dtype=bool)
    for cut in (None, 0, n // 2, min(8191, n - 1)):
        ic = n - 1 if cut is None else cut
        got = yk_pair_dot_batch_on_grid(P, Q, P, Q, a, b, ks, ok, W, ptr, cons, r, i_cut=cut)
        size = np.empty_like(got)
        ref = oracle.yk_pair_dot_batch_on_grid(P, Q, P, Q, a, b, ks, ok, W, ptr, cons, r, i_cut=cut)
        for m in range(rows):
            y = oracle.yk_on_grid(P[a[m]] * P[b[m]] + Q[a[m]] * Q[b[m]], r, int(ks[m]), i_cut=cut)
            for s in range(ptr[m], ptr[m + 1]):
                size[s] = np.abs(W[cons[s], :ic + 1]) @ np.abs(y[:ic + 1])
        assert np.all(np.abs(got - ref) <= 1e-13 * size + 1e-300)
        d = [torch.as_tensor(np.ascontiguousarray(x), device="cuda") for x in
             (P, Q, a, b, ks, ok.astype(np.uint8), W, ptr, cons)]
        tab, val = GridTables.get(r, k_max, d[0].device), torch.zeros(len(got), dtype=torch.float64, device="cuda")
        work = torch.empty((1, n), dtype=torch.float64, device="cuda")
        L = _native.require_device()
        _native.check(L.rkb_grid_pair_dot_batch(
            d[0].data_ptr(), d[1].data_ptr(), d[0].data_ptr(), d[1].data_ptr(), n, d[2].data_ptr(), d[3].data_ptr(),
            d[4].data_ptr(), d[5].data_ptr(), rows, d[6].data_ptr(), n, d[7].data_ptr(), d[8].data_ptr(),
            tab.r.data_ptr(), n, tab.RK.data_ptr(), tab.inverse.data_ptr(), tab.cuts.data_ptr(), tab.ncuts,
            tab.transfers.data_ptr(), tab.ntr, ic, val.data_ptr(), work.data_ptr(), 1, _native.stream_handle()),
            "rkb_grid_pair_dot_batch")
        assert np.all(np.abs(val.cpu().numpy() - got) <= 1e-13 * size + 1e-300)
