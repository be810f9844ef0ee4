"""Y^k rows do not depend on the path that a row count takes.

Few rows go through a block per row, more through a warp per row, with the
nodes' powers evaluated or read from a table: every product and sum is the
same in the same order, so the rows are equal to the bit, over node counts
(compiled and general), cells around the chunks of 32, and beyond the sixteen
chunks that a block takes.  Against the oracle: 1e-13 of each row's largest.
"""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("ng", [1, 2, 5, 8, 11, 14, 17])
@pytest.mark.parametrize("nv", [1, 31, 32, 33, 100, 513])
def test_paths_agree(ng, nv):
    from atomx_b200 import _native
    from atomx_b200.yk import compute_yk, compute_yk_rows, yk_partial_matrices
    L = _native.require_device()
    rng = np.random.default_rng(100 * ng + nv)
    edges = np.concatenate([[0.0], np.geomspace(1e-3, 30.0, nv)])
    x, w = np.polynomial.legendre.leggauss(ng)
    half = 0.5 * np.diff(edges)[:, None]
    gr, grw = 0.5 * (edges[1:] + edges[:-1])[:, None] + half * x, half * w
    n, rows, k_max = nv * ng, 1500, 12
    rho = rng.normal(size=(rows, n)) * np.exp(-gr.reshape(1, -1) / 5)
    ks = rng.integers(0, k_max + 1, rows).astype(np.int32)
    d = torch.as_tensor(rho, device="cuda")
    many = compute_yk_rows(d, ks, gr, grw)                       # a warp per row, power table
    few = compute_yk_rows(d[:40].contiguous(), ks[:40], gr, grw)  # a block per row where it fits
    one = compute_yk(d[7].view(nv, ng), gr, grw, nv, ng, int(ks[7]))
    assert torch.equal(many[:40], few) and torch.equal(one.reshape(-1), many[7])
    mo, mi = (torch.as_tensor(m.copy(), device="cuda") for m in yk_partial_matrices(ng))
    r, wt = (torch.as_tensor(a.reshape(-1), device="cuda") for a in (gr, grw))
    kt = torch.as_tensor(ks, device="cuda")
    ld = n + 3
    for short in (None, 4):  # powers evaluated; a table that ends before some rows' multipole
        pw = None if short is None else torch.empty(2 * (short + 1) * n, dtype=torch.float64, device="cuda")
        out = torch.full((rows, ld), 7.0, dtype=torch.float64, device="cuda")
        _native.check(L.rkb_yk_rows_pow(d.data_ptr(), n, kt.data_ptr(), rows, r.data_ptr(), wt.data_ptr(), nv, ng,
                                        mo.data_ptr(), mi.data_ptr(), out.data_ptr(), ld, _native.ptr(pw),
                                        -1 if short is None else short, _native.stream_handle()), "rkb_yk_rows_pow")
        assert torch.equal(out[:, :n], many) and not bool(out[:, n:].any())
    ref = oracle.yk_rows(rho[:40], ks[:40], gr, grw, nv, ng)
    got = few.cpu().numpy()
    assert np.all(np.abs(got - ref) <= 1e-13 * np.abs(ref).max(axis=1, keepdims=True))
