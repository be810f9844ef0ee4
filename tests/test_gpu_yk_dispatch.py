"""Y^k rows at the row counts where the kernel changes are equal to the bit.

A block per row is taken up to 16 rows per SM without a power table, up to 12
with one, and up to 8 from 13 nodes a cell on; no table is read below five
nodes a cell.  Rows of each count, with and without a table, densities given or formed
from orbital pairs, against a launch of 3 rows per SM, which every node count
sends to the block form.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("ng", [2, 4, 5, 8, 12, 13, 17])
def test_rows_around_the_limits(ng):
    from atomx_b200 import _native
    from atomx_b200.yk import yk_partial_matrices
    L = _native.require_device()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    nv, k_max, n_orb = 37, 6, 9
    n, ld = nv * ng, nv * ng + 5
    gen = torch.Generator(device="cuda").manual_seed(ng)

    def rand(*shape):
        return torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64)
    r, w = torch.sort(20 * rand(n) + 1e-3).values, 0.02 * rand(n)
    mo, mi = (torch.as_tensor(m.copy(), device="cuda") for m in yk_partial_matrices(ng))
    pw = torch.empty(2 * (k_max + 1) * n, dtype=torch.float64, device="cuda")
    top = 16 * sms + 1
    rho, P, Q = rand(top, n) - 0.5, rand(n_orb, n) - 0.5, rand(n_orb, n) - 0.5
    ks = torch.randint(0, k_max + 1, (top,), generator=gen, device="cuda", dtype=torch.int32)
    pairs = torch.randint(0, n_orb, (n_orb * n_orb, 2), generator=gen, device="cuda", dtype=torch.int64)
    pair = torch.randint(0, n_orb * n_orb, (top,), generator=gen, device="cuda", dtype=torch.int64)

    def given(rows, table):
        y = torch.full((rows, ld), 7.0, dtype=torch.float64, device="cuda")
        _native.check(L.rkb_yk_rows_pow(rho.data_ptr(), n, ks.data_ptr(), rows, r.data_ptr(), w.data_ptr(), nv, ng,
                                        mo.data_ptr(), mi.data_ptr(), y.data_ptr(), ld,
                                        pw.data_ptr() if table else 0, k_max if table else -1,
                                        _native.stream_handle()), "rkb_yk_rows_pow")
        return (y,)

    def formed(rows, table):
        g, y = (torch.full((rows, ld), 7.0, dtype=torch.float64, device="cuda") for _ in range(2))
        _native.check(L.rkb_table_rows_fp64_pow(P.data_ptr(), Q.data_ptr(), n, pairs.data_ptr(), pair.data_ptr(),
                                                ks.data_ptr(), rows, r.data_ptr(), w.data_ptr(), nv, ng,
                                                mo.data_ptr(), mi.data_ptr(), g.data_ptr(), y.data_ptr(), ld,
                                                pw.data_ptr() if table else 0, k_max if table else -1,
                                                _native.stream_handle()), "rkb_table_rows_fp64_pow")
        return g, y

    for f in (given, formed):
        few = f(3 * sms, False)
        assert all(not bool(x[:, n:].any()) for x in few)
        for per_sm in (8, 12, 16):
            for rows in (per_sm * sms, per_sm * sms + 1):
                for table in (False, True):
                    got = f(rows, table)
                    for a, b in zip(got, few):
                        assert torch.equal(a[:3 * sms], b)
        # the whole of the largest count, block form against warp form, a power table against none
        parts = [f(top, t) for t in (False, True)]
        assert all(torch.equal(a, b) for a, b in zip(*parts))
