"""The cell row kernel with few rows: a block per row, equal to the bit.

Rows of one ion from the start of a multipole, across changes of multipole and
to the end, in launches that a block takes row by row, against the launch over
all rows, which takes several a block: residues, scales, core vectors and row
records.
"""
import dataclasses

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("ng", [5, 8, 9, 11])
def test_row_by_row(ng):
    from atomx_b200 import _native
    from atomx_b200 import workloads as W
    from atomx_b200.split import CB_STRIDE, SplitEngine
    from atomx_b200.tables import upload_ion
    L = _native.require_device()
    spec = dataclasses.replace(W.uneven_batch()[1], ns=60, n_gauss=ng, ks=min(ng, 9), k_max=6,
                               shells=W._spread(40, W.kappa_ladder(5)))
    dev = upload_ion(W.build_ion(spec))
    eng = SplitEngine(dev, rows_kernel="cells")
    plan, R = dev.plan, eng.ion_rows
    rows = (4 if ng <= 8 else 2) * torch.cuda.get_device_properties(0).multi_processor_count
    assert plan.n_rows > 2 * rows
    eng.rows()
    starts = [plan.k_row_offset[k] for k in plan.ks]
    for q0, m in ((0, 1), (starts[1] - 3, 7), (starts[2] - 1, rows), (plan.n_rows - 5, 5), (plan.n_rows - rows, rows)):
        A = torch.full_like(eng.resA, 99)
        B = torch.full_like(eng._resB, 99) if eng._resB is not None else None
        rs, lf, rt, cb = (torch.full_like(t, 7.0) for t in (eng.rowscale, eng.left, eng.right, eng.cbound))
        _native.check(L.rkb_split_rows_cells_z(
            dev.Pv.data_ptr(), dev.Qv.data_ptr(), dev.n, dev.pairs.data_ptr(), dev.row_pair.data_ptr() + 8 * q0,
            dev.row_k.data_ptr() + 4 * q0, m, dev.w.data_ptr(), dev.nv, dev.ng, R.ktab.data_ptr(), R.koff.data_ptr(),
            R.ktab_t.data_ptr(), R.koff_t.data_ptr(), R.max_z, eng.bits, eng.n_mod, eng._mod_c[0], A.data_ptr(),
            _native.ptr(B), eng.kpad, eng.b_col0, eng.b_ld, q0, eng.rows_alloc, rs.data_ptr(), lf.data_ptr(),
            rt.data_ptr(), cb.data_ptr(), eng.cwp, _native.stream_handle()), "rkb_split_rows_cells_z")
        s = slice(q0, q0 + m)
        assert torch.equal(A[:, s], eng.resA[:, s])
        assert B is None or torch.equal(B[:, s], eng._resB[:, s])
        for got, want in ((rs, eng.rowscale), (lf, eng.left), (rt, eng.right),
                          (cb.view(-1, CB_STRIDE), eng.cbound.view(-1, CB_STRIDE))):
            assert torch.equal(got[s], want[s]) and bool((got[:q0] == 7.0).all()) and bool((got[q0 + m:] == 7.0).all())
        assert bool((A[:, :q0] == 99).all()) and bool((A[:, q0 + m:] == 99).all())
