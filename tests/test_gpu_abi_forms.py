"""Entry points of the C interface that the package itself no longer calls.

Each against the form that the package runs, equal to the bit: the row kernel
with a whole B and the contraction that reads it (and the batch's resB).
"""
import ctypes

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _ion(index):
    from atomx_b200 import workloads as W
    from atomx_b200.tables import upload_ion
    return upload_ion(W.build_ion(W.uneven_batch()[index]))


def test_split_with_a_whole_b():
    from atomx_b200 import _native
    from atomx_b200.batch import SplitBatch
    from atomx_b200.split import IonRows, SplitEngine
    L = _native.require_device()
    dev = _ion(4)
    eng = SplitEngine(dev, rows_kernel="cells", cert_limit=float("inf"))
    eng.run()
    assert eng._resB is not None and eng.b_col0 > 0
    R, plan, h = eng.ion_rows, dev.plan, _native.stream_handle()
    A, B = (torch.zeros((eng.n_mod, eng.rows_alloc, eng.kpad), dtype=torch.int8, device="cuda") for _ in range(2))
    rs, lf, rt, cb = (torch.empty_like(t) for t in (eng.rowscale, eng.left, eng.right, eng.cbound))
    _native.check(L.rkb_split_rows_cells(
        dev.Pv.data_ptr(), dev.Qv.data_ptr(), dev.n, dev.pairs.data_ptr(), dev.row_pair.data_ptr(),
        dev.row_k.data_ptr(), plan.n_rows, dev.w.data_ptr(), dev.nv, dev.ng, R.ktab.data_ptr(), R.koff.data_ptr(),
        R.ktab_t.data_ptr(), R.koff_t.data_ptr(), R.max_z, eng.bits, eng.n_mod, eng._mod_c[0], A.data_ptr(),
        B.data_ptr(), eng.kpad, 0, eng.rows_alloc, rs.data_ptr(), lf.data_ptr(), rt.data_ptr(), cb.data_ptr(), eng.cwp,
        h), "rkb_split_rows_cells")
    assert torch.equal(A, eng.resA) and torch.equal(B[:, :plan.n_rows], eng.resB[:, :plan.n_rows])
    assert all(torch.equal(a, b) for a, b in ((rs, eng.rowscale), (lf, eng.left), (rt, eng.right), (cb, eng.cbound)))
    out, status = torch.empty_like(eng.out), torch.zeros(1, dtype=torch.int32, device="cuda")
    some = (ctypes.c_int * 8)()
    _native.check(L.rkb_split_contract(
        A.data_ptr(), B.data_ptr(), eng.kpad, eng.rows_alloc, eng.n_mod, eng._mod_c[0], some, some, some, eng.M,
        rs.data_ptr(), lf.data_ptr(), rt.data_ptr(), cb.data_ptr(), eng.corr_floor, eng.cw, eng.cwp,
        eng.grp_row0.data_ptr(), eng.grp_n.data_ptr(), eng.grp_kdim.data_ptr(), eng.grp_out.data_ptr(),
        eng.tasks.data_ptr(), eng.n_tasks, out.data_ptr(), status.data_ptr(), h), "rkb_split_contract")
    assert torch.equal(out, eng.out) and int(status) == 0
    # a batch's B, of ions whose own parts start at different columns
    other = _ion(5)
    batch = SplitBatch([dev, other], bits=eng.bits, n_mod=eng.n_mod, cert_limit=float("inf"),
                       ion_rows=[IonRows(d, rows_kernel="cells") for d in (dev, other)])
    batch.step()
    batch.check_status()
    whole = batch.resB
    assert whole.shape == batch.resA.shape and len(set(batch.b_col0)) == 2
    assert torch.equal(whole[:, :plan.n_rows, :eng.kpad], B[:, :plan.n_rows])
    z = batch.ions[1]
    rows, c0 = slice(plan.n_rows, plan.n_rows + other.plan.n_rows), z.kbody
    assert torch.equal(whole[:, rows, :c0], batch.resA[:, rows, :c0])
    neg = -batch.resA[:, rows, c0:c0 + z.max_z].to(torch.int16)
    diff = (whole[:, rows, c0:c0 + z.max_z].to(torch.int16) - neg).abs()
    m = torch.as_tensor(batch.moduli, device="cuda")[:, None, None]
    assert bool(((diff == 0) | (diff == m)).all())
