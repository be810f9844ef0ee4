"""Entry points of the C interface that the package itself no longer calls.

Each against the form that the package runs, equal to the bit: the row kernel
with a whole B and the contraction that reads it (and the batch's resB), the
Y^k rows without a power table, and the Fock blocks built from the single
kernels, one component block and multipole at a time.
"""
import ctypes

import numpy as np
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


def test_yk_rows_without_a_table():
    from atomx_b200 import _native
    from atomx_b200.yk import compute_yk_rows, yk_partial_matrices
    L = _native.require_device()
    dev = _ion(4)
    rows, n = 400, dev.n
    gen = torch.Generator(device="cuda").manual_seed(2)
    rho = torch.rand((rows, n), generator=gen, device="cuda", dtype=torch.float64) - 0.5
    ks = np.arange(rows, dtype=np.int32) % 7
    want = compute_yk_rows(rho, ks, dev.r.view(dev.nv, dev.ng).cpu().numpy(), dev.w.view(dev.nv, dev.ng).cpu().numpy())
    mo, mi = (torch.as_tensor(m.copy(), device="cuda") for m in yk_partial_matrices(dev.ng))
    kt, out = torch.as_tensor(ks, device="cuda"), torch.empty_like(rho)
    _native.check(L.rkb_yk_rows(rho.data_ptr(), n, kt.data_ptr(), rows, dev.r.data_ptr(), dev.w.data_ptr(), dev.nv,
                                dev.ng, mo.data_ptr(), mi.data_ptr(), out.data_ptr(), n, _native.stream_handle()),
                  "rkb_yk_rows")
    assert torch.equal(out, want.view(rows, n))


@pytest.mark.parametrize("skip", [False, True])
def test_fock_blocks_from_single_kernels(skip):
    from atomx_b200 import _native, basis
    from atomx_b200 import convol as C
    L = _native.require_device()
    ns, n, ks = 37, 5, [0, 1, 3]
    bd = basis.prepare_bspline_data(basis.make_exponential_knots(ns, 7, 1e-3, 20.0), ns, 7, n_gauss=7,
                                    kinetic_balance=True)
    rng = np.random.default_rng(8)
    Ph, Qh = rng.normal(size=(n, ns)), 0.1 * rng.normal(size=(n, ns))
    ad, ax = rng.normal(size=(2, n, n, 4)) * (rng.random((2, n, n, 4)) < 0.7)
    norms, targets = 0.5 + rng.random(n), np.array([3, 0, 4])
    want = C.build_hf_matrices_dbsr(targets, Ph, Qh, ad, ax, ks, norms[targets], bd, skip_pq_exchange=skip)
    cache, nt, s = C.ConvolCache(bd), 3, _native.stream_handle()
    dev = want.device
    P, Q = C._stack(list(Ph), ns, dev), C._stack(list(Qh), ns, dev)
    comp, ld = {1: P, 2: Q}, P.shape[1]
    tgt = torch.as_tensor(targets.astype(np.int32), device=dev)
    H = torch.zeros((nt, 4, ns, ns), dtype=torch.float64, device=dev)
    kinds = {(1, 1): ("pppp", 0), (1, 2): ("pqpq", 2), (2, 1): ("qpqp", 3), (2, 2): ("qqqq", 1)}

    def buf(*shape):
        return torch.zeros(shape, dtype=torch.float64, device=dev)
    for (i, j), (itype, slot) in kinds.items():
        for k in ks:
            bank = cache.bank(k)
            r0, c0, bra, ket = bank.offsets(itype)
            coef = torch.as_tensor(np.ascontiguousarray(ad[targets, :, k]), device=dev)
            kp = C._round16(ket * ns)
            dd, v, J = buf(nt, kp), buf(nt, bra * ns), buf(nt, ns, ns)
            _native.check(L.rkb_cell_direct_density(comp[j].data_ptr(), ld, n, coef.data_ptr(), n, tgt.data_ptr(), nt,
                                                    ns, ket, dd.data_ptr(), kp, s), "rkb_cell_direct_density")
            kb = bank.K[r0:r0 + bra * ns, c0:]
            _native.check(L.rkb_gemm_nt_fp64(dd.data_ptr(), kp, kb.data_ptr(), bank.kdim, v.data_ptr(), bra * ns, nt,
                                             bra * ns, kp, 0, s), "rkb_gemm_nt_fp64")
            _native.check(L.rkb_cell_banded_to_full(v.data_ptr(), ns, bra, nt, J.data_ptr(), s),
                          "rkb_cell_banded_to_full")
            H[:, 0 if i == 1 else 1] += J
            if skip and (i, j) == (1, 2):
                continue
            coef = torch.as_tensor(np.ascontiguousarray(ax[targets, :, k]), device=dev)
            xx, K = buf(nt, ns, ns), buf(nt, ns, ns)
            _native.check(L.rkb_cell_exchange_density(comp[i].data_ptr(), comp[j].data_ptr(), ld, n, coef.data_ptr(),
                                                      n, nt, ns, xx.data_ptr(), s), "rkb_cell_exchange_density")
            at = torch.full((nt,), r0 * bank.kdim + c0, dtype=torch.int64, device=dev)
            _native.check(L.rkb_cell_exchange(bank.K.data_ptr(), bank.kdim, at.data_ptr(), xx.data_ptr(), nt, ns, bra,
                                              ket, int(i == j), 0, K.data_ptr(), s), "rkb_cell_exchange")
            H[:, slot] += K
    out, nrm = torch.empty_like(H), torch.as_tensor(norms[targets], device=dev)
    _native.check(L.rkb_cell_fock_finish(H.data_ptr(), nrm.data_ptr(), ns, int(skip), nt, out.data_ptr(), s),
                  "rkb_cell_fock_finish")
    assert torch.equal(out, want)
