"""The cell row kernel at every Gauss order it takes, against the two-kernel path.

The rows of a small ion at ng = 5..11: the row count is no multiple of the
kernel's block of rows, and multipoles change inside blocks.  Both paths sum
a row's X in other orders, so the rebuilt integers may differ by the rounding
of an X near a half: |x_cells - x_two| <= 1 quantum.  The scales are equal
(powers of two of the same maxima), the core vectors and records agree to
1e-12 of their own size, and B equals A but for the negated Z columns.
"""
import numpy as np
import pytest

from split_emulation import crt_exact

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("ng", range(5, 12))
@pytest.mark.parametrize("ns", [23, 61])
def test_rows_of_every_gauss_order(ng, ns):
    from atomx_b200 import workloads as W
    from atomx_b200.split import SplitEngine
    from atomx_b200.tables import upload_ion
    ion = W.build_ion(W.IonSpec(Z=18, ns=ns, ks=7, n_gauss=ng, r_min=1e-4, r_max=30.0,
                                shells=((-1, 3), (1, 2), (-2, 2), (2, 1)), k_max=3, seed=ng))
    dev = upload_ion(ion)
    cells, two = (SplitEngine(dev, rows_kernel=kind) for kind in ("cells", "two"))
    for eng in (cells, two):
        eng.rows()
    torch.cuda.synchronize()
    plan = dev.plan
    n = plan.n_rows
    assert n % 4 and any(plan.k_row_offset[k] % 4 for k in plan.ks)
    a, b = (crt_exact([e.resA[m, :n].cpu().numpy().astype(np.int64) for m in range(e.n_mod)], e.moduli)
            for e in (cells, two))
    assert np.array_equal(cells.rowscale.cpu().numpy(), two.rowscale.cpu().numpy())
    assert np.max(np.abs(a - b)) <= 1.0
    for x, y in ((cells.left, two.left), (cells.right, two.right), (cells.cbound, two.cbound)):
        x, y = x.cpu().numpy(), y.cpu().numpy()
        big = np.isinf(y)
        assert np.array_equal(big, np.isinf(x))
        scale = np.where(big, 0.0, np.abs(y)).max(axis=1, keepdims=True)
        assert np.all(np.abs(np.where(big, 0.0, x) - np.where(big, 0.0, y)) <= 1e-12 * scale)
    if cells.has_z:
        B = cells.resB[:, :n].cpu().numpy().astype(np.int64)
        A = cells.resA[:, :n].cpu().numpy().astype(np.int64)
        kb = cells.kbody
        assert np.array_equal(A[:, :, :kb], B[:, :, :kb])
        for i, m in enumerate(cells.moduli):
            assert not np.any((A[i, :, kb:] + B[i, :, kb:]) % int(m))
