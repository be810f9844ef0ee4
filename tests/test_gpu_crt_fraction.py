"""Tables whose moduli hold far more than their width needs.

24-bit splits recombined from 12 moduli (explicit bits and n_mod): the products
lie below 2^-34 of M, where a fraction kept to 2^-64 would be the largest
error.  Every entry against the exact integer CRT of the device's own residues:
2^-71 of M for the fraction, and the roundings of the value (2^-51 of it) and
of the FP64 core term.
"""
import numpy as np
import pytest

from split_emulation import crt_exact

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("bits,n_mod", [(24, 12), (30, 12), (16, 8)])
def test_narrow_splits_of_many_moduli(bits, n_mod):
    from atomx_b200 import workloads as W
    from atomx_b200.split import SplitEngine
    from atomx_b200.tables import upload_ion
    eng = SplitEngine(upload_ion(W.build_ion(W.neon_small())), bits=bits, n_mod=n_mod, corr_floor=0.0,
                      cert_limit=float("inf"))
    eng.run()
    plan = eng.dev.plan
    A = eng.resA.cpu().numpy().astype(np.int64)
    B = A if eng.resB is None else eng.resB.cpu().numpy().astype(np.int64)
    rs, lf, rt = (t.cpu().numpy() for t in (eng.rowscale, eng.left[:, :eng.cw], eng.right[:, :eng.cw]))
    for k in plan.ks:
        o, n = plan.k_row_offset[k], plan.n_of_k(k)
        x = crt_exact([A[m, o:o + n] @ B[m, o:o + n].T for m in range(n_mod)], eng.moduli)
        scale = np.outer(rs[o:o + n], rs[o:o + n])
        core = lf[o:o + n] @ rt[o:o + n].T
        terms = np.abs(lf[o:o + n]) @ np.abs(rt[o:o + n]).T
        T = eng.out[eng.offsets[k]:eng.offsets[k] + n * n].view(n, n).cpu().numpy()
        bound = 2.0 ** -71 * eng.M * scale + 2.0 ** -51 * np.abs(x * scale) + (eng.cw + 2) * 2.0 ** -52 * terms
        assert np.all(np.abs(T - (x * scale + core)) <= bound), k
