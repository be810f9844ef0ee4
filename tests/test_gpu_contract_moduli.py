"""The contraction's CRT for every number of moduli it takes.

Every entry of the Z=10 ion's tables against the exact integer CRT (Python
integers) of the device's own residues.  Bound, per entry, in units of the
entry's row-scale product: the fraction x / M is kept to 2^-64 with one
rounding per digit (three digits, each half a unit plus the weight's own
2^-97 times a digit below 2^32: below 3 * 2^-64 in all), and the result in
double precision (three roundings of the value, and the FP64 core term).
"""
import numpy as np
import pytest

from split_emulation import crt_exact

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n_mod", range(4, 13))
def test_every_entry_matches_exact_crt(n_mod):
    from atomx_b200 import workloads as W
    from atomx_b200.split import SplitEngine
    from atomx_b200.tables import upload_ion
    eng = SplitEngine(upload_ion(W.build_ion(W.neon_small())), n_mod=n_mod, corr_floor=0.0, cert_limit=float("inf"))
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
        bound = 3 * 2.0 ** -64 * eng.M * scale + 2.0 ** -51 * np.abs(x * scale) + (eng.cw + 2) * 2.0 ** -52 * terms
        assert np.all(np.abs(T - (x * scale + core)) <= bound), (n_mod, k)
