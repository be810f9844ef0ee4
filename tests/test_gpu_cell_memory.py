"""Cell tables, key batches and Fock blocks where device memory is short.

The allocator is limited to less than one pass over all multipoles (targets)
takes and more than one multipole's (target's) does: the calls go through, in
smaller passes, with the same results.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

NS, N, K_MAX = 60, 120, 4


class _Limit:
    """At most ``extra`` bytes more than what is in use now."""

    def __init__(self, extra):
        self.extra = extra

    def __enter__(self):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        total = torch.cuda.get_device_properties(0).total_memory
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + self.extra) / total)

    def __exit__(self, *exc):
        torch.cuda.set_per_process_memory_fraction(1.0)


@pytest.fixture(scope="module")
def problem():
    from atomx_b200 import basis
    t = basis.make_exponential_knots(NS, 7, 1e-3, 20.0)
    bd = basis.prepare_bspline_data(t, NS, 7, n_gauss=7, kinetic_balance=True)
    rng = np.random.default_rng(5)
    return bd, rng.normal(size=(N, NS)), 0.1 * rng.normal(size=(N, NS))


def test_tables_and_keys(problem):
    from atomx_b200 import convol as C
    from atomx_b200.plan import make_plan
    bd, P, Q = problem
    kappa = np.array([-1, 1, -2, 2, -3] * 24)
    plan = make_plan(kappa, K_MAX)
    want = C.cell_tables(P, Q, kappa, bd, K_MAX)
    kdim = C.ConvolCache(bd).bank(0).kdim
    sizes = [plan.n_of_k(k) for k in plan.ks]
    one, all_ = (16 * kdim * f(sizes) for f in (max, sum))
    out = 8 * sum(n * n for n in sizes)
    assert all_ > one + (48 << 20)
    with _Limit(out + one + (40 << 20)):
        got = C.cell_tables(P, Q, kappa, bd, K_MAX)
    assert torch.equal(got.values, want.values)
    del got, want
    od = {i: (P[i], Q[i]) for i in range(N)}
    rng = np.random.default_rng(6)
    keys = [(*rng.integers(0, N, 4).tolist(), int(k)) for k in rng.integers(0, K_MAX + 1, 4000)]
    want = C.compute_slater_rk_cell_batch(od, keys, bd)
    per = 3 * 8 * kdim * 1000  # bytes of one multipole's rows, at most
    with _Limit(per + (24 << 20)):  # of five such
        got = C.compute_slater_rk_cell_batch(od, keys, bd)
    assert got == want


def test_fock_blocks(problem):
    from atomx_b200 import convol as C
    bd, P, Q = problem
    rng = np.random.default_rng(7)
    ad, ax = rng.normal(size=(2, N, N, K_MAX + 1))
    ks = list(range(K_MAX + 1))
    args = (range(N), P, Q, ad, ax, ks, 0.5 + rng.random(N), bd)
    want = C.build_hf_matrices_dbsr(*args)
    out, one = 32 * N * NS * NS, 32 * (len(ks) + 1) * NS * NS
    assert one * N > 72 << 20
    with _Limit(out + (64 << 20)):
        got = C.build_hf_matrices_dbsr(*args)
    assert torch.equal(got, want)
