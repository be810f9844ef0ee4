"""The FP64 GEMM tiles (32 x 32 and 64 x 64) at their edges.

Against torch in float64.  Bound per entry: K products and sums of either
order are off by at most K 2^-52 sum |a||b| (twice, for the two results).
Tables must not depend on the tile that a launch picks.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _rand(*shape, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


@pytest.mark.parametrize("m,n,k", [(1, 1, 16), (24, 1080, 1088), (31, 33, 48), (32, 64, 0), (65, 127, 32),
                                   (222, 2049, 160), (1089, 1151, 64)])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_gemm_nt(m, n, k, accumulate):
    from atomx_b200 import _native
    L = _native.require_device()
    A, B = _rand(m, k + 2, seed=m), _rand(n, k + 2, seed=n + 7)
    C0 = _rand(m, n + 3, seed=5)
    C = C0.clone()
    _native.check(L.rkb_gemm_nt_fp64(A.data_ptr(), k + 2, B.data_ptr(), k + 2, C.data_ptr(), n + 3, m, n, k, accumulate,
                                     _native.stream_handle()), "rkb_gemm_nt_fp64")
    a, b = A[:, :k], B[:, :k]
    ref = a @ b.T + (C0[:, :n] if accumulate else 0.0)
    bound = 2.0 * (k + 1) * 2.0 ** -52 * (a.abs() @ b.abs().T + C0[:, :n].abs())
    assert bool(((C[:, :n] - ref).abs() <= bound).all())
    assert torch.equal(C[:, n:], C0[:, n:])  # nothing beside the result


@pytest.mark.parametrize("n", [1, 31, 64, 65, 129, 200])
def test_contraction_does_not_depend_on_the_tile(n):
    from atomx_b200 import _native
    from atomx_b200.tables import tile_tasks
    L = _native.require_device()
    groups, k = 300, 48
    G, Y = _rand(groups * n, k, seed=1), _rand(groups * n, k, seed=2)
    row0 = torch.arange(groups, device="cuda") * n
    size = torch.full((groups,), n, dtype=torch.int64, device="cuda")
    off = torch.arange(groups, device="cuda") * n * n

    def run(sizes, g0):
        tasks = tile_tasks(sizes)
        t = torch.as_tensor(tasks.reshape(-1), device="cuda")
        out = torch.full((len(sizes) * n * n,), float("nan"), dtype=torch.float64, device="cuda")
        _native.check(L.rkb_table_contract_fp64(G.data_ptr(), Y.data_ptr(), k, k, row0[g0:].data_ptr(), size.data_ptr(),
                                                off.data_ptr(), t.data_ptr(), tasks.shape[0], out.data_ptr(),
                                                _native.stream_handle()), "rkb_table_contract_fp64")
        return out.view(-1, n, n)

    many, one = run([n] * groups, 0), run([n], 3)  # 64 x 64 and 32 x 32 tiles
    assert torch.equal(many[3], one[0])
    assert torch.equal(many, many.transpose(1, 2))
    g, y = G[3 * n:4 * n], Y[3 * n:4 * n]
    up = torch.triu(torch.ones(n, n, dtype=torch.bool, device="cuda"))
    err = (one[0] - g @ y.T).abs()
    assert bool((err <= 2.0 * (k + 1) * 2.0 ** -52 * (g.abs() @ y.abs().T))[up].all())


@pytest.mark.parametrize("rows", [[5], [0, 33, 0, 64, 1], [700, 0, 900], [3] * 70])
def test_grouped_gemm_equals_single_ones(rows):
    """Empty groups, groups that share no tile, more groups than one launch takes."""
    from atomx_b200 import _native
    L = _native.require_device()
    n, k = 1100, 32
    r0 = np.concatenate([[0], np.cumsum(rows)]).astype(np.int64)
    A, C = _rand(max(int(r0[-1]), 1), k, seed=3), torch.full((int(r0[-1]), n), float("nan"), dtype=torch.float64, device="cuda")
    Bs = [_rand(n, k, seed=10 + i) for i in range(len(rows))]
    ptrs = np.array([b.data_ptr() for b in Bs], dtype=np.int64)
    _native.check(L.rkb_gemm_nt_fp64_groups(A.data_ptr(), k, ptrs.ctypes.data, r0.ctypes.data, len(rows), k, C.data_ptr(),
                                            n, n, k, _native.stream_handle()), "rkb_gemm_nt_fp64_groups")
    for g, b in enumerate(Bs):
        one = torch.empty(rows[g], n, dtype=torch.float64, device="cuda")
        _native.check(L.rkb_gemm_nt_fp64(A[int(r0[g]):].data_ptr(), k, b.data_ptr(), k, one.data_ptr(), n, rows[g], n, k,
                                         0, _native.stream_handle()), "rkb_gemm_nt_fp64")
        assert torch.equal(one, C[int(r0[g]):int(r0[g + 1])])
