"""Fock blocks of many targets in one call, against single kernels and oracle.

The launch over all blocks, multipoles and targets keeps the summation order
of one (block, multipole, target) at a time, so every result is equal to the
bit: over target counts that leave a group of the kernel's targets partly
empty, odd basis sizes, the grouping of targets, and a skipped PQ exchange.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _problem(ns, n, k_max):
    from atomx_b200 import basis
    t = basis.make_exponential_knots(ns, 7, 1e-3, 20.0)
    bd = basis.prepare_bspline_data(t, ns, 7, n_gauss=7, kinetic_balance=True)
    rng = np.random.default_rng(ns + n)
    P, Q = rng.normal(size=(n, ns)), 0.1 * rng.normal(size=(n, ns))
    ad, ax = rng.normal(size=(2, n, n, k_max + 1)) * (rng.random((2, n, n, k_max + 1)) < 0.7)
    return bd, P, Q, ad, ax, 0.5 + rng.random(n)


@pytest.mark.parametrize("ns,n", [(17, 1), (23, 5), (66, 9)])
@pytest.mark.parametrize("skip", [False, True])
def test_targets_together_equal_one_at_a_time(ns, n, skip, monkeypatch):
    from atomx_b200 import convol as C
    bd, P, Q, ad, ax, norms = _problem(ns, n, 3)
    ks = [0, 2, 3]
    H = C.build_hf_matrices_dbsr(range(n), P, Q, ad, ax, ks, norms, bd, skip_pq_exchange=skip)
    for i in range(n):
        one = C.build_hf_matrix_dbsr(i, P, Q, ad, ax, ks, norms[i], bd, skip_pq_exchange=skip)
        assert np.array_equal(np.stack(one), H[i].cpu().numpy())
    monkeypatch.setattr(C, "_FOCK_BYTES", 32 * 3 * ns * ns * 2)  # two targets a launch
    assert torch.equal(H, C.build_hf_matrices_dbsr(range(n), P, Q, ad, ax, ks, norms, bd, skip_pq_exchange=skip))


@pytest.mark.parametrize("ns", [17, 66])
def test_exchange_equals_the_single_contraction(ns):
    """With unit norms, no direct part and one multipole, the blocks are the
    exchange contractions of the outer-product densities (the kernel behind
    compute_exchange_matrix_cell, bit-identical to the reference's), made
    symmetric."""
    from atomx_b200 import convol as C
    bd, P, Q, _, _, _ = _problem(ns, 2, 2)
    ax = np.zeros((2, 2, 3))
    ax[0, 1, 2] = 1.0
    H = C.build_hf_matrices_dbsr([0], P, Q, np.zeros_like(ax), ax, [2], [1.0], bd)[0].cpu().numpy()
    b = (P[1], Q[1])
    kpp, kqq, kpq, _ = C.compute_exchange_matrix_cell(*b, *b, bd, 2)
    assert np.array_equal(H[0], 0.5 * (kpp + kpp.T)) and np.array_equal(H[1], 0.5 * (kqq + kqq.T))
    # the two mixed blocks come from the two mixed banks, equal to rounding
    assert np.max(np.abs(H[2] - kpq)) <= 1e-13 * np.abs(kpq).max() and np.array_equal(H[3], H[2].T)
    empty = C.build_hf_matrices_dbsr([0, 1], P, Q, ax, ax, [], [1.0, 2.0], bd)
    assert empty.shape == (2, 4, ns, ns) and not bool(empty.any())
    with pytest.raises(ValueError):
        C.build_hf_matrices_dbsr([0, 1], P, Q, ax, ax, [2], [1.0], bd)
