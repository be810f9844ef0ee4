"""Cell tables and Fock blocks on a stream of their own equal the default's.

The given stream is held back behind a long kernel while the caller goes on:
blocks that the call has freed are written over on the caller's stream, inputs
are still being made there when the call starts, banks are built on one stream
and used from another at once.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

NS, N, K_MAX = 48, 6, 4
WAIT = 40_000_000  # clocks of torch.cuda._sleep: some 20 ms


@pytest.fixture(scope="module")
def problem():
    from atomx_b200 import basis
    t = basis.make_exponential_knots(NS, 7, 1e-3, 20.0)
    bd = basis.prepare_bspline_data(t, NS, 7, n_gauss=7, kinetic_balance=True)
    rng = np.random.default_rng(3)
    ad, ax = rng.normal(size=(2, N, N, K_MAX + 1))
    return bd, rng.normal(size=(N, NS)), 0.1 * rng.normal(size=(N, NS)), ad, ax, 0.5 + rng.random(N)


KAPPA = [-1, -1, 1, -2, -2, 2]


def _tables(problem, **kw):
    from atomx_b200 import convol as C
    bd, P, Q = problem[:3]
    return C.cell_tables(P, Q, KAPPA, bd, K_MAX, **kw).values


def _fock(problem, **kw):
    from atomx_b200 import convol as C
    bd, P, Q, ad, ax, norms = problem
    return C.build_hf_matrices_dbsr(range(N), P, Q, ad, ax, [0, 1, 3], norms, bd, **kw)


def _churn():
    """Write over what the current stream's allocator has free."""
    return [torch.full((n,), 7, dtype=torch.int64, device="cuda") for n in (8, 64, 256, 1024, 4096, 1 << 16, 1 << 20)
            for _ in range(8)]


@pytest.mark.parametrize("call", [_tables, _fock])
@pytest.mark.parametrize("fresh", [False, True])
def test_side_stream(problem, call, fresh):
    from atomx_b200.convol import ConvolCache
    want = call(problem)
    side = torch.cuda.Stream()
    for _ in range(3):
        torch.cuda.synchronize()
        if fresh:
            ConvolCache(problem[0]).release_shared_banks()
        with torch.cuda.stream(side):
            torch.cuda._sleep(WAIT)
        got = call(problem, stream=side)
        _churn()
        side.synchronize()
        assert torch.equal(got, want)


def test_inputs_of_the_callers_stream(problem):
    """Coefficient stacks that a queued kernel of the caller's stream still writes."""
    from atomx_b200 import convol as C
    bd, P, Q = problem[:3]
    want = _tables(problem)
    Pd, Qd = (torch.as_tensor(x, device="cuda") for x in (P, Q))
    side, out = torch.cuda.Stream(), torch.zeros((2, N, NS), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    torch.cuda._sleep(WAIT)
    out[0].copy_(Pd)
    out[1].copy_(Qd)
    got = C.cell_tables(out[0], out[1], KAPPA, bd, K_MAX, stream=side).values
    side.synchronize()
    assert torch.equal(got, want)


def test_bank_of_another_stream(problem):
    """A bank whose build is queued behind other work is waited for."""
    from atomx_b200.convol import ConvolCache
    want = _tables(problem)
    cache = ConvolCache(problem[0])
    for home, user in ((torch.cuda.Stream(), None), (None, torch.cuda.Stream())):
        torch.cuda.synchronize()
        cache.release_shared_banks()
        with torch.cuda.stream(home or torch.cuda.current_stream()):
            cache.bank(0)  # one-time uploads, so that the next builds only queue
            torch.cuda._sleep(WAIT)
        for k in range(1, K_MAX + 1):
            cache.bank(k, home)
        got = _tables(problem, stream=user)
        torch.cuda.synchronize()
        assert torch.equal(got, want)


def test_densities_of_a_side_stream(problem):
    from atomx_b200 import convol as C
    bd, P, Q = problem[:3]
    bank = C.ConvolCache(bd).bank(1)
    Pd, Qd = (torch.as_tensor(x, device="cuda") for x in (P, Q))
    pairs = [(a, b) for a in range(N) for b in range(a + 1)]
    want, side = C.cell_densities(bank, Pd, Qd, pairs, NS, NS), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(WAIT)
    got = C.cell_densities(bank, Pd, Qd, pairs, NS, NS, side)
    _churn()
    side.synchronize()
    assert torch.equal(got, want)
