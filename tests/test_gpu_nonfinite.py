"""A non-finite orbital does not stop the split contraction.

The status word reports RKB_ENONFINITE (FloatingPointError), the rows of that
orbital come out as NaN, and every other entry equals, to the bit, the table
without it: the launch runs to its end, in a table of many more tiles than
SMs, in the launches after it that find the word set, and beside other ions
of a batch.  corr_floor = 0 keeps every core correction, so that an entry does
not depend on the other rows of its block.
"""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

ORBITAL = 17


@pytest.fixture(scope="module")
def ions():
    """(ion with a NaN, the same ion without, a small clean ion)"""
    from atomx_b200 import workloads as W
    from atomx_b200.tables import upload_values

    def values(spec):
        ion = W.build_ion(spec)
        return ion, *(np.array([f(c, ion.bsp).ravel() for c in x]) for f, x in
                      ((oracle.eval_P, ion.P), (oracle.eval_Q, ion.Q)))

    def up(ion, P, Q, k_max):
        return upload_values(P, Q, ion.kappa, ion.bsp["gr"], ion.bsp["grw"], k_max)
    spec = W.uneven_batch()[1]
    ion, P, Q = values(spec)
    bad = P.copy()
    bad[ORBITAL, 211] = np.nan
    small = W.uneven_batch()[4]
    return (up(ion, bad, Q, spec.k_max), up(ion, P, Q, spec.k_max), up(*values(small), small.k_max))


def _check(plan, got, want):
    """``got``, ``want``: {k: table}."""
    for k in plan.ks:
        hit = torch.as_tensor([ORBITAL in plan.pairs[p] for p in plan.pairs_of_k[k]], device="cuda")
        touched = hit[:, None] | hit[None, :]
        assert bool(torch.isnan(got[k][touched]).all())
        assert torch.equal(got[k][~touched], want[k][~touched]), k


def _tables(eng):
    plan = eng.dev.plan
    return {k: eng.out[eng.offsets[k]:eng.offsets[k] + plan.n_of_k(k) ** 2].view(plan.n_of_k(k), -1)
            for k in plan.ks}


def test_whole_table_and_table_by_table(ions):
    from atomx_b200.split import SplitEngine
    bad, clean, _ = ions
    opts = dict(corr_floor=0.0, cert_limit=float("inf"))
    want = SplitEngine(clean, **opts)
    want.run()
    eng = SplitEngine(bad, **opts)
    assert eng.n_tasks > 3 * torch.cuda.get_device_properties(0).multi_processor_count
    for _ in range(3):
        eng.out.fill_(7.0)
        with pytest.raises(FloatingPointError):
            eng.run()
        _check(bad.plan, _tables(eng), _tables(want))
    # a launch per table: the later ones start with the word set
    eng.out.fill_(7.0)
    host = torch.empty(eng.total, dtype=torch.float64, pin_memory=True)
    with pytest.raises(FloatingPointError):
        eng.run_to_host(host)
    _check(bad.plan, _tables(eng), _tables(want))
    assert torch.equal(torch.nan_to_num(host, nan=-1.0), torch.nan_to_num(eng.out.cpu(), nan=-1.0))
    want.run()  # the device is as good as before


def test_other_ions_of_a_batch(ions):
    from atomx_b200.batch import SplitBatch
    bad, clean, small = ions
    opts = dict(corr_floor=0.0, cert_limit=float("inf"))
    want, got = (SplitBatch([small, x, small], **opts) for x in (clean, bad))
    want.step()
    want.check_status()
    got.out.fill_(7.0)
    got.step()
    with pytest.raises(FloatingPointError):
        got.check_status()
    for i in (0, 2):
        for k in small.plan.ks:
            assert torch.equal(got.table(i, k), want.table(i, k))
    _check(bad.plan, *({k: b.table(1, k) for k in bad.plan.ks} for b in (got, want)))
