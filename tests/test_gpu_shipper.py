"""PackedShipper used table by table: each table alone, in any buffer order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_one_table_at_a_time():
    from atomx_b200.plan import make_plan
    from atomx_b200.tables import PackedShipper, packed_offsets
    plan = make_plan(np.array([-1, 1, -2, 2, -3, -1, 1]), 4)
    gen = torch.Generator(device="cuda").manual_seed(1)
    tables = {}
    for k in plan.ks:
        n = plan.n_of_k(k)
        t = torch.rand((n, n), generator=gen, device="cuda", dtype=torch.float64)
        tables[k] = t + t.T
    host = torch.full((plan.unique_entries,), -1.0, dtype=torch.float64, pin_memory=True)
    s, cs = torch.cuda.current_stream(), torch.cuda.Stream()
    shipper = PackedShipper(plan, host, torch.device("cuda", 0), cs)
    for k in plan.ks:
        shipper.ship(k, tables[k].data_ptr(), s)
    cs.synchronize()
    offs = packed_offsets(plan)
    for k in plan.ks:
        n = plan.n_of_k(k)
        got = host[offs[k]:offs[k] + n * (n + 1) // 2]
        i, j = np.triu_indices(n)
        assert torch.equal(got, tables[k].cpu()[i, j])
