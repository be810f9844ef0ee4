"""Tile lists belong to their caller: a list in blocks, whose order is kept per
set of sizes, may be written to and is not shared with the next call."""
import numpy as np
import pytest


@pytest.mark.parametrize("block", [None, 2, 8])
def test_the_callers_own_list(block):
    from atomx_b200.tables import tile_tasks
    sizes = [300, 1, 700]
    first = tile_tasks(sizes, block=block)
    want = first.copy()
    assert first.flags.writeable
    first[:] = -1
    assert np.array_equal(tile_tasks(sizes, block=block), want)
