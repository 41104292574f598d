"""The batch's automatic split along x: any split gives the same states.

A cell's update does not depend on the item it falls in, so the automatic
split, chosen from the sizes and the number of SMs, must equal whole columns
and single planes bit for bit: for one grid, for a few and for more items than
SMs, with extents below, at and above a tile.
"""
import numpy as np
import pytest

from deepgreen import batch, capi

pytestmark = pytest.mark.gpu

BATCHES = [
    [(6, 14, 64)],
    [(24, 15, 65), (5, 4, 7)],
    [(40, 31, 70)] * 12,
    [(70, 45, 129), (33, 60, 66), (9, 100, 40)] * 8,
]


@pytest.mark.parametrize("shapes", BATCHES)
@pytest.mark.parametrize("bcs", [(capi.OUTFLOW,) * 6, (capi.PERIODIC,) * 6])
def test_automatic_split_equals_any_other(shapes, bcs):
    states, chunks = [], []
    for chunk in (0, 1, 1000):
        bt, _, _ = batch.make_batch(shapes, seed=3, bcs=bcs)
        if chunk:
            bt.set_tiling(14, chunk)
        bt.step(3)
        chunks.append(bt.tiling()[1])
        states.append([bt.get_conserved(i) for i in range(len(shapes))])
    assert 1 <= chunks[0] <= 64
    for other in states[1:]:
        for a, b in zip(states[0], other):
            assert np.array_equal(a, b)
