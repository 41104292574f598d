"""The production step's split of x into blocks (choose_chunk): grids without
interior tiles take chunks down to single planes when SMs would idle.  Every
chunking computes each cell with the same arithmetic, so the automatic split
must equal one whole-column block per tile bit for bit."""
import numpy as np
import pytest

from conftest import random_primitives
from deepgreen import capi


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2, 5, 3), (3, 14, 64), (17, 29, 66), (48, 15, 65), (40, 60, 130), (149, 14, 64)])
@pytest.mark.parametrize("bcs", [(capi.PERIODIC,) * 6, (capi.OUTFLOW,) * 6, (capi.WALL,) * 6])
def test_automatic_chunks_equal_whole_columns_bitwise(shape, bcs):
    prim = random_primitives(shape, 17)
    out = []
    for chunk in (0, shape[0]):
        ctx = capi.Context(shape, 0.05, bcs, gamma=1.4, cfl=0.4, limiter=capi.LIMITER_MINMOD, precision=capi.F32)
        ctx.set_primitives(prim)
        ctx.set_chunk(chunk)
        out.append((ctx.compute_step(4), ctx.get_conserved()))
        ctx.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    for a, b in zip(out[0][1], out[1][1]):
        np.testing.assert_array_equal(a, b)
