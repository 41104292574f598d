"""Heat through a conducting lower z face in the FP32 step: it joins the first
column's z balance before that balance joins the cell's sum, one addition in
all.  The energies of the first column are compared bit for bit with stored
ones (golden/heat_f32.npz: this library's, with that order; the sum with the
heat added last takes one rounding more)."""
from pathlib import Path

import numpy as np
import pytest

from conftest import random_primitives
from deepgreen import capi

GOLDEN = Path(__file__).parent / "golden" / "heat_f32.npz"
C, O, W, P = capi.CONDUCTING_WALL, capi.OUTFLOW, capi.WALL, capi.PERIODIC
CASES = {
    "odd": ((9, 20, 41), (O, O, W, W, C, O), 1, False),
    "even": ((7, 31, 64), (C, W, C, C, C, C), 0, False),
    "gravity": ((12, 15, 33), (P, P, O, W, C, W), 1, True),
    "narrow": ((6, 14, 3), (W, C, P, P, C, C), 0, True),
}


def first_column(shape, bcs, limiter, gravity):
    prim = [p.astype(np.float32) for p in random_primitives(shape, 21)]
    prim[4] = prim[4] * np.float32(80000)              # air near 273 K, as wall_heat takes it
    ctx = capi.Context(shape, 0.5 / max(shape), bcs, gamma=1.4, cfl=0.2, limiter=limiter, gravity=gravity,
                       precision=capi.F32)
    ctx.set_primitives(prim)
    ctx.compute_step(1)
    energy = ctx.get_conserved()[4][2:-2, 2:-2, 2].copy()
    ctx.close()
    return energy


@pytest.mark.gpu
@pytest.mark.parametrize("case", list(CASES))
def test_first_column(case):
    with np.load(GOLDEN) as g:
        np.testing.assert_array_equal(first_column(*CASES[case]), g[case])
