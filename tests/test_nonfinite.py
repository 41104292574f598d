"""A state with a cell that is not finite, one step: which cells it reaches.

The limiter is zero beside a NaN difference (the product test of minmod fails),
so a cell next to the NaN keeps a finite prediction and finite faces on its
other sides: the cell itself and its six neighbours become NaN, no others, in
every kernel as in the oracle.  Without a limiter the slopes themselves carry
it on, in every kernel alike."""
import numpy as np
import pytest

from conftest import INTERIOR, random_primitives
from deepgreen import capi

KINDS = [(capi.F64, capi.ROUNDING_REFERENCE), (capi.F64, capi.ROUNDING_FAST), (capi.F32, capi.ROUNDING_REFERENCE),
         (capi.F32, capi.ROUNDING_FAST)]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("limiter", [capi.LIMITER_NONE, capi.LIMITER_MINMOD])
@pytest.mark.parametrize("at", [(6, 9, 12), (6, 15, 34)])
def test_reach_of_a_nan(kind, limiter, at):
    import pyoracle
    precision, rounding = kind
    dtype = np.float64 if precision == capi.F64 else np.float32
    shape = (9, 20, 40)
    prim = [np.asarray(a, dtype) for a in random_primitives(shape, 12)]
    prim[4][at] = np.nan
    # NaN in the state: dt = cfl (physics.rs:191-195), kept well inside ds
    kw = dict(gamma=1.4, cfl=0.01, limiter=limiter)
    o = pyoracle.Oracle(shape, 1.0, (capi.OUTFLOW,) * 6, dtype=dtype, threads=pyoracle.ALL_PARALLEL, **kw)
    o.set_primitives(prim)
    o.step(1)
    want = [~np.isfinite(c[INTERIOR]) for c in o.conserved()]
    ctx = capi.Context(shape, 1.0, (capi.OUTFLOW,) * 6, precision=precision, rounding=rounding, **kw)
    ctx.set_primitives(prim)
    ctx.enqueue_steps(1)
    got = [~np.isfinite(c[INTERIOR]) for c in ctx.get_conserved()]
    assert want[4].any()
    for f in range(5):
        np.testing.assert_array_equal(got[f], want[f], err_msg=f"field {f}")
