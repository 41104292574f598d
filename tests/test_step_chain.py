"""Steps enqueued together equal steps taken one by one, bit for bit.

Consecutive steps of one call overlap: a step's blocks take SMs as the step
before it leaves them and wait there for its end.  Steps of separate calls,
synchronised in between, do not.  For each step kernel, with fewer blocks than
SMs, about as many, and (FP32) with interior tiles, both must give the same
states and the same dt history.
"""
import numpy as np
import pytest

from deepgreen import capi

pytestmark = pytest.mark.gpu

KINDS = {
    "f32": dict(precision=capi.F32),
    "f64": dict(precision=capi.F64),
    "f64-fast": dict(precision=capi.F64, rounding=capi.ROUNDING_FAST),
    "f32-reference": dict(precision=capi.F32, rounding=capi.ROUNDING_REFERENCE),
}


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("shape", [(5, 6, 7), (40, 33, 70), (64, 64, 64), (24, 120, 200)])
def test_steps_of_one_call_equal_single_steps(kind, shape):
    rng = np.random.default_rng(4)
    ghosted = tuple(n + 4 for n in shape)
    prim = [1 + 0.2 * rng.random(ghosted)] + [0.2 * rng.random(ghosted) for _ in range(3)] + [1 + 0.2 * rng.random(ghosted)]
    runs = []
    for calls in ((12,), (1,) * 12, (5, 7)):
        ctx = capi.Context(shape, 1 / 64, (capi.PERIODIC,) * 6, **KINDS[kind])
        ctx.set_primitives([p.astype(ctx.dtype) for p in prim])
        dts = np.concatenate([ctx.compute_step(n) for n in calls])
        runs.append((ctx.get_conserved(), dts))
        ctx.close()
    for state, dts in runs[1:]:
        assert np.array_equal(dts, runs[0][1])
        for a, b in zip(state, runs[0][0]):
            assert np.array_equal(a, b)
