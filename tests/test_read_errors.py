"""Which error a read reports: a context without a state says so, whatever the
field pointers are; with one, a null field is an invalid argument."""
import pytest

from conftest import random_primitives
from deepgreen import capi


@pytest.mark.gpu
@pytest.mark.parametrize("call", ["dg_get_conserved", "dg_get_conserved_device", "dg_get_primitives"])
def test_no_state_comes_before_null_fields(call):
    shape = (4, 3, 5)
    ctx = capi.Context(shape, 0.1, (capi.PERIODIC,) * 6, gamma=1.4, cfl=0.4)
    fields = capi._PP5(*[None] * 5)
    read = getattr(ctx.lib, call)
    assert read(ctx.h, fields) == capi.DG_ERR_NO_STATE
    ctx.set_primitives(random_primitives(shape, 1))
    assert read(ctx.h, fields) == capi.DG_ERR_INVALID
    assert b"null field" in ctx.lib.dg_last_error(ctx.h)
    ctx.compute_step(1)                        # the state is as it was
