"""The one-cell-per-lane step kernel (FP64, and FP32 with the reference's
rounding): sizes around its 14-row x 32-column tiles and short chunks, bit for
bit against the oracle; states whose quotients leave the range in which a
shared reciprocal is exact (they take the plain division); and, on the CPU,
the quotient scheme itself."""
import ctypes
import ctypes.util

import numpy as np
import pytest

from conftest import INTERIOR, random_primitives, rel_l1
from deepgreen import capi

P, O, W, C = capi.PERIODIC, capi.OUTFLOW, capi.WALL, capi.CONDUCTING_WALL
KINDS = [(capi.F64, capi.ROUNDING_REFERENCE), (capi.F32, capi.ROUNDING_REFERENCE), (capi.F64, capi.ROUNDING_FAST)]
BCS = [(P,) * 6, (O,) * 6, (W, W, O, O, P, P), (C, W, W, C, C, W)]
# each axis below, at and above a tile (rows 14, columns 32), several tiles, the smallest grid
SHAPES = [(2, 2, 2), (3, 13, 31), (5, 14, 32), (4, 15, 33), (9, 29, 64), (7, 28, 66), (30, 3, 97)]


def run_both(shape, ds, bcs, prim, steps, kind, limiter, gravity, chunk=0):
    import pyoracle
    precision, rounding = kind
    exact = rounding == capi.ROUNDING_REFERENCE
    dtype = np.float64 if precision == capi.F64 else np.float32
    prim = [np.asarray(a, dtype=dtype) for a in prim]
    o = pyoracle.Oracle(shape, ds, bcs, gamma=1.4, cfl=0.3, limiter=limiter, gravity=gravity, dtype=dtype,
                        threads=pyoracle.ALL_PARALLEL)
    o.set_primitives(prim)
    ref_dts = o.step(steps)
    ctx = capi.Context(shape, ds, bcs, gamma=1.4, cfl=0.3, limiter=limiter, gravity=gravity, precision=precision,
                       rounding=rounding)
    ctx.set_chunk(chunk)
    ctx.set_primitives(prim)
    dts = ctx.compute_step(steps)
    cons = ctx.get_conserved()
    ref = o.conserved()
    if not exact and not all(np.isfinite(r[INTERIOR]).all() for r in ref):
        # a conducting wall next to a unit gas heats the smallest grids until
        # the oracle's own state is not finite: nothing to compare but that
        assert not all(np.isfinite(c[INTERIOR]).all() for c in cons)
        return
    for f in range(5):
        if exact:
            np.testing.assert_array_equal(cons[f][INTERIOR], ref[f][INTERIOR], err_msg=f"field {f}")
        else:
            assert rel_l1(cons[f], ref[f]) <= 1e-12
    if exact:
        np.testing.assert_array_equal(dts, ref_dts)
    else:
        np.testing.assert_allclose(dts, ref_dts, rtol=1e-13)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("bcs", BCS)
@pytest.mark.parametrize("shape", SHAPES)
def test_tile_edges(shape, bcs, kind):
    for limiter in (0, 1):
        run_both(shape, 0.05, bcs, random_primitives(shape, 31), 3, kind, limiter, limiter == 0, chunk=limiter * 2)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [capi.F64, capi.F32])
@pytest.mark.parametrize("case", ["tiny_ds", "huge_ds", "tiny_velocity", "zero_velocity", "tiny_slopes", "huge_state"])
def test_quotients_outside_the_shared_range(case, precision):
    shape = (6, 15, 34)
    f64 = precision == capi.F64
    prim = random_primitives(shape, 5)
    ds = 0.05
    if case == "tiny_ds":
        ds = 1e-95 if f64 else 1e-11
    elif case == "huge_ds":
        ds = 1e99 if f64 else 1e9
    elif case == "tiny_velocity":
        s = 1e-160 if f64 else 1e-24
        prim = [prim[0]] + [p * s for p in prim[1:4]] + [prim[4]]
    elif case == "zero_velocity":
        prim = [prim[0]] + [p * 0 for p in prim[1:4]] + [prim[4]]
    elif case == "tiny_slopes":
        s = 1e-200 if f64 else 1e-28
        prim = [np.ones_like(prim[0]), np.zeros_like(prim[1]), prim[2] * s, prim[3] * s, np.ones_like(prim[4])]
    else:
        s = 1e65 if f64 else 1e9
        prim = [prim[0]] + [p * s for p in prim[1:4]] + [prim[4] * s * s]
    for limiter in (0, 1):
        run_both(shape, ds, (P,) * 6, prim, 2, (precision, capi.ROUNDING_REFERENCE), limiter, False)


@pytest.mark.parametrize("dtype,name", [(np.float32, "fmaf"), (np.float64, "fma")])
def test_shared_divisor_quotient_is_the_ieee_quotient(dtype, name):
    """q0 = RN(a y), y = RN(1/b); RN(q0 - (b q0 - a) y) == RN(a / b), on random
    mantissas and the divisors next to a power of two, where q0 is furthest
    off; zeros keep their sign."""
    libm = ctypes.CDLL(ctypes.util.find_library("m"))
    fma = getattr(libm, name)
    ct = ctypes.c_float if dtype == np.float32 else ctypes.c_double
    fma.restype, fma.argtypes = ct, [ct] * 3
    rng = np.random.default_rng(3)
    eps = np.finfo(dtype).eps
    one, two = dtype(1), dtype(2)
    edge_b = [two - dtype(k) * eps for k in range(1, 40)] + [one + dtype(k) * eps for k in range(40)]
    pairs = [(dtype(rng.uniform(1, 2)), dtype(rng.uniform(1, 2))) for _ in range(8000)]
    pairs += [(dtype(rng.uniform(1.9, 2)), b) for b in edge_b for _ in range(40)]
    pairs += [(dtype(0.0), b) for b in edge_b] + [(-dtype(0.0), b) for b in edge_b]
    for a, b in pairs:
        y = one / b
        q0 = a * y
        nr = dtype(fma(float(b), float(q0), float(-a)))
        q = dtype(fma(float(-nr), float(y), float(q0)))
        ref = a / b
        assert q == ref and np.signbit(q) == np.signbit(ref), (a, b)
