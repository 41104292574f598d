"""Setting a state from device arrays and reading it back: the row kernels with
16-byte accesses (aligned rows) and without (odd rows, unaligned pointers),
every ghost cell from its interior source, bit for bit; the dt of the set
state against the host's."""
import numpy as np
import pytest

from conftest import random_primitives
from deepgreen import capi, setups

P, O, W = capi.PERIODIC, capi.OUTFLOW, capi.WALL


def axis_source(n, lo, hi):
    """Source index and mirror flag of every ghosted index of an axis."""
    src, flip = list(range(n)), [False] * n
    for g, low in ((0, True), (1, True), (n - 2, False), (n - 1, False)):
        bc, k = (lo, g) if low else (hi, n - 1 - g)       # k: distance from the edge, 0 or 1
        edge = 2 if low else n - 3
        step = 1 if low else -1
        if bc == P:
            src[g] = (n - 4 + k) if low else (3 - k)
        elif bc == O:
            src[g] = edge
        else:
            src[g], flip[g] = edge + step * (1 - k), True
    return np.array(src), np.array(flip)


def with_ghosts(cons, bcs):
    idx = [axis_source(cons[0].shape[a], bcs[2 * a], bcs[2 * a + 1]) for a in range(3)]
    out = [c[np.ix_(*(s for s, _ in idx))].copy() for c in cons]
    for a in range(3):
        sh = [1, 1, 1]
        sh[a] = -1
        out[1 + a] = np.where(idx[a][1].reshape(sh), -out[1 + a], out[1 + a])
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [capi.F32, capi.F64])
@pytest.mark.parametrize("bcs", [(P,) * 6, (O,) * 6, (W,) * 6, (W, O, P, P, O, W)])
@pytest.mark.parametrize("shape,offset", [((2, 2, 4), 0), ((5, 3, 28), 0), ((3, 6, 124), 0), ((4, 5, 129), 0),
                                          ((5, 4, 28), 1), ((3, 3, 2), 0), ((2, 7, 61), 3)])
def test_device_state_round_trip(shape, offset, bcs, precision):
    import torch
    dtype = np.float32 if precision == capi.F32 else np.float64
    prim = [np.asarray(a, dtype) for a in random_primitives(shape, 8)]
    ds, gamma, cfl = 0.125, 1.4, 0.4
    cons = [np.asarray(c, dtype) for c in setups.conserved_from_primitives(prim, ds, gamma)]
    cells = cons[0].size
    flat = torch.zeros(5 * cells + 8, dtype=torch.float32 if precision == capi.F32 else torch.float64, device="cuda")
    out = torch.zeros_like(flat)
    flat[offset:offset + 5 * cells] = torch.from_numpy(np.concatenate([c.reshape(-1) for c in cons])).cuda()
    torch.cuda.synchronize()
    ctx = capi.Context(shape, ds, bcs, gamma=gamma, cfl=cfl, precision=precision)
    elem = flat.element_size()
    ptrs = lambda t: [t.data_ptr() + (offset + f * cells) * elem for f in range(5)]  # noqa: E731
    ctx.set_conserved_device(ptrs(flat))
    ctx.get_conserved_device(ptrs(out))
    got = out.cpu().numpy()
    want = np.concatenate([c.reshape(-1) for c in with_ghosts(cons, bcs)])
    np.testing.assert_array_equal(got[offset:offset + 5 * cells], want)
    assert not got[:offset].any() and not got[offset + 5 * cells:].any()
    # host arrays take the same kernels
    ctx.set_conserved(cons)
    for g, w in zip(ctx.get_conserved(), with_ghosts(cons, bcs)):
        np.testing.assert_array_equal(g, w)
    i = (slice(2, -2),) * 3
    r, vx, vy, vz, p = (np.asarray(a, np.float64)[i] for a in prim)
    dt = cfl * (ds / (np.sqrt(gamma * p / r) + np.sqrt(vx * vx + vy * vy + vz * vz))).min()
    # FP32: totals, primitives and speeds each round a few times (2^-24 each)
    np.testing.assert_allclose(ctx.next_dt(), dt, rtol=2e-6 if precision == capi.F32 else 1e-14)
