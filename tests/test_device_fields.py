"""dg_set_conserved_device / dg_get_conserved_device on fields that a copy
serves and a kernel's loads and stores do not: the rule that tells them apart
(CPU; fields on another GPU only here), and a round trip through fields off
their elements' alignment and through fields that end with their allocation."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

from conftest import random_primitives
from deepgreen import capi, setups

ROOT = Path(__file__).resolve().parents[1]

MB = 1 << 20
# device memory?, its GPU, foreign context?, allocation's start and size, p, bytes, element, context's GPU
OWN = (1, 0, 0, MB, MB, MB, 4096, 4, 0)
RULE = [
    (OWN, 1),
    ((1, 0, 0, MB, MB, MB + 8, 4096, 8, 0), 1),
    ((1, 3, 0, MB, MB, MB, 4096, 4, 3), 1),
    ((1, 0, 0, MB, MB, 2 * MB - 4096, 4096, 4, 0), 1),         # ends with its allocation
    ((1, 0, 0, MB, MB, 2 * MB - 4092, 4096, 4, 0), 0),         # ends behind it
    ((1, 0, 0, MB, MB, MB, 2 * MB, 4, 0), 0),
    ((1, 0, 0, MB, MB, 2 ** 64 - 4, 4096, 4, 0), 0),
    ((1, 0, 0, MB, MB, MB - 4, 4096, 4, 0), 0),                # begins before it
    ((1, 1, 0, MB, MB, MB, 4096, 4, 0), 0),                    # on another GPU
    ((0, 0, 0, MB, MB, MB, 4096, 4, 0), 0),                    # host or managed memory
    ((1, 0, 1, MB, MB, MB, 4096, 4, 0), 0),                    # another context's
    ((1, 0, 0, MB, MB, MB + 2, 4096, 4, 0), 0),                # off its elements' alignment
    ((1, 0, 0, MB, MB, MB + 4, 4096, 8, 0), 0),
    ((0, -1, 0, 0, 0, MB, 4096, 4, 0), 0),                     # nothing known
]


def test_rule(tmp_path):
    exe = tmp_path / "pointer_rule"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", "-I",
                        str(ROOT / "deep-green_b200" / "csrc"), str(ROOT / "tests" / "cpp" / "pointer_rule.cpp"), "-o",
                        str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    lines = "\n".join(" ".join(map(str, case)) for case, _ in RULE)
    out = subprocess.run([str(exe)], input=lines, capture_output=True, text=True, check=True).stdout
    assert [int(v) for v in out.split()] == [want for _, want in RULE]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [capi.F32, capi.F64])
@pytest.mark.parametrize("offset", [0, 1, 2, 4, 12])
def test_round_trip_at_any_byte_offset(precision, offset):
    import torch
    shape = (5, 4, 28)
    dtype = np.float32 if precision == capi.F32 else np.float64
    prim = [np.asarray(a, dtype) for a in random_primitives(shape, 8)]
    cons = [np.asarray(c, dtype) for c in setups.conserved_from_primitives(prim, 0.125, 1.4)]
    nbytes = cons[0].nbytes
    raw = np.concatenate([c.reshape(-1).view(np.uint8) for c in cons])
    # one allocation, the last field at its end
    src = torch.zeros(offset + 5 * nbytes, dtype=torch.uint8, device="cuda")
    out = torch.zeros(offset + 5 * nbytes, dtype=torch.uint8, device="cuda")
    src[offset:] = torch.from_numpy(raw).cuda()
    torch.cuda.synchronize()
    ctx = capi.Context(shape, 0.125, (capi.PERIODIC,) * 6, gamma=1.4, cfl=0.4, precision=precision)
    ctx.set_conserved(cons)                    # host arrays: what the device arrays must give
    want, dt = ctx.get_conserved(), ctx.next_dt()
    ptrs = lambda t: [t.data_ptr() + offset + f * nbytes for f in range(5)]  # noqa: E731
    ctx.set_conserved_device(ptrs(src))
    assert ctx.next_dt() == dt
    ctx.get_conserved_device(ptrs(out))
    got = out.cpu().numpy()
    assert not got[:offset].any()
    for f in range(5):
        field = got[offset + f * nbytes:offset + (f + 1) * nbytes].copy().view(dtype).reshape(want[f].shape)
        np.testing.assert_array_equal(field, want[f])
    # and from a state set through unaligned fields, a step
    a = ctx.compute_step(2)
    ctx.set_conserved(cons)
    np.testing.assert_array_equal(a, ctx.compute_step(2))
