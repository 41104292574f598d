"""Which grids the no-allocation step takes: every answer stays what it was when
its scratch held 56 bytes per block of the kernels of that time, 18134 blocks in
all.  The counts below come from those kernels' own rules."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

from conftest import random_primitives
from deepgreen import capi, setups

ROOT = Path(__file__).resolve().parents[1]

# kernel (0: reference rounding FP64, 1: FP32, 2: fused FP32, 3: FP64), nx, ny, nz, blocks
GRIDS = [
    (0, 41, 1071, 1877, 15812),
    (0, 37, 705, 2818, 15753),
    (0, 364, 2496, 811, 16224),
    (0, 187, 1265, 1623, 16167),
    (0, 62, 1438, 1584, 18000),
    (0, 18, 1887, 1194, 17936),
    (0, 395, 1685, 1351, 18146),
    (0, 9, 778, 2977, 18330),
    (1, 23, 3389, 1182, 15688),
    (1, 77, 2226, 1766, 15624),
    (1, 290, 1611, 2516, 15958),
    (1, 361, 1608, 2623, 16482),
    (1, 20, 2837, 1606, 18105),
    (1, 50, 3055, 1480, 17954),
    (1, 81, 2395, 1945, 18300),
    (1, 57, 1878, 2493, 18330),
    (2, 211, 3898, 3009, 16173),
    (2, 259, 3718, 2945, 16046),
    (3, 28, 2152, 1840, 15602),
    (3, 82, 2987, 1192, 15721),
    (3, 40, 2436, 1690, 16443),
    (3, 359, 2023, 1391, 16392),
    (3, 46, 2256, 2004, 18048),
    (3, 13, 3777, 1180, 17955),
    (3, 238, 3638, 844, 18272),
    (3, 305, 2061, 1710, 18360),
    (0, 2, 2, 2, 1),
    (1, 2, 2, 2, 1),
    (2, 2, 2, 2, 1),
    (3, 2, 2, 2, 1),
    (0, 48, 48, 48, 48),
    (1, 48, 48, 48, 24),
    (2, 48, 48, 48, 8),
    (3, 48, 48, 48, 24),
    (0, 508, 508, 508, 6096),
    (1, 508, 508, 508, 5120),
    (2, 508, 508, 508, 898),
    (3, 508, 508, 508, 2878),
    (0, 1000, 1000, 1000, 8000),
    (1, 1000, 1000, 1000, 8000),
    (2, 1000, 1000, 1000, 3732),
    (3, 1000, 1000, 1000, 11920),
    (0, 100000, 4, 4, 4000),
    (1, 100000, 4, 4, 4000),
    (2, 100000, 4, 4, 64),
    (3, 100000, 4, 4, 64),
    (0, 4, 4, 100000, 3125),
    (1, 4, 4, 100000, 3125),
    (2, 4, 4, 100000, 1563),
    (3, 4, 4, 100000, 1563),
    (0, 4, 30000, 60, 15000),
    (1, 4, 30000, 60, 7500),
    (2, 4, 30000, 60, 2143),
    (3, 4, 30000, 60, 7500),
    (0, 700, 700, 700, 7700),
    (1, 700, 700, 700, 5808),
    (2, 700, 700, 700, 1730),
    (3, 700, 700, 700, 5605),
]


def test_counts_and_answers(tmp_path):
    exe = tmp_path / "noalloc_limit"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", "-I",
                        str(ROOT / "deep-green_b200" / "csrc"), str(ROOT / "tests" / "cpp" / "noalloc_limit.cpp"), "-o",
                        str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    lines = "\n".join(f"{nx} {ny} {nz} {int(k in (0, 3))} {int(k >= 2)}" for k, nx, ny, nz, _ in GRIDS)
    out = subprocess.run([str(exe)], input=lines, capture_output=True, text=True, check=True).stdout.split()
    assert list(zip(map(int, out[::2]), map(int, out[1::2]))) == [(b, int(b <= 18134)) for *_, b in GRIDS]
    assert any(15867 < b <= 18134 for *_, b in GRIDS)


@pytest.mark.gpu
@pytest.mark.parametrize("precision,shape", [(capi.F64, (2, 536, 4288)), (capi.F32, (2, 1072, 4288))])
def test_step_just_below_the_limit(precision, shape):
    import torch
    dtype = np.float64 if precision == capi.F64 else np.float32
    cons = [np.asarray(c, dtype) for c in setups.conserved_from_primitives(random_primitives(shape, 4), 0.5, 1.4)]
    bcs = (capi.PERIODIC,) * 6
    ctx = capi.Context(shape, 0.5, bcs, gamma=1.4, cfl=0.3, precision=precision, rounding=capi.ROUNDING_REFERENCE)
    ctx.set_conserved(cons)
    want_dt = ctx.compute_step(1)[0]
    want = ctx.get_conserved()
    info = ctx.info
    a = torch.from_numpy(np.stack(cons)).cuda()
    b = torch.zeros_like(a)
    torch.cuda.synchronize()
    dt = ctypes.c_double()
    rc = ctx.lib.dg_compute_step_noalloc(ctypes.byref(info), ctypes.c_void_p(a.data_ptr()),
                                         ctypes.c_void_p(b.data_ptr()), ctypes.byref(dt), None)
    assert rc == capi.DG_OK, ctx.lib.dg_last_error(None)
    assert dt.value == want_dt
    got = b.cpu().numpy()
    for f in range(5):
        np.testing.assert_array_equal(got[f], want[f])
