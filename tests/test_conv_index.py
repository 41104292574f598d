"""Output positions of the convolutions in 64 bits, on the CPU: planes of as
many positions as the entry points accept (up to 2^30), where a plane of 32
channels passes 2^31 elements."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "deep-green_b200" / "csrc"

# (batch, x, y, z) of a network input: small, just below and above 2^31
# elements per plane of 32 and of 16 channels, the widest plane accepted
INPUTS = [(3, 12, 30, 41), (1, 9, 8193, 8193), (1, 9, 8195, 8195), (2, 11, 11589, 11587), (1, 9, 9, 119304647)]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = tmp_path_factory.mktemp("conv_index") / "conv_index"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", "-I", str(CSRC),
                        str(ROOT / "tests" / "cpp" / "conv_index.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    return exe


@pytest.mark.parametrize("shape", INPUTS)
def test_output_positions(program, shape):
    n, x, y, z = shape
    lines, want = [], []
    for layer in range(4):
        ch = 32 if layer < 3 else 16
        ex, ey, ez = x - 2 * (layer + 1), y - 2 * (layer + 1), z - 2 * (layer + 1)
        for pad in (0, 2):                       # dense outputs; gradients padded by 2
            nx, ny, nz = ex + 2 * pad, ey + 2 * pad, ez + 2 * pad
            for x0 in (0, ex - 1):
                for py, pz in ((0, 0), (ey - 1, ez - 1)):
                    for c0 in (0, ch // 2):
                        for k in (0, ex - 1 - x0):
                            at = (n - 1, x0 + pad, py + pad, pz + pad, nx, ny, nz, ch, c0, k)
                            lines.append(" ".join(map(str, at)))
                            want.append(((((n - 1) * nx + x0 + pad + k) * ny + py + pad) * nz + pz + pad) * ch + c0)
    out = subprocess.run([str(program)], input="\n".join(lines), capture_output=True, text=True, check=True).stdout
    assert [int(v) for v in out.split()] == want


def test_the_epilogue_takes_its_positions_from_there():
    """No product of two extents and the channel count in the kernel's own
    arithmetic: it passes 2^31 within the sizes that are accepted."""
    text = (CSRC / "dg_conv.cuh").read_text()
    for line in text.splitlines():
        code = line.split("//")[0]
        assert not ("* COUT" in code and ("a.oy" in code or "a.yo" in code or "a.oz" in code or "a.zo" in code)), line
    assert text.count("PlaneIndex") >= 2
