"""How the convolutions divide their work among the blocks (CPU): every plane of
every column once, and the busiest block marches no more planes than with
whole columns dealt out in turn, nor more than the start of one piece above the
fixed chunks of 8 to 64 planes that the same kernels once took."""
import random
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
SMS = 148


def layers(shape):
    """Columns and their length in the four convolutions of a forward pass."""
    n, x, y, z = shape
    for _ in range(4):
        yield n * -(-((y - 2) * z) // 128), x - 2
        x, y, z = x - 2, y - 2, z - 2


def fixed_chunks(columns, length, blocks):
    for chunk in (64, 32, 16, 8):
        units = columns * -(-length // chunk)
        if units >= 4 * SMS:
            break
    per, rest = divmod(units, blocks)
    pieces = -(-length // chunk)
    most = 0
    for b in range(min(blocks, units)):
        mine = sum(min(chunk, length - u % pieces * chunk) + 2 for u in range(b, units, blocks))
        most = max(most, mine)
    return most


@pytest.fixture(scope="module")
def shares(tmp_path_factory):
    exe = tmp_path_factory.mktemp("conv_share") / "conv_share"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", "-I",
                        str(ROOT / "deep-green_b200" / "csrc"), str(ROOT / "tests" / "cpp" / "conv_share.cpp"), "-o",
                        str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]

    def run(cases):
        out = subprocess.run([str(exe)], input="\n".join("%d %d %d" % c for c in cases), capture_output=True, text=True,
                             check=True).stdout.split()
        return list(zip(map(int, out[::2]), map(int, out[1::2])))
    return run


def cases():
    rng = random.Random(5)
    shapes = [(1, 9, 9, 9), (1, 264, 264, 264), (8, 73, 73, 73), (4, 12, 300, 300), (1, 13, 400, 400), (1, 20, 400, 400),
              (200, 12, 16, 24), (64, 20, 20, 20), (16, 40, 40, 40)]
    shapes += [(rng.choice([1, 1, 2, 8, 40]), int(2 ** rng.uniform(3.2, 8)), int(2 ** rng.uniform(3.2, 8)),
                int(2 ** rng.uniform(3.2, 8))) for _ in range(60)]
    for s in shapes:
        for columns, length in layers(s):
            blocks = min(columns * length, SMS)
            if blocks > 0 and length > 0 and columns * length < 1 << 22:
                yield columns, length, blocks


def test_every_step_once_and_no_block_behind(shares):
    todo = list(cases())
    for (columns, length, blocks), (once, most) in zip(todo, shares([(c * n, n, b) for c, n, b in todo])):
        assert once, (columns, length)
        assert most <= -(-columns // blocks) * (length + 2), (columns, length, most)
        assert most <= fixed_chunks(columns, length, blocks) + 2, (columns, length, most)
