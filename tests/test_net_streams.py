"""The corrector runs the network on its grid's stream; optimizer updates run on
the network's own.  Neither stream waits for the other by itself: a corrected
step behind an update takes the new weights, an update behind a corrected step
leaves it the old ones, also where the stream in front is busy."""
import numpy as np
import pytest

from conftest import random_primitives
from deepgreen import learned
from deepgreen import net as dnet

pytestmark = pytest.mark.gpu

N = 24


def corrected_state(update_first, wait):
    import torch

    net = dnet.Net(learned.INPUTS, learned.OUTPUTS, seed=5, out_scale=1.0)
    grid = learned.grid(N)
    norm = learned.Norm.identity()
    for c in range(5):
        norm.out_std[c] = 1e-4
    cor = learned.Corrector(grid, net, norm, tolerance=1.0)
    # a training pass of the corrector's extents: gradients, and a workspace
    # that the corrector need not replace
    gen = torch.Generator().manual_seed(1)
    feat = torch.randn(1, N + 8, N + 8, N + 8, 16, generator=gen).to(torch.bfloat16).cuda()
    tgt = torch.randn(1, N, N, N, 16, generator=gen).cuda()
    net.forward_backward(feat, tgt)
    grid.set_primitives(random_primitives((N,) * 3, 9))
    torch.cuda.synchronize()
    first = net.stream() if update_first else grid.stream()
    if not wait:
        with torch.cuda.stream(torch.cuda.ExternalStream(int(first))):
            torch.cuda._sleep(20_000_000)      # ~10 ms
    for step in (("update", "correct") if update_first else ("correct", "update")):
        if step == "update":
            net.adam_step(0.1)
        else:
            cor.step(1)
        if wait:
            torch.cuda.synchronize()
    torch.cuda.synchronize()
    state = grid.get_conserved()
    assert cor.stats()["fallback_steps"] == 0
    cor.close()
    return state


def test_updates_and_corrected_steps_keep_their_order():
    states = {}
    for update_first in (True, False):
        a, b = (corrected_state(update_first, wait) for wait in (True, False))
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
        states[update_first] = a
    assert any(not np.array_equal(x, y) for x, y in zip(states[True], states[False]))   # the update matters
