"""The first batch of a training run.  Batcher zeroes its buffers on the
default stream, so the crops have to be written behind that work: on the
default stream too, which a training pass waits for."""
import pytest

from deepgreen import learned
from deepgreen import net as dnet


def test_batches_are_filled_where_their_buffers_are_zeroed(monkeypatch):
    streams = []

    class Batches:
        feat = tgt = None

        def __init__(self, *a):
            pass

        def fill(self, norm, stream=None):
            streams.append(stream)

    class OwnStreamNet:
        def stream(self):
            return 0x5000

        def forward_backward_flux(self, feat, tgt, balance):
            return 1.0

        def adam_step(self, rate):
            pass

    monkeypatch.setattr(learned, "Batcher", Batches)
    assert learned.train(OwnStreamNet(), None, None, 3, log=lambda *a: None) == [1.0] * 3
    assert streams == [None] * 3


@pytest.mark.gpu
def test_first_batch_behind_a_busy_default_stream():
    import torch

    quiet = lambda *a: None  # noqa: E731
    ps = learned.make_pairs(32, [("kh", 1)], 2, 2, 4, 0, log=quiet)
    norm = learned.fit_norm(ps, 8, 16, 0)
    losses = []
    for busy in (False, True, True):
        net = dnet.Net(learned.INPUTS, learned.OUTPUTS, seed=0, out_scale=0.1)
        torch.cuda.synchronize()
        if busy:
            torch.cuda._sleep(20_000_000)      # ~10 ms ahead of the buffers' zeroing
        losses.append(learned.train(net, ps, norm, 2, batch=4, crop=24, seed=0, log=quiet))
    assert losses[1] == losses[0] and losses[2] == losses[0]
