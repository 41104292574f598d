"""A training pass waits for the batch that the default stream still fills.

dg_learned_features and dg_learned_targets with stream NULL, and torch, work on
the default stream; the network has a stream of its own.  The batch is
overwritten behind a long kernel on the default stream and the pass called at
once: loss and gradients must be those of the new batch.  And two equal
training runs give equal weights.
"""
import numpy as np
import pytest

from deepgreen import learned
from deepgreen import net as dnet

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flux", [False, True])
def test_pass_waits_for_the_default_stream(flux):
    import torch

    net = dnet.Net(14, 15, seed=2, out_scale=1.0)
    g = torch.Generator().manual_seed(3)
    feat = torch.randn(2, 20, 20, 20, 16, generator=g).to(torch.bfloat16).cuda()
    t = 11 if flux else 12
    tgt = torch.randn(2, t, t, t, 16, generator=g).cuda()
    run = net.forward_backward_flux if flux else net.forward_backward
    torch.cuda.synchronize()
    want = run(feat, tgt), [a.copy() for l in range(4) for a in net.get_grad(l)]
    f, q = torch.zeros_like(feat), torch.zeros_like(tgt)
    run(f, q)
    torch.cuda.synchronize()
    torch.cuda._sleep(20_000_000)              # ~10 ms
    f.copy_(feat)
    q.copy_(tgt)
    got = run(f, q), [a for l in range(4) for a in net.get_grad(l)]
    assert got[0] == want[0]
    for a, b in zip(got[1], want[1]):
        assert np.array_equal(a, b)


def test_training_is_reproducible():
    quiet = lambda *a: None
    ps = learned.make_pairs(32, [("kh", 1), ("fourier", 2)], 2, 2, 4, 0, log=quiet)
    norm = learned.fit_norm(ps, 8, 16, 0)
    runs = []
    for _ in range(3):
        net = dnet.Net(learned.INPUTS, learned.OUTPUTS, seed=0, out_scale=0.1)
        hist = learned.train(net, ps, norm, 60, batch=8, crop=24, lr=1e-3, seed=0, log=quiet)
        runs.append((hist, net.params()))
    for hist, params in runs[1:]:
        assert hist == runs[0][0]
        for (w, b), (w0, b0) in zip(params, runs[0][1]):
            assert np.array_equal(w, w0) and np.array_equal(b, b0)
