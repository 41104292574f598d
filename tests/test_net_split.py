"""The convolutions' division of work, at the sizes where it changes.

The forward kernel gives each block an equal share of all output planes; a
plane's values do not depend on the share it falls in, so a batch must equal
its entries run alone, bit for bit, with fewer columns of tiles than SMs, as
many, and more.
"""
import numpy as np
import pytest

from deepgreen import net as dnet

pytestmark = pytest.mark.gpu

def features(shape, inputs, seed):
    import torch

    g = torch.Generator().manual_seed(seed)
    f = torch.zeros(*shape, dnet.IO_CHANNELS, dtype=torch.bfloat16)
    f[..., :inputs] = torch.randn(*shape, inputs, generator=g).to(torch.bfloat16)
    return f


@pytest.mark.parametrize("shape", [(1, 9, 9, 9), (3, 12, 30, 41), (37, 11, 20, 26), (5, 10, 70, 73)])
def test_batch_equals_its_entries(shape):
    import torch

    net = dnet.Net(14, 15, seed=6, out_scale=1.0)
    f = features(shape, 14, 1).cuda()
    out = net.forward(f)
    net.synchronize()
    out = out.clone()
    for b in range(shape[0]):
        one = net.forward(f[b:b + 1].contiguous())
        net.synchronize()
        assert torch.equal(one[0], out[b]), b


def test_update_packs_the_weights_it_writes():
    import torch

    f = features((2, 12, 12, 12), 14, 5).cuda()
    t = torch.randn(2, 4, 4, 4, dnet.IO_CHANNELS, generator=torch.Generator().manual_seed(6)).cuda()
    net = dnet.Net(14, 15, seed=7, out_scale=1.0)
    net.forward_backward(f, t)
    net.adam_step(1e-2)
    other = dnet.Net(14, 15, seed=8, out_scale=1.0)
    other.set_params(net.params())
    for n in (net, other):
        n.forward_backward(f, t)
    for l in range(4):
        k = 2 * (l + 1)
        shape = (2, 12 - k, 12 - k, 12 - k, 32 if l < 3 else 16)
        assert np.array_equal(net.get_tensor(l, 3, shape), other.get_tensor(l, 3, shape)), l
        for a, b in zip(net.get_grad(l), other.get_grad(l)):
            assert np.array_equal(a, b), l
