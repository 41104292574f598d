"""The convolutions' division of work, at the sizes where it changes.

The forward kernel gives each block an equal share of all output planes; a
plane's values do not depend on the share it falls in, so a batch must equal
its entries run alone, bit for bit, with fewer columns of tiles than SMs, as
many, and more.

The weight-gradient kernel copies rows of z rounded up to 16 positions (128 at
most) into a ring as deep as they leave room for.  Row lengths on both sides
of those steps are compared with the weight gradient of the very tensors that
the pass stored, in float64.  Every step of 16 positions and every block's
partial is one FP32 addition, off by at most 2^-22 of the sum of the products'
magnitudes.
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


@pytest.mark.parametrize("shape", [(1, 9, 9, 9), (8, 20, 9, 10), (2, 10, 12, 24), (1, 11, 10, 25), (1, 10, 11, 136),
                                   (1, 10, 11, 137)])
def test_weight_gradients_over_row_lengths(shape):
    import torch
    from torch.nn.grad import conv3d_weight

    inputs, outputs = 14, 5
    net = dnet.Net(inputs, outputs, seed=12, out_scale=1.0)
    f = features(shape, inputs, 3)
    n, x, y, z = shape
    t = torch.zeros(n, x - 8, y - 8, z - 8, dnet.IO_CHANNELS)
    t[..., :outputs] = torch.randn(n, x - 8, y - 8, z - 8, outputs, generator=torch.Generator().manual_seed(4))
    net.forward_backward(f.cuda(), t.cuda())

    def first(a):
        return torch.as_tensor(a).double().permute(0, 4, 1, 2, 3)

    for l in range(4):
        k = 2 * (l + 1)
        a = first(f.float() if l == 0 else net.get_tensor(l - 1, 0, (n, x - k + 2, y - k + 2, z - k + 2, 32)))
        g = first(net.get_tensor(l, 3, (n, x - k, y - k, z - k, 32 if l < 3 else 16)))
        gw, gb = net.get_grad(l)
        co, ci = gw.shape[:2]
        a, g = a[:, :ci], g[:, :co]
        rows = n * (x - k) * (y - k)
        steps = rows * -(-(z - k) // 16)
        eps = (steps + 148) * 2.0 ** -22
        size = (co, ci, 3, 3, 3)
        err = (torch.as_tensor(gw).double() - conv3d_weight(a, size, g)).abs()
        assert bool((err <= eps * conv3d_weight(a.abs(), size, g.abs())).all()), ("gw", l)
        err = (torch.as_tensor(gb).double() - g.sum(dim=(0, 2, 3, 4))).abs()
        assert bool((err <= eps * g.abs().sum(dim=(0, 2, 3, 4))).all()), ("gb", l)


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
