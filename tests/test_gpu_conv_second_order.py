"""Differentiable gradients of the convolution block (create_graph) and their own
gradients, against the module's layers."""
import pytest
import torch

from dtvb200 import conv
from dtvb200.nets import ConvBlock

pytestmark = pytest.mark.gpu
bf = torch.bfloat16


@pytest.mark.parametrize("features,batch,size", [(16, 1, (5, 9, 17)), (32, 2, (9, 18, 20))])
@pytest.mark.parametrize("wanted", ["all", "x", "body.2.weight"])
def test_second_order(cuda, features, batch, size, wanted):
    torch.manual_seed(9)
    block = ConvBlock(features).to(cuda)
    x = torch.randn((batch, 1) + size, device=cuda, requires_grad=True)
    gy = torch.randn((batch, 1) + size, device=cuda).to(bf).requires_grad_()
    named = {"x": x, **dict(block.named_parameters())}
    first = list(named.values()) if wanted == "all" else [named[wanted]]
    c = [torch.randn_like(t) for t in first]
    got = []
    for f in (block, block.body):
        with torch.autocast("cuda", dtype=bf):
            assert conv.supported(block.body, x)
            y = f(x)
        g = torch.autograd.grad(y, first, gy, create_graph=True)
        total = sum((a.float() * b).sum() for a, b in zip(g, c))
        second = torch.autograd.grad(total, list(named.values()) + [gy], allow_unused=True)
        got.append((g, second))
    for a, b in zip(got[0][0], got[1][0]):
        assert float((a - b).detach().norm()) < 2.0 ** -6 * float(b.detach().norm())  # the first-order tolerance
    for name, a, b in zip(list(named) + ["gy"], got[0][1], got[1][1]):
        assert (a is None) == (b is None), name
        if a is not None:  # twice as many layers of BF16 roundings
            assert float((a - b).detach().norm()) <= 2.0 ** -5 * float(b.detach().norm()), name
