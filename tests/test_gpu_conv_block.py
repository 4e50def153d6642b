"""The BF16 convolution block's kernels at sizes around their tiles (8 x 16 columns,
z chunks, 16-wide tiles of the first and last convolution), forward and gradients,
against the block with the same roundings in FP32 sums; and the calls that stay with
the general path."""
import pytest
import torch
import torch.nn.functional as F

from dtvb200 import conv
from dtvb200.nets import ConvBlock

pytestmark = pytest.mark.gpu
bf = torch.bfloat16


class _Conv(torch.autograd.Function):
    """One convolution as BF16 autocast rounds it: FP32 sums, BF16, plus the BF16 bias, BF16."""

    @staticmethod
    def forward(ctx, x, w, b):
        ctx.save_for_backward(x, w)
        y = F.conv3d(x.double(), w.double(), padding=1).to(bf)
        return y + b.view(1, -1, 1, 1, 1)

    @staticmethod
    def backward(ctx, g):
        x, w = ctx.saved_tensors
        g = g.double()
        return (torch.nn.grad.conv3d_input(x.shape, w.double(), g, padding=1).to(bf),
                torch.nn.grad.conv3d_weight(x.double(), w.shape, g, padding=1).to(bf),
                g.sum((0, 2, 3, 4)).to(bf))


def _reference(block, x):
    p = [t.to(bf) for i in (0, 2, 4) for t in (block.body[i].weight, block.body[i].bias)]
    h = F.relu(_Conv.apply(x.to(bf), p[0], p[1]))
    h = F.relu(_Conv.apply(h, p[2], p[3]))
    return _Conv.apply(h, p[4], p[5])


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30))


SIZES = [(1, 1, 1), (8, 16, 4), (9, 17, 5), (7, 15, 33), (16, 4, 8), (17, 5, 9), (33, 18, 70),
         (40, 1, 3), (1, 40, 3)]


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("features,batch,last", [(16, 1, False), (32, 2, True)])
def test_block(cuda, size, features, batch, last):
    X, Y, Z = size
    torch.manual_seed(3)
    block = ConvBlock(features).to(cuda)
    if last:
        block.to(memory_format=torch.channels_last_3d)
    x = torch.randn(batch, 1, Z, Y, X, device=cuda, requires_grad=True)
    gy = torch.randn(batch, 1, Z, Y, X, device=cuda).to(bf)
    ref = _reference(block, x)
    wanted = [x] + list(block.parameters())
    gref = torch.autograd.grad(ref, wanted, gy)
    with torch.autocast("cuda", dtype=bf):
        assert conv.supported(block.body, x)
        y = block(x)
    assert y.dtype == bf and y.shape == ref.shape
    # both round to BF16 at the same places; FP32 sums next to a rounding edge move a
    # few values by one step of 2^-8, three layers deep
    assert _rel(y, ref) < 2.0 ** -8
    for g, r in zip(torch.autograd.grad(y, wanted, gy), gref):
        assert g.dtype == r.dtype and _rel(g, r) < 2.0 ** -6


@pytest.mark.parametrize("wanted", [("x",), ("body.4.weight",), ("body.4.bias",), ("body.2.bias",),
                                    ("body.2.weight", "body.4.bias"), ("body.0.bias", "x"),
                                    ("body.0.weight",)])
def test_some_gradients(cuda, wanted):
    """Any subset of the gradients has the bits it has among all of them."""
    torch.manual_seed(4)
    block = ConvBlock(16).to(cuda)
    x = torch.randn(1, 1, 9, 18, 20, device=cuda, requires_grad=True)
    named = {"x": x, **dict(block.named_parameters())}
    with torch.autocast("cuda", dtype=bf):
        y = block(x)
    gy = torch.randn_like(y)
    full = dict(zip(named, torch.autograd.grad(y, list(named.values()), gy)))
    for k, t in named.items():
        t.requires_grad_(k in wanted)
    with torch.autocast("cuda", dtype=bf), torch.autograd.graph.save_on_cpu():
        y = block(x)
    for k, g in zip(wanted, torch.autograd.grad(y, [named[k] for k in wanted], gy)):
        assert torch.equal(g, full[k]), k


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("at", [(0, 0, 0), (4, 9, 12), (8, 17, 19)])
def test_not_finite(cuda, value, at):
    """One infinite or NaN voxel reaches the outputs that the module's own layers let
    it reach, and one such output gradient the same input gradients."""
    torch.manual_seed(5)
    block = ConvBlock(32).to(cuda)
    x = torch.randn(1, 1, 9, 18, 20, device=cuda)
    gy = torch.randn(1, 1, 9, 18, 20, device=cuda).to(bf)
    bad_x, bad_gy = x.clone(), gy.clone()
    bad_x[0, 0][at] = value
    bad_gy[0, 0][at] = value
    for xi, g in ((bad_x, None), (x, bad_gy)):
        got = []
        for f in (block, block.body):
            xi = xi.detach().requires_grad_()
            with torch.autocast("cuda", dtype=bf):
                y = f(xi)
            if g is not None:
                y, = torch.autograd.grad(y, xi, g)
            got.append(y.detach().float())
        assert torch.equal(torch.isnan(got[0]), torch.isnan(got[1]))
        assert torch.equal(torch.isinf(got[0]), torch.isinf(got[1]))


@pytest.mark.parametrize("mode", [torch.inference_mode, torch.no_grad])
def test_without_gradients(cuda, mode):
    block = ConvBlock(16).to(cuda)
    x = torch.randn(2, 1, 5, 6, 7, device=cuda)
    with torch.autocast("cuda", dtype=bf):
        y = block(x)
        with mode():
            z = block(x)
    assert torch.equal(y, z)


def test_what_stays_general(cuda):
    block = ConvBlock(16).to(cuda)
    x = torch.randn(1, 1, 6, 5, 7, device=cuda)
    assert not conv.supported(block.body, x)  # no autocast
    with torch.autocast("cuda", dtype=torch.float16):
        assert not conv.supported(block.body, x)
    with torch.autocast("cuda", dtype=bf):
        assert conv.supported(block.body, x)
        assert not conv.supported(ConvBlock(8).to(cuda).body, x)
        assert not conv.supported(block.body, x[0])
        assert not conv.supported(block.body, x[:0])
        assert not conv.supported(block.body, x.half())
        seen = []
        h = block.body[2].register_forward_hook(lambda *a: seen.append(1))
        block(x)
        assert seen
        h.remove()
        with torch.autograd.forward_ad.dual_level():
            d = torch.autograd.forward_ad.make_dual(x, torch.ones_like(x))
            assert torch.autograd.forward_ad.unpack_dual(block(d)).tangent is not None
    x.requires_grad_()
    with torch.autocast("cuda", dtype=bf):
        g, = torch.autograd.grad(block(x).float().sum(), x, create_graph=True)
        assert g.requires_grad
        g.pow(2).sum().backward()  # through the gradient
