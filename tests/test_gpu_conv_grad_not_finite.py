"""The convolution block's gradients where an activation or an output gradient is
infinite or NaN, on the volume's faces and inside: NaN and infinities where the
module's own layers give them, and the other weight gradients unharmed."""
import pytest
import torch

from dtvb200.nets import ConvBlock

pytestmark = pytest.mark.gpu
bf = torch.bfloat16
SIZE = (9, 18, 20)  # remainders of the 8 x 16 columns in both directions


@pytest.mark.parametrize("features", [16, 32])
@pytest.mark.parametrize("positive", [True, False])  # weights of one sign: infinities stay infinite
@pytest.mark.parametrize("which", ["x", "gy"])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("at", [(0, 0, 0), (8, 17, 19), (4, 9, 0), (4, 9, 19), (4, 0, 7), (4, 17, 7),
                                (0, 5, 7), (8, 5, 7), (4, 9, 1), (4, 8, 12)])
def test_gradients(cuda, features, positive, which, value, at):
    torch.manual_seed(5)
    block = ConvBlock(features).to(cuda)
    if positive:
        with torch.no_grad():
            for p in block.parameters():
                p.abs_()
    x = torch.rand((1, 1) + SIZE, device=cuda) + 0.1
    gy = (torch.rand((1, 1) + SIZE, device=cuda) + 0.1).to(bf)
    (x if which == "x" else gy)[0, 0][at] = value
    x.requires_grad_()
    wanted = [x] + list(block.parameters())
    got = []
    for f in (block, block.body):
        with torch.autocast("cuda", dtype=bf):
            y = f(x)
        got.append(torch.autograd.grad(y, wanted, gy))
    for a, b in zip(*got):
        assert torch.equal(torch.isnan(a), torch.isnan(b))
        assert torch.equal(torch.isinf(a), torch.isinf(b))
        ok = torch.isfinite(b)
        if positive and ok.any():
            # sums of one sign: both round them, and three layers of terms, to 2^-9
            assert ((a - b)[ok].abs() <= 2.0 ** -6 * b[ok].abs()).all()
