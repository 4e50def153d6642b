"""Checkpointed convolution blocks whose calls are watched in the forward pass only, or
in the backward pass only: the repetition takes the forward pass's path, and the
gradients are those of a step that nothing watches."""
import contextlib

import pytest
import torch
from torch.utils.checkpoint import checkpoint
from torch.utils.flop_counter import FlopCounterMode

import dtvb200
from dtvb200 import conv
from dtvb200.nets import ConvBlock, UnrolledPDHG

pytestmark = pytest.mark.gpu
bf = torch.bfloat16


@contextlib.contextmanager
def watched(how, net):
    with contextlib.ExitStack() as stack:
        if how == "mode":
            stack.enter_context(FlopCounterMode(display=False))
        elif how == "hook":
            for m in net.modules():
                if isinstance(m, torch.nn.Conv3d):
                    stack.callback(m.register_forward_hook(lambda *a: None).remove)
        elif how == "global hook":
            register = torch.nn.modules.module.register_module_forward_hook
            stack.callback(register(lambda *a: None).remove)
        yield


def close(a, b):
    # two paths round the blocks' BF16 values at the same places and sum in other orders
    return all(float((x.double() - y.double()).norm()) <= 2.0 ** -6 * float(y.double().norm())
               for x, y in zip(a, b))


@pytest.mark.parametrize("how", ["mode", "hook", "global hook"])
@pytest.mark.parametrize("when", ["forward", "backward"])
@pytest.mark.parametrize("outer", [False, True])  # the caller checkpoints the whole network too
def test_network(cuda, how, when, outer):
    torch.manual_seed(7)
    geo = dtvb200.circular([0.0, 50.0, 100.0, 140.0], (18, 16, 12), (1.0,) * 3, (24, 20), (1.5, 1.5),
                           60, 120)
    net = UnrolledPDHG(dtvb200.Projector(geo), stages=2, features=16, tau=0.1).to(cuda)
    x, p = (torch.rand(s, device=cuda) for s in (geo.vol_shape(), geo.sino_shape()))

    def step(fwd, bwd):
        with watched(how if fwd else None, net):
            y = checkpoint(net, x, p, use_reentrant=False) if outer else net(x, p)
        with watched(how if bwd else None, net):
            return torch.autograd.grad(y.pow(2).sum(), list(net.parameters()))

    assert close(step(when == "forward", when == "backward"), step(False, False))


@pytest.mark.parametrize("how", ["mode", "hook", "global hook"])
def test_block_in_own_checkpoint(cuda, how):
    torch.manual_seed(8)
    block = ConvBlock(16).to(cuda)
    x = torch.rand(1, 1, 9, 10, 11, device=cuda, requires_grad=True)
    grads = []
    for h in (how, None):
        with torch.autocast("cuda", dtype=bf):
            with watched(h, block):
                y = checkpoint(block, x, use_reentrant=False)
        grads.append(torch.autograd.grad(y.float().sum(), [x] + list(block.parameters())))
    assert close(*grads)


def test_kernels_in_network(cuda, monkeypatch):
    """A checkpointed network's blocks run on the kernels in both passes."""
    calls = []
    monkeypatch.setattr(conv, "conv_block", lambda body, x, f=conv.conv_block: calls.append(1) or f(body, x))
    geo = dtvb200.circular([0.0, 90.0], (10, 10, 8), (1.0,) * 3, (12, 10), (1.5, 1.5), 60, 120)
    net = UnrolledPDHG(dtvb200.Projector(geo), stages=2, features=16).to(cuda)
    y = net(torch.rand(geo.vol_shape(), device=cuda), torch.rand(geo.sino_shape(), device=cuda))
    assert len(calls) == 2
    y.sum().backward()
    assert len(calls) == 4
