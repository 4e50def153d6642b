"""The convolution block under torch's compilers on the CPU: its modules run as before."""
import pytest
import torch

from dtvb200.nets import ConvBlock


@pytest.mark.parametrize("how", ["script", "trace", "fx", "compile"])
def test_compilers(how):
    torch.manual_seed(6)
    block = ConvBlock(8)
    x = torch.randn(1, 1, 4, 5, 6)
    f = {"script": lambda: torch.jit.script(block), "trace": lambda: torch.jit.trace(block, x),
         "fx": lambda: torch.fx.symbolic_trace(block),
         "compile": lambda: torch.compile(block, fullgraph=True, backend="eager")}[how]()
    assert torch.allclose(f(x), block.body(x), atol=1e-6)
