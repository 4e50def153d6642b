"""The names that torch does not publish and the convolution block's choice of path
reads: without one of them the block keeps its modules."""
import importlib.util
import sys

import pytest
import torch

import dtvb200.conv


@pytest.mark.parametrize("where,name", [
    (torch._C._functorch, "peek_interpreter_stack"), (torch.autograd.forward_ad, "_current_level"),
    (torch._C, "_len_torch_dispatch_stack"), (torch._C, "_len_torch_function_stack"),
    (torch.nn.modules.module, "_has_any_global_hook"), (None, None)])
def test_missing_name(monkeypatch, where, name):
    # modules call _has_any_global_hook's data, not the function, so it can go for the test
    spec = importlib.util.spec_from_file_location("dtvb200.conv_copy", dtvb200.conv.__file__)
    conv = importlib.util.module_from_spec(spec)
    monkeypatch.setitem(sys.modules, spec.name, conv)
    if where is not None:
        monkeypatch.delattr(where, name)
    spec.loader.exec_module(conv)
    assert conv._special_modes() is (where is not None)
