"""The FBP filter with eight and with two outputs per thread and parity: numbers of rows
on both sides of the line, against the FP64 oracle."""
import numpy as np
import pytest
import torch

import dtvb200
import oracle as O
from helpers import rel_rmse

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [2, 6, 18, 34, 250, 290, 1022, 1024, 1026])
@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("few", [True, False])
def test_rows(cuda, width, adjoint, few):
    rows = 10000 // ((width // 2 + 7) // 8) + (-1 if few else 1)
    x = np.random.default_rng(4).standard_normal((1, 1, 1, rows, width)).astype(np.float32)
    out = dtvb200.fbp_filter(torch.from_numpy(x).to(cuda), 900.0, rows, rows / 2, width / 2, adjoint=adjoint)
    # the tolerance of the other filter tests
    assert rel_rmse(out.cpu().numpy(), O.fbp_filter(x, rows, 900.0, rows / 2, width / 2, adjoint=adjoint)) < 1e-6
