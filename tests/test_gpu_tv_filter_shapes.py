"""The ASD-POCS TV descent step at sizes around its warps' 30 columns, a thread's 4
rows and its z-slabs, with the clean D_y and the wrap (square slices take the
row-marching kernel, others the general one), and the FBP filter at row widths
around a thread's 8 outputs per parity, each against FP64."""
import numpy as np
import pytest
import torch

import dtvb200
import oracle as O
from dtvb200 import _lib
from dtvb200.geometry import _ptr, _stream
from helpers import rel_rmse

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1, 1), (7, 1, 1), (1, 6, 1), (1, 1, 9), (30, 30, 5),
                                  (31, 31, 9), (61, 17, 8), (29, 33, 17), (5, 5, 33), (64, 64, 3),
                                  (90, 4, 7)])
@pytest.mark.parametrize("quirk", [True, False])
def test_tv_descent(cuda, size, quirk):
    X, Y, Z = size
    f = np.random.default_rng(3).standard_normal((2, 1, Z, Y, X)).astype(np.float32)
    ds = [O.diff(f, size, a, quirk) for a in range(3)]
    g = np.sqrt(sum(d * d for d in ds)) + 1
    step = 0.3
    ref = f - step * sum(O.diff(ds[a] / g, size, a, quirk, True) for a in range(3))
    fin = torch.from_numpy(f).to(cuda)
    out = torch.full_like(fin, float("nan"))
    davg = torch.tensor([step], device=cuda)
    _lib.call("dtv_tv_descent", _ptr(fin), _ptr(out), _lib.ivec(size), 2, int(quirk), _ptr(davg),
              _stream(cuda))
    # about ten roundings of O(1) terms, each 2^-24
    assert np.abs(out.cpu().numpy() - ref).max() < 2e-6


@pytest.mark.parametrize("width", [2, 6, 16, 18, 34, 250, 290, 2064, 8192])
@pytest.mark.parametrize("adjoint", [False, True])
def test_filter_widths(cuda, width, adjoint):
    x = np.random.default_rng(4).standard_normal((1, 1, 3, 5, width)).astype(np.float32)
    out = dtvb200.fbp_filter(torch.from_numpy(x).to(cuda), 900.0, 5, 2.5, width / 2, adjoint=adjoint)
    # the tolerance of the other filter tests
    assert rel_rmse(out.cpu().numpy(), O.fbp_filter(x, 5, 900.0, 2.5, width / 2, adjoint=adjoint)) < 1e-6
