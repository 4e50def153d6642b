"""The ASD-POCS TV descent step on values whose squared differences overflow and on
infinite and NaN voxels: square slices and the clean D_y (row-marching kernel) and the
wrap on other slices (general kernel) alike give what the formula gives in FP32, where
a finite gradient over an overflowed norm is zero."""
import numpy as np
import pytest
import torch

import oracle as O
from dtvb200 import _lib
from dtvb200.geometry import _ptr, _stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,quirk", [((33, 33, 9), True), ((33, 33, 9), False),
                                        ((61, 17, 9), False), ((33, 29, 9), True)])
@pytest.mark.parametrize("value", [3e19, -3e19, float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("at", [(0, 0, 0), (4, 7, 30), (8, 16, 32)])
def test_tv_descent_large(cuda, size, quirk, value, at):
    X, Y, Z = size
    f = np.random.default_rng(3).standard_normal((1, 1, Z, Y, X)).astype(np.float32)
    f[(0, 0) + tuple(min(a, n - 1) for a, n in zip(at, (Z, Y, X)))] = value
    step = np.float32(0.3)
    with np.errstate(all="ignore"):
        ds = [O.diff(f, size, a, quirk).astype(np.float32) for a in range(3)]
        n = np.sqrt(sum(d * d for d in ds)) + np.float32(1)
        assert n.dtype == np.float32 and not np.isfinite(n).all()
        ref = f - step * sum(O.diff(ds[a] / n, size, a, quirk, True) for a in range(3))
    fin = torch.from_numpy(f).to(cuda)
    out = torch.zeros_like(fin)
    davg = torch.tensor([step], device=cuda)
    _lib.call("dtv_tv_descent", _ptr(fin), _ptr(out), _lib.ivec(size), 1, int(quirk), _ptr(davg),
              _stream(cuda))
    out = out.cpu().numpy()
    assert np.array_equal(np.isnan(out), np.isnan(ref))
    assert np.array_equal(np.isinf(out), np.isinf(ref))
    ok = np.isfinite(ref)
    # about ten roundings of O(1) terms, each 2^-24, and one of the large voxel itself
    assert (np.abs(out[ok] - ref[ok]) <= 2e-6 + 2.0 ** -23 * np.abs(ref[ok])).all()
