"""Volumes with more tiles along y or z than a grid's second or third dimension holds:
staging, projection, backprojection and the exact adjoint against the FP64 oracle."""
import numpy as np
import pytest
import torch

import dtvb200
import oracle as O
from helpers import rel_rmse

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sampler", ["soft", "exact"])
@pytest.mark.parametrize("size", [(2, 300_000, 1), (1, 600_000, 2)])
def test_long_y(cuda, sampler, size):
    # thin voxels along y, rays across it
    args = ([90.0, 92.0], size, (1.0, 50.0 / size[1], 1.0), (33, 2), (2.0, 0.5), 60, 120)
    geo, og = dtvb200.circular(*args), O.circular_geometry(*args)
    vol = np.linspace(1.0, 2.0, size[1], dtype=np.float32)
    vol = np.broadcast_to(vol[None, :, None], (size[2], size[1], size[0])).copy()
    if sampler == "exact":
        vol = vol.astype(np.float16).astype(np.float32)
    plan = dtvb200.Plan(geo, sampler=sampler, adjoint=True, device=cuda)
    out = plan.forward(torch.from_numpy(vol.reshape(geo.vol_shape(1))).to(cuda))
    ref = O.forward(og, vol)
    assert (ref > 0).sum() > 16
    # some 1e4 FP32 terms per ray, coordinates of 3e-2 voxels on smooth data
    assert rel_rmse(out.cpu().numpy().reshape(ref.shape), ref) < 1e-4
    y = np.random.default_rng(2).random(geo.sino_shape(1)).astype(np.float32)
    dev = torch.from_numpy(y).to(cuda)
    ref = O.backward(og, y)
    assert rel_rmse(plan.backward(dev).cpu().numpy().reshape(ref.shape), ref) < 1e-5
    back = plan.adjoint(dev).cpu().numpy().reshape(ref.shape)
    # the transpose: equal products with the smooth volume
    a, b = float((back.astype(np.float64) * vol).sum()), float((O.forward(og, vol).ravel() * y.ravel()).sum())
    assert abs(a / b - 1) < 1e-4
