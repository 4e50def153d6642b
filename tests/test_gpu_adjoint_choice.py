"""The exact adjoint on both sides of each line that chooses its scatter (detector rows
per voxel, rows, number of rays, pairs of batch items), against the FP64 oracle, and the
plain scatter in z-slabs against the bricks, which take the same FP32 positions."""
import numpy as np
import pytest
import torch

import dtvb200
import oracle as O
from dtvb200 import _lib
from helpers import rel_rmse

pytestmark = pytest.mark.gpu

# volume, detector, views, rows per voxel at magnification 2
CASES = {"few_rays": ((40, 38, 36), (50, 46), 13, 1.0), "rays": ((40, 38, 36), (90, 50), 40, 1.0),
         "four_rows": ((60, 50, 5), (160, 4), 190, 0.8), "five_rows": ((60, 50, 5), (160, 5), 190, 0.8),
         "sparse": ((45, 40, 60), (90, 31), 60, 0.38), "less_sparse": ((45, 40, 60), (90, 33), 60, 0.42),
         "dense": ((50, 40, 45), (110, 70), 60, 1.3), "one_row": ((70, 60, 1), (150, 1), 60, 0.8),
         "row": ((300, 7, 5), (64, 16), 33, 1.0)}


@pytest.mark.parametrize("kind", sorted(CASES))
@pytest.mark.parametrize("batch", [1, 3])
def test_adjoint(cuda, kind, batch):
    vs, ds, views, rows = CASES[kind]
    far = 3.0 * max(vs)
    args = (np.linspace(0, 360, views, endpoint=False), vs, (1.0,) * 3, ds,
            (2.6 * max(vs[:2]) / ds[0], 2.0 / rows), far, 2 * far)
    geo, og = dtvb200.circular(*args), O.circular_geometry(*args)
    y = np.random.default_rng(7).random(geo.sino_shape(batch)).astype(np.float32)
    plan = dtvb200.Plan(geo, batch, sampler="soft", adjoint=True, device=cuda)
    out = plan.adjoint(torch.from_numpy(y).to(cuda)).cpu().numpy()
    ref = O.adjoint(og, y).reshape(out.shape)
    assert np.abs(ref).max() > 0
    # FP32 positions on rays of up to 600 voxels: the tolerance of the other adjoint tests
    assert rel_rmse(out, ref) < 1e-5


@pytest.mark.parametrize("batch", [1, 3])
def test_slabs(cuda, batch):
    vs, ds = (601, 590, 12), (70, 9)  # 5.7 MB of records per slice and item, 72 MB per slab
    geo = dtvb200.circular(np.linspace(0, 360, 8, endpoint=False), vs, (1.0,) * 3, ds, (22.3, 6.7),
                           1803, 3606)
    plan = dtvb200.Plan(geo, batch, sampler="soft", adjoint=True, device=cuda)
    y = torch.rand(plan.sino_shape(batch), device=cuda)
    out = plan.adjoint(y)
    plan.set_tuning(_lib.DTV_TUNE_ADJOINT, 0)
    ref = plan.adjoint(y)
    # a few FP32 terms of one sign per voxel, in other orders
    assert float(ref.max()) > 0 and rel_rmse(out.cpu().numpy(), ref.cpu().numpy()) < 1e-6
