"""The exact adjoint of a scan with more views than a grid's second dimension holds."""
import numpy as np
import pytest
import torch

import dtvb200
import oracle as O
from helpers import rel_rmse

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 2, 3])
def test_many_views(cuda, batch):
    n = 66_001
    args = (np.linspace(0, 360, n, endpoint=False), (8, 7, 5), (1.0,) * 3, (4, 3), (3.0, 3.0), 60, 120)
    geo, og = dtvb200.circular(*args), O.circular_geometry(*args)
    y = np.random.default_rng(6).random(geo.sino_shape(batch)).astype(np.float32)
    plan = dtvb200.Plan(geo, batch, sampler="soft", adjoint=True, device=cuda)
    out = plan.adjoint(torch.from_numpy(y).to(cuda)).cpu().numpy()
    ref = O.adjoint(og, y).reshape(out.shape)
    # some 1e4 FP32 terms of one sign per voxel, added in any order
    assert rel_rmse(out, ref) < 1e-4
