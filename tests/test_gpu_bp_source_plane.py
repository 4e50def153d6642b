"""Backprojection of a tilted detector's view whose source plane passes exactly through
voxel centres: there h = 0 and the detector coordinates are infinite, which the extent
test leaves out. Every such voxel is zero, with samples from records or a texture."""
import numpy as np
import pytest
import torch

import dtvb200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sampler", ["soft", "exact", "tex", "pairs"])
def test_source_plane(cuda, sampler):
    n, sx = 16, -3.0
    # source in the plane x = sx, detector parallel to it, its rows tilted within it
    pv = np.array([[sx, 0.25, 0.25, 13.0, 0.0, 0.0, 0.0, 0.25, 1.0, 0.0, 1.0, 0.0]] * 21, np.float32)
    geo = dtvb200.vector(pv, (n, n, n), (24, 20))
    plan = dtvb200.Plan(geo, sampler=sampler, device=cuda)
    sino = torch.rand(plan.sino_shape(1), device=cuda) + 0.5
    out = plan.backward(sino).cpu().numpy()[0, 0]
    # h along x, from the plan's own map: zero in one slice, positive beyond it
    plane = int(round(sx + n / 2.0 - geo.struct.vol_offset[0]))
    assert 0 < plane < n - 1
    assert np.isfinite(out).all()
    assert (out[:, :, plane] == 0).all()
    assert (out[:, :, plane + 1:] != 0).any()
