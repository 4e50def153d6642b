"""Volumes and detectors with more than 2^22 elements along an axis, where FP32 sums
with a large constant no longer give floors: projection, backprojection (z-affine and
tilted) and the exact adjoint on smooth data, against the FP64 oracle. An FP32
coordinate there is good to half an element, some 1e-7 of the data's range."""
import numpy as np
import pytest
import torch

import dtvb200
import oracle as O
from helpers import rel_max

pytestmark = pytest.mark.gpu
N = 5_000_000


@pytest.mark.parametrize("sampler", ["soft", "exact"])
@pytest.mark.parametrize("tilted", [False, True])
def test_backward(cuda, sampler, tilted):
    vs, ds, pitch = (21, 18, 5), (N, 3), (50.0 / N, 20.0)
    if tilted:
        pv = np.array([[-60, 0, 0, 60, 0, 0, 0, 0.2 * pitch[1], pitch[1], 0, pitch[0], 0]], np.float32)
        geo, og = dtvb200.vector(pv, vs, ds), O.vector_geometry(pv, vs, ds)
        # without the layer's test of detector coordinates against the volume's size
        geo.struct.bp_extent_check = og.og.bp_extent = 0
        geo.struct.bp_scale = og.og.bp_scale = 0.7
    else:
        args = ([0.0, 70.0], vs, (1.0,) * 3, ds, pitch, 60, 120)
        geo, og = dtvb200.circular(*args), O.circular_geometry(*args)
    ramp = np.linspace(0.5, 1.5, N, dtype=np.float32)
    sino = np.stack([ramp, 1.2 * ramp, 0.9 * ramp])[None].repeat(geo.n_views, 0)
    ref = O.backward(og, sino)
    out = dtvb200.Plan(geo, sampler=sampler, device=cuda).backward(
        torch.from_numpy(sino.reshape(geo.sino_shape(1))).to(cuda))
    assert np.abs(ref).max() > 0 and rel_max(out.cpu().numpy().reshape(ref.shape), ref) < 1e-5


@pytest.mark.parametrize("sampler", ["soft", "exact"])
def test_forward_and_adjoint(cuda, sampler):
    # rays across the long axis, whose voxels are thin
    args = ([0.0], (N, 1, 1), (50.0 / N, 1.0, 1.0), (33, 1), (2.4, 1.0), 60, 120)
    geo, og = dtvb200.circular(*args), O.circular_geometry(*args)
    vol = np.linspace(1.0, 2.0, N, dtype=np.float32).reshape(geo.vol_shape(1))
    ref = O.forward(og, vol.astype(np.float16) if sampler == "exact" else vol)
    plan = dtvb200.Plan(geo, sampler=sampler, adjoint=True, device=cuda)
    out = plan.forward(torch.from_numpy(vol).to(cuda)).cpu().numpy()
    assert (ref > 0).sum() > 16
    # some 1e5 FP32 terms per ray
    assert rel_max(out.reshape(ref.shape), ref) < 1e-4
    y = np.random.default_rng(2).random(geo.sino_shape(1)).astype(np.float32)
    back = plan.adjoint(torch.from_numpy(y).to(cuda))
    smooth = torch.from_numpy(vol).to(cuda).double()
    forward = float((O.forward(og, vol).ravel() * y.astype(np.float64).ravel()).sum())
    assert abs(float((back.double() * smooth).sum()) / forward - 1) < 1e-4
