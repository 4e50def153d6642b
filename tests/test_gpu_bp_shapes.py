"""The backprojector's launch shapes against the FP64 oracle: one, two, four and
eight view groups per block (by volume size), z-affine and tilted detectors,
detectors smaller than the volume's shadow (runs across an edge, runs wholly
beside it), and the many-module scans whose blocks first look for the views
they meet."""
import math

import numpy as np
import pytest
import torch

import dtvb200
import oracle as O
from helpers import rel_max, rel_rmse

pytestmark = pytest.mark.gpu


def modules(angles, planes, W, H, n, nz):
    """[angles * planes, 12] vectors: per angle `planes` flat modules on an arc
    about the source, rows tilted towards it; each sees a slice of the fan."""
    sod, sdd = 1.6 * n, 2.8 * n
    fan = 2 * math.asin(0.72 / 1.6)
    du, dv = 2 * sdd * math.tan(fan / planes / 2) / W, 1.1 * nz * sdd / sod / H
    pv = np.zeros((angles, planes, 12))
    for a in range(angles):
        t = 2 * math.pi * a / angles
        src = -sod * np.array([math.cos(t), math.sin(t), 0.0])
        for j in range(planes):
            g = t + fan * ((j + 0.5) / planes - 0.5)
            ex = np.array([math.cos(g), math.sin(g), 0.0])
            ey = np.array([-math.sin(g), math.cos(g), 0.0])
            pv[a, j] = np.concatenate([src, src + sdd * ex,
                                       dv * (np.array([0, 0, 1.0]) + 0.05 * ex), du * ey])
    return pv.reshape(-1, 12).astype(np.float32)


def case(kind):
    if kind == "modules":
        pv = modules(6, 11, 12, 18, 48, 20)
        return dtvb200.vector(pv, (48, 45, 20), (12, 18)), O.vector_geometry(pv, (48, 45, 20),
                                                                            (12, 18))
    vs, ds, views = {"one_group": ((131, 126, 62), (151, 97), 7),
                     "two_groups": ((97, 95, 63), (120, 90), 9),
                     "four_groups": ((65, 62, 61), (90, 100), 11),
                     "eight_groups": ((33, 30, 17), (40, 30), 13),
                     "two_views": ((19, 21, 9), (30, 20), 2),
                     "small_detector": ((64, 61, 33), (37, 23), 10)}[kind]
    args = (np.linspace(0, 360, views, endpoint=False), vs, (1.0,) * 3, ds, (1.2, 1.2), 500, 1000)
    return dtvb200.circular(*args), O.circular_geometry(*args)


@pytest.mark.parametrize("kind", ["one_group", "two_groups", "four_groups", "eight_groups",
                                  "two_views", "small_detector", "modules"])
def test_backward_shapes(cuda, kind):
    geo, og = case(kind)
    sino = np.random.default_rng(5).random((1, 1) + tuple(og.sino_shape)).astype(np.float32)
    dev = torch.from_numpy(sino).to(cuda)
    ref = O.backward(og, sino).reshape((1, 1) + tuple(og.vol_shape))
    assert np.abs(ref).max() > 0
    outs = {}
    for sampler in ("soft", "exact", "tex"):
        outs[sampler] = dtvb200.Plan(geo, sampler=sampler, device=cuda).backward(dev)
    # FP32 weights: the tolerances of the other software-projector tests
    assert rel_rmse(outs["soft"].cpu().numpy(), ref) < 1e-5
    assert rel_max(outs["soft"].cpu().numpy(), ref) < 1e-4
    assert torch.equal(outs["soft"], outs["exact"])
    refq = O.backward(og, sino, q=True).reshape(ref.shape)
    assert rel_rmse(outs["tex"].cpu().numpy(), refq) < 5e-3
    # the correction pass: both sums of one launch have the separate passes' bits
    fast, exact = (dtvb200.Plan(geo, sampler=s, device=cuda) for s in ("pairs", "exact"))
    out, e_b = torch.empty_like(outs["soft"]), torch.empty_like(outs["soft"])
    dtvb200.backward_refresh(fast, exact, dev, out, e_b)
    assert torch.equal(out, outs["exact"])
    assert torch.equal(e_b, out - fast.backward(dev))
