"""Backprojection into volumes of few slices (two per thread up to four slices, eight
beyond): against the FP64 oracle, with the bits of the launches that take eight per
thread throughout (the correction pass, several plans at once)."""
import numpy as np
import pytest
import torch

import dtvb200
import oracle as O
from helpers import rel_rmse
from test_gpu_bp_shapes import modules

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("kind", ["small", "large", "modules"])
def test_flat(cuda, nz, kind):
    if kind == "modules":
        pv = modules(6, 11, 12, 18, 48, nz)
        geo, og = dtvb200.vector(pv, (48, 45, nz), (12, 18)), O.vector_geometry(pv, (48, 45, nz), (12, 18))
    else:
        vs, ds = ((33, 30, nz), (40, 3)) if kind == "small" else ((371, 290, nz), (90, 2))
        args = (np.linspace(0, 360, 13, endpoint=False), vs, (1.0,) * 3, ds, (2.6 * vs[0] / ds[0], nz), 900, 1800)
        geo, og = dtvb200.circular(*args), O.circular_geometry(*args)
    sino = np.random.default_rng(5).random((1, 1) + tuple(og.sino_shape)).astype(np.float32)
    dev = torch.from_numpy(sino).to(cuda)
    plans = {s: dtvb200.Plan(geo, sampler=s, device=cuda) for s in ("soft", "exact", "pairs")}
    outs = {s: p.backward(dev) for s, p in plans.items()}
    ref = O.backward(og, sino).reshape(outs["soft"].shape)
    assert np.abs(ref).max() > 0
    assert rel_rmse(outs["soft"].cpu().numpy(), ref) < 1e-5  # the software projectors' tolerance
    out, e_b = torch.empty_like(outs["soft"]), torch.empty_like(outs["soft"])
    dtvb200.backward_refresh(plans["pairs"], plans["exact"], dev, out, e_b)
    assert torch.equal(out, outs["exact"]) and torch.equal(out, outs["soft"])
    assert torch.equal(e_b, out - outs["pairs"])
    many = dtvb200.backward_many([plans["pairs"]], [dev])
    assert torch.equal(many[0], outs["pairs"])
