"""Record projectors on detectors of few rows, whose warps and blocks take no more rows
than there are, against the FP64 oracle; the correction pass has the separate
projections' bits there too."""
import numpy as np
import pytest
import torch

import dtvb200
import oracle as O
from helpers import blob_volume, rel_rmse

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 2, 3, 4, 5, 9])
@pytest.mark.parametrize("nz", [1, 7])
def test_forward(cuda, rows, nz):
    size, det = (37, 33, nz), (70, rows)
    args = (np.linspace(0, 360, 9, endpoint=False), size, (1.0,) * 3, det, (1.4, 2.2 * nz / rows), 100, 200)
    geo, og = dtvb200.circular(*args), O.circular_geometry(*args)
    vol = blob_volume(np.random.default_rng(8), size[::-1], 2).astype(np.float16).astype(np.float32)
    dev = torch.from_numpy(vol).to(cuda)
    ref = O.forward(og, vol).reshape(geo.sino_shape(2))
    outs = {s: dtvb200.Plan(geo, 2, sampler=s, device=cuda).forward(dev) for s in ("soft", "exact")}
    for out in outs.values():
        assert rel_rmse(out.cpu().numpy(), ref) < 1e-5  # the software projectors' tolerance
    fast, exact = (dtvb200.Plan(geo, 2, sampler=s, device=cuda) for s in ("pairs", "exact"))
    g, w = torch.rand_like(outs["exact"]), torch.zeros_like(outs["exact"])
    g_eff = torch.empty_like(g)
    dtvb200.geometry.forward_refresh(fast, exact, dev, g, w, g_eff, 1.0)
    assert torch.equal(w, (outs["exact"] - g) / 2)
    assert torch.equal(g_eff, g + (fast.forward(dev) - outs["exact"]))
