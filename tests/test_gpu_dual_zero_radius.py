"""The DTV dual step where some or all of the three L1 balls have radius zero (a zero
image's first steps: the projection is zero, the dual is its ascent point), in the
one-voxel and the four-voxel kernels, against the update order of the reference
(DTVCP.py:41-54) in FP64."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from dtvb200 import _lib
from dtvb200.geometry import _ptr, _stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1, 1), (33, 9, 17), (32, 8, 8), (64, 64, 5)])
@pytest.mark.parametrize("zeros", [(0,), (1,), (2,), (0, 2), (0, 1, 2)])
def test_zero_radius(cuda, size, zeros):
    X, Y, Z = size
    rng = np.random.default_rng(8)
    shp = (1, 1, Z, Y, X)
    f = {k: (rng.standard_normal(shp) * 0.01).astype(np.float32) for k in ("fbar", "f", "recon")}
    d = [(rng.standard_normal(shp) * 0.01).astype(np.float32) for _ in range(4)]
    sg, tau, mu, v = 0.05, 0.02, 0.7, (0.4, 0.3, 0.2)
    t = [0.0 if a in zeros else np.abs(O.diff(f["f"], size, a, True)).sum() * 0.5 for a in range(3)]
    ref = []
    for a in range(3):
        u = d[a] + v[a] * sg * O.diff(f["fbar"], size, a, True)
        if a not in zeros:
            lam = O.l1ball_lambda_exact(np.abs(u) / sg, v[a] * t[a])
            u = u - sg * np.sign(u) * np.maximum(np.abs(u) / sg - lam, 0)
        ref.append(u)
    prm = _lib.dtv_pdhg_params()
    prm.sigma, prm.tau, prm.mu, prm.quirk, prm.f_dtype = sg, tau, mu, 1, _lib.DTV_F32
    prm.v[:] = v
    fd = {k: torch.from_numpy(a).to(cuda) for k, a in f.items()}
    dd = [torch.from_numpy(a).to(cuda) for a in d]
    tt = torch.tensor(t, dtype=torch.float64, device=cuda)
    ws = torch.zeros(_lib.load().dtv_pdhg_workspace_bytes(), dtype=torch.uint8, device=cuda)
    args = [_ptr(x) for x in dd] + [_lib.ivec(size), 1, ctypes.byref(prm)]
    _lib.call("dtv_pdhg_dual", _ptr(fd["fbar"]), *args, _ptr(tt), _ptr(ws), _stream(cuda))
    _lib.call("dtv_pdhg_primal", _ptr(fd["f"]), _ptr(fd["fbar"]), _ptr(fd["recon"]), *args,
              _ptr(ws), _stream(cuda))
    for a in range(3):
        # the tolerance of the dual step's other tests
        assert np.abs(dd[a].cpu().numpy() - ref[a]).max() <= 1e-5 * max(np.abs(ref[a]).max(), 1e-3)
