"""The exact adjoint's cell-record scatter against the FP64 oracle where its warps
merge differently: many rays per voxel along v (long runs of one record), about
one, fewer than one, detector rows that run down instead of up, rays that miss,
and zero rays between live ones."""
import numpy as np
import pytest
import torch

import dtvb200
import oracle as O
from helpers import rel_max, rel_rmse, vector_views

pytestmark = pytest.mark.gpu


def case(kind):
    if kind == "rows_down":
        pv = vector_views(9, 40.0, 70.0, 1.1, 1.2, 1.5)
        pv[:, 6:9] *= -1  # V points down
        return dtvb200.vector(pv, (18, 15, 21), (33, 41)), O.vector_geometry(pv, (18, 15, 21),
                                                                            (33, 41))
    vs, ds, pitch = {"long_runs": ((12, 14, 11), (40, 150), (1.0, 0.2)),
                     "one_per_voxel": ((30, 26, 33), (50, 47), (1.6, 2.0)),
                     "sparse_rays": ((40, 37, 50), (20, 19), (4.0, 5.0)),
                     "wide": ((9, 11, 7), (60, 33), (2.0, 1.2))}[kind]
    args = (np.linspace(0, 360, 8, endpoint=False), vs, (1.0,) * 3, ds, pitch, 500, 1000)
    return dtvb200.circular(*args), O.circular_geometry(*args)


@pytest.mark.parametrize("kind", ["long_runs", "one_per_voxel", "sparse_rays", "wide", "rows_down"])
@pytest.mark.parametrize("holes", [False, True])
@pytest.mark.parametrize("batch", [1, 2, 3])  # pairs of items share threads, an odd one runs alone
def test_adjoint_runs(cuda, kind, holes, batch):
    geo, og = case(kind)
    rng = np.random.default_rng(11)
    y = rng.standard_normal((batch, 1) + tuple(og.sino_shape)).astype(np.float32)
    if holes:
        y *= rng.random(y.shape) < 0.6
    plan = dtvb200.Plan(geo, max_batch=batch, device=cuda, adjoint=True)
    out = plan.adjoint(torch.from_numpy(y).to(cuda)).cpu().numpy()
    ref = O.adjoint(og, y).reshape(out.shape)
    assert np.abs(ref).max() > 0
    # the tolerances of the other adjoint and software-projector tests
    assert rel_rmse(out, ref) < 1e-5
    assert rel_max(out, ref) < 1e-4
