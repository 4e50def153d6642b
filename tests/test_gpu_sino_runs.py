"""Plans whose sinogram's records exceed their limit of 4 GB stage and project it in runs
of views: no more memory than that, and the sum over two scans of half the views each."""
import numpy as np
import pytest
import torch

import dtvb200

pytestmark = pytest.mark.gpu


def scan(angles, det):
    return dtvb200.circular(angles, (21, 18, 13), (1.0,) * 3, det, (40.0 / det[0], 40.0 / det[1]),
                            60, 120)


# one run of 31 views and nine more; runs of more views than one launch's maps
@pytest.mark.parametrize("det,views", [((4096, 2048), 40), ((700, 550), 800)])
def test_long_scan(cuda, det, views):
    angles = np.linspace(0, 360, views, endpoint=False)
    geo = scan(angles, det)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    plan = dtvb200.Plan(geo, sampler="soft", device=cuda)
    assert free - torch.cuda.mem_get_info()[0] <= (4 << 30) + (64 << 20)
    sino = torch.rand(plan.sino_shape(1), device=cuda)
    out = plan.backward(sino)
    ref = torch.zeros_like(out, dtype=torch.float64)
    h = views // 2
    for part in (slice(0, h), slice(h, views)):
        g = scan(angles[part], det)
        r = dtvb200.Plan(g, sampler="soft", device=cuda).backward(sino[:, :, part].contiguous())
        ref += r.double() * (geo.struct.bp_scale / g.struct.bp_scale)
    # FP32 sums of `views` positive terms in other orders
    assert float((out - ref).abs().max()) < 1e-5 * float(ref.abs().max())
    # onto a base, and the correction pass of a texture plan
    base = torch.rand_like(out)
    assert torch.allclose(plan.backward(sino, base=base), base + out, rtol=1e-6, atol=1e-6)
    fast, exact = (dtvb200.Plan(geo, sampler=s, device=cuda) for s in ("pairs", "exact"))
    both, e_b = torch.empty_like(out), torch.empty_like(out)
    dtvb200.backward_refresh(fast, exact, sino, both, e_b)
    assert torch.equal(both, out)
    assert float((both - e_b - fast.backward(sino)).abs().max()) < 1e-5 * float(ref.abs().max())
