"""The FBP filter on rows with one infinite or NaN column: it reaches the outputs whose
taps meet it, the centre one and those at odd offsets up to half the row, and no other."""
import numpy as np
import pytest
import torch

import dtvb200
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [2, 6, 16, 18, 34, 250, 290, 1680, 8192])
@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("where", [0.0, 0.37, 1.0])
def test_one_column(cuda, width, adjoint, value, where):
    x = np.random.default_rng(4).standard_normal((1, 1, 3, 5, width)).astype(np.float32)
    c = int(round(where * (width - 1)))
    clean = O.fbp_filter(x, 5, 900.0, 2.5, width / 2, adjoint=adjoint)
    x[0, 0, 1, 2, c] = value
    out = dtvb200.fbp_filter(torch.from_numpy(x).to(cuda), 900.0, 5, 2.5, width / 2,
                             adjoint=adjoint).cpu().numpy()
    d = np.abs(np.arange(width) - c)
    reached = np.zeros(x.shape, bool)
    reached[0, 0, 1, 2] = (d == 0) | ((d % 2 == 1) & (d <= width // 2))
    assert np.array_equal(~np.isfinite(out), reached)
    # FP32 sums of a row: the tolerance of the other filter tests, 1e-6 of the row's scale, by element
    scale = np.abs(clean).max()
    assert (np.abs(out - clean)[~reached] <= 1e-5 * scale).all()
