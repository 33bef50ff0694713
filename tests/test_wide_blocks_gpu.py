"""Grid-wide solves at the edges of their 128-column blocks and 32-row strips:
pivot counts around one and two blocks, 2x2 pivots across a block's end, one and
several fronts a level, FP64 and FP32 factors.  The relative residual is <= 1e-10
(FP64) and a right-hand side solved among others equals the same one solved alone
bit for bit."""
import numpy as np
import pytest
import torch

from test_panel_rows_gpu import arrow
from test_solve_front_gpu import handle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("width,rows", [(1, 2), (31, 97), (127, 34), (128, 1), (129, 63),
                                        (200, 57), (256, 33)])
def test_block_edges(width, rows, precision):
    K = arrow(width, rows, 3 * width + rows, 0.5)
    ldl = handle(K, precision, 1)
    ldl.set_wide_threshold(1)
    B = np.random.RandomState(width).randn(3, K.shape[0])
    x = torch.from_numpy(B.copy()).cuda()
    ldl.solve_device(x)
    got = x.cpu().numpy()
    for k in range(3):
        y = torch.from_numpy(B[k]).cuda()
        ldl.solve_device(y)
        assert np.array_equal(got[k], y.cpu().numpy())
    if precision == "fp64":
        r = np.abs(K @ got.T - B.T).max()
        assert r <= 1e-10 * (abs(K).sum(axis=1).max() * np.abs(got).max() + np.abs(B).max())
