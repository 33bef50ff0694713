"""Element kernels of the SIMP models on meshes whose colours are empty or hold
one element, and on odd ones, against the numpy restatement
oracle/simp2d_oracle.py: FP64 with different summation order, rtol 1e-13
relative to the largest entry; two passes give the same bits."""
import numpy as np
import pytest
import torch

from amigo_b200.problems.simp2d import Simp2D
from amigo_b200.problems.simp3d import Simp3D
from oracle import simp2d_oracle as O
from test_simp3d_gpu import rand_point

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", [(2, 1), (3, 2), (13, 5), (1, 2, 2), (2, 1, 3), (5, 4, 3)])
def test_small_and_odd_meshes(mesh):
    m = (Simp2D if len(mesh) == 2 else Simp3D)(*mesh, seed=1)
    dm = m.device_model("cuda:0")
    x = rand_point(m, 7)
    xd = torch.from_numpy(x).cuda()
    g = torch.full((m.n,), 3.0, dtype=torch.float64, device="cuda:0")
    vals = torch.full((m.nnz,), 7.0, dtype=torch.float64, device="cuda:0")
    dm.gradient(xd, 1.1, g)
    dm.hessian(xd, 1.1, vals)
    for got, want in ((g, O.gradient_fixed(m, x, 1.1)), (vals, O.hessian_values(m, x))):
        assert np.abs(got.cpu().numpy() - want).max() <= 1e-13 * max(1.0, np.abs(want).max())
    g2, vals2 = torch.zeros_like(g), torch.zeros_like(vals)
    dm.gradient(xd, 1.1, g2)
    dm.hessian(xd, 1.1, vals2)
    assert torch.equal(g, g2) and torch.equal(vals, vals2)
