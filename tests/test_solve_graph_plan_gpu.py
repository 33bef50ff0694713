"""A captured solve (linalg.SolveGraph) after eager solves that change what it
holds on to: another number of right-hand sides moves the handle's update
vectors, another threshold its list of fronts.  The graph is captured again and
gives the eager solve's bits; without a factorization it raises.  (Replayed as
captured, it would read the other solve's offsets or a buffer that was freed.)"""
import numpy as np
import pytest
import torch

from matrices import csr_arrays
from test_panel_rows_gpu import arrow

pytestmark = pytest.mark.gpu


def handle(K):
    from amigo_b200 import linalg
    n, rp, ci, v = csr_arrays(K)
    ldl = linalg.SparseLDL(linalg.CSRMat(n, n, rp, ci, v),
                           order=linalg.OrderingType.NATURAL)
    assert ldl.factor() == 0
    return ldl


def eager(ldl, b):
    x = b.clone()
    ldl.solve_device(x)
    return x


@pytest.mark.parametrize("nrhs,other", [(1, 8), (8, 1), (3, 17)])
def test_other_number_of_right_hand_sides(nrhs, other):
    from amigo_b200 import linalg
    K = arrow(90, 70, 5, 0.4)
    n = K.shape[0]
    ldl = handle(K)
    b = torch.from_numpy(np.random.RandomState(1).randn(nrhs, n)).cuda()
    want = eager(ldl, b)
    x = b.clone()
    g = linalg.SolveGraph(ldl, x)
    g()
    assert torch.equal(x, want)
    eager(ldl, torch.ones(other, n, dtype=torch.float64, device="cuda"))
    for captures in (2, 2):  # once more, then replayed
        x.copy_(b)
        g()
        assert torch.equal(x, want)
        assert g.captures == captures


def test_other_threshold():
    from amigo_b200 import linalg
    K = arrow(180, 60, 6, 0.4)
    n = K.shape[0]
    ldl = handle(K)
    b = torch.from_numpy(np.random.RandomState(2).randn(n)).cuda()
    x = b.clone()
    g = linalg.SolveGraph(ldl, x)
    for wide in (1 << 62, 1, 1 << 12):
        ldl.set_wide_threshold(wide)
        want = eager(ldl, b)
        x.copy_(b)
        g()
        assert torch.equal(x, want)
    ldl.solve_status()


def test_no_factorization():
    from amigo_b200 import linalg
    K = arrow(100, 500, 11, 0.4)
    ldl = handle(K)
    x = torch.ones(K.shape[0], dtype=torch.float64, device="cuda")
    g = linalg.SolveGraph(ldl, x)
    g()
    ldl.set_wait_limit(0)  # the panels' messages are given up: no factor
    with pytest.raises(RuntimeError):
        ldl.factor()
    with pytest.raises(RuntimeError):
        g()
