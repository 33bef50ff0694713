"""The cluster threshold set on a handle that has solved already takes effect
with the next solve, as the wide threshold does: with every front on a cluster
and a message limit of 0 polls, whether clusters ran shows in solve_status()."""
import numpy as np
import pytest
import torch

from matrices import csr_arrays
from test_panel_rows_gpu import arrow

pytestmark = pytest.mark.gpu

NEVER = 1 << 62


def clusters_run(ldl, n):
    """Whether a solve of the current schedule waits for a cluster's message."""
    x = torch.ones(n, dtype=torch.float64, device="cuda:0")
    ldl.set_wait_limit(0)
    ldl.solve_device(x)
    ldl.set_wait_limit(1 << 20)
    try:
        ldl.solve_status()
    except RuntimeError:
        return True
    return False


@pytest.mark.parametrize("width,rows", [(40, 70), (180, 60)])
def test_cluster_threshold_after_a_solve(width, rows):
    from amigo_b200 import linalg
    K = arrow(width, rows, 12, 0.5)
    n, rp, ci, v = csr_arrays(K)
    ldl = linalg.SparseLDL(linalg.CSRMat(n, n, rp, ci, v),
                           order=linalg.OrderingType.NATURAL)
    ldl.set_wide_threshold(NEVER)
    ldl.set_cluster_threshold(NEVER)
    assert ldl.factor() == 0
    assert not clusters_run(ldl, n)
    ldl.set_cluster_threshold(1)
    assert clusters_run(ldl, n)
    ldl.set_cluster_threshold(NEVER)
    assert not clusters_run(ldl, n)
