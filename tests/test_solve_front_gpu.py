"""Solves of narrow fronts with their pivot columns in shared memory against
the general form, which reads them from global memory, at the edges of its
blocks: pivot counts around 32-column blocks, 2x2 pivots across a block's end
(33-column blocks), right-hand sides around the eight solved at a time, FP64
and FP32 factors.  A cluster threshold of 2^62 keeps every front on one CTA; a
front of more rows than the launch's shared memory takes takes the general
form.  The relative residual of every solution is <= 1e-10 (FP64) and a
right-hand side solved among others equals the same one solved alone bit for
bit."""
import numpy as np
import pytest
import torch

from test_panel_rows_gpu import arrow

pytestmark = pytest.mark.gpu


def handle(K, precision, cluster):
    from amigo_b200 import linalg
    from matrices import csr_arrays
    n, rp, ci, v = csr_arrays(K)
    mat = linalg.CSRMat(n, n, rp, ci, v)
    ldl = linalg.SparseLDL(mat, order=linalg.OrderingType.NATURAL)
    ldl.set_precision(precision)
    ldl.set_cluster_threshold(cluster)
    assert ldl.factor() == 0
    return ldl


@pytest.mark.parametrize("width,rows", [(1, 3), (31, 20), (32, 33), (33, 5), (34, 64),
                                        (65, 40), (97, 150), (180, 60)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("cluster", [1 << 62, 1])
def test_blocks_and_right_hand_sides(width, rows, precision, cluster):
    K = arrow(width, rows, 7 * width + rows, 0.5)
    ldl = handle(K, precision, cluster)
    n = K.shape[0]
    B = np.random.RandomState(width).randn(17, n)
    alone = []
    for k in range(17):
        x = torch.from_numpy(B[k]).cuda()
        ldl.solve_device(x)
        alone.append(x.cpu().numpy())
    for nrhs in (1, 2, 7, 8, 9, 17):
        x = torch.from_numpy(B[:nrhs].copy()).cuda()
        ldl.solve_device(x)
        got = x.cpu().numpy()
        for k in range(nrhs):
            assert np.array_equal(got[k], alone[k])
    ldl.solve_status()
    if precision == "fp64":
        norm = abs(K).sum(axis=1).max()
        for k in range(17):
            r = np.abs(K @ alone[k] - B[k]).max()
            assert r <= 1e-10 * (norm * np.abs(alone[k]).max() + np.abs(B[k]).max())
