"""The forms of a front's factorization and solves against each other.

Small fronts in shared memory and solves with staged pivot columns against the
general kernels: inertia, pivot and delay counts and every solution are equal bit
for bit, FP64 and FP32, at the edges of the row chunks (32 rows) and of the
32-column blocks (33 with a 2x2 pivot across the end), one right-hand side and
nine, as a work queue and a launch per level.

Solves of one factor by one CTA a front, by clusters and by the grid: each sums
in FP64 whatever the factor's precision, so two of them differ by no more than
1e3 n u cond(K) of the largest entry (n u cond for backward stable solves, 1e3
for the growth of |L| |D| |L^T| with pivots down to 0.01 of their column)."""
import numpy as np
import pytest
import torch

from matrices import csr_arrays
from test_panel_rows_gpu import arrow

pytestmark = pytest.mark.gpu

NEVER = 1 << 62


def handle(K, precision, forms, cluster=NEVER, wide=NEVER, queue=1):
    from amigo_b200 import linalg
    n, rp, ci, v = csr_arrays(K)
    ldl = linalg.SparseLDL(linalg.CSRMat(n, n, rp, ci, v),
                           order=linalg.OrderingType.NATURAL)
    ldl.set_precision(precision)
    ldl.set_general_forms(forms)
    ldl.set_cluster_threshold(cluster)
    ldl.set_wide_threshold(wide)
    ldl.set_solve_queue(queue)
    assert ldl.factor() == 0
    return ldl


def solution(ldl, b):
    x = torch.from_numpy(b.copy()).cuda()
    ldl.solve_device(x)
    ldl.solve_status()
    return x.cpu().numpy()


SIZES = [(1, 1), (1, 3), (20, 11), (20, 12), (21, 12), (31, 20), (32, 33), (33, 5), (40, 24),
         (34, 64), (60, 5), (30, 66), (90, 7), (64, 64), (64, 65), (65, 40), (118, 20)]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("width,rows", SIZES)
def test_small_fronts_equal_general_form(width, rows, precision):
    K = arrow(width, rows, 9 * width + rows, 0.4)
    b = np.random.RandomState(5).randn(2, K.shape[0])
    a, g = handle(K, precision, 0), handle(K, precision, 1)
    assert a.get_inertia() == g.get_inertia()
    for u, w in zip(a.node_pivots(), g.node_pivots()):
        assert np.array_equal(u, w)
    assert np.array_equal(solution(a, b), solution(g, b))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("queue", [0, 1, 2])
@pytest.mark.parametrize("width,rows", SIZES + [(97, 50), (180, 30)])
def test_staged_solves_equal_general_form(width, rows, queue, precision):
    K = arrow(width, rows, 7 * width + rows, 0.5)
    a, g = handle(K, precision, 0, queue=queue), handle(K, precision, 2, queue=queue)
    for nrhs in (1, 9):
        b = np.random.RandomState(nrhs).randn(nrhs, K.shape[0])
        assert np.array_equal(solution(a, b), solution(g, b))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("width,rows", [(1, 3), (31, 97), (32, 33), (33, 5), (65, 40),
                                        (97, 150), (128, 1), (129, 63), (180, 60), (256, 33)])
def test_cluster_and_grid_solves_agree_with_one_cta(width, rows, precision):
    K = arrow(width, rows, 7 * width + rows, 0.5)
    n = K.shape[0]
    b = np.random.RandomState(6).randn(9, n)
    want = solution(handle(K, precision, 2), b)
    bound = 1e3 * n * 1.1e-16 * np.linalg.cond(K.toarray()) * np.abs(want).max(axis=1)
    assert bound.max() <= 1e-2 * np.abs(want).max()
    for cluster, wide in ((1, NEVER), (1, 1)):
        d = np.abs(solution(handle(K, precision, 0, cluster, wide), b) - want).max(axis=1)
        assert np.all(d <= bound)
