"""Waits for messages between the CTAs of a front's cluster that run out: with a
limit of 0 polls every wait gives up at once.  The factorization raises and
leaves the handle unfactored, a solve is reported by solve_status(), and the
device stays usable: with the default limit again, the results equal those of a
fresh handle bit for bit."""
import numpy as np
import pytest
import torch

from matrices import csr_arrays
from test_panel_rows_gpu import arrow

pytestmark = pytest.mark.gpu

DEFAULT = 1 << 20


def handle(K, precision):
    from amigo_b200 import linalg
    n, rp, ci, v = csr_arrays(K)
    ldl = linalg.SparseLDL(linalg.CSRMat(n, n, rp, ci, v),
                           order=linalg.OrderingType.NATURAL)
    ldl.set_precision(precision)
    return ldl


def solution(ldl, b):
    x = torch.from_numpy(b.copy()).cuda()
    ldl.solve_device(x)
    return x.cpu().numpy()


# fronts of 600 rows (clusters of 4 CTAs) and 500 (2), of 2,600 (16) and 2,500
@pytest.mark.parametrize("width,rows", [(100, 500), (100, 2500)])
def test_panel_wait_runs_out(width, rows):
    K = arrow(width, rows, 11, 0.4)
    b = np.random.RandomState(1).randn(K.shape[0])
    ldl, fresh = handle(K, "fp64"), handle(K, "fp64")
    ldl.set_wait_limit(0)
    for _ in range(2):
        with pytest.raises(RuntimeError):
            ldl.factor()
        with pytest.raises(RuntimeError):
            solution(ldl, b)
    ldl.set_wait_limit(DEFAULT)
    assert ldl.factor() == 0 and fresh.factor() == 0
    assert ldl.get_inertia() == fresh.get_inertia()
    assert np.array_equal(solution(ldl, b), solution(fresh, b))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("width,rows", [(200, 60), (400, 5), (270, 100)])
def test_small_front_above_a_wait_that_ran_out(width, rows, precision):
    """The front above is one of the small ones, which are assembled from their
    children's pivot counts: it is skipped (in a new handle the counts are 0,
    and a child's rows would be more than the front has)."""
    K = arrow(width, rows, 13, 0.4)
    b = np.random.RandomState(3).randn(K.shape[0])
    ldl, fresh = handle(K, precision), handle(K, precision)
    ldl.set_wait_limit(0)
    with pytest.raises(RuntimeError):
        ldl.factor()
    ldl.set_wait_limit(DEFAULT)
    assert ldl.factor() == 0 and fresh.factor() == 0
    assert ldl.get_inertia() == fresh.get_inertia()
    assert np.array_equal(solution(ldl, b), solution(fresh, b))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nrhs", [1, 17])
def test_solve_wait_runs_out(precision, nrhs):
    K = arrow(180, 60, 12, 0.5)
    b = np.random.RandomState(2).randn(nrhs, K.shape[0])
    ldl = handle(K, precision)
    ldl.set_cluster_threshold(1)
    assert ldl.factor() == 0
    want = solution(ldl, b)
    ldl.solve_status()
    ldl.set_wait_limit(0)
    solution(ldl, b)
    with pytest.raises(RuntimeError):
        ldl.solve_status()
    ldl.set_wait_limit(DEFAULT)
    assert np.array_equal(solution(ldl, b), want)
    ldl.solve_status()
