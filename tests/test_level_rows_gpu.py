"""A front that its child's delayed pivots grow past the room its static size
leaves (64 rows): its panels are launched for the rows that the level below
reports.  The child holds the multipliers of a saddle point, a zero block of
which no pivot can be taken, so all of them are delayed.  Panel modes 0 and 3
agree bit for bit (inertia, pivots, delays, solution), the inertia is that of the
saddle point and the relative residual <= 1e-10."""
import numpy as np
import pytest
import scipy.sparse as sp

from matrices import csr_arrays
from test_panel_rows_gpu import factor_solve

pytestmark = pytest.mark.gpu


def saddle(width, rows, seed):
    """[[0, 0, B^T], [0, P, C^T], [B, C, S]] in natural order: `width`
    multipliers, as many primal variables and `rows` shared ones, P and S - C
    P^-1 C^T positive definite, B of full rank: `width` negative eigenvalues."""
    r = np.random.RandomState(seed)
    n = 2 * width + rows
    A = np.zeros((n, n))
    M, P, S = slice(0, width), slice(width, 2 * width), slice(2 * width, n)
    A[S, M] = np.linalg.qr(r.randn(rows, width))[0]
    A[P, P] = np.eye(width) * 4.0 + 0.5 / width * np.ones((width, width))
    A[S, P] = 0.5 * np.linalg.qr(r.randn(rows, width))[0]
    A[S, S] = np.eye(rows) * 2.0 + 0.5 / rows * np.ones((rows, rows))
    A = np.tril(A) + np.tril(A, -1).T
    Z = A != 0.0
    Z[M, M] = True
    rr, cc = np.nonzero(Z)
    K = sp.csr_matrix((A[rr, cc], (rr, cc)), shape=(n, n))
    K.sort_indices()
    return K


@pytest.mark.parametrize("width,rows", [(70, 90), (100, 300), (190, 200)])
def test_grown_front(width, rows):
    K = saddle(width, rows, width)
    b = K @ np.random.RandomState(3).randn(K.shape[0])
    i0, p0, d0, x0 = factor_solve(K, 0, "fp64", b)
    i3, p3, d3, x3 = factor_solve(K, 3, "fp64", b)
    assert sum(d0) == width
    assert i0 == i3 == (width + rows, width)
    assert np.array_equal(p0, p3) and np.array_equal(d0, d3) and np.array_equal(x0, x3)
    r = np.abs(K @ x0 - b).max()
    assert r <= 1e-10 * (abs(K).sum(axis=1).max() * np.abs(x0).max() + np.abs(b).max())
