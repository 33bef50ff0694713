"""The large-front panel with one row per thread (panel mode 0) at the edges
of its rows: 256 threads a CTA on clusters of 1, 2, 4, 8 and 16 CTAs, then two
rows a thread.  Every row gets the operations of the global-scratch cluster
panel (panel mode 3) in the same order, so inertia, per-node pivot and delay
counts and the solution are equal bit for bit; the relative residual of the
solution is <= 1e-10."""
import numpy as np
import pytest
import scipy.sparse as sp

from matrices import csr_arrays

pytestmark = pytest.mark.gpu


def arrow(width, rows, seed, zero_share):
    """Two dense blocks of `width` variables coupled to the same `rows` shared
    variables (natural order: two fronts of width + rows rows, then a root of
    `rows`), with a share of zero diagonals (2x2 pivots and interchanges) and
    columns that are large only in the shared rows (delayed pivots)."""
    r = np.random.RandomState(seed)
    n = 2 * width + rows
    A = np.zeros((n, n))
    S = slice(2 * width, n)
    for b in range(2):
        B = slice(b * width, (b + 1) * width)
        A[B, B] = r.randn(width, width)
        A[S, B] = r.randn(rows, width) * 0.1
        late = b * width + r.choice(width, max(1, width // 8), replace=False)
        A[B, late] *= 1e-3
        A[late, B] *= 1e-3
        A[2 * width:, late] *= 100.0
    A[S, S] = r.randn(rows, rows) * 0.1
    A = np.tril(A) + np.tril(A, -1).T
    d = r.randn(n)
    d[r.rand(n) < zero_share] = 0.0
    A[np.arange(n), np.arange(n)] = d
    K = sp.csr_matrix(A)
    # the whole block pattern, explicit zeros included
    P = np.zeros((n, n), bool)
    for b in range(2):
        i = np.r_[b * width:(b + 1) * width, 2 * width:n]
        P[np.ix_(i, i)] = True
    rr, cc = np.nonzero(P)
    K = sp.csr_matrix((A[rr, cc], (rr, cc)), shape=(n, n))
    K.sort_indices()
    return K


def factor_solve(K, mode, precision, b):
    from amigo_b200 import linalg
    n, rp, ci, v = csr_arrays(K)
    mat = linalg.CSRMat(n, n, rp, ci, v)
    ldl = linalg.SparseLDL(mat, order=linalg.OrderingType.NATURAL)
    ldl.set_panel_mode(mode, 1)
    ldl.set_precision(precision)
    assert ldl.factor() == 0
    x = b.copy()
    ldl.solve(x)
    npiv, ndel = ldl.node_pivots()
    return ldl.get_inertia(), npiv, ndel, x


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("width,rows", [(31, 225), (40, 217), (70, 442), (65, 448),
                                        (100, 924), (130, 895), (33, 2015), (32, 2017)])
def test_rows_panel_equals_global_form(width, rows, precision):
    K = arrow(width, rows, width + rows, 0.4)
    b = K @ np.random.RandomState(3).randn(K.shape[0])
    i0, p0, d0, x0 = factor_solve(K, 0, precision, b)
    i3, p3, d3, x3 = factor_solve(K, 3, precision, b)
    assert i0 == i3
    assert np.array_equal(p0, p3) and np.array_equal(d0, d3)
    assert np.array_equal(x0, x3)
    if precision == "fp64":
        r = np.abs(K @ x0 - b).max()
        assert r <= 1e-10 * (abs(K).sum(axis=1).max() * np.abs(x0).max() + np.abs(b).max())


def test_two_rows_a_thread():
    """A 3D KKT with fronts past 4,096 rows (two rows a thread)."""
    from test_cluster_panel_gpu import check_global_form, simp3d_kkt
    check_global_form(simp3d_kkt(20, 10, 10), 1)
