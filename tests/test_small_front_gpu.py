"""Fronts factored in shared memory at the edges of their row chunks (32, 64,
96, 128 rows, and the largest that is scheduled so), with 2x2 pivots,
interchanges and delayed pivots: the inertia is that of the eigenvalues, and the
relative residual of a solution <= 1e-10 (FP64 fronts) or 1e-3 (FP32: 6e-8 times
an element growth of a few hundred, times the rows' accumulation)."""
import numpy as np
import pytest

from matrices import csr_arrays, eig_inertia
from test_panel_rows_gpu import arrow

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,bound", [("fp64", 1e-10), ("fp32", 1e-3)])
@pytest.mark.parametrize("width,rows", [(1, 1), (20, 11), (20, 12), (21, 12), (40, 24), (60, 5),
                                        (30, 66), (90, 7), (64, 64), (64, 65), (118, 20)])
def test_chunk_edges(width, rows, precision, bound):
    from amigo_b200 import linalg
    K = arrow(width, rows, 5 * width + rows, 0.4)
    n, rp, ci, v = csr_arrays(K)
    mat = linalg.CSRMat(n, n, rp, ci, v)
    ldl = linalg.SparseLDL(mat, order=linalg.OrderingType.NATURAL)
    ldl.set_precision(precision)
    assert ldl.factor() == 0
    b = K @ np.random.RandomState(3).randn(n)
    x = b.copy()
    ldl.solve(x)
    r = np.abs(K @ x - b).max()
    assert r <= bound * (abs(K).sum(axis=1).max() * np.abs(x).max() + np.abs(b).max())
    if precision == "fp64":
        assert ldl.get_inertia() == eig_inertia(K.toarray())
