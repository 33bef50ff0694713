"""The rows that a level reports for the level above: a root that its child's
delayed pivots grow past its static size and the 64 rows of room has its panels
launched for the rows it has, so none falls back to one CTA (panel_fallbacks).
The roots are large fronts statically (130 rows and more), their children too, and
the delays are more than the room."""
import numpy as np
import pytest

from matrices import csr_arrays
from test_level_rows_gpu import saddle

pytestmark = pytest.mark.gpu


def check(K, width, rows):
    from amigo_b200 import linalg
    n, rp, ci, v = csr_arrays(K)
    ldl = linalg.SparseLDL(linalg.CSRMat(n, n, rp, ci, v),
                           order=linalg.OrderingType.NATURAL)
    assert ldl.factor() == 0
    _, ndel = ldl.node_pivots()
    assert sum(ndel) == width
    assert ldl.get_inertia() == (width + rows, width)
    b = K @ np.random.RandomState(4).randn(n)
    x = b.copy()
    ldl.solve(x)
    r = np.abs(K @ x - b).max()
    assert r <= 1e-10 * (abs(K).sum(axis=1).max() * np.abs(x).max() + np.abs(b).max())
    return ldl.panel_fallbacks()


@pytest.mark.parametrize("width,rows", [(70, 130), (190, 200), (100, 300), (400, 450)])
def test_rows_are_known(width, rows):
    assert check(saddle(width, rows, width), width, rows) == 0
