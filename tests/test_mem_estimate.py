"""The workspace estimate (ab_ldl_mem_estimate) against what a handle allocates,
counted here from the symbolic analysis: the front and integer pools, the plan's
arrays (a node's 27 ints among them), the done flags of two sweeps and eight
right-hand-side slices, the update vectors, and the panels' global scratch, which
fronts past 8,192 rows use (delayed pivots included).  No GPU needed."""
import numpy as np
import pytest

from amigo_b200 import linalg


def star(n, m):
    """n variables: the first is coupled to the next m - 1, the rest to none."""
    cols = [np.r_[0:m]] + [np.array([0, i]) for i in range(1, m)]
    cols += [np.array([i]) for i in range(m, n)]
    rp = np.r_[0, np.cumsum([len(c) for c in cols])].astype(np.int32)
    return rp, np.concatenate(cols).astype(np.int32)


def allocated(n, rp, ci, growth, bytes_per_entry):
    S = linalg.analyze(n, rp, ci, linalg.OrderingType.NATURAL)
    ns = np.diff(S["node_ptr"]).astype(np.int64)
    nc = np.diff(S["contrib_ptr"]).astype(np.int64)
    f = ns + nc
    pools = growth * (bytes_per_entry * np.sum(f * f + 32 * f + 8) + 4 * np.sum(4 * f + 16))
    plan = (27 * 4 + 2 * 8 * 4) * (len(f) + 1) + 8 * nc.sum() + 4 * n + 12 * np.sum(ns * f)
    rows = max(int(growth * f.max()), f.max() + 64)
    groups = -(-rows // 32)
    scratch = 2 * 32 * 32 * (16 * -(-groups // 16)) * bytes_per_entry if rows > 8192 else 0
    return pools + plan + 8 * f.sum() + scratch


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("n,m,growth", [(4000, 3, 1.0),    # many nodes: flags and plan
                                        (3500, 3500, 1.0), (8128, 8128, 1.0),  # no scratch
                                        (8129, 8129, 1.0), (9000, 9000, 1.0),
                                        (4095, 4095, 2.0), (4200, 4200, 2.0), (9000, 9000, 2.0)])
def test_estimate_is_what_is_allocated(n, m, growth, precision):
    rp, ci = star(n, m)
    want = allocated(n, rp, ci, growth, precision // 8)
    got = linalg.mem_estimate(n, rp, ci, precision=precision, delay_growth=growth,
                              order=linalg.OrderingType.NATURAL)
    # (each term is truncated to whole bytes)
    assert abs(got - want) <= 8
