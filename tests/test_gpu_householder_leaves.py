"""Householder TSQR with more than 32 leaves (Cholesky QR off), where Q is
formed by a launch for the first five levels and one for each further level: 64
to 512 leaves, with and without empty ones, one and two 64-row chunks a node.
Against the oracle, with test_gpu_householder_apply's bounds."""
import numpy as np
import pytest

import paratt_b200 as P
from oracle import tt_oracle as O
from test_gpu_round import gapped_tt

pytestmark = pytest.mark.gpu

CASES = [
    ([64, 128, 40], [1, 64, 50, 1], [1, 30, 20, 1]),      # 8192 x 50: 64 leaves, all with rows
    ([50, 85, 37], [1, 50, 60, 1], [1, 25, 36, 1]),       # 4250 x 60: 33 of 64 leaves
    ([40, 701, 40], [1, 40, 37, 1], [1, 20, 17, 1]),      # 28040 x 37: 219 of 256
    ([64, 1024, 64], [1, 64, 64, 1], [1, 31, 33, 1]),     # 65536 x 64: 512
    ([100, 93, 90], [1, 100, 90, 1], [1, 15, 60, 1]),     # 9300 x 90: 36 of 64, two chunks per node
    ([96, 300, 128], [1, 96, 128, 1], [1, 40, 70, 1]),    # 28800 x 128: 112 of 128
]


@pytest.mark.parametrize("dims,ranks,keep", CASES)
def test_householder_leaves(ctx, dims, ranks, keep):
    x = gapped_tt(dims, ranks, 17, keep)
    tol = 1e-6 * O.norm(x)
    ref = O.round_tt(x, tol, 128)
    ctx.cholqr(False)
    try:
        before = ctx.qr_counts()
        X = P.TT.from_cores(ctx, x)
        X.round(tol, 128)
        got = X.get()
        X.close()
        assert ctx.qr_counts() == before  # the Householder tree ran
    finally:
        ctx.cholqr(True)
    assert O.ranks_of(got) == O.ranks_of(ref)
    assert O.rel_diff_exact(got, ref) <= 1e-12
    for c in got[1:]:
        m = O.right_unfold(c)
        np.testing.assert_allclose(m @ m.T, np.eye(m.shape[0]), atol=1e-12)
