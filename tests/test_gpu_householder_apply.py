"""The Householder TSQR of unfoldings with more than 32 columns on its own
(Cholesky QR off): Q and Q V_r are formed by blocks that walk the tree from the
root to their leaf.  Leaf counts that are and are not a power of two (empty
leaves), one leaf, one and two 64-row chunks per node, against the oracle:
ranks equal, difference <= 1e-12 of ||X|| as in the other rounding tests, and
cores 1..d-1 right-orthonormal."""
import numpy as np
import pytest

import paratt_b200 as P
from oracle import tt_oracle as O
from test_gpu_round import gapped_tt

pytestmark = pytest.mark.gpu

CASES = [
    ([64, 64, 40], [1, 64, 50, 1], [1, 30, 20, 1]),     # 4096 x 50: 32 leaves, all with rows
    ([50, 50, 37], [1, 50, 60, 1], [1, 25, 36, 1]),     # 2500 x 60: 19 of 32 leaves
    ([48, 3, 48], [1, 48, 40, 1], [1, 20, 17, 1]),      # 144 x 40: one leaf of a two-leaf tree
    ([40, 40, 100], [1, 40, 100, 1], [1, 15, 60, 1]),   # 1600 x 100, two chunks per node
    ([96, 11, 128], [1, 96, 128, 1], [1, 40, 70, 1]),   # 1056 x 128
]


@pytest.mark.parametrize("dims,ranks,keep", CASES)
def test_householder_apply(ctx, dims, ranks, keep):
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
