"""The run-walking kernels of the formal product and of the all-modes stencil
operator in trains with enough runs to take them: one large core among many
small ones (which go fiber by fiber in the same call), runs of 16 fibers with a
last one that is full, ragged, one fiber or the only one, and one row less of
ranks than the even 32 they need.  Against the oracle, with
test_gpu_formal_runs's bounds; the second call reads what the first one's last
block published."""
import numpy as np
import pytest

import paratt_b200 as P
from oracle import tt_oracle as O

pytestmark = pytest.mark.gpu

D, AT = 100, 50  # runs count 100-fold: 2048 and 4096 are reached from r1 = 21 and 41 on


@pytest.mark.parametrize("n,r1", [(13, 34), (16, 21), (16, 20), (23, 66), (63, 60), (177, 64), (353, 37), (241, 65)])
@pytest.mark.parametrize("r", [30, 32, 33, 34, 66])
def test_op_sum(ctx, n, r1, r):
    dims = [3] * D
    dims[AT] = n
    ranks = [1] + [2] * (D - 1) + [1]
    ranks[AT], ranks[AT + 1] = r, r1
    x = O.random_tt(dims, ranks, 5)
    sten = [0.7, -1.9, 0.4]
    X, Y = P.TT.from_cores(ctx, x), P.TT(ctx, dims, [1] * (D + 1))
    for _ in range(2):
        P.op_sum(X, sten, 0.3, Y)
    ref = O.op_sum_apply(x, [sten] * D, 0.3)
    mag = O.op_sum_apply([np.abs(c) for c in x], [np.abs(sten)] * D, 0.3)
    for a, b, m in zip(Y.get(), ref, mag):
        assert a.shape == b.shape
        assert np.all(np.abs(a - b) <= 6 * 1.2e-16 * m)
    X.close()
    Y.close()


@pytest.mark.parametrize("n,r1,q1", [(13, 2, 17), (15, 6, 7), (16, 5, 8), (23, 6, 11), (63, 6, 10), (177, 8, 8), (241, 7, 9)])
@pytest.mark.parametrize("r,q", [(4, 8), (5, 14), (33, 2), (5, 9)])
def test_hadamard(ctx, n, r1, q1, r, q):
    dims = [3] * D
    dims[AT] = n
    rx, ry = [1] + [2] * (D - 1) + [1], [1] + [1] * (D - 1) + [1]
    rx[AT], rx[AT + 1], ry[AT], ry[AT + 1] = r, r1, q, q1
    x, y = O.random_tt(dims, rx, 6), O.random_tt(dims, ry, 7)
    X, Y = P.TT.from_cores(ctx, x), P.TT.from_cores(ctx, y)
    Z = P.TT(ctx, dims, [1] * (D + 1))
    for _ in range(2):
        P.hadamard(X, Y, Z)
    for a, b in zip(Z.get(), O.hadamard(x, y)):
        assert np.array_equal(a, b)
    for t in (X, Y, Z):
        t.close()
