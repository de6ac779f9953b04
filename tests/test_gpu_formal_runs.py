"""The run-walking branches of the formal product and of the all-modes stencil
operator (even ranks from 32 on, runs of 16 fibers) at their edges, against the
oracle: mode sizes below, at and beyond a run, ranks beyond one 64-row block,
odd neighbour ranks.  The product is one multiplication per element (equal); the
stencil is three terms, so both sides are within 3 u of the sum of magnitudes."""
import numpy as np
import pytest

import paratt_b200 as P
from oracle import tt_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 15, 16, 17, 50])
@pytest.mark.parametrize("r", [30, 32, 34, 64, 66, 130])
def test_op_sum(ctx, n, r):
    x = O.random_tt([n, n + 1, n, n], [1, r, r - 3, r, 1], 5)
    sten = [0.7, -1.9, 0.4]
    X, Y = P.TT.from_cores(ctx, x), P.TT(ctx, [n, n + 1, n, n], [1, 1, 1, 1, 1])
    P.op_sum(X, sten, 0.3, Y)
    ref = O.op_sum_apply(x, [sten] * 4, 0.3)
    mag = O.op_sum_apply([np.abs(c) for c in x], [np.abs(sten)] * 4, 0.3)
    for a, b, m in zip(Y.get(), ref, mag):
        assert a.shape == b.shape
        assert np.all(np.abs(a - b) <= 6 * 1.2e-16 * m)
    X.close()
    Y.close()


@pytest.mark.parametrize("n", [1, 16, 33])
@pytest.mark.parametrize("r,q", [(4, 8), (6, 6), (3, 12), (5, 14), (8, 8), (9, 10), (7, 5), (33, 2)])
def test_hadamard(ctx, n, r, q):
    x, y = O.random_tt([n, n, n], [1, r, r, 1], 6), O.random_tt([n, n, n], [1, q, q + 1, 1], 7)
    X, Y = P.TT.from_cores(ctx, x), P.TT.from_cores(ctx, y)
    Z = P.TT(ctx, [n, n, n], [1, 1, 1, 1])
    P.hadamard(X, Y, Z)
    for a, b in zip(Z.get(), O.hadamard(x, y)):
        assert np.array_equal(a, b)
    for t in (X, Y, Z):
        t.close()
