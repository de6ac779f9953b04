"""Inner products at the edges of the fused contraction (8 x 8 tiles, ranks to
64, one CTA per mode index and fewer) and one rank beyond it, which takes the
general kernels, against the oracle.  Both sum n r products of rounded terms per
core in another order: the difference is a few u times the sum of magnitudes,
below 1e-13 ||x|| ||y|| here as in test_gpu_ops."""
import numpy as np
import pytest

import paratt_b200 as P
from oracle import tt_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 150, 301])
@pytest.mark.parametrize("r,q", [(1, 1), (2, 9), (7, 8), (8, 16), (17, 5), (31, 64), (63, 64), (64, 64), (65, 3)])
def test_dot(ctx, n, r, q):
    dims = [n, 5, n, 4]
    x = O.random_tt(dims, [1, r, max(1, r - 1), r, 1], 3, std=0.3)
    y = O.random_tt(dims, [1, q, q, max(1, q - 3), 1], 4, std=0.3)
    X, Y = P.TT.from_cores(ctx, x), P.TT.from_cores(ctx, y)
    tol = 1e-13 * O.norm(x) * O.norm(y)
    assert abs(X.dot(Y) - O.dot(x, y)) <= tol
    assert abs(Y.dot(X) - O.dot(x, y)) <= tol
    assert abs(X.norm() - O.norm(x)) <= 1e-13 * O.norm(x)
    need = 2 * r * q + max(max(r, q) ** 2 * n, r * q * n)
    if need <= 1 << 18:
        assert abs(X.dot_noalloc(Y) - O.dot(x, y)) <= tol
    # a capacity above the ranks does not change the value
    Z = P.TT.from_cores(ctx, x, [1] + [64 if r <= 64 else r] * 3 + [1])
    assert Z.dot(Y) == X.dot(Y)
    for t in (X, Y, Z):
        t.close()
