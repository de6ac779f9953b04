"""Inner products: infinite entries at ranks that are no multiple of the tiles,
where the kernel's padding must not turn an infinity into a NaN."""
import numpy as np
import pytest

import paratt_b200 as P
from oracle import tt_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r", [1, 2, 3, 5, 6, 7, 9, 15, 33, 63, 64, 65])
@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("side", ["x", "y", "both"])
def test_infinite_entry(ctx, r, mode, side):
    """Positive entries and one infinite one: every term is positive, so the
    inner product is infinite."""
    rng = np.random.default_rng(r)
    dims, ranks = [5, 6, 4], [1, r, max(1, r - 1), 1]
    x, y = ([0.5 + rng.random((ranks[k], dims[k], ranks[k + 1])) for k in range(3)] for _ in "xy")
    for t in ((x,) if side == "x" else (y,) if side == "y" else (x, y)):
        t[mode][-1, 1, -1] = np.inf
    X, Y = P.TT.from_cores(ctx, x), P.TT.from_cores(ctx, y)
    assert X.dot(Y) == np.inf
    assert X.dot_noalloc(Y) == np.inf
    X.close()
    Y.close()


@pytest.mark.parametrize("dims,r,q", [([40, 5, 40, 4], 1, 1), ([256, 5, 150, 4], 7, 20), ([9, 5, 9, 4], 63, 64),
                                      ([12, 5, 9, 4], 64, 64), ([16, 5, 9, 4], 20, 65)])
def test_capacity_does_not_matter(ctx, dims, r, q):
    """The same bits whatever the buffers hold, by either entry point."""
    x = O.random_tt(dims, [1, r, max(1, r - 1), r, 1], 3, std=0.3)
    y = O.random_tt(dims, [1, q, q, max(1, q - 3), 1], 4, std=0.3)
    X, Y = P.TT.from_cores(ctx, x), P.TT.from_cores(ctx, y)
    want = X.dot(Y)
    assert abs(want - O.dot(x, y)) <= 1e-13 * O.norm(x) * O.norm(y)
    assert X.dot_noalloc(Y) == want
    for cx in (max(r, 64), 65, 128):
        Z = P.TT.from_cores(ctx, x, [1] + [cx] * 3 + [1])
        assert Z.dot(Y) == want
        assert Z.norm() == X.norm()
        Z.close()
    X.close()
    Y.close()
