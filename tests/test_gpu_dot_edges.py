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
