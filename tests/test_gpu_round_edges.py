"""Rounding at the edges of the 8-wide tiles of the contractions that carry a
bond's R (or U_r S_r) into the neighbour core: ranks 1, 7/8/9, 16/17, 24/25 and
32, mode sizes that leave ragged last tiles, and single rows.  Against the
oracle on gapped trains: ranks equal and a difference <= 1e-12 of ||X||, as in
the other rounding tests."""
import pytest

import paratt_b200 as P
from oracle import tt_oracle as O
from test_gpu_round import gapped_tt

pytestmark = pytest.mark.gpu

CASES = [
    ([9, 7, 11, 9], [1, 8, 7, 9, 1], [1, 3, 4, 4, 1], 64),
    ([17, 5, 19, 16], [1, 16, 17, 15, 1], [1, 7, 9, 8, 1], 64),
    ([31, 3, 29, 25], [1, 24, 25, 23, 1], [1, 8, 16, 9, 1], 64),
    ([33, 2, 37, 32], [1, 32, 31, 32, 1], [1, 17, 24, 25, 1], 64),
    ([33, 1, 3, 32], [1, 32, 32, 32, 1], [1, 8, 8, 8, 1], 5),
    ([257, 13, 130], [1, 12, 20, 1], [1, 1, 9, 1], 64),
    ([40, 600, 9], [1, 40, 9, 1], [1, 33, 8, 1], 64),       # 64-wide contractions, ranks on both sides of 8
    ([70, 19, 65], [1, 63, 65, 1], [1, 31, 33, 1], 64),     # 128-wide
    ([127, 9, 128], [1, 127, 121, 1], [1, 64, 57, 1], 128),
    ([40, 5000, 40], [1, 32, 32, 1], [1, 9, 17, 1], 64),    # 160000 rows: the block-level tree at 32 columns
]


@pytest.mark.parametrize("dims,ranks,keep,maxr", CASES)
def test_round_tile_edges(ctx, dims, ranks, keep, maxr):
    x = gapped_tt(dims, ranks, 19, keep)
    tol = 1e-6 * O.norm(x)
    ref = O.round_tt(x, tol, maxr)
    X = P.TT.from_cores(ctx, x)
    X.round(tol, maxr)
    got = X.get()
    X.close()
    assert O.ranks_of(got) == O.ranks_of(ref)
    assert O.rel_diff_exact(got, ref) <= 1e-12
