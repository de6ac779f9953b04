"""Sketch rounding at small ranks, where the contractions of a core are fused
per mode index: around the edges of its tiles (ranks 8/9, 16/17, 24/25, 32 for
one train; 8 and sketch rank 16 for a product), of its split over warps and
CTAs (mode sizes 1, 7, 8, 9, 256, 257, 1025, 2048) and one past each limit
(ranks 33 and 9, sketch rank 17, mode size 2049: the general contractions).

The trains have true ranks t hidden in ranks r by orthonormal gauges, and
sketch ranks t + 6 or more, so the sketch spans the train: a Gaussian sketch
with 6 columns to spare has a condition number of some tens, the result is the
train itself to about 100 u per core, and the bound is 1e-12 of its norm as in
the other rounding tests.  The ranks found are t (or the modes' own limit)."""
import numpy as np
import pytest

import paratt_b200 as P
from oracle import tt_oracle as O

pytestmark = pytest.mark.gpu


def hidden(dims, r, t, seed):
    """Train of true ranks <= t stored with ranks r (a list, ends 1)."""
    rng = np.random.default_rng(seed)
    d = len(dims)
    tr = [1] + [min(t, r[k]) for k in range(1, d)] + [1]
    E = [np.ones((1, 1))] + [np.linalg.qr(rng.standard_normal((r[k], tr[k])))[0] for k in range(1, d)] + [np.ones((1, 1))]
    out = []
    for k, n in enumerate(dims):
        c = rng.standard_normal((tr[k], n, tr[k + 1])) / np.sqrt(n * tr[k])
        out.append(np.einsum("ia,anb,jb->inj", E[k], c, E[k + 1]))
    return out


ONE = [
    # dims, ranks, t, ell
    ([6, 8, 9, 7, 5], [1, 6, 8, 8, 5, 1], 3, 9),
    ([256, 7, 257, 12], [1, 9, 16, 12, 1], 4, 10),
    ([40, 1, 33, 40], [1, 16, 16, 17, 1], 5, 12),
    ([64, 20, 9, 64], [1, 24, 24, 24, 1], 14, 22),
    ([1025, 8, 30], [1, 25, 24, 1], 10, 17),
    ([2048, 9, 40], [1, 32, 32, 1], 18, 32),
    ([40, 24, 40, 17], [1, 32, 19, 5, 1], 16, 24),
    ([2049, 8, 30], [1, 17, 9, 1], 3, 9),           # general: mode size
    ([40, 40, 40], [1, 33, 32, 1], 6, 12),          # general: rank
    ([30, 40], [1, 13, 1], 4, 10),
]


@pytest.mark.parametrize("dims,r,t,ell", ONE)
def test_sketch_one_train(ctx, dims, r, t, ell):
    x = hidden(dims, r, t, 3)
    tol = 1e-10 * O.norm(x)
    ref = O.round_tt(x, tol, 64)
    X = P.TT.from_cores(ctx, x)
    Z = P.TT(ctx, dims, [1] + [40] * (len(dims) - 1) + [1])
    P.round_sketch(X, None, Z, ell, 11, tol, 64, pad=2)
    got = Z.get()
    assert O.ranks_of(got) == O.ranks_of(ref)
    assert O.rel_diff_exact(got, x) <= 1e-12
    X.close()
    Z.close()


TWO = [
    # dims, ranks of x, of y, t of x, of y, ell
    ([6, 8, 9, 7, 5], [1, 6, 8, 8, 5, 1], [1, 6, 8, 7, 5, 1], 2, 3, 12),
    ([256, 7, 257, 12], [1, 8, 1, 5, 1], [1, 3, 8, 8, 1], 2, 2, 16),
    ([40, 1, 33, 40], [1, 4, 4, 8, 1], [1, 2, 2, 1, 1], 3, 2, 13),
    ([1025, 8, 30], [1, 8, 8, 1], [1, 8, 8, 1], 3, 3, 16),
    ([40, 9, 40], [1, 9, 8, 1], [1, 8, 8, 1], 2, 2, 12),   # general: rank of x
    ([40, 9, 40], [1, 8, 8, 1], [1, 8, 9, 1], 2, 2, 12),   # general: rank of y
    ([40, 9, 40], [1, 8, 8, 1], [1, 8, 8, 1], 3, 3, 17),   # general: sketch rank
]


@pytest.mark.parametrize("dims,rx,ry,tx,ty,ell", TWO)
def test_sketch_product(ctx, dims, rx, ry, tx, ty, ell):
    x, y = hidden(dims, rx, tx, 5), hidden(dims, ry, ty, 6)
    full = O.hadamard(x, y)
    tol = 1e-10 * O.norm(full)
    ref = O.round_tt(full, tol, 64)
    X, Y = P.TT.from_cores(ctx, x), P.TT.from_cores(ctx, y)
    Z = P.TT(ctx, dims, [1] + [40] * (len(dims) - 1) + [1])
    P.round_sketch(X, Y, Z, ell, 11, tol, 64, pad=2)
    got = Z.get()
    assert O.ranks_of(got) == O.ranks_of(ref)
    assert O.rel_diff_exact(got, full) <= 1e-12
    for t in (X, Y, Z):
        t.close()
