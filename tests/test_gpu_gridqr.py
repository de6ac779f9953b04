"""The grid Cholesky QR (33 to 128 columns) against the oracle and against the
Householder TSQR: roundings whose bonds sit at the edges of its column blocks
(8), of its 64- and 128-column kernels and of its rows per CTA (16, 112, 128),
for spectra that its Gram stages treat differently -- well conditioned, decaying
by 2^-j over more than double precision holds, exactly repeated, and with exactly
zero columns (the last two lose columns in the sequence).  Every factorisation
of an unfolding with at least as many rows as columns must finish there.

Tolerance: both sides truncate the same tensor at a gap of 1e-9 (or of a factor
2 at 1e-8 of the norm), so they differ by rounding only: a few u sqrt(c) per
bond, below 1e-12 of the norm for three bonds, as in test_gpu_round."""
import numpy as np
import pytest

import paratt_b200 as P
from oracle import tt_oracle as O
from test_gpu_round import gapped_tt

pytestmark = pytest.mark.gpu


def make(kind, n, c):
    dims, ranks = [n, n, n + 1, n], [1, min(c, n), c, min(c, n), 1]
    keep = [1] + [max(1, r // 2) for r in ranks[1:-1]] + [1]
    if kind == "decay":
        rng = np.random.default_rng(5)
        x = [np.linalg.qr(rng.standard_normal((ranks[k] * dims[k], ranks[k + 1])))[0] for k in range(4)]
        x = [q * 2.0 ** -np.arange(q.shape[1]) if k < 3 else q for k, q in enumerate(x)]
        return [q.reshape(ranks[k], dims[k], ranks[k + 1], order="F") for k, q in enumerate(x)], 1e-8
    if kind == "repeated":  # x + 2 x at ranks c / 2 + c / 2
        half = [1, (min(c, n - 1) + 1) // 2, (c + 1) // 2, (min(c, n - 1) + 1) // 2, 1]
        x = gapped_tt(dims, half, 7, half)
        return O.axpby(1.0, x, 2.0, x), 1e-10
    x = gapped_tt(dims, ranks, 7, keep)
    if kind == "zero":  # three columns of the middle unfoldings are exactly zero
        x[1][:, :, [0, c // 2, c - 1]] = 0.0
    return x, 1e-6


@pytest.mark.parametrize("n,c", [(40, 33), (40, 40), (64, 57), (64, 63), (64, 64), (65, 65), (72, 72), (90, 81),
                                 (101, 96), (130, 127), (128, 128)])
@pytest.mark.parametrize("kind", ["gap", "decay", "repeated", "zero"])
def test_round_parity(ctx, kind, n, c):
    x, rtol = make(kind, n, c)
    tol = rtol * O.norm(x)
    ref = O.round_tt(x, tol, 128)
    before = ctx.qr_counts()
    X = P.TT.from_cores(ctx, x)
    X.round(tol)
    got = X.get()
    after = ctx.qr_counts()
    assert O.ranks_of(got) == O.ranks_of(ref)
    assert O.rel_diff_exact(got, ref) <= 1e-12
    for u in got[1:]:
        m = O.right_unfold(u)
        np.testing.assert_allclose(m @ m.T, np.eye(m.shape[0]), atol=1e-12)
    assert after[1] == before[1] and after[0] - before[0] == 6  # three bonds, both sweeps, none fell back
    H = P.TT.from_cores(ctx, x)
    ctx.cholqr(False)
    try:
        H.round(tol)
    finally:
        ctx.cholqr(True)
    hh = H.get()
    assert O.ranks_of(hh) == O.ranks_of(got)
    assert O.rel_diff_exact(got, hh) <= 1e-12
    X.close()
    H.close()


@pytest.mark.parametrize("n,c", [(300, 64), (515, 96)])
def test_tall_unfolding(ctx, n, c):
    """More row tiles than SMs (several waves of CTAs), ragged last CTA."""
    x = gapped_tt([c, n, c], [1, c, c, 1], 9, [1, c // 2, c // 3, 1])
    tol = 1e-6 * O.norm(x)
    ref = O.round_tt(x, tol, 128)
    X = P.TT.from_cores(ctx, x)
    X.round(tol)
    got = X.get()
    assert O.ranks_of(got) == O.ranks_of(ref)
    assert O.rel_diff_exact(got, ref) <= 1e-12
    X.close()
