"""The bond SVD (block Jacobi in registers) at the edges of its kernels (16, 32,
48, 64, 96, 128 columns), of its groups of four columns and of both pair
orders: roundings of two-mode trains against the oracle, and the singular
values it reports against numpy's of the same matrix.  "noise": columns below
the numerical-rank threshold, which take no part in the sweeps.

Tolerances: a Jacobi SVD's values are within a few c u of the largest one (1e-13
allows c = 128 with a factor of 7); the truncated product is cut at a gap, so
both sides differ by rounding (1e-12, as in test_gpu_round)."""
import numpy as np
import pytest

import paratt_b200 as P
from oracle import tt_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [1, 2, 3, 4, 5, 7, 8, 12, 13, 16, 17, 20, 24, 28, 31, 32, 33, 47, 48, 49, 60, 64, 65, 95, 96,
                               97, 128])
@pytest.mark.parametrize("kind", ["flat", "decay", "noise"])
def test_two_modes(ctx, c, kind):
    rng = np.random.default_rng(100 * c + len(kind))
    n = c + 9
    q1 = np.linalg.qr(rng.standard_normal((n, c)))[0]
    q2 = np.linalg.qr(rng.standard_normal((n, c)))[0]
    s = {"flat": 1.0 + rng.random(c), "decay": 2.0 ** -np.arange(c),
         "noise": np.where(np.arange(c) % 3 == 1, 1e-18, 1.0 + rng.random(c))}[kind]
    mix = np.linalg.qr(rng.standard_normal((c, c)))[0] if kind == "flat" else np.eye(c)
    keep = max(1, (2 * c) // 3)
    sv = np.sort(s)[::-1]
    if kind == "flat":  # a gap at the cutoff
        s = np.where(np.arange(c) < keep, s, 1e-7 * s)
        sv = np.sort(s)[::-1]
    x = [(q1 @ mix).reshape(1, n, c, order="F"), ((mix.T * s) @ q2.T).reshape(c, n, 1, order="F")]
    tol = 1e-5 * O.norm(x)
    ref = O.round_tt(x, tol, 128)
    X = P.TT.from_cores(ctx, x)
    X.round(tol)
    got = X.get()
    assert O.ranks_of(got) == O.ranks_of(ref)
    assert O.rel_diff_exact(got, ref) <= 1e-12
    top = ctx.round_stats(2)[1][8:8 + min(c, 16)]
    assert np.all(np.abs(top - sv[:16][:len(top)]) <= 1e-13 * sv[0])
    m = O.right_unfold(got[1])
    np.testing.assert_allclose(m @ m.T, np.eye(m.shape[0]), atol=1e-12)
    X.close()
