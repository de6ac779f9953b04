"""Sketch rounding of trains whose bond has a numerical rank below its rank:
the QR of a core drops noise columns, some in the stage that ends the
factorisation, and the sketch uses the Q it gets as a projector.  Two modes,
sketch rank = bond rank, so the sketch spans the train and the result is Q Q^T
x: it differs from x by rounding only, by about 100 u per core as in
test_gpu_sketch_fused, 2.5e-14 for two.  The noise levels lie around u, where a
column is dropped late or not depending on its last bits, so each size takes
many draws (kept in Q, the columns cost one draw in a hundred up to 1e-12).

Near-square and tall unfoldings, for the cluster's kernels (16, 24, 32 columns)
and the grid's (64, 128)."""
import numpy as np
import pytest

import paratt_b200 as P
from oracle import tt_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,c,keep,draws", [(12, 12, 6, 600), (24, 24, 4, 300), (32, 32, 8, 300), (300, 30, 8, 60),
                                            (33, 33, 8, 300), (33, 33, 30, 300), (40, 40, 8, 300), (64, 64, 8, 200),
                                            (400, 48, 8, 60), (80, 80, 20, 100)])
def test_projector(ctx, m, c, keep, draws):
    X = P.TT(ctx, [m, c + 3], [1, c, 1])
    Z = P.TT(ctx, [m, c + 3], [1, c, 1])
    worst = 0.0
    for seed in range(draws):
        rng = np.random.default_rng([seed, c])
        q1 = np.linalg.qr(rng.standard_normal((m, c)))[0]
        q2 = np.linalg.qr(rng.standard_normal((c, c)))[0]
        s = np.ones(c)
        s[keep:] = 10.0 ** -rng.uniform(15.5, 16.5, c - keep)
        a = (q1 * s) @ q2
        b = np.linalg.qr(rng.standard_normal((c + 3, c)))[0].T
        x = [a.reshape(1, m, c, order="F"), b.reshape(c, c + 3, 1, order="F")]
        X.set(x)
        P.round_sketch(X, None, Z, c, seed, 0.0, c)
        got = Z.get()
        full = np.einsum("ij,jk->ik", got[0][0], got[1][:, :, 0])
        worst = max(worst, np.linalg.norm(full - a @ b) / np.linalg.norm(a @ b))
    X.close()
    Z.close()
    assert worst <= 2.5e-14
