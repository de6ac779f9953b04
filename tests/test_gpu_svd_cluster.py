"""The bond SVD on clustered singular values: factors Q (I + eps E), where every
cosine is tiny from the start but the rotations are not, so that sweeps whose
cosines are small must not be taken for the last one.

Tolerance: as in test_gpu_svd, 1e-13 of the largest value (a few c u at 128
columns, with a factor of 7); the values differ by eps, up to 1e3 times that."""
import numpy as np
import pytest

import paratt_b200 as P
from oracle import tt_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [2, 3, 4, 5, 8, 13, 16, 17, 20, 32, 33, 48, 49, 64, 65, 96, 97, 128])
@pytest.mark.parametrize("eps", [1e-10, 1e-12])
@pytest.mark.parametrize("kind", ["one", "two"])
def test_cluster(ctx, c, eps, kind):
    rng = np.random.default_rng([c, int(-np.log10(eps)), len(kind)])
    n = c + 9
    q1 = np.linalg.qr(rng.standard_normal((n, c)))[0]
    q2 = np.linalg.qr(rng.standard_normal((n, c)))[0]
    mix = np.linalg.qr(rng.standard_normal((c, c)))[0]
    a = np.eye(c) + eps * rng.standard_normal((c, c))
    if kind == "two":  # half of the values near 1, half near 1/2, the spaces mixed
        a = mix @ (a * np.where(np.arange(c) % 2, 0.5, 1.0)) @ mix.T
    b = a @ q2.T
    x = [q1.reshape(1, n, c, order="F"), b.reshape(c, n, 1, order="F")]
    sv = np.linalg.svd(b, compute_uv=False)
    X = P.TT.from_cores(ctx, x)
    X.round(1e-6 * O.norm(x))
    got = X.get()
    assert O.ranks_of(got) == [1, c, 1]
    top = ctx.round_stats(2)[1][8:8 + min(c, 16)]
    assert np.all(np.abs(top - sv[:16][:len(top)]) <= 1e-13 * sv[0])
    assert O.rel_diff_exact(got, x) <= 1e-12
    m = O.right_unfold(got[1])
    np.testing.assert_allclose(m @ m.T, np.eye(c), atol=1e-12)
    u = got[0].reshape(n, c, order="F")  # U S: orthogonal columns
    g = u.T @ u
    np.testing.assert_allclose(g - np.diag(np.diag(g)), 0.0, atol=1e-12)
    X.close()
