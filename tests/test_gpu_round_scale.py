"""A factorisation must not stretch or shrink a train on average: a program
rounds the same state thousands of times, and a factor next to 1 in each adds up
where rounding errors average out.

Trains of rank 1, whose bond SVDs rotate nothing: what a rounding with tolerance
0 changes is the product of a column's pivot and its inverse.  Per train <x,
round(x)> / <x, x> - 1 in extended precision; a factorisation rounds some five
times by at most u / 2 (rms u / 2 sqrt(3)), 22 of them scatter one train's value
by u sqrt(110) / 3.5 = 3.3e-16, and the mean of 100 trains by 3.3e-17; the bound
is 2e-16, six of them.  A pivot off by its inverse by 1.2e-16 on average gives
2.6e-15, and -1.5e-15 was seen for cores of norm 1."""
import numpy as np
import pytest

import paratt_b200 as P

pytestmark = pytest.mark.gpu


def inner(x, y):
    v = np.longdouble(1)
    for a, b in zip(x, y):
        v = v * np.sum(a.astype(np.longdouble) * b.astype(np.longdouble))
    return v


@pytest.mark.parametrize("n", [6, 64, 700])
@pytest.mark.parametrize("kind", ["signed", "scaled", "unit"])
def test_no_drift(ctx, n, kind):
    d = 12
    X = P.TT(ctx, [n] * d, [1] * (d + 1))
    s = []
    for seed in range(100):
        rng = np.random.default_rng([seed, n])
        x = [rng.standard_normal((1, n, 1)) for _ in range(d)]
        if kind == "scaled":
            x = [np.abs(c) * np.exp(rng.uniform(-3, 3)) for c in x]
        if kind == "unit":
            x = [c / np.linalg.norm(c) for c in x]
        X.set(x)
        X.round(0.0, 1)
        s.append(float(inner(x, X.get()) / inner(x, x) - 1))
    X.close()
    assert abs(np.mean(s)) <= 2e-16
