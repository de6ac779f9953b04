"""The Gram stages of the Cholesky-QR factorisations (ptt_gramstage.cuh), as a
numpy model of their rules: both the cluster's limits (7 stages, done at 1e-15)
and the grid's (6 stages, done at 1e-14), on well conditioned, graded, exactly
repeated, rank-deficient and noisy unfoldings, near-square and tall.

Bounds: the columns of Q that are kept are orthonormal to the level at which a
stage is taken as done plus the rounding of the products, below 1e-13 for 40
columns; A = Q R holds to a few u per stage (1e-14 of each column)."""
import numpy as np
import pytest

U = 1.1102230246251565e-16
FIRST, FIRST_DONE, PIV, DROP, SMALL, LARGE = 1e-7, 1e-8, 1e-13, 0.5 * U, 1e-280, 1e300
GRID, CLUSTER = (6, 1e-14), (7, 1e-15)


def factor(H, on):
    """chol(H), weak pivots set to PIV with a zero row, zero rows where not on; inverse pivots."""
    c = len(H)
    g, R, inv = H.copy(), np.zeros((c, c)), np.zeros(c)
    for j in np.flatnonzero(on):
        good = g[j, j] > PIV
        R[j, j] = np.sqrt(g[j, j] if good else PIV)
        inv[j] = 1.0 / R[j, j]
        if good:
            R[j, j + 1:] = g[j, j + 1:] * inv[j]
            g[j + 1:, j + 1:] -= np.outer(R[j, j + 1:], R[j, j + 1:])
    return R, inv


def solve(X, R, inv):
    Y = X.copy()
    for j in range(X.shape[1]):
        Y[:, j] = (X[:, j] - Y[:, :j] @ R[:j, j]) * inv[j]
    return Y


def stages(A, maxst, tau, clear=True):
    """(state, Q, R, stages); clear=False keeps a column that the deciding stage drops."""
    c = A.shape[1]
    Q, T = A.copy(), None
    for s in range(maxst):
        G = Q.T @ Q
        g = np.diag(G).copy()
        d = np.sqrt(np.maximum(g, 0.0))
        on = g > 0.0
        if s > 0:
            on &= d * tm > DROP * np.sqrt(c)
        else:
            an = np.where(on, 1.0 / np.where(on, d, 1.0), 0.0)
        if not np.isfinite(G).all() or (g >= LARGE).any() or ((g != 0.0) & (g < SMALL)).any() or not on.any():
            return "fallback", Q, T, s
        both = np.outer(on, on)
        e = (np.abs(G - np.eye(c)) * both).max()
        if s >= 1 and e <= tau:
            return "done", Q * on if clear else Q, T * on[:, None], s
        if s == maxst - 1:
            return "fallback", Q, T, s
        first = s >= 1 and e <= FIRST
        if first:
            diag = np.where(on, 1.0 + 0.5 * (g - 1.0), 0.0)
            F = np.triu(G, 1) * both + np.diag(diag)
            inv = np.where(on, 1.0 / np.where(on, diag, 1.0), 0.0)
        else:
            p2 = 2.0 ** np.frexp(np.where(on, d, 1.0))[1]  # D: the powers of two above the norms
            R1, inv = factor(G / np.outer(p2, p2), on)
            F, inv = R1 * np.where(on, p2, 0.0), inv / p2
        T = F if s == 0 else F @ T
        tm = (np.abs(T) * an).max(axis=1)
        Q = solve(Q, F, inv)
        if first and e <= FIRST_DONE:
            return "done", Q, T, s
    raise AssertionError


def unfolding(kind, m, c, rng):
    k = max(1, c // 2)
    if kind == "full":
        return rng.standard_normal((m, c))
    if kind == "graded":  # down to 1e-24 of the largest
        q = np.linalg.qr(rng.standard_normal((m, c)))[0]
        return q * 10.0 ** (-24.0 * np.arange(c) / c) @ np.linalg.qr(rng.standard_normal((c, c)))[0]
    if kind == "repeated":
        a = rng.standard_normal((m, (c + 1) // 2))
        return np.hstack([a, 2.0 * a])[:, :c]
    a = rng.standard_normal((m, k)) @ rng.standard_normal((k, c))
    if kind == "noise":
        a = a + 10.0 ** rng.uniform(-17, -12) * rng.standard_normal((m, c))
    if kind == "scaled":
        a = a * 10.0 ** rng.uniform(-8, 8, c)
    if kind == "zero":
        a[:, ::3] = 0.0
    return a


KINDS = ["full", "graded", "repeated", "product", "noise", "scaled", "zero"]


def spoilt(Q):
    """Largest entry of Q^T Q - I over the columns that are not zero."""
    q = Q[:, np.linalg.norm(Q, axis=0) > 0.0]
    return np.abs(q.T @ q - np.eye(q.shape[1])).max()


@pytest.mark.parametrize("limits", [GRID, CLUSTER], ids=["grid", "cluster"])
@pytest.mark.parametrize("kind", KINDS)
def test_factorisation(limits, kind):
    for seed in range(60):
        rng = np.random.default_rng([seed, KINDS.index(kind)])
        c = int(rng.integers(2, 41))
        m = c + int(rng.integers(0, 3 if seed % 2 else 100))
        A = unfolding(kind, m, c, rng)
        state, Q, R, _ = stages(A, *limits)
        assert state == "done"  # zero and repeated columns as well
        assert spoilt(Q) <= 1e-13
        err, size = np.linalg.norm(Q @ R - A, axis=0), np.linalg.norm(A, axis=0)
        assert (err <= 1e-14 * size).all()
        assert np.linalg.norm(Q @ (Q.T @ A) - A) <= 1e-14 * np.linalg.norm(A)  # Q alone is a projector onto A's range


def test_column_dropped_by_the_deciding_stage():
    """Kept in Q, it is neither of unit norm nor orthogonal to the others."""
    worst = 0.0
    for seed in range(60):
        rng = np.random.default_rng([seed, KINDS.index("product")])
        A = unfolding("product", 14, 12, rng)
        worst = max(worst, spoilt(stages(A, *GRID, clear=False)[1]))
        assert spoilt(stages(A, *GRID)[1]) <= 1e-13
    assert worst > 1e-13  # beyond the bound above


def test_no_finite_factorisation():
    A = np.random.default_rng(0).standard_normal((9, 4))
    A[3, 1] = np.nan
    assert stages(A, *GRID)[0] == "fallback"
    assert stages(np.zeros((9, 4)), *GRID)[0] == "fallback"
    assert stages(1e-150 * np.ones((9, 4)), *GRID)[0] == "fallback"  # squares that lose digits
    with np.errstate(over="ignore"):
        assert stages(1e155 * np.ones((9, 4)), *GRID)[0] == "fallback"
