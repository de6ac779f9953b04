"""The pair order of the bond SVD's sweeps (ptt_svd.cuh: circle_blk, ring_blks,
svd_pair), which the replay of the rotations relies on, mirrored in Python for
every number of columns the kernels take: each pair of columns is rotated
exactly once a sweep, the pairs of a step are disjoint, the blocks that move
between the groups are where the order says, and the sizes of the replay's
tables hold."""
import pytest

CIRCLE, RING = 2, 3


def circle_blk(pos, s, nblk):
    return 0 if pos == 0 else 1 + (pos - 1 + s) % (nblk - 1)


def ring_blks(g, s, G):
    lg = (2 * G - 1 - s).bit_length() - 1
    hb = 1 << lg
    sh, i, b0 = s - (2 * G - 2 * hb), g & (hb - 1), (g >> lg) << (lg + 1)
    return b0 + i, b0 + hb + ((i + sh) & (hb - 1))


def svd_pair(pr, st, G, order):
    g, k, ns = pr >> 1, pr & 1, 2 * G - 1
    if st == 2 * ns:
        blk = pr if order == RING else (2 * G - 1 - g if k else g)
        return 2 * blk, 2 * blk + 1
    if order == RING:
        a, b = ring_blks(g, st >> 1, G)
    else:
        a, b = circle_blk(g, st >> 1, 2 * G), circle_blk(2 * G - 1 - g, st >> 1, 2 * G)
    return 2 * a + k, 2 * b + (k ^ (st & 1))


def groups(qa, rb):
    """(groups, order) for qa columns in the kernel of rb rows."""
    gc = (qa + 3) >> 2 if qa > 4 else 1
    gr = 1 << (gc - 1).bit_length() if gc > 1 else 1
    ring = 4 * gr <= rb and 20 * (4 * gr - 1) <= 23 * (4 * gc - 1)
    return (gr, RING) if ring else (gc, CIRCLE)


CHOICES = sorted({groups(qa, rb) for rb in (16, 32, 48, 64, 96, 128) for qa in range(1, rb + 1)})


@pytest.mark.parametrize("G,order", CHOICES)
def test_every_pair_once(G, order):
    n = 4 * G
    seen = set()
    for st in range(4 * G - 1):
        cols = []
        for pr in range(2 * G):
            p, q = svd_pair(pr, st, G, order)
            cols += [p, q]
            seen.add((min(p, q), max(p, q)))
        assert sorted(cols) == list(range(n))
    assert len(seen) == n * (n - 1) // 2


@pytest.mark.parametrize("G,order", CHOICES)
def test_moves_follow_the_order(G, order):
    ns = 2 * G - 1
    A, B = list(range(G)), [G + g if order == RING else 2 * G - 1 - g for g in range(G)]
    home = A[:], B[:]
    s = 0
    if order == RING:
        hb = G
        while hb >= 1:
            for _ in range(hb):
                assert [(A[g], B[g]) for g in range(G)] == [ring_blks(g, s, G) for g in range(G)]
                s += 1
                if hb > 1:
                    B = [B[g - (g & (hb - 1)) + (((g & (hb - 1)) + 1) & (hb - 1))] for g in range(G)]
            if hb >= 2:
                h = hb >> 1
                low = [(g & (hb - 1)) < h for g in range(G)]
                put = [B[g] if low[g] else A[g] for g in range(G)]
                A, B = ([A[g] if low[g] else put[g ^ h] for g in range(G)],
                        [put[g ^ h] if low[g] else B[g] for g in range(G)])
            hb >>= 1
        slots = [v for g in range(G) for v in (A[g], B[g])]
        assert slots == list(range(2 * G))  # group g: blocks 2 g, 2 g + 1
        A, B = slots[:G], slots[G:]
    else:
        for s in range(ns):
            assert [(A[g], B[g]) for g in range(G)] == [
                (circle_blk(g, s, 2 * G), circle_blk(2 * G - 1 - g, s, 2 * G)) for g in range(G)]
            if G > 1:
                slot = A + B
                A, B = ([A[0]] + [slot[G + g if g == G - 1 else g + 1] for g in range(1, G)],
                        [slot[G + g - 1 if g > 0 else 1] for g in range(G)])
        s = ns
    assert s == ns and (A, B) == home


@pytest.mark.parametrize("rb,ct", [(16, 32), (32, 32), (48, 64), (64, 64), (96, 128), (128, 128)])
def test_replay_tables(rb, ct):
    for qa in range(1, rb + 1):
        G, _ = groups(qa, rb)
        assert 4 * G >= qa and 4 * G <= rb
        assert 4 * G - 1 <= ct + 1 and 2 * G <= (ct + 2) // 2  # steps and pairs a sweep may have
        assert 2 * G <= 64  # two pairs a lane of the replaying warp
    assert ct | ct << 8 < 1 << 16  # two columns, or "none" (ct), in 16 bits
