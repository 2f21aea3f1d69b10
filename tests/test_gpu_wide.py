"""Counts-tier pushes whose child is wide: 48 to 128 kept rows that most of the
candidates meet in two rows or more, below, inside and above the sizes from
which a warp's bitmap-tier scratch would not hold a level per kept row, several
such pushes in one task."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def nested(nV, nL, kept, n, seed):
    """A row of all nL U vertices, one of the first `kept`, n rows that hold two
    or more of those (prefixes; a third of them with one U vertex beyond, so
    that they outlive the first push), a second row of `kept` that overlaps the
    first, and pairs outside up to nV rows."""
    rng = np.random.default_rng(seed)
    adj = [np.arange(nL), np.arange(kept)]
    for i in range(n):
        r = np.arange(2 + i % (kept - 2))
        if i % 3 == 0:
            r = np.append(r, rng.integers(kept, nL))
        adj.append(r)
    adj.append(np.arange(nL - kept, nL))
    while len(adj) < nV:
        adj.append(np.sort(rng.choice(np.arange(kept, nL), size=2, replace=False)))
    ro = np.zeros(len(adj) + 1, np.int32)
    ro[1:] = np.cumsum([len(r) for r in adj])
    return ro, np.concatenate(adj).astype(np.int32), nL


SHAPES = [(700, 140, 100, 560), (700, 140, 100, 608), (700, 140, 100, 680),
          (900, 140, 128, 560), (900, 140, 128, 608), (900, 140, 128, 800),
          (1000, 140, 128, 997), (5000, 130, 128, 4990), (8000, 140, 48, 7000),
          (8000, 140, 48, 7800), (2500, 150, 64, 2450)]


@pytest.mark.parametrize("nV,nL,kept,n", SHAPES)
def test_wide_children_match_oracle(nV, nL, kept, n):
    import gmbe_b200 as gm
    g = nested(nV, nL, kept, n, seed=n)
    for order in (0, 1):
        want = oracle.gmbe(*g, uvtrans=0, order=order)
        with gm.Graph.from_csr(*g, uvtrans=0, order=order) as G:
            runs = [dict(), dict(share_counts=-1), dict(share_min_work=1), dict(direct_max_c=1)]
            if nV <= 1000:  # (a tree thousands of times as large at 8,000)
                runs.append(dict(prune=0))
            for params in runs:
                r = G.enumerate(wait_limit_ns=30 * 10**9, time_limit_ns=60 * 10**9, **params)
                assert (r.count, r.set_hash) == (want.count, want.set_hash), (order, params)
            if nV <= 1000:
                r, found = G.enumerate_emit(1 << 22, time_limit_ns=60 * 10**9)
                assert len(set(found)) == len(found) == want.count
                assert r.set_hash == want.set_hash


def test_wide_children_in_a_batch():
    import gmbe_b200 as gm
    graphs = [nested(700, 140, 100, n, seed=n) for n in (560, 608, 680)]
    want = [oracle.gmbe(*g) for g in graphs]
    batch = gm.Batch([gm.BipartiteCSR(*g) for g in graphs])
    for _ in range(2):
        per, _ = batch.run()
        assert [(r.count, r.set_hash) for r in per] == [(w.count, w.set_hash) for w in want]
    batch.free()


# Rejected pushes with pruning off, as the engine counted them when the bitmap
# tier walked single candidates (which tier runs a child decides the order of
# its pushes, and with it this count).
@pytest.mark.parametrize("nV,nL,kept,n,nonmax", [
    (700, 140, 100, 560, 68424), (700, 140, 100, 680, 88800),
    (900, 140, 128, 560, 82175), (900, 140, 128, 800, 112055), (1000, 140, 128, 997, 136975)])
def test_wide_children_stay_in_the_bitmap_tier(nV, nL, kept, n, nonmax):
    import gmbe_b200 as gm
    g = nested(nV, nL, kept, n, seed=n)
    with gm.Graph.from_csr(*g, uvtrans=0, order=0) as G:
        r = G.enumerate(prune=0, wait_limit_ns=30 * 10**9)
        assert r.non_maximal == nonmax
        # pruning on: the first level's pushes only
        r = G.enumerate(split_mode=1, bound_height=1 << 20, bound_size=1 << 30)
        assert r.max_task_pushes1 < nV
        assert r.non_maximal == G.enumerate(share_min_work=1).non_maximal
