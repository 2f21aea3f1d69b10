"""Counts-tier pushes that keep one or two rows, walked without a sub-problem:
rows of 1, 31..33, 127..129 and 257 candidates (rounds of 32 and of 4 x 32
entries), candidates of one row, of two and of more, with and without Q
candidates before them."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def hub(nL, lens, seed, extra):
    """One V vertex adjacent to all nL U vertices; U vertex i is met by lens[i]
    others of one or two U vertices; `extra` rows of 3 to 8."""
    rng = np.random.default_rng(seed)
    adj = [np.arange(nL, dtype=np.int32)]
    for i, n in enumerate(lens):
        for k in range(n):
            other = int(rng.integers(nL))
            adj.append(np.unique(np.array([i] if k % 3 == 0 else [i, other], np.int32)))
    for _ in range(extra):
        adj.append(np.sort(rng.choice(nL, size=int(rng.integers(3, 9)), replace=False)))
    order = np.concatenate([[0], 1 + rng.permutation(len(adj) - 1)])
    adj = [np.asarray(adj[i], np.int32) for i in order]
    ro = np.zeros(len(adj) + 1, np.int32)
    ro[1:] = np.cumsum([len(r) for r in adj])
    return ro, np.concatenate(adj), nL


@pytest.mark.parametrize("nL,lens,extra", [
    (130, (1, 31, 32, 33), 40),
    (160, (127, 128, 129, 2), 200),
    (300, (257, 64, 65, 1, 1, 300), 400),
])
def test_narrow_pushes_match_oracle(nL, lens, extra):
    import gmbe_b200 as gm
    g = hub(nL, lens, nL, extra)
    for order in (0, 1):
        want = oracle.gmbe(*g, uvtrans=0, order=order)
        with gm.Graph.from_csr(*g, uvtrans=0, order=order) as G:
            plain = None
            for params in (dict(), dict(bitmap_max_l=1), dict(bitmap_max_l=32), dict(prune=0),
                           dict(share_min_work=1), dict(share_counts=-1)):
                r = G.enumerate(wait_limit_ns=30 * 10**9, **params)
                assert (r.count, r.set_hash) == (want.count, want.set_hash), (order, params)
                if not params:
                    plain = r.non_maximal
                elif params.get("prune", 1) and "bitmap_max_l" not in params:
                    assert r.non_maximal == plain, (order, params)
            r, found = G.enumerate_emit(1 << 20)
            assert len(found) == want.count and r.set_hash == want.set_hash


@pytest.mark.parametrize("nL,singles,extra", [
    (40, 100, 3),      # fewer entries than a compaction starts from
    (40, 170, 12),     # about that many
    (40, 1000, 60),    # several compactions in one task
    (200, 5000, 300),
])
def test_retired_entries_dropped_match_oracle(nL, singles, extra):
    """Most candidates on two hub rows and on nothing else: the first push that
    keeps such a row retires them, and the rows are compacted under the pushes
    that follow (counts tier, also for short L: bitmap_max_l)."""
    import gmbe_b200 as gm
    rng = np.random.default_rng(nL + singles)
    adj = [np.arange(nL, dtype=np.int32)]
    adj += [np.array([i % 7 == 0], np.int32) for i in range(singles)]
    for _ in range(extra):
        rest = 2 + rng.choice(nL - 2, size=int(rng.integers(1, 12)), replace=False)
        hubs = np.nonzero(rng.random(2) < 0.7)[0]
        adj.append(np.sort(np.concatenate([hubs, rest])).astype(np.int32))
    ro = np.zeros(len(adj) + 1, np.int32)
    ro[1:] = np.cumsum([len(r) for r in adj])
    g = (ro, np.concatenate(adj).astype(np.int32), nL)
    for order in (0, 1):
        want = oracle.gmbe(*g, uvtrans=0, order=order)
        with gm.Graph.from_csr(*g, uvtrans=0, order=order) as G:
            for params in (dict(), dict(bitmap_max_l=1), dict(bitmap_max_l=16),
                           dict(bitmap_max_l=16, share_min_work=1), dict(direct_max_c=1),
                           dict(direct_max_c=1, range_split_work=100, range_chunk=8),
                           dict(bitmap_max_l=4, touch_scan=1)):
                r = G.enumerate(wait_limit_ns=30 * 10**9, **params)
                assert (r.count, r.set_hash) == (want.count, want.set_hash), (order, params)
