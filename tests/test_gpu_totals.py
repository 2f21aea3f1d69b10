"""Sub-problems of many more pushes than a walk makes between two looks at the
stop flag (4,096), when its counts go to the warp's 64-bit totals: whole roots
on one warp each against the same roots shared out, leaves only (crown graph)
and levels above leaves."""
import numpy as np
import pytest

import oracle
from util import random_bipartite

pytestmark = pytest.mark.gpu


def crown(n):
    """Every vertex but its own on the other side: 2^n - 2 maximal bicliques."""
    adj = [np.delete(np.arange(n), i) for i in range(n)]
    ro = np.zeros(n + 1, np.int32)
    ro[1:] = np.cumsum([len(r) for r in adj])
    return ro, np.concatenate(adj).astype(np.int32), n


@pytest.mark.parametrize("make", [lambda: crown(18), lambda: random_bipartite(60, 40, 0.6, 1)],
                         ids=["crown", "levels"])
def test_totals_of_long_walks(make):
    import gmbe_b200 as gm
    g = make()
    want = oracle.gmbe(*g, uvtrans=0)
    alone = dict(split_mode=1, bound_height=1 << 20, bound_size=1 << 30)
    with gm.Graph.from_csr(*g, uvtrans=0) as G:
        nonmax = set()
        for params in (alone, dict(), dict(share_min_work=1), dict(alone, bitmap_max_l=16)):
            r = G.enumerate(wait_limit_ns=30 * 10**9, **params)
            assert (r.count, r.set_hash) == (want.count, want.set_hash), params
            if "bitmap_max_l" not in params:  # (the counts tier pushes in another order)
                nonmax.add(r.non_maximal)
            if params is alone:  # the longest walk takes many looks
                assert r.max_task_pushes2 > 8 * 4096
        assert len(nonmax) == 1
