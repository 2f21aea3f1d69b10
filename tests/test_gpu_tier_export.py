"""Two scratch tiers: a counts-tier child that a big warp shares out is laid out
anew from the graph's whole rows, by a warp sized for the small tier's two-hop
bound.  Dead entries that the big warp has dropped from its own rows count."""
import numpy as np
import pytest

import oracle

pytestmark = [pytest.mark.gpu, pytest.mark.last]

SINGLES, BOUND = 6000, 3000


def hub_then_wide():
    """Root 0 holds 300 U vertices.  Thousands of rows hold U vertex 0 alone:
    the first push retires them and their entries go.  The next one keeps 200
    rows (the counts tier again), of well below BOUND entries then and of more
    than twice as many in the graph.  A last row has a degree above 200 and a
    two-hop multiset below BOUND, so that every warp takes 200 rows in."""
    rng = np.random.default_rng(7)
    adj = [np.arange(300)]
    adj += [np.array([0])] * SINGLES
    adj += [np.arange(200)]
    for _ in range(60):
        adj.append(np.sort(rng.choice(300, size=int(rng.integers(10, 40)), replace=False)))
    adj.append(np.arange(300, 560))
    ro = np.zeros(len(adj) + 1, np.int32)
    ro[1:] = np.cumsum([len(r) for r in adj])
    return ro, np.concatenate(adj).astype(np.int32), 560


@pytest.mark.parametrize("big_warps", [1, 8])
def test_child_of_compacted_rows_shared_out(big_warps):
    import gmbe_b200 as gm
    ro, co, nU = hub_then_wide()
    rows = [co[a:b] for a, b in zip(ro[:-1], ro[1:])]
    deg = np.bincount(co, minlength=nU)
    child = rows[SINGLES + 1]
    assert deg[child].sum() > BOUND > deg[child].sum() - SINGLES  # whole rows / without the dead
    assert deg[rows[-1]].sum() <= BOUND and len(rows[-1]) >= len(child)
    want = oracle.gmbe(ro, co, nU, uvtrans=0, order=0)
    with gm.Graph.from_csr(ro, co, nU, uvtrans=0, order=0) as G:
        for extra in (dict(), dict(share_min_work=1), dict(share_counts=-1)):
            r = G.enumerate(big_two_hop=BOUND, big_warps=big_warps, wait_limit_ns=30 * 10**9,
                            **extra)
            assert (r.count, r.set_hash) == (want.count, want.set_hash), extra
