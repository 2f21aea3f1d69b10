"""Set-up of roots on their way to the bitmap tier: at and above the number of
entries from which no copy of them is kept (4,096), with the counts tier taking
such a root over, and class lists of above 1,024 candidates with few and with
many different masks."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def below_one_row(rows, nL):
    """One row of all nL U vertices, then `rows`."""
    adj = [np.arange(nL)] + [np.asarray(r) for r in rows]
    ro = np.zeros(len(adj) + 1, np.int32)
    ro[1:] = np.cumsum([len(r) for r in adj])
    return ro, np.concatenate(adj).astype(np.int32), nL


def by_entries(entries, nL=8):
    """The full row's root has exactly that many entries: rows of three U
    vertices, then single ones."""
    rng = np.random.default_rng(entries)
    left = entries - nL
    rows = [np.sort(rng.choice(nL, 3, replace=False)) for _ in range(left // 3 - 20)]
    rows += [rng.choice(nL, 1) for _ in range(left - 3 * len(rows))]
    return below_one_row([rows[i] for i in rng.permutation(len(rows))], nL)


def by_masks(n, masks, nL=60, seed=5):
    """n rows, `masks` different ones of 2 to 4 U vertices."""
    rng = np.random.default_rng(seed)
    kinds = [np.sort(rng.choice(nL, int(rng.integers(2, 5)), replace=False)) for _ in range(masks)]
    return below_one_row([kinds[i] for i in rng.integers(0, masks, n)], nL)


CASES = {"entries 4096": lambda: by_entries(4096), "entries 4097": lambda: by_entries(4097),
         "masks 30 of 1025": lambda: by_masks(1025, 30),
         "masks 1500 of 3000": lambda: by_masks(3000, 1500),
         "masks 200 of 9000": lambda: by_masks(9000, 200)}


@pytest.mark.parametrize("name", CASES)
def test_root_setup_matches_oracle(name):
    import gmbe_b200 as gm
    g = CASES[name]()
    if name.startswith("entries"):
        deg = np.bincount(g[1], minlength=g[2])
        assert deg.sum() == int(name.split()[1])
    for order in (0, 1):
        want = oracle.gmbe(*g, uvtrans=0, order=order)
        with gm.Graph.from_csr(*g, uvtrans=0, order=order) as G:
            for params in (dict(), dict(direct_max_c=1), dict(bitmap_max_l=4),
                           dict(touch_scan=1), dict(share_min_work=1),
                           dict(range_split_work=100, range_chunk=16)):
                r = G.enumerate(wait_limit_ns=30 * 10**9, time_limit_ns=60 * 10**9, **params)
                assert (r.count, r.set_hash) == (want.count, want.set_hash), (order, params)
