"""Bitmap tier over classes of equal candidates: mask words at |L| 32/33, 64/65
and 128/129, lists of 31..33, 128..129 and over 1,024 classes (one lane each, a
child found through its table, a merge in several parts), every row twice so
that classes hold several candidates."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def one_root(nL, rows, seed):
    """`rows` short rows below one row that holds every U vertex; each is there
    twice, so the full row's root has |L| = nL and at least `rows` classes."""
    rng = np.random.default_rng(seed)
    adj = [np.arange(nL, dtype=np.int32)]
    for i in range(rows):
        k = int(rng.integers(2, 4 if rows > 200 else 6))
        r = np.sort(rng.choice(nL, size=k, replace=False)).astype(np.int32)
        adj += [r, r]
    ro = np.zeros(len(adj) + 1, np.int32)
    ro[1:] = np.cumsum([len(r) for r in adj])
    return ro, np.concatenate(adj), nL


@pytest.mark.parametrize("nL,rows", [(31, 31), (32, 32), (33, 33), (64, 128), (65, 129),
                                     (128, 1100), (129, 300)])
def test_class_lists_match_oracle(nL, rows):
    import gmbe_b200 as gm
    g = one_root(nL, rows, seed=nL + rows)
    for order in (0, 1):
        want = oracle.gmbe(*g, uvtrans=0, order=order)
        with gm.Graph.from_csr(*g, uvtrans=0, order=order) as G:
            for params in (dict(), dict(prune=0), dict(share_min_work=1, slot_records=8),
                           dict(bound_height=1 << 20, bound_size=1 << 20)):
                r = G.enumerate(wait_limit_ns=30 * 10**9, **params)
                assert (r.count, r.set_hash) == (want.count, want.set_hash), (order, params)
