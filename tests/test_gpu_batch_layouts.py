"""A batch's captured launch starts from all-zero count maps wherever its own
scratch layout puts them: launches with other layouts in between (another
batch, a single graph) must not change its results."""
import pytest

import oracle
from util import planted, random_bipartite

pytestmark = pytest.mark.gpu


def test_batches_and_single_graphs_in_turn():
    import gmbe_b200 as gm

    sets = [[planted(200 + 60 * k, 150 + 40 * k, blocks=4, seed=3 * k + j, bsize=12)
             for j in range(3)] for k in range(3)]
    want = [[(w.count, w.set_hash) for w in (oracle.gmbe(*g) for g in gs)] for gs in sets]
    one = random_bipartite(60, 90, 0.2, 5)
    w1 = oracle.gmbe(*one)
    batches = [gm.Batch([gm.BipartiteCSR(*g) for g in gs]) for gs in sets]
    with gm.Graph.from_csr(*one, uvtrans=1) as G:
        for rep in range(3):  # the first run of each captures, later ones replay
            for b, w in zip(batches, want):
                per, _ = b.run()
                assert [(r.count, r.set_hash) for r in per] == w, rep
                if rep == 1:
                    r = G.enumerate()
                    assert (r.count, r.set_hash) == (w1.count, w1.set_hash)
    for b in batches:
        b.free()
