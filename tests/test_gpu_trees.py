"""The search tree itself: the number of rejected (non-maximal) pushes, as the
engine counted them when the bitmap tier walked single candidates.  Merging
equal candidates, walking leaves in registers, summing up narrow pushes and
dropping retired entries must leave it as it is, however a launch shares work."""
import pytest

from test_gpu_classes import one_root
from test_gpu_narrow import hub
from util import hub_graph, planted, random_bipartite

pytestmark = pytest.mark.gpu

# graph: per order 0, 1 (rejected pushes with pruning, without)
TREES = {
    "classes 31": (lambda: one_root(31, 31, 62), ((108, 512), (80, 442))),
    "classes 33": (lambda: one_root(33, 33, 66), ((113, 531), (83, 421))),
    "classes 64": (lambda: one_root(64, 128, 192), ((561, 4172), (449, 3914))),
    "classes 65": (lambda: one_root(65, 129, 194), ((537, 3185), (403, 2747))),
    "classes 128": (lambda: one_root(128, 1100, 1228), ((4549, None), (3591, None))),
    "classes 129": (lambda: one_root(129, 300, 429), ((1069, 5053), (789, 4377))),
    "narrow 130": (lambda: hub(130, (1, 31, 32, 33), 130, 40), ((260, 1150), (159, 886))),
    "narrow 300": (lambda: hub(300, (257, 64, 65, 1, 1, 300), 300, 400),
                   ((3399, 47960), (2602, 41403))),
    "planted": (lambda: planted(300, 200, blocks=6, seed=3, bsize=14),
                ((4281, 155436), (2909, 66140))),
    "hubs": (lambda: hub_graph(1), ((5555, 24511), (2128, 12286))),
    "dense": (lambda: random_bipartite(60, 40, 0.6, 1), ((966127, 5069848), (759777, 4003977))),
}


@pytest.mark.parametrize("name", TREES)
def test_rejected_pushes(name):
    import gmbe_b200 as gm
    make, want = TREES[name]
    g = make()
    for order in (0, 1):
        pruned, whole = want[order]
        with gm.Graph.from_csr(*g, uvtrans=0, order=order) as G:
            for params in (dict(), dict(share_min_work=1), dict(share_min_work=1, slot_records=8),
                           dict(share_counts=-1),
                           dict(split_mode=1, bound_height=1 << 20, bound_size=1 << 30)):
                r = G.enumerate(wait_limit_ns=30 * 10**9, **params)
                assert r.non_maximal == pruned, (order, params)
            if whole is not None:
                assert G.enumerate(prune=0, wait_limit_ns=30 * 10**9).non_maximal == whole, order
            if name.startswith("classes"):
                r, found = G.enumerate_emit(1 << 20)
                assert r.non_maximal == pruned and len(set(found)) == len(found) == r.count
