"""A launch whose scratch cannot be had gives the workspace's scratch up all the
same: a batch captured before must not be replayed on it."""
import numpy as np
import pytest

import oracle
from util import planted

pytestmark = [pytest.mark.gpu, pytest.mark.last]


def test_batch_after_another_ran_out_of_memory():
    import torch
    import gmbe_b200 as gm
    gm.release_device()
    graphs = [planted(200, 150, blocks=4, seed=s) for s in (1, 2, 3)]
    want = [(w.count, w.set_hash) for w in (oracle.gmbe(*g) for g in graphs)]
    small = gm.Batch([gm.BipartiteCSR(*g) for g in graphs])

    def run_small():
        per, _ = small.run()
        assert [(r.count, r.set_hash) for r in per] == want

    run_small()
    # 400,000 rows of one vertex: count maps of 1.6 MB a warp, gigabytes in all
    nV = 400000
    wide = gm.Batch([gm.BipartiteCSR(np.arange(nV + 1, dtype=np.int32),
                                     np.arange(nV, dtype=np.int32) // 4, nV // 4)], uvtrans=0)
    free, _ = torch.cuda.mem_get_info()
    held = torch.empty(free - (1 << 30), dtype=torch.uint8, device="cuda")
    with pytest.raises(gm.MBEError) as ei:
        wide.run()
    assert ei.value.name == "MBE_ERR_NOMEM"
    del held
    torch.cuda.empty_cache()
    # the failed allocation is reported once: the launches of a device build find
    # no error that is not theirs
    with gm.Graph.build_on_device(*graphs[0]) as G:
        r = G.enumerate()
        assert (r.count, r.set_hash) == want[0]
    run_small()
    # with memory the other one runs, on scratch of its own, and the first again
    per, _ = wide.run()
    assert per[0].count == nV // 4
    run_small()
    small.free()
    wide.free()
