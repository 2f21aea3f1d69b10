"""The largest V side whose first-touch bitmaps lie in shared memory (3,584 words
a warp: with the kernel's own variables, all that a block may have), and the
next larger one, which has them in global memory."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nV", [3584 * 32 - 1, 3584 * 32, 3584 * 32 + 1])
def test_shared_bitmap_limit(nV):
    import gmbe_b200 as gm
    rng = np.random.default_rng(nV)
    nU = 2000
    rows = rng.integers(0, nU, size=(nV, 2), dtype=np.int32)
    rows[:, 1] = np.where(rows[:, 0] == rows[:, 1], (rows[:, 1] + 1) % nU, rows[:, 1])
    rows.sort(axis=1)
    g = np.arange(nV + 1, dtype=np.int32) * 2, rows.ravel(), nU
    want = oracle.gmbe(*g, uvtrans=0)
    with gm.Graph.from_csr(*g, uvtrans=0) as G:
        assert G.info().V_size == nV
        for params in (dict(), dict(sm_timing=1, bitmap_max_l=16)):
            r = G.enumerate(wait_limit_ns=30 * 10**9, **params)
            assert (r.count, r.set_hash) == (want.count, want.set_hash), params
