"""The kernel's shared memory limit is one setting of the process: launches of
different bitmap sizes from several threads, and the no-allocation entry point
recorded into a graph, must not take it from one another."""
import ctypes as C
import threading

import numpy as np
import pytest

import oracle
from util import planted

pytestmark = [pytest.mark.gpu, pytest.mark.last]


def _pairs(nV, nU=500):
    rng = np.random.default_rng(nV)
    a = rng.integers(0, nU, nV, dtype=np.int32)
    rows = np.stack([a, (a + 1 + rng.integers(0, nU - 1, nV, dtype=np.int32)) % nU], 1)
    return np.arange(nV + 1, dtype=np.int32) * 2, np.sort(rows, 1).astype(np.int32).ravel(), nU


class NoAlloc:
    """One graph in device buffers of the test's own, enumerated without allocation."""

    def __init__(self, gm, ro, co, nU):
        import torch
        nV = len(ro) - 1
        order = np.lexsort((np.repeat(np.arange(nV), np.diff(ro)), co))
        rco = np.repeat(np.arange(nV, dtype=np.int32), np.diff(ro))[order]
        rro = np.concatenate([[0], np.cumsum(np.bincount(co, minlength=nU))]).astype(np.int32)
        self.t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (ro, co, rro, rco)]
        self.out = torch.zeros(4, dtype=torch.int64, device="cuda")
        self.n = (nV, nU, len(co))
        self.f = C.CDLL(gm.LIB_PATH).mbe_enumerate_device_noalloc
        self.f.restype = C.c_int
        self.f.argtypes = [C.c_void_p, C.c_void_p, C.c_int32, C.c_void_p, C.c_void_p, C.c_int32,
                           C.c_int64, C.c_int64, C.c_void_p, C.c_void_p, C.c_void_p]

    def __call__(self, stream):
        p = [x.data_ptr() for x in self.t]
        nV, nU, nE = self.n
        return self.f(p[0], p[1], nV, p[2], p[3], nU, nE, 0, None, self.out.data_ptr(),
                      stream.cuda_stream)

    def result(self):
        c, h, _, status = (int(x) for x in self.out.cpu())
        return c, h & ((1 << 64) - 1), status


def test_threads_with_different_bitmap_sizes():
    import torch
    import gmbe_b200 as gm
    big, mid, small = _pairs(3584 * 32), _pairs(90000), planted(200, 150, blocks=4, seed=3)
    want = [oracle.gmbe(*g, uvtrans=0) for g in (big, mid, small)]
    errors = []

    def allocating(g, w):
        with gm.Graph.from_csr(*g, uvtrans=0) as G:
            for _ in range(10):
                r = G.enumerate(wait_limit_ns=30 * 10**9)
                assert (r.count, r.set_hash) == (w.count, w.set_hash)

    def without(g, w):
        one = NoAlloc(gm, *g)
        s = torch.cuda.Stream()
        torch.cuda.synchronize()
        for _ in range(10):
            assert one(s) == 0
            s.synchronize()
            assert one.result() == (w.count, w.set_hash, 0)

    def guarded(f, *a):
        try:
            f(*a)
        except BaseException as e:  # noqa: BLE001 (reported by the test's own thread)
            errors.append(e)

    ts = [threading.Thread(target=guarded, args=a)
          for a in ((allocating, big, want[0]), (allocating, mid, want[1]),
                    (without, small, want[2]))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors


def test_no_alloc_recorded_into_a_graph():
    import torch
    import gmbe_b200 as gm
    g = planted(200, 150, blocks=4, seed=5)
    w = oracle.gmbe(*g, uvtrans=0)
    one = NoAlloc(gm, *g)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    assert one(s) == 0
    s.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        assert one(torch.cuda.current_stream()) == 0
    for _ in range(2):
        one.out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert one.result() == (w.count, w.set_hash, 0)
