"""The work a user of this engine has it do, as timed cases.

Every case goes through the package's public entry points (``Graph``,
``Batch``, ``Server``) with the flags the engine is run with in earnest
(``-t 1 -o 1 -f``, pruning on, bounds 20/1500) unless the case says otherwise.
Outputs are whole numbers: [count, set hash, non-maximal count] per graph (the
64-bit words as int64), and for emission every biclique's ids; none of them
has a value that 64-bit floating point would give more exactly.

Graphs are the seeded Chung-Lu families of ``gmbe_b200/workloads.json`` and of
the batched workload, the same families at other sizes, and the small random
graphs of the tests.  The seed makes the graph.
"""
import math

import numpy as np
import torch

import gmbe_b200 as gm

# The named workloads as families over |U|: exponents of the degree
# distributions, |V| and edges per U vertex, degree cap as a share of |U|.
FAMILIES = {
    "small": dict(gu=2.1, gv=2.1, v_per_u=1.5, e_per_u=10.0, cap=0.1),      # 2,000 x 3,000, 20k edges
    "serve": dict(gu=2.1, gv=2.1, v_per_u=4.0, e_per_u=15.0, cap=0.1),      # 20,000 x 80,000, 300k
    "medium": dict(gu=2.0, gv=2.4, v_per_u=4.0, e_per_u=20.0, cap=0.05),    # 100,000 x 400,000, 2M
    "large": dict(gu=2.1, gv=2.2, v_per_u=4.0, e_per_u=30.0, cap=0.025),    # 2M x 8M, 60M
}


def listed():
    return [
        # The smallest call: a graph of a few dozen vertices a side, resident.
        # The launch and the host path around it are the whole cost.
        {"name": "tiny", "kind": "random", "nV": 40, "nU": 48, "p": 0.2},
        # The small configuration, resident: a few thousand light roots.
        {"name": "small", "kind": "graph", "family": "small", "nU": 2000},
        # A small dense graph: few roots, hundreds of thousands of bicliques
        # under them, so the whole launch is sub-problems shared between warps.
        {"name": "dense", "kind": "random", "nV": 28, "nU": 40, "p": 0.8},
        # One request served by plain calls: a graph of the batched workload
        # from host arrays (host build, upload, enumeration, release).
        {"name": "request", "kind": "graph", "family": "small", "nU": 3500, "build": "host"},
        # The 300,000-edge serving graph, resident.
        {"name": "serve_graph", "kind": "graph", "family": "serve", "nU": 20000},
        # The medium configuration, resident: the reference's kind of skewed
        # graph with planted blocks, millions of bicliques, hub roots.
        {"name": "medium", "kind": "graph", "family": "medium", "nU": 100000},
        # The same from host arrays: device build, enumeration, release.
        {"name": "medium_build", "kind": "graph", "family": "medium", "nU": 100000,
         "build": "device"},
        # One GPU's share of the medium configuration split over eight.
        {"name": "medium_shard", "kind": "graph", "family": "medium", "nU": 100000,
         "shards": 8, "shard": 3},
        # Every biclique handed back, not only counted.
        {"name": "emit", "kind": "graph", "family": "small", "nU": 1000, "emit": True},
        # Many small graphs in one launch (the batched workload), resident.
        {"name": "batch", "kind": "batch", "graphs": 256},
        # A burst of requests to a running server: the serving mix (95 %
        # batched-workload graphs, 5 % 300,000-edge graphs).
        {"name": "serving", "kind": "server", "requests": 160},
        # The large configuration, resident: one interleaved root shard (about
        # 100 of 2 million roots, over the whole degree order), as the headline
        # benchmark steps through it.
        {"name": "large_shard", "kind": "large", "nU": 2000000, "shards": 20000, "shard": 12345},
    ]


# Words of the caller's record buffer in the emission cases.
EMIT_WORDS = 1 << 20


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["random", "graph", "graph", "graph", "batch", "server", "medium", "large"])
    if kind == "random":
        # from a handful of vertices to the dense graphs of the tests
        nV = _log(rng, 6, 200)
        p = rng.uniform(0.1, 0.8) if nV < 28 else rng.uniform(0.05, 0.25)
        nU = rng.randint(nV, 2 * nV) if nV < 28 else _log(rng, 28, 300)
        return {"kind": "random", "nV": nV, "nU": min(nU, 40) if p > 0.25 else nU,
                "p": round(p, 3)}
    if kind == "batch":
        return {"kind": "batch", "graphs": _log(rng, 8, 256), "first": rng.randint(0, 100000)}
    if kind == "server":
        return {"kind": "server", "requests": _log(rng, 8, 160), "first": rng.randint(0, 100000)}
    if kind == "large":
        # The lower two fifths of the interleaved shards: the others' heaviest
        # roots can take a shard past two seconds.
        return {"kind": "large", "nU": 2000000, "shards": 20000, "shard": rng.randint(12000, 19999)}
    if kind == "medium":
        c = {"kind": "graph", "family": "medium", "nU": _log(rng, 20000, 100000)}
    else:
        fam = rng.choice(["small", "serve"])
        c = {"kind": "graph", "family": fam,
             "nU": _log(rng, 100, 5000) if fam == "small" else _log(rng, 1000, 20000)}
        c["order"] = rng.choice([1, 1, 1, 2])
        c["uvtrans"] = rng.choice([1, 1, 1, 2]) if fam == "small" else 1
        if fam == "small" and c["nU"] < 1200 and rng.random() < 0.3:
            c["emit"] = True
    if "emit" not in c:
        c["build"] = rng.choice(["", "", "host" if c["family"] != "medium" else "device", "device"])
        if rng.random() < 0.3:
            c["shards"] = rng.randint(2, 16)
            c["shard"] = rng.randint(0, c["shards"] - 1)
    return c


# ---------------------------------------------------------------------------
# Inputs.

def _family_spec(family, nU, seed):
    f = FAMILIES[family]
    cap = max(2, int(f["cap"] * nU))
    blocks = int(round(64 * nU / 100000)) if family == "medium" else 0
    return gm.GenSpec(nU=nU, nV=int(round(f["v_per_u"] * nU)), n_edges=int(round(f["e_per_u"] * nU)),
                      gamma_u=f["gu"], gamma_v=f["gv"], max_deg_u=cap, max_deg_v=cap,
                      seed=seed, n_blocks=blocks, block_u=24 if blocks else 0,
                      block_v=24 if blocks else 0, reserved=0, block_p=0.7 if blocks else 0.0,
                      pair_p_max=0.1)


def _random_graph(nV, nU, p, seed):
    """Independent edges, no vertex of either side without one."""
    rng = np.random.default_rng(seed)
    A = rng.random((nV, nU)) < p
    A[np.arange(nV), rng.integers(nU, size=nV)] |= ~A.any(axis=1)
    A[rng.integers(nV, size=nU), np.arange(nU)] |= ~A.any(axis=0)
    ro = np.concatenate([[0], np.cumsum(A.sum(axis=1))]).astype(np.int32)
    return gm.BipartiteCSR(ro, np.nonzero(A)[1].astype(np.int32), nU)


def _large_graph(nU, seed):
    """The large configuration's family, drawn on the GPU: 60 million edges
    take the package's generator a quarter of a minute.  Same law: Chung-Lu
    ends in proportion to capped power-law weights, duplicates dropped, and
    pairs above probability 0.1 thinned to it."""
    f = FAMILIES["large"]
    nV, nE, cap = int(f["v_per_u"] * nU), int(f["e_per_u"] * nU), f["cap"] * nU
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)

    def weights(n, gamma):
        base = torch.arange(1, n + 1, device=dev, dtype=torch.float64) ** (-1.0 / (gamma - 1.0))
        lo, hi = 0.0, float(nE)
        for _ in range(100):
            c = 0.5 * (lo + hi)
            if float((base * c).clamp(max=cap).sum()) < nE:
                lo = c
            else:
                hi = c
        return (base * hi).clamp(max=cap)

    wu, wv = weights(nU, f["gu"]), weights(nV, f["gv"])
    # In integers: a floating-point scan on the GPU may round differently twice.
    cu, cv = ((w * 2.0 ** 24).to(torch.int64).cumsum(0) for w in (wu, wv))

    def pick(m, c):
        r = torch.rand(m, generator=gen, device=dev, dtype=torch.float64)
        return (r * float(c[-1])).to(torch.int64)

    lmax = -math.log(0.9)
    keys = []
    for _ in range(8):  # in pieces: the device's memory is the enumeration's
        m = nE // 8
        u = torch.searchsorted(cu, pick(m, cu), right=True)
        v = torch.searchsorted(cv, pick(m, cv), right=True)
        u, v = u.clamp_(max=nU - 1), v.clamp_(max=nV - 1)
        lam = wu[u] * wv[v] / nE
        keep = torch.rand(m, generator=gen, device=dev, dtype=torch.float64) * lam < lmax
        keys.append((v * nU + u)[keep])
        del u, v, lam, keep
    keys = torch.unique(torch.cat(keys))
    v, u = keys // nU, keys % nU
    del keys
    used = torch.zeros(nU, device=dev, dtype=torch.bool)
    used[u] = True
    col = (torch.cumsum(used, 0) - 1)[u].to(torch.int32)
    deg = torch.bincount(v, minlength=nV)
    ro = torch.cat([deg.new_zeros(1), deg[deg > 0].cumsum(0)]).to(torch.int32)
    g = gm.BipartiteCSR(ro.cpu().numpy(), col.cpu().numpy(), int(used.sum()))
    del u, v, col, deg, ro, used, wu, wv, cu, cv
    torch.cuda.empty_cache()
    return g


def _opts(case):
    return dict(uvtrans=case.get("uvtrans", 1), order=case.get("order", 1))


def _params(case):
    n = case.get("shards", 0)
    return dict(shard_count=n, shard_index=case["shard"]) if n else {}


def prepare(case, seed):
    state = _state(case, seed)
    state["case"] = case
    return state


def _state(case, seed):
    kind = case["kind"]
    if kind == "batch":
        # Graphs of the batched workload from another place of its seed line,
        # and one heavier graph that is the same in every batch: it is the
        # largest in every capacity, so that a program which keeps several
        # batches runs all of them in one scratch layout.
        first = 1000 + case.get("first", 0) + seed * 4096
        graphs = [gm.batch_graph(first + i) for i in range(case["graphs"] - 1)]
        graphs.append(gm.generate(_family_spec("small", 20000, 1)))
        return {"batch": gm.Batch(graphs)}
    if kind == "server":
        first = 1000 + case.get("first", 0) + seed * 4096
        n = case["requests"]
        medium = [gm.generate(_family_spec("serve", 20000, seed * 16 + k)) for k in range(2)]
        graphs = [medium[i // 20 % 2] if i % 20 == 10 else gm.batch_graph(first + i)
                  for i in range(n)]
        # A server is sized for the graphs it is to take; memory that plain
        # calls of this process have cached goes back first.
        gm.release_device()
        return {"server": gm.Server(max_v=32768, max_degree=4096, max_two_hop=1 << 17),
                "graphs": graphs}
    if kind == "random":
        g = _random_graph(case["nV"], case["nU"], case["p"], seed)
    elif kind == "large":
        g = _large_graph(case["nU"], seed)
    else:
        g = gm.generate(_family_spec(case["family"], case["nU"], seed))
    if case.get("build"):
        return {"csr": g}
    make = gm.Graph.build_on_device if kind == "large" else gm.Graph.from_csr
    return {"graph": make(g.row_off, g.col, g.nU, **_opts(case))}


def _words(results):
    return np.array([(r.count, r.set_hash, r.non_maximal) for r in results],
                    np.uint64).view(np.int64)


def run(state):
    case = state["case"]
    if "batch" in state:
        per, _ = state["batch"].run()
        return _words(per)
    if "server" in state:
        srv = state["server"]
        ids = [srv.submit(g.row_off, g.col, g.nU) for g in state["graphs"]]
        return _words([srv.wait(i) for i in ids])
    if case.get("emit"):
        # The order bicliques arrive in is the schedule's: sorted to compare.
        r, found = state["graph"].enumerate_emit(EMIT_WORDS)
        found.sort()
        flat = np.fromiter((x for us, vs in found for x in (len(us), len(vs), *us, *vs)), np.int32)
        records = np.zeros(EMIT_WORDS, np.int32)
        records[:len(flat)] = flat
        return {"result": _words([r]), "bicliques": records}
    if case.get("build"):
        g = state["csr"]
        make = gm.Graph.from_csr if case["build"] == "host" else gm.Graph.build_on_device
        with make(g.row_off, g.col, g.nU, **_opts(case)) as G:
            return _words([G.enumerate(**_params(case))])
    return _words([state["graph"].enumerate(**_params(case))])


# ---------------------------------------------------------------------------
# What a pass cannot do without.

def work(case):
    """Each input edge read once in either direction (the two CSRs the
    enumeration works on) and the result words written once; integer work, no
    floating-point operations."""
    kind = case["kind"]
    if kind == "batch":
        edges, out = 17000 * case["graphs"], 24 * case["graphs"]
    elif kind == "server":
        edges, out = (17000 + 15000) * case["requests"], 24 * case["requests"]
    elif kind == "random":
        edges, out = case["nV"] * case["nU"] * case["p"], 24
    else:
        fam = "large" if kind == "large" else case["family"]
        edges, out = FAMILIES[fam]["e_per_u"] * case["nU"], 24
    return {"bytes": float(8 * edges + out), "flops": 0.0}
