"""Workloads of the betweenness-centrality framework, through its public entry points.

A case is one call that a user of the framework makes, on a seeded road-like grid
(``synth.grid_graph``): every vertex as a source or a sample of them, over a label index
(``mhl``, ``h2h``) or the label-free index (``csr``) of a graph with long shortcuts, returning BC of
all vertices, BC of query sets, or the per-source rows.  The graph, the source sample and the members of
the query sets follow from the seed.

Fields: ``call`` (what is called), ``index``, ``n`` (target vertex count of the grid), ``shortcuts``
(fraction of n added as random long edges), ``ns`` (sources, 0 = every vertex), ``sets`` and
``set_hi`` (query sets and the largest size of one; sizes are log-uniform from 16).
"""
from __future__ import annotations

import numpy as np
import torch

import gpu_betweennesscentrality_b200 as q
from gpu_betweennesscentrality_b200 import synth

KINDS = {"mhl": q.QBC_INDEX_MHL, "h2h": q.QBC_INDEX_H2H, "csr": q.QBC_INDEX_CSR}


def _case(call, index, n, shortcuts=0.0, ns=0, sets=0, set_hi=0, name=None):
    c = dict(call=call, index=index, n=n, shortcuts=shortcuts, ns=ns, sets=sets, set_hi=set_hi)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # QBC of a small road network from its order file, every vertex a source: milliseconds,
        # where launches and latency count
        _case("bc_all", "h2h", 2000, name="qbc_all_2k"),
        # the headline workload: MHL-QBC of the 50k grid, every vertex a source
        _case("bc_all", "mhl", 50000, name="mhl_all_50k"),
        # an interactive update: the contributions of a handful of sources that a GPU-side program
        # holds on the device, added into its own BC vector on its own stream
        _case("device", "mhl", 50000, ns=16, name="mhl_device_16_of_50k"),
        # a sampled BC estimate (host list of sources, BC of all vertices back) at an ordinary size
        _case("sources", "mhl", 21013, ns=1000, name="mhl_sources_1k_of_21k"),
        # RQ: one query set against every source of a district-sized network
        _case("query", "mhl", 6007, sets=1, set_hi=256, name="rq_all_6k"),
        # batched RQ: 64 query sets answered by one sweep over a source sample
        _case("query", "mhl", 50000, ns=4096, sets=64, set_hi=16384, name="rq_batch_4k_of_50k"),
        # sampled BC of a large network without shortcuts
        _case("sources", "mhl", 500000, ns=1024, name="mhl_sources_1k_of_500k"),
        # the label-free index: a small graph with 2 % shortcuts, every vertex a source
        _case("bc_all", "csr", 5003, shortcuts=0.02, name="csr_all_5k"),
        # RQ of 4,096 query vertices on 200k vertices with 2 % shortcuts, sampled sources
        _case("query", "csr", 200000, shortcuts=0.02, ns=4096, sets=1, set_hi=4096, name="csr_rq_4k_of_200k"),
        # the largest: sampled BC of 1M vertices with 2 % shortcuts
        _case("sources", "csr", 1000000, shortcuts=0.02, ns=2048, name="csr_sources_2k_of_1m"),
        # distance / path count / hop rows of a few sources, copied back to the host
        _case("rows", "mhl", 50000, ns=48, name="rows_48_of_50k"),
        # the served loop: requests that arrive together share one turn over the sources
        _case("served", "mhl", 10007, sets=16, set_hi=2048, name="served_16_on_10k"),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    """One more case of the same ranges: n from 400 to 500k, 1 to 4,096 sources or all of them."""
    call = rng.choice(["bc_all", "device", "sources", "sources", "query", "query", "rows", "served"])
    index = rng.choice(["mhl", "mhl", "mhl", "h2h", "csr", "csr"]) if call != "served" else "mhl"
    shortcuts = round(rng.uniform(0.0, 0.05), 3) if index == "csr" else 0.0
    if call in ("bc_all", "served"):
        return _case(call, index, _log_int(rng, 400, 40000 if index == "mhl" else 12000), shortcuts,
                     sets=rng.randint(1, 24) if call == "served" else 0,
                     set_hi=_log_int(rng, 32, 4096) if call == "served" else 0)
    # order files are those of small networks; label rows in vertex order are a few sources' worth
    hi = 20000 if index == "h2h" else 60000 if call == "rows" else 500000 if index == "mhl" else 300000
    n = _log_int(rng, 1000, hi)
    ns = _log_int(rng, 1, min(64 if call == "rows" else 4096, max(1, 500000000 // n)))
    if call == "query":
        return _case(call, index, n, shortcuts, ns=min(n // 2, ns), sets=rng.randint(1, 64), set_hi=_log_int(rng, 32, 16384))
    return _case(call, index, n, shortcuts, ns=min(n // 2, ns))


def _edges(case, seed):
    return synth.grid_graph(case["n"], seed=seed % (1 << 31), shortcut_frac=case["shortcuts"])


def _sample(case, seed, n):
    """The case's source sample as 0-based ids in random order, or None for every vertex."""
    if not case["ns"]:
        return None
    rng = np.random.default_rng([seed, 7])
    return rng.choice(n, size=min(case["ns"], n), replace=False).astype(np.int32)


def _sets(case, seed, n):
    rng = np.random.default_rng([seed, 11])
    if case["sets"] == 1:
        return [np.sort(rng.choice(n, size=min(case["set_hi"], n), replace=False)).astype(np.int32)]
    sizes = np.minimum(synth.log_uniform_sizes(case["sets"], 16, case["set_hi"]), n)
    return [np.sort(rng.choice(n, size=int(k), replace=False)).astype(np.int32) for k in sizes]


def _index(case, edges):
    u, v, w = edges.arcs()
    g = q.Graph(device=0)
    g.ReadLines(edges.n, u, v, w)
    order = g.min_degree_order() if case["index"] == "h2h" else None
    return g.build_index(KINDS[case["index"]], order, on_device=True)


def prepare(case, seed):
    edges = _edges(case, seed)
    s = {"call": case["call"], "idx": _index(case, edges), "src": _sample(case, seed, edges.n)}
    if case["call"] in ("query", "served"):
        s["sets"] = _sets(case, seed, edges.n)
    if case["call"] == "device":
        s["stream"] = torch.cuda.Stream()
        s["src"] = torch.from_numpy(s["src"]).cuda()
        s["bc"] = torch.zeros(edges.n, dtype=torch.float64, device="cuda")
    if case["call"] == "served":
        s["server"] = s["idx"].serve()
    return s


def run(state):
    call, idx, src = state["call"], state["idx"], state["src"]
    if call == "bc_all":
        return idx.bc_all()
    if call == "sources":
        return idx.bc_sources(src)
    if call == "query":
        return np.concatenate(idx.bc_query_batch(state["sets"], src))
    if call == "rows":
        return list(idx.rows(src))
    if call == "served":
        srv = state["server"]
        tickets = [srv.submit(s) for s in state["sets"]]
        return np.concatenate([srv.wait(t)[0] for t in tickets])
    with torch.cuda.stream(state["stream"]):
        bc = state["bc"].zero_()
        idx.bc_sources_device(src.data_ptr(), src.numel(), bc.data_ptr(), state["stream"].cuda_stream)
    return bc


def _size(case):
    """Vertices and arcs of the case's grid (its recipe keeps 73 % of the lattice edges)."""
    rows = int(np.floor(np.sqrt(case["n"])))
    cols = int(np.ceil(case["n"] / rows))
    n = rows * cols
    lattice = rows * (cols - 1) + cols * (rows - 1)
    return n, 2 * int(round(0.73 * lattice) + round(case["shortcuts"] * n))


def work(case):
    """Bytes: the arc list read once, the result written once.  Operations: per source, every arc
    relaxed once (an add and a comparison) and visited once more for counts and dependencies (a
    comparison, an add), and four per vertex for its own dependency."""
    n, arcs = _size(case)
    ns = case["ns"] or n
    out = 12 * n * ns if case["call"] == "rows" else 8 * n
    return {"bytes": 12 * arcs + 4 * ns + out, "flops": ns * (4 * arcs + (0 if case["call"] == "rows" else 4 * n))}


def _dependencies(n, u, v, w, sources, dev):
    """BC(v) = 0.5 * sum over the sources of delta_s(v), in 64 bits: all sources' distances by
    repeated relaxation, then path counts and dependencies by repeated substitution on the
    shortest-path DAG (each reaches its fixed point after as many rounds as the DAG has layers)."""
    deg = np.bincount(u, minlength=n)
    order = np.argsort(u, kind="stable")
    slot = np.arange(order.size) - np.repeat(np.cumsum(deg) - deg, deg)
    k = int(deg.max())
    nbr = np.tile(np.arange(n)[:, None], (1, k))
    wt = np.full((n, k), 1 << 40, np.int64)
    nbr[u[order], slot], wt[u[order], slot] = v[order], w[order]
    nbr, wt = torch.from_numpy(nbr).to(dev), torch.from_numpy(wt).to(dev)
    bc = torch.zeros(n, dtype=torch.float64, device=dev)
    step = max(1, 60_000_000 // (n * k))
    for b in range(0, len(sources), step):
        src = torch.as_tensor(np.asarray(sources[b:b + step], np.int64), device=dev)
        rows = torch.arange(src.numel(), device=dev)
        dist = torch.full((src.numel(), n), 1 << 50, dtype=torch.int64, device=dev)
        dist[rows, src] = 0
        while True:
            new = dist
            for j in range(k):
                new = torch.minimum(new, dist[:, nbr[:, j]] + wt[:, j])
            if torch.equal(new, dist):
                break
            dist = new
        into = [dist[:, nbr[:, j]] + wt[:, j] == dist for j in range(k)]
        first = torch.zeros(src.numel(), n, dtype=torch.float64, device=dev)
        first[rows, src] = 1.0
        sigma = first
        while True:
            new = first.clone()
            for j in range(k):
                new += into[j] * sigma[:, nbr[:, j]]
            if torch.equal(new, sigma):
                break
            sigma = new
        del into
        out = [dist + wt[:, j] == dist[:, nbr[:, j]] for j in range(k)]
        delta = torch.zeros_like(sigma)
        while True:
            share = (1.0 + delta) / sigma
            new = torch.zeros_like(delta)
            for j in range(k):
                new += out[j] * share[:, nbr[:, j]]
            new *= sigma
            if torch.equal(new, delta):
                break
            delta = new
        delta[rows, src] = 0.0
        bc += delta.sum(0)
    return (0.5 * bc).cpu().numpy()


def exact(case, seed):
    n, arcs = _size(case)
    ns = case["ns"] or n
    # relaxation rounds grow with the grid's side; beyond this many arc visits it takes too long
    if case["call"] == "rows" or ns * arcs * 3 * int(np.sqrt(n)) > 6e10:
        return None
    edges = _edges(case, seed)
    u, v, w = edges.arcs()
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    src = _sample(case, seed, edges.n)
    bc = _dependencies(edges.n, u - 1, v - 1, w, np.arange(edges.n) if src is None else src, dev)
    if case["call"] in ("query", "served"):
        return np.concatenate([bc[s] for s in _sets(case, seed, edges.n)])
    return torch.from_numpy(bc) if case["call"] == "device" else bc
