"""GPU: BC of the label-free index over its core graph (core.cuh) against the oracle's
Dijkstra-Brandes, and against the sweep of the whole graph (dep_form=4 asks for it).

The graphs meet the edges of the split into core and bottoms: bottoms at the limit of their rows
(paths), none at all (cliques, hubs), core vertices with more than eight arcs, sources in the core and
in bottoms, source lists that do not fill a group of 64, little scratch; and what has no core plan or
voids one: lengths and distances past the keys, counts past 2^31.
Both sides add the same FP64 terms in other orders: BC_RTOL."""
import numpy as np
import pytest

import gpu_betweennesscentrality_b200 as Q
import pyoracle as O
from conftest import rel_err
from test_gpu_tree import GRAPHS
from util import BC_RTOL, grid_lines, lines_of, unit_grid_lines

pytestmark = pytest.mark.gpu


def _hubs():
    rng = np.random.default_rng(4)
    e = {(int(a), int(b)) if a < b else (int(b), int(a)) for a, b in rng.integers(0, 400, (900, 2)) if a != b}
    e |= {(i, i + 1) for i in range(399)} | {(7, i) for i in range(9, 400, 3)} | {(300, i) for i in range(0, 280, 9)}
    return [(a, b, int(rng.integers(1, 4))) for a, b in sorted(e)]


MORE = {
    "hubs": (400, _hubs),
    "path_3000": (3000, lambda: [(i, i + 1, 1 + i % 5) for i in range(2999)]),
    # the longest length that a bottom takes is 1,973,790; distances of a core vertex end at 33,554,432
    "long_arcs": (60, lambda: [(i, i + 1, 1973790 + i % 2) for i in range(59)] + [(0, 30, 9000000)]),
    "far_apart": (300, lambda: [(i, i + 1, 1900000) for i in range(299)]),
    "far_core": (120, lambda: [(i, j, 1900000 + i) for i in range(0, 20) for j in range(i)] +
                 [(i, i + 1, 1800000) for i in range(19, 119)]),
}
ALL = {**GRAPHS, **MORE}


def _index(n, u, v, w, **tuning):
    g = Q.Graph(device=0)
    g.ReadLines(n, u, v, w)
    idx = g.build_index(Q.QBC_INDEX_CSR)
    if tuning:
        idx.set_tuning(**tuning)
    return idx


@pytest.mark.parametrize("name", sorted(ALL))
def test_small_graphs(name):
    n, edges = ALL[name]
    nn, u, v, w = lines_of(edges(), n)
    arcs = O.Arcs(nn, u, v, w)
    idx = _index(nn, u, v, w)
    assert rel_err(idx.bc_all(), arcs.bc()) <= BC_RTOL
    srcs = np.random.default_rng(3).choice(n, 2 * n + 1, replace=True).astype(np.int32)  # repeats, any count
    want = _index(nn, u, v, w, dep_form=4).bc_sources(srcs)
    assert rel_err(idx.bc_sources(srcs), want) <= BC_RTOL
    for s in (0, n // 2, n - 1):
        one = np.array([s], np.int32)
        assert rel_err(idx.bc_sources(one), arcs.bc(one)) <= BC_RTOL


@pytest.mark.parametrize("threads", [0, 256, 512, 1024, 2048])
@pytest.mark.parametrize("shortcuts,ns", [(0.0, 63), (0.02, 64), (0.02, 65), (0.05, 700)])
def test_grids(shortcuts, ns, threads):
    n, u, v, w = grid_lines(3000, seed=8, shortcut_frac=shortcuts)
    srcs = np.random.default_rng(ns).choice(n, ns, replace=False).astype(np.int32)
    want = O.Arcs(n, u, v, w).bc(srcs)
    idx = _index(n, u, v, w, sweep_threads=threads)
    assert rel_err(idx.bc_sources(srcs), want) <= BC_RTOL
    for delta in (1, 1 << 20):
        idx.set_tuning(sweep_threads=threads, sweep_delta=delta)
        assert rel_err(idx.bc_sources(srcs), want) <= BC_RTOL
    idx.set_tuning(sweep_threads=threads, chunk=32)  # the least scratch
    assert rel_err(idx.bc_sources(srcs), want) <= BC_RTOL


@pytest.mark.parametrize("diamonds", [14, 30, 31, 33, 40])
def test_counts_up_to_and_past_2_31(diamonds):
    """2^k shortest paths along a chain of k diamonds, with dense ends so that both lie in the core"""
    ends = 12
    e, at = [(i, j, 3) for i in range(ends) for j in range(i)], 0
    nxt = ends
    for _ in range(diamonds):
        a, b, c = nxt, nxt + 1, nxt + 2
        e += [(at, a, 1), (at, b, 1), (a, c, 1), (b, c, 1)]
        at, nxt = c, nxt + 3
    e += [(at, nxt + i, 2) for i in range(ends)] + [(nxt + i, nxt + j, 3) for i in range(ends) for j in range(i)]
    n, u, v, w = lines_of(e, nxt + ends)
    idx, general = _index(n, u, v, w), _index(n, u, v, w, dep_form=4)
    want = general.bc_all()

    def same(got, want):  # (a 32-bit count that wraps to 0 makes both sides' shares 0 / 0)
        return np.array_equal(np.isnan(got), np.isnan(want)) and rel_err(np.nan_to_num(got), np.nan_to_num(want)) <= BC_RTOL

    for _ in range(2):  # and again after a plan was given up
        assert same(idx.bc_all(), want)
    q = np.arange(0, n, 3, dtype=np.int32)
    assert same(_index(n, u, v, w).bc_query(q), want[q])


def test_wrap_on_every_entry_point():
    """the 24 x 24 unit grid: without a host check in between, the whole graph's sweep follows"""
    import torch

    n, u, v, w = unit_grid_lines()
    want = _index(n, u, v, w, dep_form=4).bc_all()
    d_src = torch.arange(n, dtype=torch.int32, device="cuda:0")
    d_bc = torch.zeros(n, dtype=torch.float64, device="cuda:0")
    torch.cuda.synchronize()
    idx = _index(n, u, v, w)
    for k in (1, 2):
        idx.bc_sources_device(d_src.data_ptr(), n, d_bc.data_ptr())
        torch.cuda.synchronize()
        assert rel_err(d_bc.cpu().numpy(), k * want) <= BC_RTOL
    q = np.arange(0, n, 5, dtype=np.int32)
    with _index(n, u, v, w).serve(chunk=192) as srv:
        for _ in range(2):
            assert rel_err(srv.wait(srv.submit(q))[0], want[q]) <= BC_RTOL
    assert rel_err(_index(n, u, v, w).bc_sources(np.arange(n, dtype=np.int32)), want) <= BC_RTOL


def test_loaded_index(tmp_path):
    """the plan comes from the arcs, so an index read from a file has it too"""
    n, u, v, w = grid_lines(2000, seed=9, shortcut_frac=0.02)
    idx = _index(n, u, v, w)
    path = str(tmp_path / "i.qbc")
    idx.save(path)
    assert rel_err(Q.Index.load(path).bc_all(), idx.bc_all()) <= BC_RTOL
