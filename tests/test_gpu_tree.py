"""GPU: BC over the elimination tree (tree.cu) against the oracle's Dijkstra-Brandes.

The tree path answers large calls; QBC_TREE_MIN_PAIRS=0 sends the small graphs here through it, so
that the edges of its pieces are met: whole trees inside one bottom subtree, trunks without bottoms,
long paths, vertices whose shortest paths come from many separator entries (unit weights), source
lists that do not fill a group of 64, repeats, and counts past 2^31.
"""
import os

import numpy as np
import pytest

import gpu_betweennesscentrality_b200 as Q
import pyoracle as O
from conftest import rel_err
from util import BC_RTOL, grid_lines, lines_of, unit_grid_lines

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def always_tree(monkeypatch):
    monkeypatch.setenv("QBC_TREE_MIN_PAIRS", "0")


def _grid_edges(rows, cols, weight):
    e = [(r * cols + c, r * cols + c + 1) for r in range(rows) for c in range(cols - 1)]
    e += [(r * cols + c, (r + 1) * cols + c) for r in range(rows - 1) for c in range(cols)]
    return [(a, b, weight(a, b)) for a, b in e]


def _clique(n):
    rng = np.random.default_rng(5)
    return [(i, j, int(rng.integers(1, 10))) for i in range(n) for j in range(i)]


GRAPHS = {
    "two": (2, lambda: [(0, 1, 5)]),
    "one_bottom": (20, lambda: [(i, i + 1, 1 + i % 3) for i in range(19)]),
    "path_31": (31, lambda: [(i, i + 1, 2) for i in range(30)]),
    "path_34": (34, lambda: [(i, i + 1, 1 + i % 2) for i in range(33)]),
    "path_700": (700, lambda: [(i, i + 1, 1 + i % 3) for i in range(699)]),
    "star": (300, lambda: [(0, i, 1 + i % 2) for i in range(1, 300)]),
    "ring": (129, lambda: [(i, (i + 1) % 129, 3) for i in range(129)]),
    "clique": (70, lambda: _clique(70)),
    "unit_grid": (14 * 13, lambda: _grid_edges(14, 13, lambda a, b: 1)),
    "two_weights": (40 * 30, lambda: _grid_edges(40, 30, lambda a, b: 1 + (a * 7 + b) % 2)),
}


def _graph(n, u, v, w):
    g = Q.Graph(device=0)
    g.ReadLines(n, u, v, w)
    return g


@pytest.mark.parametrize("on_device", [False, True])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_small_graphs(name, on_device):
    n, edges = GRAPHS[name]
    nn, u, v, w = lines_of(edges(), n)
    arcs = O.Arcs(nn, u, v, w)
    g = _graph(nn, u, v, w)
    idx = g.build_index(on_device=on_device)
    assert rel_err(idx.bc_all(), arcs.bc()) <= BC_RTOL
    srcs = np.random.default_rng(3).choice(n, 2 * n + 1, replace=True).astype(np.int32)  # repeats, any count
    want = idx.n * [0.0]
    for s, c in zip(*np.unique(srcs, return_counts=True)):
        want = want + c * arcs.bc(np.array([s], np.int32))
    assert rel_err(idx.bc_sources(srcs), want) <= BC_RTOL
    one = np.array([n // 2], np.int32)
    assert rel_err(idx.bc_sources(one), arcs.bc(one)) <= BC_RTOL


@pytest.mark.parametrize("kind", [Q.QBC_INDEX_MHL, Q.QBC_INDEX_H2H])
@pytest.mark.parametrize("shortcuts,ns", [(0.0, 63), (0.0, 64), (0.0, 65), (0.0, 700), (0.02, 333)])
def test_grids(kind, shortcuts, ns):
    n, u, v, w = grid_lines(3000, seed=8, shortcut_frac=shortcuts)
    g = _graph(n, u, v, w)
    idx = g.build_index(kind, g.min_degree_order() if kind == Q.QBC_INDEX_H2H else None, on_device=True)
    srcs = np.random.default_rng(ns).choice(n, ns, replace=False).astype(np.int32)
    want = O.Arcs(n, u, v, w).bc(srcs)
    assert rel_err(idx.bc_sources(srcs), want) <= BC_RTOL
    try:
        idx.set_tuning(chunk=32)  # the least scratch: few groups at a time, or the label kernels
        assert rel_err(idx.bc_sources(srcs), want) <= BC_RTOL
    finally:
        idx.set_tuning()


def test_counts_that_wrap_are_answered_by_the_label_path():
    """an H2H index has no count labels, so the sweep itself meets counts past 2^31 (24 x 24 unit
    grid): every entry point returns what the label kernels return"""
    import torch

    n, u, v, w = unit_grid_lines()
    g = _graph(n, u, v, w)
    order = g.min_degree_order()
    label = g.build_index(Q.QBC_INDEX_H2H, order)
    label.set_tuning(queue_depth=64)  # a label-path field: that path answers
    want = label.bc_all()
    q = np.arange(0, n, 5, dtype=np.int32)

    def fresh():
        return g.build_index(Q.QBC_INDEX_H2H, order, on_device=True)

    idx = fresh()
    for _ in range(2):
        assert rel_err(idx.bc_all(), want) <= BC_RTOL
    assert rel_err(fresh().bc_sources(np.arange(n, dtype=np.int32)), want) <= BC_RTOL
    assert rel_err(fresh().bc_query(q), want[q]) <= BC_RTOL
    idx = fresh()
    d_src = torch.arange(n, dtype=torch.int32, device="cuda:0")
    d_bc = torch.zeros(n, dtype=torch.float64, device="cuda:0")
    torch.cuda.synchronize()
    for k in (1, 2):
        idx.bc_sources_device(d_src.data_ptr(), n, d_bc.data_ptr())
        torch.cuda.synchronize()
        assert rel_err(d_bc.cpu().numpy(), k * want) <= BC_RTOL
    idx = fresh()
    with idx.serve(chunk=192) as srv:
        for _ in range(2):
            assert rel_err(srv.wait(srv.submit(q))[0], want[q]) <= BC_RTOL


def test_saved_index_uses_the_label_path(tmp_path):
    """an index file holds no separators: a loaded index answers as before"""
    n, u, v, w = grid_lines(2000, seed=9)
    idx = _graph(n, u, v, w).build_index()
    path = str(tmp_path / "i.qbc")
    idx.save(path)
    assert rel_err(Q.Index.load(path).bc_all(), idx.bc_all()) <= BC_RTOL
