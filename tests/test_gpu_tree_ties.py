"""GPU: the way back of the U rows (k_up_back, tree.cu) where its lists of entries do not suffice: more
than 160 entries on shortest paths in 32 consecutive ancestors of a source, and more than 160 of one
ancestor.  Complete multipartite graphs of unit weight: nearly all of a source's ancestors are at
distance 1, the rest at 2 over every ancestor between."""
import numpy as np
import pytest

import gpu_betweennesscentrality_b200 as Q
import pyoracle as O
from conftest import rel_err
from util import BC_RTOL, lines_of

pytestmark = pytest.mark.gpu


def _multipartite(n, parts, tail):
    """vertex i is of part i % parts; a path of `tail` vertices hangs on vertex 0"""
    e = [(i, j, 1) for i in range(n) for j in range(i) if (i - j) % parts]
    e += [(0 if k == 0 else n + k - 1, n + k, 1) for k in range(tail)]
    return lines_of(e, n + tail)


@pytest.mark.parametrize("n,parts,tail", [(220, 110, 0), (180, 15, 0), (240, 16, 3)])
@pytest.mark.parametrize("kind", [Q.QBC_INDEX_MHL, Q.QBC_INDEX_H2H])
def test_many_tied_ancestors(kind, n, parts, tail, monkeypatch):
    monkeypatch.setenv("QBC_TREE_MIN_PAIRS", "0")
    n, u, v, w = _multipartite(n, parts, tail)
    g = Q.Graph(device=0)
    g.ReadLines(n, u, v, w)
    idx = g.build_index(kind, g.min_degree_order() if kind == Q.QBC_INDEX_H2H else None, on_device=True)
    want = O.Arcs(n, u, v, w).bc()
    assert want.max() > 0
    assert rel_err(idx.bc_all(), want) <= BC_RTOL  # eight warps per source
    many = np.repeat(np.arange(n, dtype=np.int32), 8)  # enough sources for four
    assert many.size >= 148 * 8
    assert rel_err(idx.bc_sources(many), 8 * want) <= BC_RTOL
