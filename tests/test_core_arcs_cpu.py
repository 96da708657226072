"""CPU: a label-free index file may hold arcs that the graph reader would refuse (one-way, repeated, of
two weights, a loop).  It loads as ever, but its arcs are marked, so that no core plan is made from them:
the elimination takes every arc's reverse for granted.  Read through a small program over the loader."""
import os
import subprocess

import numpy as np
import pytest

import gpu_betweennesscentrality_b200 as Q
from gpu_betweennesscentrality_b200 import build, capi
from test_index_file import _word_hash
from util import grid_lines

PROGRAM = r"""
#include <cstdio>
#include "host.h"
int main(int argc, char **argv) {
  for (int i = 1; i < argc; i++) std::printf("%d\n", (int)qbc::index_load(argv[i]).arcs_paired);
}
"""


@pytest.fixture(scope="module")
def paired(tmp_path_factory):
    """paths -> their indexes' arcs_paired"""
    d = tmp_path_factory.mktemp("arcs")
    (d / "main.cpp").write_text(PROGRAM)
    exe = str(d / "main")
    cxx = build._cxx()
    r = subprocess.run([cxx, "-std=c++17", "-O1", "-I", build.CSRC, "-I", build.INCLUDE, str(d / "main.cpp"),
                        os.path.join(build.CSRC, "index_file.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return lambda *p: [x == "1" for x in subprocess.run([exe, *p], capture_output=True, text=True, check=True).stdout.split()]


@pytest.fixture(scope="module")
def saved(tmp_path_factory):
    """a CSR index file and its arrays' places: (path, n, arc_off, bytes before arc_head, arcs)"""
    n, u, v, w = grid_lines(300, seed=6, shortcut_frac=0.02)
    g = Q.Graph()
    g.ReadLines(n, u, v, w)
    p = str(tmp_path_factory.mktemp("file") / "s.qbcidx")
    g.build_index(Q.QBC_INDEX_CSR, upload=False).save(p)
    off = np.asarray(g.arcs()[0], np.int32)
    return p, n, off, 56 + 20 * n + 8 * (n + 1) + 4 * (n + 1), int(off[-1])


def _edited(saved, path, edit):
    p, n, off, at, arcs = saved
    raw = bytearray(open(p, "rb").read()[:-8])
    a = np.frombuffer(raw, np.int32, 2 * arcs, at).reshape(2, arcs)
    off_in = np.frombuffer(raw, np.int32, n + 1, at - 4 * (n + 1))
    assert np.array_equal(off_in, off)
    edit(off, a[0], a[1])
    open(path, "wb").write(bytes(raw) + _word_hash(bytes(raw)).to_bytes(8, "little"))
    return path


def _vertex(off, degree):
    return int(np.flatnonzero(np.diff(off) >= degree)[0])


def one_way(off, head, w):
    v = _vertex(off, 2)
    b = off[v]
    head[b] = next(x for x in range(len(off) - 1) if x != v and x not in head[b:off[v + 1]])


def repeated(off, head, w):
    b = off[_vertex(off, 2)]
    head[b + 1], w[b + 1] = head[b], w[b]


def two_weights(off, head, w):
    w[off[_vertex(off, 2)]] += 1


def loop(off, head, w):
    v = _vertex(off, 2)
    head[off[v]] = v


def crossed(off, head, w):
    """as many arcs in as out at every vertex, none repeated, but v1 - x1 and v2 - x2 cross on one side"""
    n = len(off) - 1
    v1 = _vertex(off, 1)
    x1 = head[off[v1]]
    near = set(head[off[v1]:off[v1 + 1]]) | {v1}
    for v2 in range(v1 + 1, n):
        x2 = head[off[v2]]
        if x2 not in near and x2 != x1 and x1 != v2 and x1 not in head[off[v2]:off[v2 + 1]]:
            head[off[v1]], head[off[v2]] = x2, x1
            return
    raise AssertionError("no pair of arcs to cross")


@pytest.mark.parametrize("edit", [one_way, repeated, two_weights, loop, crossed])
def test_unpaired_arcs_are_marked(saved, paired, tmp_path, edit):
    bad = _edited(saved, str(tmp_path / "bad.qbcidx"), edit)
    assert paired(saved[0], bad) == [True, False]
    assert Q.Index.load(bad, device=None).n == saved[1]  # accepted as before


@pytest.mark.parametrize("first", [-1, 1])
def test_arcs_that_do_not_start_at_0_are_refused(saved, tmp_path, first):
    p, n, off, at, arcs = saved
    raw = bytearray(open(p, "rb").read()[:-8])
    np.frombuffer(raw, np.int32, n + 1, at - 4 * (n + 1))[0] = first
    bad = str(tmp_path / "bad.qbcidx")
    open(bad, "wb").write(bytes(raw) + _word_hash(bytes(raw)).to_bytes(8, "little"))
    with pytest.raises(Q.QbcError) as e:
        Q.Index.load(bad, device=None)
    assert e.value.code == capi.QBC_EIO


def test_every_recipe_is_paired(paired, tmp_path):
    paths = []
    for k, (n, sc) in enumerate([(1, 0.0), (50, 0.0), (2000, 0.05)]):
        nn, u, v, w = grid_lines(n, seed=k, shortcut_frac=sc) if n > 1 else (1, *(np.empty(0, np.int32),) * 3)
        g = Q.Graph()
        g.ReadLines(nn, u, v, w)
        paths.append(str(tmp_path / f"{k}.qbcidx"))
        g.build_index(Q.QBC_INDEX_CSR, upload=False).save(paths[-1])
    assert paired(*paths) == [True] * len(paths)
