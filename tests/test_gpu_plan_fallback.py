"""GPU: what a call over an elimination-tree or core-graph plan leaves behind.  One index, several
entry points, and a plan that is given up between them (a path count past 2^31, a core distance from
2^25 on): a call that was captured while the plan was in use has to be answered as before, by the label
or sweep kernels.  And a source id out of range in a device list, which only the device can find."""
import numpy as np
import pytest

import gpu_betweennesscentrality_b200 as Q
import pyoracle as O
from conftest import rel_err
from gpu_betweennesscentrality_b200 import capi
from util import BC_RTOL, grid_lines, lines_of, unit_grid_lines

pytestmark = pytest.mark.gpu


def _far_lines(blocks=40, step=1000000):
    """Cliques of seven, a leaf at each vertex, in a chain with long links: the core is the cliques;
    from the ends distances reach 39M, from the middle 20M, either side of 2^25"""
    rng, e = np.random.default_rng(6), []
    for b in range(blocks):
        c = range(14 * b, 14 * b + 7)
        e += [(i, j, int(rng.integers(1, 9))) for i in c for j in range(14 * b, i)]
        e += [(i, i + 7, int(rng.integers(1, 9))) for i in c]
        if b:
            e.append((14 * b, 14 * b - 13, step))
    return lines_of(e, 14 * blocks)


def _far():
    """label-free index: harmless sources, sources that give the plan up"""
    n, u, v, w = _far_lines()
    g = Q.Graph(device=0)
    g.ReadLines(n, u, v, w)
    middle = np.arange(n // 2 - 20, n // 2 + 20, dtype=np.int32)
    return n, O.Arcs(n, u, v, w), g.build_index(Q.QBC_INDEX_CSR), middle, np.arange(12, dtype=np.int32)


def _unit_grid():
    """H2H index of the 24 x 24 unit grid: counts from its middle end at C(24, 12), from a corner pass 2^31"""
    n, u, v, w = unit_grid_lines()
    g = Q.Graph(device=0)
    g.ReadLines(n, u, v, w)
    idx = g.build_index(Q.QBC_INDEX_H2H, g.min_degree_order(), on_device=True)
    middle = np.array([24 * r + c for r in (11, 12) for c in (11, 12)], np.int32)
    return n, O.Arcs(n, u, v, w), idx, middle, np.arange(24, dtype=np.int32)


def _device_call(idx, n, srcs):
    import torch

    d_src = torch.from_numpy(srcs).cuda()
    d_bc = torch.zeros(n, dtype=torch.float64, device="cuda:0")
    torch.cuda.synchronize()
    idx.bc_sources_device(d_src.data_ptr(), len(srcs), d_bc.data_ptr())
    torch.cuda.synchronize()
    return d_bc.cpu().numpy()


BETWEEN = {
    "sources": lambda idx, n, middle, void: idx.bc_sources(void),
    "device_rows": lambda idx, n, middle, void: (_device_call(idx, n, void), idx.rows(middle[:2])),
    "device_plain": lambda idx, n, middle, void: (_device_call(idx, n, void), idx.bc_plain(middle[:2])),
    "device_only": lambda idx, n, middle, void: _device_call(idx, n, void),
    "query": lambda idx, n, middle, void: idx.bc_query_batch([middle], void),
    "autotune": lambda idx, n, middle, void: idx.autotune(void),
}


@pytest.mark.parametrize("between", sorted(BETWEEN))
@pytest.mark.parametrize("make", [_far, _unit_grid])
def test_captured_call_after_the_plan_is_given_up(make, between, monkeypatch):
    monkeypatch.setenv("QBC_TREE_MIN_PAIRS", "0")
    n, arcs, idx, middle, void = make()
    sets = [np.arange(0, n, 3, dtype=np.int32), np.arange(n, dtype=np.int32)]
    want = arcs.bc(middle)
    assert want.any()

    def answered():
        """right twice (captured, then replayed), and with how many launches"""
        for _ in range(2):
            idx.profile(True)
            for s, got in zip(sets, idx.bc_query_batch(sets, middle)):
                assert rel_err(got, want[s]) <= BC_RTOL
        return idx.stats()["launches"]

    with_plan = answered()
    BETWEEN[between](idx, n, middle, void)
    assert answered() != with_plan
    assert rel_err(idx.bc_sources(middle), want) <= BC_RTOL


def test_captured_call_after_the_threshold_moves(monkeypatch):
    """a graph captured with the tree's launches is not the one for a call that the rule sends elsewhere"""
    n, arcs, idx, middle, _ = _unit_grid()
    want = arcs.bc(middle)
    launches = []
    for pairs in ("0", "1000000000", "0"):
        monkeypatch.setenv("QBC_TREE_MIN_PAIRS", pairs)
        idx.bc_query_batch([middle], middle)  # captures
        idx.profile(True)
        assert rel_err(idx.bc_query_batch([middle], middle)[0], want[middle]) <= BC_RTOL
        launches.append(idx.stats()["launches"])
    assert launches[0] == launches[2] != launches[1]


@pytest.mark.parametrize("bad", [-1, "n"])
@pytest.mark.parametrize("kind", [Q.QBC_INDEX_MHL, Q.QBC_INDEX_H2H, Q.QBC_INDEX_CSR])
def test_bad_device_source_leaves_the_vector(kind, bad, monkeypatch):
    """an id out of range is found on the device: nothing is added, the next host call reports it, the
    one after that is right"""
    import torch

    monkeypatch.setenv("QBC_TREE_MIN_PAIRS", "0")
    n, u, v, w = grid_lines(1500, seed=5, shortcut_frac=0.02 if kind == Q.QBC_INDEX_CSR else 0.0)
    g = Q.Graph(device=0)
    g.ReadLines(n, u, v, w)
    idx = g.build_index(kind, g.min_degree_order() if kind == Q.QBC_INDEX_H2H else None, on_device=True)
    srcs = np.arange(0, n, 9, dtype=np.int32)
    with_bad = srcs.copy()
    with_bad[7] = n if bad == "n" else bad
    before = np.arange(n, dtype=np.float64)
    d_bc = torch.from_numpy(before).cuda()
    d_src = torch.from_numpy(with_bad).cuda()
    torch.cuda.synchronize()
    idx.bc_sources_device(d_src.data_ptr(), len(srcs), d_bc.data_ptr())
    torch.cuda.synchronize()
    assert np.array_equal(d_bc.cpu().numpy(), before)
    with pytest.raises(Q.QbcError, match="out of range"):
        idx.bc_sources(srcs)
    assert rel_err(idx.bc_sources(srcs), O.Arcs(n, u, v, w).bc(srcs)) <= BC_RTOL


def _launches(idx, call):
    call()  # captures
    idx.profile(True)
    call()
    return idx.stats()["launches"]


def test_autotune_on_a_short_list_keeps_the_plan_for_longer_ones(tmp_path):
    n, u, v, w = grid_lines(6007, seed=3)
    g = Q.Graph(device=0)
    g.ReadLines(n, u, v, w)
    idx = g.build_index(on_device=True)
    few = np.arange(5, n, n // 15, dtype=np.int32)
    all_tree, want = _launches(idx, idx.bc_all), idx.bc_all()
    few_want = O.Arcs(n, u, v, w).bc(few)
    path = str(tmp_path / "tuning.json")
    idx.autotune(few, path=path)
    assert _launches(idx, idx.bc_all) == all_tree
    assert rel_err(idx.bc_all(), want) <= BC_RTOL
    assert rel_err(idx.bc_sources(few), few_want) <= BC_RTOL
    idx.set_tuning()
    idx.load_tuning(path)
    assert _launches(idx, idx.bc_all) == all_tree
    idx.set_tuning(label_sources=16, label_warps=16, label_stream=1, keep_plan=1)
    assert _launches(idx, idx.bc_all) == all_tree and idx.label_group() == 16
    assert rel_err(_device_call(idx, n, few), few_want) <= BC_RTOL
    idx.set_tuning(label_sources=16, label_warps=16, label_stream=1)
    assert _launches(idx, idx.bc_all) != all_tree
    idx.set_tuning()
    idx.autotune(np.arange(0, n, 3, dtype=np.int32))  # long enough for the tree: it wins
    t = idx.get_tuning()
    assert t["keep_plan"] == t["label_warps"] == t["split"] == t["dep_form"] == 0


@pytest.mark.parametrize("kind,n,shortcuts,ns,waits,plan", [
    # below and above the rule's line where a call waits, and where it only enqueues
    (Q.QBC_INDEX_MHL, 2000, 0.0, 800, True, False), (Q.QBC_INDEX_MHL, 2000, 0.0, 1500, True, True),
    (Q.QBC_INDEX_MHL, 6000, 0.0, 416, True, False), (Q.QBC_INDEX_MHL, 6000, 0.0, 600, True, True),
    (Q.QBC_INDEX_MHL, 45000, 0.0, 20, True, False), (Q.QBC_INDEX_MHL, 45000, 0.0, 40, True, True),
    (Q.QBC_INDEX_MHL, 90000, 0.0, 1, True, True),
    (Q.QBC_INDEX_MHL, 6000, 0.0, 333, False, False), (Q.QBC_INDEX_MHL, 6000, 0.0, 600, False, True),
    (Q.QBC_INDEX_MHL, 45000, 0.0, 40, False, False), (Q.QBC_INDEX_MHL, 45000, 0.0, 60, False, True),
    (Q.QBC_INDEX_CSR, 100, 0.02, 1, True, True), (Q.QBC_INDEX_CSR, 100, 0.02, 1, False, True)])
def test_route_by_size(kind, n, shortcuts, ns, waits, plan, monkeypatch):
    n, u, v, w = grid_lines(n, seed=4, shortcut_frac=shortcuts)
    g = Q.Graph(device=0)
    g.ReadLines(n, u, v, w)
    idx = g.build_index(kind, on_device=True)
    srcs = np.random.default_rng(ns).choice(n, ns, replace=False).astype(np.int32)
    call = (lambda: idx.bc_sources(srcs)) if waits else (lambda: _device_call(idx, n, srcs))
    took, got = _launches(idx, call), call()
    monkeypatch.setenv("QBC_TREE_MIN_PAIRS", "0")
    with_plan, other = _launches(idx, call), call()
    monkeypatch.setenv("QBC_TREE_MIN_PAIRS", str(1 << 50))
    without, want = _launches(idx, call), call()
    assert with_plan != without
    assert took == (with_plan if plan else without)
    assert rel_err(got, want) <= BC_RTOL and rel_err(other, want) <= BC_RTOL


def test_chunk_that_does_not_fit_leaves_the_scratch():
    """200,000 slots of 200,000 vertices are 1.4 TB: refused, and the next calls are answered as before"""
    n, u, v, w = grid_lines(200000, seed=4, shortcut_frac=0.02)
    g = Q.Graph(device=0)
    g.ReadLines(n, u, v, w)
    idx = g.build_index(Q.QBC_INDEX_CSR)
    srcs = np.arange(0, n, n // 40, dtype=np.int32)
    want, size = idx.bc_sources(srcs), idx.info()
    for _ in range(2):
        with pytest.raises(Q.QbcError) as e:
            idx.set_tuning(chunk=200000)
        assert e.value.code == capi.QBC_ENOMEM
        assert np.array_equal(idx.info(), size)  # the same device bytes
        assert rel_err(idx.bc_sources(srcs), want) <= BC_RTOL
        assert rel_err(idx.bc_query_batch([srcs], srcs)[0], want[srcs]) <= BC_RTOL
    idx.set_tuning(chunk=64)
    assert rel_err(idx.bc_sources(srcs), want) <= BC_RTOL
