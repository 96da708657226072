"""CPU: the tuning field that keeps label-kernel fields from asking for those kernels (keep_plan)."""
import pytest

import gpu_betweennesscentrality_b200 as Q
from gpu_betweennesscentrality_b200 import capi
from gpu_betweennesscentrality_b200.capi import i32p, ptr
from util import grid_lines


def _index():
    n, u, v, w = grid_lines(200, seed=2)
    g = Q.Graph()
    g.ReadLines(n, u, v, w)
    return g.build_index(upload=False)


def test_keep_plan_round_trip():
    idx = _index()
    assert idx.get_tuning()["keep_plan"] == 0
    idx.set_tuning(label_warps=16, keep_plan=1)
    assert idx.get_tuning()["keep_plan"] == 1
    idx.set_tuning(**idx.get_tuning())
    assert idx.get_tuning()["keep_plan"] == 1 and idx.get_tuning()["label_warps"] == 16
    with pytest.raises(Q.QbcError) as e:
        idx.set_tuning(keep_plan=2)
    assert e.value.code == capi.QBC_EINVAL
    idx.set_tuning()
    assert idx.get_tuning()["keep_plan"] == 0


@pytest.mark.parametrize("nparams", [1, 8, 14])
def test_shorter_lists_ask_for_the_kernels_they_name(nparams):
    idx = _index()
    idx.set_tuning(label_warps=16, keep_plan=1)
    p = Q.i32([0] * 7 + [12] + [0] * 6)
    capi.check(capi.lib().qbc_index_set_tuning(idx.h, ptr(p, i32p), nparams))
    assert idx.get_tuning()["keep_plan"] == 0
