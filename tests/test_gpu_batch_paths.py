"""The batch's two force kernels (boxes on the mixed hi/lo displacement, and
those whose cutoff is close to half an edge) and its per-box cut of the work
items: a box gives the same bits alone and among boxes of the other path, at
the sizes where the cut changes, and when it comes into a batch whose step
graphs were captured without it.  Equality is exact: a box's items, their
order of summation and its kernel depend on the box only.
"""
import numpy as np
import pytest

from yukawamd_b200 import abi, configs
from yukawamd_b200.engine import Batch, SlotBatch

pytestmark = pytest.mark.gpu

PRECS = pytest.mark.parametrize("prec", [abi.YK_PREC_FP64, abi.YK_PREC_MIXED], ids=["fp64", "mixed"])


def _box(n, seed, half_edge):
    w = configs.pure_ion(n, 8, 16, 1.5, 120.0, seed=seed)
    L = w.params["xl"][0]
    w.params["rccut"] = 0.5 * L if half_edge else 0.3 * L
    return w


@PRECS
def test_both_paths_at_the_cuts(gpu, prec):
    """Tiles 1, 2, 16 and 17 (one source tile per item up to 16), either path."""
    boxes = [_box(n, 20 + k, k % 2 == 1) for k, n in enumerate([128, 129, 2048, 2049, 2050, 2048])]
    with Batch(boxes, precision=prec) as b:
        b.accel(True)
        b.run(9, 3, series=False)
        mix = [b.get_state(r) for r in range(b.nrep)]
    for r, w in enumerate(boxes):
        with Batch([w], precision=prec) as b:
            b.accel(True)
            b.run(9, 3, series=False)
            for A, B in zip(mix[r], b.get_state(0)):
                assert np.array_equal(A, B), r


@pytest.mark.parametrize("late_half", [True, False], ids=["half-edge-late", "short-late"])
def test_box_of_the_other_path_comes_later(gpu, late_half):
    first, late = _box(900, 31, not late_half), _box(1100, 32, late_half)

    def args(w):
        return w.yk_params(precision=abi.YK_PREC_MIXED), w.x, w.v, w.zii, w.aii

    units = 4 * SlotBatch.pair_units(1100)
    with SlotBatch(args(first)[0], 2, 4000, units) as b:
        b.admit(*args(first), 400)
        b.run(100, 0, series=False)
        slot, _ = b.admit(*args(late), 100)
        b.run(100, 0, series=False)
        got = b.retire(slot)
    with SlotBatch(args(late)[0], 2, 4000, units) as b:
        slot, _ = b.admit(*args(late), 100)
        b.run(100, 0, series=False)
        want = b.retire(slot)
    for A, B in zip(got, want):
        assert np.array_equal(A, B)
