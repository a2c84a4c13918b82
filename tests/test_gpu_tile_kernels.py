"""k_force_pairs and the batch's cut where the dispatch still takes them.  The
octet kernels serve most small boxes whatever pair_seg and source_split say, so
these choose boxes that they do not take, and assert which kernel runs.
Tolerances as in test_gpu_parity.py; between two cuts of the same pair terms the
sums differ by rounding alone (1e-13, as test_gpu_batch.py)."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from yukawamd_b200 import abi, configs
from yukawamd_b200.engine import Batch, Engine

from helpers import rel, rel_norm
from test_gpu_parity import _short_cutoff, check_accel, workload

pytestmark = pytest.mark.gpu

FP64, MIXED = abi.YK_PREC_FP64, abi.YK_PREC_MIXED
CUTS = {"default": {}, "split2": dict(source_split=2), "split4-unsorted": dict(source_split=4, sort_every=-1),
        "unsorted-seg3": dict(sort_every=-1, pair_seg=3), "seg1": dict(pair_seg=1)}


@pytest.fixture(scope="module")
def orc():
    return Oracle("double", threads=8)


def check_pairs(orc, w, prec, meas, tuning):
    with Engine(w, precision=prec) as e:
        if tuning:
            e.set_tuning(**tuning)
        assert e.force_kernel() == "k_force_pairs"
    check_accel(orc, w, prec, meas, tuning=tuning)


@pytest.mark.parametrize("cut", list(CUTS))
@pytest.mark.parametrize("meas", [True, False], ids=["meas", "force"])
@pytest.mark.parametrize("kind,n,prec", [("nn", 4097, FP64), ("nn", 4225, FP64), ("nn", 4300, FP64),
                                         ("nn", 2049, MIXED), ("nn", 2177, MIXED), ("nn", 2300, MIXED),
                                         ("mix", 6145, MIXED), ("pure", 6273, MIXED), ("mix", 6300, MIXED)])
def test_tiles_match_oracle(gpu, orc, kind, n, prec, meas, cut):
    """Last tiles of one particle, one more tile, ragged ones; ions with the
    hi/lo displacement."""
    w = workload(kind, n, 70 + n)
    check_pairs(orc, w if kind == "nn" else _short_cutoff(w, 0.4), prec, meas, CUTS[cut])


@pytest.mark.parametrize("cut", list(CUTS))
@pytest.mark.parametrize("n", [1, 2, 3, 17, 127, 128, 129, 255, 257, 513])
@pytest.mark.parametrize("kind", ["pure", "mix"])
def test_half_edge_ions_ragged(gpu, orc, kind, n, cut):
    """Mixed ions with the cutoff at half an edge, the general displacement."""
    w = _short_cutoff(workload(kind, n, 13 + n), 0.5)
    check_pairs(orc, w, MIXED, True, CUTS[cut])
    check_pairs(orc, w, MIXED, False, CUTS[cut])


@pytest.mark.parametrize("kind", ["nn", "mix"])
def test_small_boxes_of_a_batch(gpu, orc, kind):
    """Ragged small boxes against the oracle, FP64: single engines of these sizes
    no longer run the tiles."""
    boxes = [workload(kind, n, 90 + n) for n in (2, 17, 129, 257, 513, 1500)]
    with Batch(boxes, mix_mode=abi.YK_MIX_FIXED) as b:
        sc = b.accel(True)
        got = [b.get_state(r)[3] for r in range(b.nrep)]
    for r, w in enumerate(boxes):
        a_ref, s_ref = orc.accel(w.yk_params(mix_mode=abi.YK_MIX_FIXED), w.x, w.zii, w.aii, True)
        assert rel_norm(got[r][:3 * w.n], a_ref[:3 * w.n]) <= 1e-12, w.n
        assert rel(sc[r].ev, s_ref.ev) <= 1e-12 and rel(sc[r].px, s_ref.px) <= 1e-12, w.n


@pytest.mark.parametrize("prec", [FP64, MIXED], ids=["fp64", "mixed"])
def test_another_cut_of_a_batch(gpu, prec):
    """pair_seg re-cuts the items of boxes that are large enough (3,001 ions make
    items of 2 tiles at most, 6,500 of 4): the same forces to rounding, and runs
    go on from there."""
    boxes = [configs.pure_ion(n, 8, 16, 1.5, 120.0, seed=n) for n in (700, 3001, 6500)]
    acc, items, states = {}, {}, {}
    with Batch(boxes, precision=prec) as b:
        for seg in (8, 3, 2, 1, 8):
            b.set_tuning(pair_seg=seg, graph_steps=10)
            b.accel(True)
            acc[seg] = [b.get_state(r)[3] for r in range(b.nrep)]
            items[seg] = b.work_items()
    assert items[8] < items[3] < items[2] < items[1]
    assert items[1] == sum(T * (T + 1) // 2 for T in (6, 24, 51))
    for seg in (3, 2, 1):
        for r, w in enumerate(boxes):
            # (mixed: the target sums of an item are FP64, the reactions FP32 either way)
            assert rel_norm(acc[seg][r][:3 * w.n], acc[8][r][:3 * w.n]) <= 1e-13, (seg, r)
    for seg in (8, 1):
        with Batch(boxes, precision=prec) as b:
            b.set_tuning(pair_seg=seg, graph_steps=10)
            b.accel(True)
            b.run(23, 5, series=False)
            states[seg] = [b.get_state(r)[0] for r in range(b.nrep)]
    for r in range(len(boxes)):
        assert rel_norm(states[1][r], states[8][r]) <= 1e-12
