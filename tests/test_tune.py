"""The tuner's bookkeeping on fake engines: candidates that come to the same are
timed once, and a cached winner is only applied where the same kernels were the
choice."""
import json
from types import SimpleNamespace

import pytest

from yukawamd_b200 import abi, tune


class FakeEngine:
    """An ion box: the octet kernel for one target per thread, as at 55,296
    mixed ions."""
    n = 55296

    def __init__(self, auto="k_force_octets"):
        self.params = SimpleNamespace(sim_type=abi.YK_SIM_ION_MIXTURE, precision=abi.YK_PREC_MIXED)
        self.auto = auto
        self.t = dict(force_kernel=2, pair_seg=4, sort_every=4, source_split=1, targets_per_thread=1, graph_steps=50)
        self.runs = []
        self.set = []

    def set_tuning(self, **kw):
        self.set.append(kw)
        self.t.update(kw)
        if self.t["sort_every"] == 0:
            self.t["sort_every"] = 4

    def tuning(self):
        return SimpleNamespace(**self.t)

    def force_kernel(self, automatic=False):
        if automatic:
            return self.auto
        if self.t["force_kernel"] == abi.KERNEL_ROWS:
            return "k_force_rows"
        if self.t["force_kernel"] == abi.KERNEL_NEAR:
            return "k_force_near"
        return "k_force_pairs2" if self.t["targets_per_thread"] == 2 else self.auto

    def get_state(self):
        return None, None, None, None

    def set_state(self, **kw):
        pass

    def run(self, steps, meas, series):
        self.runs.append(self.force_kernel())

    def perf_enable(self, on, flush):
        pass

    def perf_read(self):
        return SimpleNamespace(run_ms=1.0 * len(self.runs), steps=1, force_ms=1.0, force_calls=1)


@pytest.fixture(autouse=True)
def cache(tmp_path, monkeypatch):
    path = tmp_path / "tune.json"
    monkeypatch.setenv("YK_TUNE_CACHE", str(path))
    monkeypatch.setattr(tune, "gpu_name", lambda device=0: "NVIDIA B200")
    return path


def test_candidates_that_come_to_the_same_are_timed_once():
    e = FakeEngine()
    best, ms, res = tune.tune(e)
    cands = [c for c in tune.CANDIDATES if c.get("source_split", 1) == 1]
    assert len(res) == len(cands)
    # the octet kernel once per sort cadence: automatic (4), 2, 8, 16, never
    assert e.runs.count("k_force_octets") == 2 * 5        # warm-up and timed run
    same = [r for r in res if r[1]["force_kernel"] == abi.KERNEL_PAIRS and r[1]["sort_every"] == 0
            and r[1]["targets_per_thread"] == 1]
    assert len(same) == 4 and len({r[0] for r in same}) == 1
    # kernels that take notice of pair_seg are timed for each
    assert e.runs.count("k_force_pairs2") == e.runs.count("k_force_near") == 2 * 3


def test_tiles_are_timed_for_each_cut():
    e = FakeEngine(auto="k_force_pairs")
    e.n = 12000
    tune.tune(e, save=False)
    # pair_seg 8, 4, 16, 2; sort 2, 8, 16, never; split 2 and 4
    assert e.runs.count("k_force_pairs") == 2 * 10


def test_winner_of_other_kernels_is_not_applied(cache):
    old = dict(force_kernel=2, pair_seg=8, sort_every=0, source_split=1, targets_per_thread=2)
    cache.write_text(json.dumps({"NVIDIA B200|sim3|prec1|nb32": old, "NVIDIA B200|sim2|prec1|nb32": old}))
    e = FakeEngine()
    assert tune.apply(e) is False and e.set == []
    # stored now, and found again, but not for a box that takes another kernel
    tune.tune(e)
    assert tune.apply(FakeEngine()) is True
    assert tune.apply(FakeEngine(auto="k_force_pairs2")) is False


def test_batch_cuts_that_come_to_the_same_are_timed_once():
    class FakeBatch:
        nrep, n = 1, [3001]
        params = [SimpleNamespace(sim_type=2, precision=1)]
        timed = 0

        def get_state(self, r):
            return None, None, None, None

        def set_state(self, r, **kw):
            pass

        def set_tuning(self, pair_seg, graph_steps):
            self.seg = pair_seg

        def work_items(self):
            return 24 * 25 // 2 // min(self.seg, 2)

        def run(self, steps, meas, series):
            self.timed += 1
            return None, 3.0 + self.seg

    b = FakeBatch()
    best, ms, res = tune.tune_batch(b, segs=(8, 4, 16, 2, 1), save=False)
    assert b.timed == 2 * 2 and len(res) == 5
    assert best == 1 and ms == 4.0 and {r[0] for r in res[:4]} == {11.0}
    assert tune.batch_key(b).startswith("r%d|" % tune.REVISION)
