"""Server(autotune=True): a slot batch is empty when its cached tuning is looked
up, so it has a kind but no sizes."""
import json
from types import SimpleNamespace

import numpy as np
import pytest

from yukawamd_b200 import abi, configs, tune
from yukawamd_b200.serve import Request, Server


class EmptySlots:
    nrep, n = 256, [0] * 256

    def __init__(self, precision=abi.YK_PREC_MIXED):
        self.params = [SimpleNamespace(sim_type=2, precision=precision)]
        self.set = None

    def set_tuning(self, **kw):
        self.set = kw


def test_empty_slots_take_the_latest_choice_of_their_kind(tmp_path, monkeypatch):
    cache = tmp_path / "tune.json"
    monkeypatch.setenv("YK_TUNE_CACHE", str(cache))
    monkeypatch.setattr(tune, "gpu_name", lambda device=0: "NVIDIA B200")
    b = EmptySlots()
    assert tune.apply_batch(b) is False and b.set is None
    full = EmptySlots()
    full.n = [7000] * 256
    full.nrep = 256
    key = tune.batch_key(full)
    other = key.rsplit("nb", 1)[0] + "nb20"
    cache.write_text(json.dumps({key: dict(pair_seg=16, graph_steps=50, when=1.0),
                                 other: dict(pair_seg=4, graph_steps=25, when=2.0),
                                 key.replace("nrep256", "nrep25"): dict(pair_seg=2, when=3.0)}))
    assert tune.apply_batch(b) is True and b.set == dict(pair_seg=4, graph_steps=25)
    assert tune.apply_batch(EmptySlots(abi.YK_PREC_FP64)) is False
    assert tune.apply_batch(full) is True and full.set == dict(pair_seg=16, graph_steps=50)


@pytest.mark.gpu
def test_autotuned_server_runs(gpu, tmp_path, monkeypatch):
    monkeypatch.setenv("YK_TUNE_CACHE", str(tmp_path / "tune.json"))
    w = configs.pure_ion(900, 6, 12, 0.8, 120.0, seed=3)
    runs = [Request(i, w, 100, abi.YK_PREC_MIXED, 0.0) for i in range(2)]
    Server(hbm_budget=2 << 30, chunk=50, autotune=True).run(runs[:1])
    Server(hbm_budget=2 << 30, chunk=50).run(runs[1:])
    assert np.array_equal(runs[0].final_x, runs[1].final_x)
