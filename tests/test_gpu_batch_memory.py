"""What a batch reserves: a serving group stays within its HBM budget, and a
batch fits wherever it fitted with whole segments of tiles per work item.  Each
measurement runs in a process of its own, so that cached memory of other
batches does not count."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

GROUP = """
import torch
from yukawamd_b200 import configs, serve
w = configs.pure_ion(512, 8, 16, 1.0, 100.0, 1)
torch.zeros(1, device="cuda")
prec, gib = {prec}, {gib}
before = torch.cuda.mem_get_info()[0]
g = serve.Group(("ion", prec), w.yk_params(precision=prec), gib << 30, 0, 256, 50, False)
used = before - torch.cuda.mem_get_info()[0]
print("reserved", used / 2 ** 30)
assert used > 0.5 * (gib << 30)
assert used <= gib << 30
"""

# 6,000 boxes of 16 tiles.  need: the bytes of a batch with whole segments of 8
# tiles (2 units / 8 + 2 tiles rows of target sums), without some small arrays.
TIGHT = """
import numpy as np
import torch
from yukawamd_b200 import abi, configs
from yukawamd_b200.engine import Batch, SlotBatch
T, boxes = 16, {boxes}
units, n = boxes * T * (T + 1) // 2, boxes * T * 128
tiles = n // 128 + boxes
w = configs.pure_ion(2048, 8, 16, 1.0, 100.0, 1)
p = w.yk_params(precision=abi.YK_PREC_MIXED)
rows = 2 * units // 8 + 2 * tiles
need = units * 128 * 3 * 4 + rows * (128 * 3 * 8 + 96) + 14 * 8 * (n + 3 * boxes) + 128 * tiles * 96 + 24 * n
torch.zeros(1, device="cuda")
hold = torch.empty(torch.cuda.mem_get_info()[0] - need - (1 << 29), dtype=torch.uint8, device="cuda")
free = torch.cuda.mem_get_info()[0]
assert need < free < need + units * 3168 * 0.9, (need, free)      # a row for each unit does not fit
with SlotBatch(p, boxes, n, units) as b:
    slot, s = b.admit(p, w.x, w.v, w.zii, w.aii, 40)
    b.run(20, 5, series=False)
    got = b.get_state(slot)
del hold
torch.cuda.empty_cache()
with Batch([w], precision=abi.YK_PREC_MIXED) as b:
    b.accel(True)
    b.run(20, 5, series=False)
    want = b.get_state(0)
for A, B in zip(got[:2], want[:2]):                               # another cut: the same to rounding
    assert np.linalg.norm(A - B) <= 1e-6 * np.linalg.norm(B)
print("ok")
"""


def _run(code):
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr[-2000:]


@pytest.mark.parametrize("prec,gib", [(1, 4), (1, 16), (0, 16)])
def test_group_stays_within_its_budget(gpu, prec, gib):
    _run(GROUP.format(prec=prec, gib=gib))


def test_batch_fits_where_whole_segments_fit(gpu):
    _run(TIGHT.format(boxes=6000))
