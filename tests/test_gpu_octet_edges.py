"""The octet kernels where an answer once depended on more than the particles:
positions a box length or more outside the box, step graphs captured before
the job table was cut, a slot order that belongs to another configuration.
Tolerances as in test_gpu_parity.py.
"""
import numpy as np
import pytest

from oracle.oracle import Oracle
from yukawamd_b200 import abi, configs
from yukawamd_b200.engine import Engine

from test_gpu_parity import check_accel, workload

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def orc():
    return Oracle("double", threads=8)


@pytest.mark.parametrize("kind,n", [("pure", 600), ("pure", 9500), ("nn", 2000)])
@pytest.mark.parametrize("edges", [1, 2, 3, -2])
@pytest.mark.parametrize("cut", [1e50, 0.4], ids=["uncut", "cut"])
def test_particles_whole_edges_apart(gpu, orc, kind, n, edges, cut):
    """Two small clusters `edges` box lengths apart.  The reference's image
    (int_ion_pure.f:149-150) takes one edge off a displacement, not the nearest
    multiple, so clusters two edges apart stay one edge apart."""
    w = workload(kind, n, 40 + n)
    L = w.params["xl"][0]
    x = (0.1 + 0.08 * np.random.default_rng(n).random((n, 3))) * L
    x[n // 2:, 0] += edges * L
    w.x = np.ascontiguousarray(x.reshape(-1))
    w.params["xmuc"] = 1.0 / L                 # the far cluster still counts
    w.params["rccut"] = cut if cut > 1 else cut * L
    check_accel(orc, w, abi.YK_PREC_FP64, True)
    check_accel(orc, w, abi.YK_PREC_FP64, False)
