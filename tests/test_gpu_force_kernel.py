"""yk_force_kernel names the kernel that a force call runs.  On each side of
every line of the dispatch, and under tunings that override it."""
import pytest

from yukawamd_b200 import abi, configs
from yukawamd_b200.engine import Engine

pytestmark = pytest.mark.gpu

FP64, MIXED = abi.YK_PREC_FP64, abi.YK_PREC_MIXED


@pytest.mark.parametrize("kind,n,prec,cut,name", [
    ("pure", 500, FP64, 0.3, "k_force_octets_all"), ("pure", 9216, FP64, 0.3, "k_force_octets_all"),
    ("pure", 9217, FP64, 0.3, "k_force_octets"), ("pure", 8704, FP64, 0.4, "k_force_octets_all"),
    ("pure", 8705, FP64, 0.4, "k_force_octets"), ("pure", 7168, FP64, None, "k_force_octets_all"),
    ("pure", 7169, FP64, None, "k_force_octets"), ("pure", 6144, MIXED, 0.3, "k_force_octets_all"),
    ("pure", 6145, MIXED, 0.3, "k_force_pairs"), ("pure", 16383, MIXED, 0.3, "k_force_pairs"),
    ("pure", 16384, MIXED, 0.3, "k_force_pairs2"), ("pure", 24575, MIXED, 0.3, "k_force_pairs2"),
    ("pure", 24576, MIXED, 0.3, "k_force_octets"), ("pure", 500, MIXED, 0.5, "k_force_pairs"),
    ("nn", 4096, FP64, None, "k_force_octets_all"), ("nn", 4097, FP64, None, "k_force_pairs"),
    ("nn", 2048, MIXED, None, "k_force_octets_all"), ("nn", 2049, MIXED, None, "k_force_pairs")])
def test_automatic_kernel(gpu, kind, n, prec, cut, name):
    w = configs.pure_ion_ocp(3, n) if kind == "pure" else configs.nucleon_matter(3, n)
    w.params["rccut"] = 1e50 if cut is None else cut * w.params["xl"][0]
    with Engine(w, precision=prec) as e:
        assert e.force_kernel() == e.force_kernel(automatic=True) == name
        e.accel(True)
        e.set_tuning(force_kernel=abi.KERNEL_ROWS)
        assert e.force_kernel() == "k_force_rows" and e.force_kernel(automatic=True) == name
        e.set_tuning(force_kernel=abi.KERNEL_NEAR)
        assert e.force_kernel() == "k_force_near"
        e.set_tuning(force_kernel=abi.KERNEL_PAIRS, targets_per_thread=2)
        two = "k_force_pairs2" if e.tuning().targets_per_thread == 2 else name
        assert e.force_kernel() == two and e.force_kernel(automatic=True) == name


def test_bfield_has_none(gpu):
    w = configs.pure_ion_ocp(3, 100)
    with Engine(w.yk_params(sim_type=abi.YK_SIM_BFIELD, bfield=1e15), w.x, w.v, w.zii, w.aii) as e:
        assert e.force_kernel() == ""
