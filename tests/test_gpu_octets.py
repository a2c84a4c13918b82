"""The octet kernels: accelerations and sums against the CPU oracle at the sizes
where the engine changes kernel (FP64: every pair from both sides up to 9,216
particles, half pairs in jobs cut by cost above; mixed: up to 6,144 and from
24,576) and at the shapes where the job table can go wrong.

Tolerances as in test_gpu_parity.py: both sides sum the same FP64 pair terms
in another order; the terms are within a few ulp of the oracle's (1e-15) and
a force is a sum of up to n of them with cancellation, which 1e-12 of the
2-norm covers (n = 24,577: sqrt(n) roundings of terms up to the norm, 4e-14).
Mixed: 1e-6, the form's bound.
"""
import numpy as np
import pytest

from oracle.oracle import Oracle
from yukawamd_b200 import abi, configs
from yukawamd_b200.engine import Engine

from test_gpu_parity import check_accel, rel_norm, workload

pytestmark = pytest.mark.gpu

PRECS = pytest.mark.parametrize("prec", [abi.YK_PREC_FP64, abi.YK_PREC_MIXED], ids=["fp64", "mixed"])


@pytest.fixture(scope="module")
def orc():
    return Oracle("double", threads=8)


@pytest.mark.parametrize("kind", ["pure", "mix", "nn"])
@pytest.mark.parametrize("n,prec", [(9216, abi.YK_PREC_FP64), (9217, abi.YK_PREC_FP64), (10369, abi.YK_PREC_FP64),
                                    (6143, abi.YK_PREC_MIXED), (6145, abi.YK_PREC_MIXED),
                                    (24575, abi.YK_PREC_MIXED), (24577, abi.YK_PREC_MIXED)])
def test_sizes_around_the_kernel_change(gpu, orc, kind, n, prec):
    """The largest all-pairs box, the smallest cost-cut one (its last tile
    holds one particle), one more tile; the mixed form's changes, with last
    tiles that end on half a source pair."""
    w = workload(kind, n, 500 + n)
    check_accel(orc, w, prec, True)
    check_accel(orc, w, prec, False)


def _clustered(kind, n, seed):
    """Half the particles in one corner of the box, the rest spread out: rows
    with everything and rows with nothing within reach."""
    w = workload(kind, n, seed)
    rng = np.random.default_rng(seed)
    L = np.array(w.params["xl"])
    x = rng.random((n, 3))
    x[: n // 2] *= 0.15
    w.x = np.ascontiguousarray((x * L).reshape(-1))
    w.params["rccut"] = 0.1 * L[0] if kind != "nn" else w.params["rccut"]
    return w


@PRECS
@pytest.mark.parametrize("sort", ["sorted", "unsorted"])
def test_uneven_work(gpu, orc, sort, prec):
    w = _clustered("mix", 15000, 3)
    check_accel(orc, w, prec, True, tuning=dict(sort_every=4 if sort == "sorted" else -1))


@pytest.mark.parametrize("n", [700, 9500])
@pytest.mark.parametrize("rccut", [1.0e50, 1.0e200], ids=["1e50", "1e200"])
def test_no_cutoff(gpu, orc, n, rccut):
    """No cutoff (rccut at its 1e50 default, and one whose square overflows):
    every pair counts, no image can be shared by a tile, and list pads and
    empty target slots must still add nothing.  FP64 (the mixed form's FP32
    energies of an uncut plasma are not held to 1e-6)."""
    w = configs.pure_ion_ocp(11, n)
    w.params["rccut"] = rccut
    check_accel(orc, w, abi.YK_PREC_FP64, True)


@PRECS
@pytest.mark.parametrize("n", [700, 24577])
def test_power_of_two_edges(gpu, orc, n, prec):
    """Box edges of 2^8 fm: an image shift of a far-away value by whole edges
    is exact, so a pad of a source list that is told by its distance alone
    must stay far away under any shift."""
    w = workload("pure", n, 77 + n)
    L = np.array(w.params["xl"])
    w.x = np.ascontiguousarray((w.x.reshape(-1, 3) / L * 256.0).reshape(-1))
    w.params["xl"] = [256.0, 256.0, 256.0]
    w.params["rccut"] = 76.8
    check_accel(orc, w, prec, True)
    check_accel(orc, w, prec, False)


@pytest.mark.parametrize("n,prec", [(100, abi.YK_PREC_FP64), (4096, abi.YK_PREC_FP64), (4097, abi.YK_PREC_FP64),
                                    (101, abi.YK_PREC_MIXED), (2047, abi.YK_PREC_MIXED), (2049, abi.YK_PREC_MIXED)])
@pytest.mark.parametrize("terms", ["both", "nuclear", "coulomb", "cut", "edges"])
def test_small_nucleon_boxes(gpu, orc, n, prec, terms):
    """Nucleons up to and past the sizes that take every pair from both sides:
    each term alone, a Coulomb cutoff inside the box, and box edges of a power
    of two with protons exactly half an edge apart (the image's boundary)."""
    w = workload("nn", n, 900 + n)
    if terms == "nuclear":
        w.params["coulomb_on"] = 0
    elif terms == "coulomb":
        w.params["nuclear_on"] = 0
    elif terms == "cut":
        w.params["rccut"] = 0.4 * w.params["xl"][0]
    elif terms == "edges":
        edge = 2.0 ** np.ceil(np.log2(w.params["xl"][0]))
        x = w.x.reshape(-1, 3) / np.array(w.params["xl"]) * edge
        protons = np.flatnonzero(np.asarray(w.zii)[:n] == 1.0)
        x[protons[1]] = (x[protons[0]] + [0.5 * edge, 1.0, 2.0]) % edge
        w.x = np.ascontiguousarray(x.reshape(-1))
        w.params["xl"] = [edge] * 3
    check_accel(orc, w, prec, True)
    check_accel(orc, w, prec, False)


@PRECS
@pytest.mark.parametrize("n", [700, 12000])
@pytest.mark.parametrize("integrator", [1, 2])
def test_another_kernel_after_octet_steps(gpu, orc, n, prec, integrator):
    """Octet steps gather the positions themselves and leave the FP32 shadow
    behind: a kernel that reads it, chosen between steps with the slot order
    kept, must see the moved positions.  (The steps move every particle by
    far more than the tolerance.)"""
    w = workload("mix", n, 40 + n)
    w.params["integrator"] = integrator
    w.params["precision"] = prec
    p = w.yk_params(precision=prec)
    with Engine(p, w.x, w.v, w.zii, w.aii) as e:
        e.set_tuning(sort_every=-1)
        e.accel(True)
        # (read now: the last entry is also e.scalars, which the next call fills)
        series = [(q.ev, q.ek) for q in e.run(12, 5, series=True)]
        e.set_tuning(force_kernel=abi.KERNEL_ROWS, sort_every=-1)
        s = e.accel(True)
        a = e.a.copy()
        x = e.get_state()[0]
    a_ref, s_ref = orc.accel(p, x, w.zii, w.aii, True)
    tol = 1e-12 if prec == abi.YK_PREC_FP64 else 1e-6
    assert rel_norm(a[:3 * n], a_ref[:3 * n]) <= tol
    assert abs(s.ev - s_ref.ev) <= tol * abs(s_ref.ev)
    # a step that measures nothing leaves zeros in its entry (integrator 2)
    for k in range(12):
        assert (series[k][0] != 0.0) == ((k + 1) % 5 == 0), k
        if integrator == 2:
            assert (series[k][1] != 0.0) == ((k + 1) % 5 == 0), k
