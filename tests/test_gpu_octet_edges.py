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


@pytest.mark.parametrize("n,prec", [(9300, abi.YK_PREC_FP64), (24700, abi.YK_PREC_MIXED)], ids=["fp64", "mixed"])
@pytest.mark.parametrize("sort_every", [4, -1])
@pytest.mark.parametrize("accel_first", [True, False], ids=["accel", "fresh"])
def test_run_equals_newton_on_cut_jobs(gpu, n, prec, sort_every, accel_first):
    """The boxes whose jobs are cut on the device: yk_run gives the bits of the
    same steps through yk_newton over several replays of its graph, also when
    the table has not been cut before the run."""
    w = configs.pure_ion_ocp(51, n)
    # in an order that is spatial without a sort, moving fast: a cut at other
    # positions is another cut
    L = w.params["xl"][0]
    x = w.x.reshape(-1, 3)
    cell = np.floor(x / L * 8).astype(int)
    w.x = np.ascontiguousarray(x[np.lexsort((cell[:, 2], cell[:, 1], cell[:, 0]))].reshape(-1))
    w.v = np.random.default_rng(5).standard_normal(3 * n) * 0.01 * L / w.params["dt"]
    w.params["rccut"] = 0.25 * L
    p = w.yk_params(precision=prec)
    steps, me = 23, 5
    out = []
    for run in (False, True):
        with Engine(p, w.x, w.v, w.zii, w.aii) as e:
            e.set_tuning(sort_every=sort_every, graph_steps=5)
            if accel_first:
                e.accel(True)
            if run:
                ser = e.run(steps, me)
            else:
                ser = [abi.YkScalars.from_buffer_copy(e.newton(g % me == 0)) for g in range(1, steps + 1)]
            out.append((e.get_state(), [bytes(t) for t in ser]))
    for A, B in zip(out[0][0], out[1][0]):
        assert np.array_equal(A, B)
    assert out[0][1] == out[1][1]


@pytest.mark.parametrize("n,prec", [(7000, abi.YK_PREC_FP64), (9000, abi.YK_PREC_FP64), (9300, abi.YK_PREC_FP64),
                                    (24700, abi.YK_PREC_MIXED)])
@pytest.mark.parametrize("calls", [1, 30], ids=["at-once", "in-steps"])
def test_other_positions_get_their_own_order(gpu, orc, n, prec, calls):
    """Positions that the host sets far from the old ones, at once or little by
    little, are put in order again before the next force call: the bits are
    those of an engine created with them.  (In 30 calls of 0.32 to 0.35
    spacings the boxes on all pairs sort at every fifth, 9,300 at every second,
    24,700 at each.)"""
    w = configs.pure_ion_ocp(61, n)
    p = w.yk_params(precision=prec)
    L = w.params["xl"][0]
    # every particle along x, calls + 1 times the same way
    step = np.zeros((n, 3))
    step[:, 0] = np.random.default_rng(7).random(n) * L / calls
    with Engine(p, w.x, w.v, w.zii, w.aii) as e:
        e.accel(True)
        for k in range(1, calls + 1):
            x = np.ascontiguousarray(np.mod(w.x.reshape(-1, 3) + k * step, L).reshape(-1))
            e.set_state(x=x)
            s = e.accel(True)
            a = e.a.copy()
            ev = s.ev
    with Engine(p, x, w.v, w.zii, w.aii) as e:
        s = e.accel(True)
        assert np.array_equal(e.a, a)
        assert s.ev == ev
    if calls == 1:
        a_ref, s_ref = orc.accel(p, x, w.zii, w.aii, True)
        tol = 1e-12 if prec == abi.YK_PREC_FP64 else 1e-6
        assert np.linalg.norm(a[:3 * n] - a_ref[:3 * n]) <= tol * np.linalg.norm(a_ref[:3 * n])
        assert abs(ev - s_ref.ev) <= tol * abs(s_ref.ev)


@pytest.mark.parametrize("n,cut", [(7168, 1e50), (7169, 1e50), (8704, 0.4), (8705, 0.4)])
def test_sizes_around_the_wide_cutoffs_change(gpu, orc, n, cut):
    """The FP64 sizes at which a box with a wide or no cutoff goes from every pair
    from both sides to half pairs; a box that comes to such a cutoff by set_box."""
    w = workload("mix", n, 800 + n)
    L = w.params["xl"][0]
    w.params["rccut"] = cut if cut > 1 else cut * L
    check_accel(orc, w, abi.YK_PREC_FP64, True)
    check_accel(orc, w, abi.YK_PREC_FP64, False)
    p = w.yk_params()
    wide = [t * 1.5 for t in w.params["xl"]]
    p2 = w.yk_params(xl=wide)
    x2 = np.ascontiguousarray(w.x * 1.5)
    with Engine(p2, x2, w.v, w.zii, w.aii) as e:
        e.accel(True)
        e.set_box(w.params["xl"])
        e.set_state(x=w.x)
        s = e.accel(True)
        a = e.a.copy()
    with Engine(p, w.x, w.v, w.zii, w.aii) as e:
        assert e.accel(True).ev == s.ev
        assert np.linalg.norm(e.a - a) <= 1e-13 * np.linalg.norm(a)


@pytest.mark.parametrize("kind,n,prec", [("pure", 349, abi.YK_PREC_FP64), ("pure", 349, abi.YK_PREC_MIXED),
                                         ("mix", 9500, abi.YK_PREC_FP64), ("mix", 24700, abi.YK_PREC_MIXED),
                                         ("nn", 700, abi.YK_PREC_FP64), ("nn", 700, abi.YK_PREC_MIXED)])
def test_coincident_particles_stay_by_themselves(gpu, orc, kind, n, prec):
    """Two particles in one place get no finite force and, a step later, no finite
    position.  The others do not notice them, as in the oracle."""
    w = workload(kind, n, 30 + n)
    m = int(np.ceil(n ** (1 / 3)))                     # apart from each other: a jittered lattice
    rng = np.random.default_rng(n)
    c = rng.permutation(m ** 3)[:n]
    x = (np.stack([c // (m * m), c // m % m, c % m], axis=1) + 0.5 + 0.2 * (rng.random((n, 3)) - 0.5)) / m
    if kind == "nn":
        w.zii[:2] = w.zii[n // 2] = 1.0
    else:
        w.params["rccut"] = 0.3 * w.params["xl"][0]
    x[n // 2] = x[1]
    w.x = np.ascontiguousarray((x * np.array(w.params["xl"])).reshape(-1))
    p = w.yk_params(precision=prec)
    xr, vr, vo = w.x.copy(), w.v.copy(), np.zeros(3 * n)
    ar, sr = orc.accel(p, xr, w.zii, w.aii, True)
    with Engine(p, w.x, w.v, w.zii, w.aii) as e:
        assert e.force_kernel().startswith("k_force_octets")
        e.accel(True)
        for step in range(3):
            e.newton(step == 1)
            orc.newton(p, xr, vr, vo, ar, w.zii, w.aii, step == 1, sr)
            gx = e.get_state()[0]
            lost = ~np.isfinite(xr)
            assert lost.sum() == 6
            assert np.array_equal(~np.isfinite(gx), lost), step


@pytest.mark.parametrize("kind,n", [("pure", 7), ("pure", 300), ("nn", 300)])
def test_negative_screening(gpu, orc, kind, n):
    """xmuc < 0 is accepted: e^{-mu r} grows, and the FP64 form follows it (the
    mixed form stays off the octets, whose far-away pads would count)."""
    w = workload(kind, n, 17 + n)
    w.params["xmuc"] = -0.3 / w.params["xl"][0]
    w.params["rccut"] = 0.3 * w.params["xl"][0]
    check_accel(orc, w, abi.YK_PREC_FP64, True)
    with Engine(w, precision=abi.YK_PREC_MIXED) as e:
        assert e.force_kernel() == "k_force_pairs"
