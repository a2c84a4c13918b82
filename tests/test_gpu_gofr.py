"""yk_gofr_counts places pairs in FP32 and takes the exact arithmetic next to a
bin edge: the counts must equal the oracle's bin for bin (integers, no
tolerance) where that could go wrong -- pairs exactly on edges, coincident
particles, coordinates on and outside the faces, unequal edges, bins below the
FP32 resolution."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from yukawamd_b200 import configs
from yukawamd_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _points(kind, n, xl, rng):
    L = np.array(xl)
    if kind == "lattice":              # distances that sit on bin edges, many exactly equal
        m = int(np.ceil(n ** (1 / 3)))
        c = rng.permutation(m ** 3)[:n]
        return np.stack([c // (m * m), c // m % m, c % m], axis=1) / m * L
    x = rng.random((n, 3)) * L
    if kind == "faces":                # on and around both faces, some coincident
        x[::3] = np.where(rng.random(x[::3].shape) < 0.5, 0.0, L)
        x[1::7] = x[0]
    if kind == "outside":              # beyond the range that the FP32 place covers
        x[::5] += (rng.random(x[::5].shape) - 0.5) * L
    return x


@pytest.mark.parametrize("nbin", [1, 100, 8192])
@pytest.mark.parametrize("kind,xl", [("lattice", (64.0, 64.0, 64.0)), ("faces", (71.3, 71.3, 71.3)),
                                     ("faces", (40.0, 71.3, 250.0)), ("outside", (71.3, 50.0, 90.0)),
                                     ("uniform", (1.7e4, 1.7e4, 1.7e4)), ("uniform", (1e-3, 2e-3, 1e-3))])
def test_counts_equal_oracle(gpu, kind, xl, nbin):
    n = 1153                           # nine tiles and one particle
    w = configs.pure_ion_ocp(3, n)
    w.x = np.ascontiguousarray(_points(kind, n, xl, np.random.default_rng(nbin)).reshape(-1))
    w.params["xl"] = list(xl)
    w.params["rccut"] = 0.3 * min(xl)
    p = w.yk_params()
    with Engine(p, w.x, w.v, w.zii, w.aii) as e:
        assert np.array_equal(e.gofr_counts(nbin), Oracle("double").gofr_counts(p, w.x, nbin))


def test_counters_hold_every_pair_of_a_cta(gpu):
    """2.8 million particles in a 1 : 1 : 60 box with the most bins (fewest
    CTAs): nearly all pairs are past the last bin's inner edge and end in that
    one 32-bit counter of each CTA, 4.3e9 of them if the resident CTAs alone
    took all units.  The counts add up to n (n - 1) / 2."""
    n = 2800000
    w = configs.pure_ion_ocp(3, 128)
    xl = np.array([100.0, 100.0, 6000.0])
    w.params["xl"] = list(xl)
    w.params["rccut"] = 30.0
    x = np.ascontiguousarray((np.random.default_rng(4).random((n, 3)) * xl).reshape(-1))
    with Engine(w.yk_params(), x, np.zeros(3 * n), np.full(n, 8.0), np.full(n, 16.0)) as e:
        c = e.gofr_counts(8192)
    assert c[-1] > 0.9 * c.sum()
    assert int(c.sum()) == n * (n - 1) // 2


@pytest.mark.parametrize("kind,xl", [("lattice", (64.0, 64.0, 64.0)), ("faces", (71.3, 71.3, 71.3)),
                                     ("outside", (71.3, 71.3, 71.3)), ("uniform", (1.7e4, 1.7e4, 1.7e4)),
                                     ("uniform", (40.0, 40.0, 2000.0))])
@pytest.mark.parametrize("n,nbin", [(1153, 80), (1153, 4100), (1153, 4200), (4097, 150), (4097, 7400), (4097, 7600)])
def test_counts_at_the_widest_place(gpu, kind, xl, n, nbin):
    """The largest bin counts that are placed in FP32 (in a cube 4,100 up to
    4,096 particles, where the bound is 0.005 of a bin, and 7,400 above, where
    it is 0.009) and the next, whose pairs are all taken exactly; 80 and 150
    bins are the largest in the 1 : 1 : 50 box."""
    w = configs.pure_ion_ocp(3, n)
    w.x = np.ascontiguousarray(_points(kind, n, xl, np.random.default_rng(nbin)).reshape(-1))
    w.params["xl"] = list(xl)
    w.params["rccut"] = 0.3 * min(xl)
    p = w.yk_params()
    with Engine(p, w.x, w.v, w.zii, w.aii) as e:
        assert np.array_equal(e.gofr_counts(nbin), Oracle("double").gofr_counts(p, w.x, nbin))
