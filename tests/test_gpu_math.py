"""Error bounds of the FP64 pair arithmetic on the GPU (yk_math_selftest), in
units in the last place of the exact value, taken from numpy's long double
(64-bit significand: 2^-11 ulp).

1/sqrt(x), octet kernels (rsqrt_h64_step in yk_octets.cuh): the estimate is
within 2^-20, so e = 1 - x y^2 is below 2^-19 and the dropped 5 e^3 / 16 below
2^-58.6 (0.02 ulp at most); x y rounds by 2^-53, which reaches the result halved
(0.5 ulp at most); the last FMA rounds by 0.5 ulp: 1.02 ulp.  The other kernels'
rsqrt_nr64 has a finer estimate and the same two roundings: 1.0 ulp.

e^-t, octet kernels (exp_neg_f64_warp): the table's entry 0.5 ulp, the last FMA
0.5; e^r - 1 is below 0.011, so its roundings and its argument's are below 0.04,
and the series truncated after r^6 drops 3.5e-18 (0.03 ulp): 1.1 ulp.  The other
kernels' exp_neg_f64 is held to 3 ulp by test_numerics.py; its table is eight
times finer and its series shorter.
"""
import ctypes as C

import numpy as np
import pytest

from yukawamd_b200 import _lib

pytestmark = pytest.mark.gpu

ESTIMATE, RSQRT, EXP, RSQRT_NR, EXP_256 = range(5)


def device(what, x):
    x = np.ascontiguousarray(x)
    out = np.empty_like(x)
    dp = C.POINTER(C.c_double)
    rc = _lib.lib().yk_math_selftest(0, what, len(x), x.ctypes.data_as(dp), out.ctypes.data_as(dp))
    _lib.check(rc)
    return out


def ulps(got, exact):
    return np.abs(got - exact) / np.spacing(exact.astype(np.float64))


def squares(seed):
    rng = np.random.default_rng(seed)
    edges = 2.0 ** np.arange(-40, 41)
    return np.concatenate([10.0 ** rng.uniform(-6, 12, 400000), rng.uniform(1, 4, 400000), edges,
                           np.nextafter(edges, 0), np.nextafter(edges, np.inf)])


def test_estimate(gpu):
    x = np.concatenate([squares(1), 2.0 ** np.random.default_rng(2).uniform(-1000, 1000, 200000)])
    exact = 1 / np.sqrt(x.astype(np.longdouble))
    assert np.abs(device(ESTIMATE, x) / exact - 1).max() <= 2.0 ** -20


@pytest.mark.parametrize("what,bound", [(RSQRT, 1.02), (RSQRT_NR, 1.0)], ids=["octets", "nr64"])
def test_reciprocal_root(gpu, what, bound):
    x = squares(3)
    assert ulps(device(what, x), 1 / np.sqrt(x.astype(np.longdouble))).max() <= bound


def test_reciprocal_root_past_fp32(gpu):
    x = 2.0 ** np.random.default_rng(4).uniform(-1000, 1000, 200000)
    assert ulps(device(RSQRT, x), 1 / np.sqrt(x.astype(np.longdouble))).max() <= 1.02


@pytest.mark.parametrize("what,bound", [(EXP, 1.1), (EXP_256, 3.0)], ids=["octets", "256-entries"])
def test_exponential(gpu, what, bound):
    rng = np.random.default_rng(5)
    half = np.arange(1, 2000) * (np.log(2.0) / 64)          # where the table index changes
    t = np.concatenate([[0.0, 1e-300, 699.9], 10.0 ** rng.uniform(-12, -1, 200000), rng.uniform(0, 30, 400000),
                        rng.uniform(0, 700, 400000), half, np.nextafter(half, 0), np.nextafter(half, np.inf)])
    assert ulps(device(what, t), np.exp(-t.astype(np.longdouble))).max() <= bound
    assert np.all(device(what, np.array([700.1, 1e4, 1e300])) == 0.0)


def test_octet_arithmetic_is_no_coarser_on_average(gpu):
    x, t = squares(6), np.random.default_rng(7).uniform(0, 690, 400000)
    root, ex = 1 / np.sqrt(x.astype(np.longdouble)), np.exp(-t.astype(np.longdouble))
    # (the mean of 800,000 errors of spread 0.2 ulp is known to 0.0003)
    assert ulps(device(RSQRT, x), root).mean() <= ulps(device(RSQRT_NR, x), root).mean() + 0.001
    assert ulps(device(EXP, t), ex).mean() <= ulps(device(EXP_256, t), ex).mean() + 0.001
