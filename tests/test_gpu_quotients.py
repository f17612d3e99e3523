"""The kernels' FP64 quotient and reciprocal against IEEE division (numpy's), over the whole range of exponents.

The hardware's estimate carries about 20 bits, a Newton step doubles that, and the last operation rounds once on top
of an error of 2^-80: the result is one of the two doubles around the exact value, at most one ulp from the
rounded one.  Operands that the estimate cannot take go through the division and agree bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ulps(a, b):
    """Distance in representable doubles (same signs)."""
    return np.abs(a.view(np.int64) - b.view(np.int64))


def same(a, b):
    return np.array_equal(np.where(np.isnan(a), 0.0, a), np.where(np.isnan(b), 0.0, b)) and \
        np.array_equal(np.isnan(a), np.isnan(b))


@pytest.mark.parametrize("seed", [0, 1])
def test_within_an_ulp_over_the_range(pkg, gpulib, seed):
    rng = np.random.default_rng(seed)
    n = 400000
    den = rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-1022, 1022, n) * rng.choice([-1.0, 1.0], n)
    num = rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-960, 1000, n)
    exponent = np.log2(num) - np.log2(np.abs(den))
    keep = np.abs(exponent) < 1020            # a normal quotient
    num, den = num[keep], den[keep]
    q, r = pkg.selftest_quotients(num, den)
    assert ulps(q, num / den).max() <= 1
    assert ulps(r, 1.0 / den).max() <= 1


def test_mobility_like_operands(pkg, gpulib):
    rng = np.random.default_rng(3)
    m0, m1 = (rng.uniform(0.0, 1.0, 300000) ** 2 * s for s in (1e3, 1e2))
    m0[:100] = 0.0
    q, _ = pkg.selftest_quotients(m0, m0 + m1)
    assert ulps(q, m0 / (m0 + m1)).max() <= 1
    assert np.all(q[:100] == 0.0) and q.max() <= 1.0


def test_operands_outside_the_estimate(pkg, gpulib):
    tiny, huge = 5e-324, np.finfo(np.float64).max
    special = np.array([0.0, -0.0, tiny, 1e-310, -1e-310, 2.0 ** 1022, 1.5 * 2.0 ** 1022, huge, -huge, np.inf, -np.inf,
                        np.nan])
    num, den = (a.ravel() for a in np.meshgrid(np.array([0.0, 1.0, 3.0, 1e-308, 1e300, huge, np.inf, np.nan]), special))
    with np.errstate(all="ignore"):
        q, r = pkg.selftest_quotients(num, den)
        assert same(q, num / den)
        assert same(r, 1.0 / den)
    # the estimate's first and last operands
    den = np.array([2.0 ** -1022, np.nextafter(2.0 ** 1022, 0.0), 1.0, 3.0])
    q, r = pkg.selftest_quotients(np.ones(4), den)
    assert ulps(r, 1.0 / den).max() <= 1 and ulps(q, 1.0 / den).max() <= 1
