"""The straight-line functions of csrc/device against long double (64 bits of
significand), on the host: random arguments over their ranges and the hard ones."""
import numpy as np
import pytest

from device_math import ulps, values

# pi/2 in long double and the rest, for the doubles nearest to its multiples
HALF_PI = np.longdouble("1.57079632679489661923132169163975144")


def near_multiples(count=20000, seed=1):
    n = np.concatenate([np.arange(1, 4001), np.exp2(np.random.default_rng(seed).uniform(0, 29.3, count)).astype(np.int64),
                        [5, 116, 105577836, 513943970, 589193354]])
    x = (n.astype(np.longdouble) * HALF_PI).astype(np.float64)
    x = np.concatenate([x, np.nextafter(x, 0), [2915.397982531328, 925515306.8978163]])
    return np.concatenate([x, -x])


@pytest.mark.parametrize("fn", ["sin", "cos"])
def test_sin_and_cos_over_their_range(fn):
    """Half an ulp for the sum's rounding, 0.87 for that of the reduced argument
    (half an ulp of it where the sine has passed to the binade below), 0.1 for
    the polynomial and its products: 1.5 ulp, next to a zero of the function too;
    the mean of the library's, 0.30; never beyond 1."""
    rng = np.random.default_rng(0)
    x = np.concatenate([rng.uniform(-r, r, 40000) for r in (1.0, 10.0, 1e3, 1e6, 2.0 ** 30)])
    y = values(fn, x)
    off = ulps(y, getattr(np, fn)(x.astype(np.longdouble)))
    assert off.max() <= 1.5 and off.mean() <= 0.30
    x = near_multiples()
    x = x[np.abs(x) <= 2.0 ** 30]
    near = values(fn, x)
    assert ulps(near, getattr(np, fn)(x.astype(np.longdouble))).max() <= 1.5
    assert max(np.abs(y).max(), np.abs(near).max()) <= 1
    small = np.array([0.0, -0.0, 5e-324, -1e-310, 1e-9, -1e-8])
    np.testing.assert_array_equal(values(fn, small), getattr(np, fn)(small))
    np.testing.assert_array_equal(np.signbit(values(fn, small)), np.signbit(getattr(np, fn)(small)))


def test_exp_over_its_range():
    """Half an ulp for the sum's rounding, a quarter for that of the reduced
    argument, the polynomial's 0.05: 0.8 ulp, and a mean below the library's."""
    rng = np.random.default_rng(2)
    x = np.concatenate([rng.uniform(-r, r, 40000) for r in (0.35, 0.7, 10.0, 707.99)])
    off = ulps(values("exp", x), np.exp(x.astype(np.longdouble)))
    assert off.max() <= 0.8 and off.mean() <= 0.257
    small = np.array([0.0, -0.0, 5e-324, -1e-310, 1e-20])
    np.testing.assert_array_equal(values("exp", small), np.ones(5))


def test_log_and_sqrt_of_the_noise():
    """The generator's arguments, multiples of 2^-54 in (0, 1), and others: half an
    ulp for the last rounding, 0.06 for the terms behind it; the root is
    correctly rounded."""
    rng = np.random.default_rng(3)
    u = (1 + rng.integers(0, 1 << 53, 100000)).astype(float) * float.fromhex("0x1.fffffffffffffp-54")
    ends = np.array([2.0 ** -54, 1 - 2.0 ** -53, 0.5, np.nextafter(0.5, 0), np.sqrt(0.5), 1e-8, 1 - 1e-8, 1.0, 1 + 1e-8, 1e300])
    x = np.concatenate([u, u ** 8, ends])
    off = ulps(values("log", x), np.log(x.astype(np.longdouble)))
    assert off.max() <= 0.56 and off[:u.size].mean() <= 0.2505
    r = -2.0 * values("log", x[x < 1])
    r = np.concatenate([r, np.exp(rng.uniform(-300, 300, 100000))])
    np.testing.assert_array_equal(values("sqrt", r), np.sqrt(r))
