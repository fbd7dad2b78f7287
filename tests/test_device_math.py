"""The straight-line functions of csrc/device against long double (64 bits of
significand), on the host: random arguments over their ranges and the hard ones."""
import numpy as np
import pytest

from device_math import call, ulps, values

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


def pairs(bits, count, seed):
    """Dividends and divisors: random significands, ones near 1 and 2, quotients
    next to the middle between two numbers (a = b m rounded, m a bit longer than a
    number), moderate and extreme exponents, and specials in every combination."""
    kind, word = (np.float64, np.int64) if bits == 53 else (np.float32, np.int32)
    rng = np.random.default_rng(seed)
    top, wide = (1 << (bits - 1)), (40 if bits == 53 else 15)

    def significand():
        m = rng.integers(top, 2 * top, count)
        near = rng.random(count)
        m = np.where(near < 0.1, top + rng.integers(0, 64, count), m)
        return np.where(near > 0.9, 2 * top - 1 - rng.integers(0, 64, count), m)

    a, b = significand().astype(kind), significand().astype(kind)
    middle = (2 * significand() + 1).astype(np.longdouble) * b.astype(np.longdouble)
    a = np.where(rng.random(count) < 0.5, a, (middle * np.ldexp(np.longdouble(1), -bits)).astype(kind))
    a = (np.ldexp(a, rng.integers(-wide, wide, count)) * rng.choice([-1, 1], count)).astype(kind)
    b = (np.ldexp(b, rng.integers(-wide, wide, count)) * rng.choice([-1, 1], count)).astype(kind)
    extreme = rng.integers(0, 1 << (63 if bits == 53 else 31), count // 10).astype(word).view(kind)
    a[:extreme.size], b[-extreme.size:] = extreme, extreme[::-1]
    i = np.finfo(kind)
    special = np.array([0.0, i.smallest_subnormal, i.tiny, i.max, np.inf, np.nan, 1.0, 3.0, 2.0, i.eps, 1 - i.epsneg], kind)
    special = np.concatenate([special, -special])
    return (np.concatenate([a, np.repeat(special, special.size)]).astype(kind),
            np.concatenate([b, np.tile(special, special.size)]).astype(kind))


def check_quotients(name, a, b, covered):
    """Bit for bit, the sign of a zero too, wherever the function does not say that it is outside."""
    q, outside = np.empty_like(a), np.empty(a.size, dtype=np.uint8)
    call(name, a, b, q, outside)
    with np.errstate(all="ignore"):
        want = a / b
    word = np.int64 if a.dtype == np.float64 else np.int32
    inside = outside == 0
    nan = np.isnan(want)
    assert np.isnan(q[inside & nan]).all()
    same = inside & ~nan
    np.testing.assert_array_equal(q[same].view(word), want[same].view(word))
    assert not outside[covered].any()


@pytest.mark.parametrize("name", ["chain", "straight"])
def test_quotients_have_the_ieee_quotients_bits(name):
    a, b = pairs(53, 2000000, 4)
    with np.errstate(all="ignore"):
        moderate = ((np.abs(a) > 1e-20) & (np.abs(a) < 1e40) | ((a == 0) & ~np.signbit(a))) & \
            (np.abs(b) > 1e-20) & (np.abs(b) < 1e28) & (np.frexp(np.abs(b))[0] != 1 - 2.0 ** -53)
    check_quotients(name + "_quotients", a, b, moderate)


def test_float_quotients_have_the_ieee_quotients_bits():
    a, b = pairs(24, 2000000, 5)
    a = np.concatenate([a, np.float32([float.fromhex("0x1.d074d8p+0")])])
    b = np.concatenate([b, np.float32([float.fromhex("0x1.527e7cp+0")])])
    moderate = ((np.abs(a) > 1e-30) & (np.abs(a) < 1e30) | ((a == 0) & ~np.signbit(a))) & (np.abs(b) > 1e-7) & (np.abs(b) < 1e7)
    check_quotients("straight_quotients_f32", a, b, moderate)
