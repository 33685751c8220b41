"""The branch-free elementary functions of the quadrature kernels against exact values (80-bit long double, whose own
error is 2^-11 of the unit used here) and against CUDA's functions on the same arguments.

Unit: 2^-53 absolute for sine and cosine, relative for the others.  Bounds: half a unit for the result's rounding (one
relative unit just above a power of two) and the roundings inside: sine and cosine 0.25 to 0.35 for the polynomials' last
sums and r^2, exp 0.2; none larger than CUDA's largest error.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.fixture(scope="module")
def ctx():
    import bem_b200 as bb
    c = bb.Context(0)
    yield c
    c.close()


def _eval(ctx, fn, x):
    import bem_b200 as bb
    x = np.ascontiguousarray(x, dtype=np.float64)
    own, ref = (np.empty((len(x), 2) if fn in (0, 3) else len(x)) for _ in range(2))
    ctx.check(bb.lib().bem_selftest_math(ctx.h, fn, x.ctypes.data, len(x), own.ctypes.data, ref.ctypes.data))
    return own, ref


def _sine_arguments():
    rng = np.random.default_rng(0)
    n = 400_000
    top = np.nextafter(2.0 ** 20, 0)
    k = rng.integers(0, 667544, n)
    near = k * np.longdouble("1.57079632679489661923132169163975144")
    return np.concatenate([
        rng.uniform(-4, 4, n), rng.uniform(-100, 100, n), rng.uniform(-top, top, n),
        np.exp(rng.uniform(-700, 0, n)), near.astype(float),                          # next to multiples of pi/2
        (near + np.longdouble("0.785398163397448309615660845819875721")).astype(float),  # the ends of the reduced range
        [0.0, -0.0, 5e-324, 2.3e-308, top, -top, np.pi / 4, -np.pi / 4, np.pi / 2, np.pi]])


def test_sine_and_cosine(ctx):
    x = _sine_arguments()
    x = x[np.abs(x) < 2.0 ** 20]
    own, ref = _eval(ctx, 0, x)
    xl = x.astype(np.longdouble)
    for c, f in enumerate((np.sin, np.cos)):
        e, r = (np.abs((v[:, c] - f(xl)).astype(float)) / U for v in (own, ref))
        assert e.max() < 1.16 and e.max() <= r.max() and np.sqrt((e ** 2).mean()) <= np.sqrt((r ** 2).mean()), \
            (e.max(), r.max(), x[e.argmax()])
    small = np.abs(x) < 1e-3  # no cancellation: relative accuracy as well
    e = np.abs((own[small, 0] - np.sin(xl[small])).astype(float))
    assert (e <= 1.01 * U * np.abs(x[small]) + 5e-324).all()
    assert np.isnan(_eval(ctx, 0, [np.nan])[0]).all()


def test_decaying_exponential(ctx):
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.uniform(0, 2, 300_000), rng.uniform(0, 708, 300_000), np.exp(rng.uniform(-700, 6, 300_000)),
                        np.arange(0, 1021) * np.log(2.0), [0.0, 5e-324, 708.0, np.nextafter(708.0, 0)]])
    x = x[x <= 708.0]
    x = np.concatenate([x, -x])
    own, ref = _eval(ctx, 1, x)
    ex = np.exp(-x.astype(np.longdouble))
    e, r = (np.abs(((v - ex) / ex).astype(float)) / U for v in (own, ref))
    assert e.max() < 1.3 and e.max() <= 1.02 * r.max(), (e.max(), r.max(), x[e.argmax()])
    assert (own[x == 0.0] == 1.0).all()
    held = _eval(ctx, 1, [708.0, 708.5, 1e4, 1e300, np.inf])[0]  # no smaller than e^-708
    assert (held == held[0]).all()


def test_reciprocal_square_root(ctx):
    rng = np.random.default_rng(2)
    x = np.concatenate([rng.uniform(0.25, 4, 600_000), np.exp(rng.uniform(-707, 709, 600_000)),
                        [1e-30, 1.0, 4.0, 2.3e-308, 1.7e308]])
    own, ref = _eval(ctx, 2, x)
    ex = 1 / np.sqrt(x.astype(np.longdouble))
    e, r = (np.abs(((v - ex) / ex).astype(float)) / U for v in (own, ref))
    assert e.max() < 1.02 and e.max() <= 1.001 * r.max(), (e.max(), r.max(), x[e.argmax()])


def test_pivot_reciprocal_is_the_division(ctx):
    # a quotient corrected by its remainder is the division's except where the remainder's own rounding meets a tie:
    # none in 1e6 random ones is expected, one unit in the last place would be the difference
    rng = np.random.default_rng(3)
    n = 200_000
    mag = np.exp(rng.uniform(-3, 3, n))[:, None]
    wide = 10.0 ** rng.uniform(-140, 140, n)[:, None]
    skew = np.stack([10.0 ** rng.uniform(-60, 0, n), np.ones(n)], axis=1)
    z = rng.standard_normal((n, 2))
    edge = np.concatenate([z[:50_000] * s for s in (0.9e-145, 1.1e-145, 0.9e145, 1.1e145)])  # |p|^2 at 1e-290 and 1e290
    p = np.concatenate([z * mag, z * wide, z * skew, edge, [[1.0, 0.0], [0.0, -1.0], [1e-300, 0.0], [3.0, 4.0]]])
    own, ref = _eval(ctx, 3, p)
    d = (own != ref) & ~(np.isnan(own) & np.isnan(ref))  # |p|^2 below the smallest number: 0 / 0 in both
    assert d.mean() < 1e-6
    assert (np.abs(own[d] - ref[d]) <= 2 * U * np.abs(ref[d])).all()
