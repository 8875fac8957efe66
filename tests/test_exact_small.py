"""The steps of gp_exact.cuh that round upwards or downwards, or that stop at an
approximation, checked for every significand of 4 to 12 bits: the same sequence of
roundings with a significand of P bits, in float64, which holds every product and
sum below exactly.

* inv_in: the last-but-one iterate is 1/b to a relative 2^-58 = 2^-(P+5), rounded
  upwards; one more Newton step then rounds correctly, for the all-ones significand
  too.  (Rounded to nearest it does not: the test says where.)
* quot_bpos: the remainder rounded to nearest or downwards, the quotient is RN(a/b).
* root: h = y/2 with y within 0.55 ulp of a^(-1/2) gives RN(sqrt(a)).

What the device's seeds have to be for that is derived in gp_exact.cuh and measured in
test_gpu_exact.py."""
import numpy as np
import pytest

P_ALL = range(4, 13)


def grid(x, P):
    """Spacing of the P-bit numbers at x > 0."""
    return np.ldexp(1.0, np.frexp(x)[1] - P)


def rnd(x, P, how=np.rint):
    """x (exact in float64) to P bits: np.rint to nearest even, np.floor, np.ceil."""
    u = grid(np.abs(x) + (x == 0), P)
    return how(x / u) * u


def significands(P):
    return np.arange(2 ** (P - 1), 2 ** P, dtype=np.float64)


def rn_quotient(a, b, P):
    """RN(a/b) of P-bit integers, from the exact comparison with the midpoint."""
    u = grid(a / b, P)
    lo = np.floor(a / b / u)
    twice, mid = 2.0 * a, (2.0 * lo + 1.0) * u * b
    up = (twice > mid) | ((twice == mid) & (lo % 2 == 1))
    return (lo + up) * u


def newton(y1, b, P):
    return rnd(y1 + rnd(1.0 - b * y1, P) * y1, P)


@pytest.mark.parametrize("P", P_ALL)
def test_reciprocal(P):
    b = significands(P)
    y = rn_quotient(np.ones_like(b), b, P)
    nearest = np.zeros(b.shape, bool)
    for k in np.linspace(-1.0, 1.0, 33):
        v = (1.0 / b) * (1.0 + k * 2.0 ** -(P + 5))
        np.testing.assert_array_equal(newton(rnd(v, P, np.ceil), b, P), y)
        nearest |= newton(rnd(v, P), b, P) != y
    # Markstein's exception, which rounding upwards removes
    assert set(b[nearest]) <= {2.0 ** P - 1}


@pytest.mark.parametrize("P", P_ALL)
def test_quotient(P):
    a = significands(P)[:, None]
    b = significands(P)[None, :]
    y = rn_quotient(np.ones_like(b), b, P)
    want = rn_quotient(a + 0 * b, b + 0 * a, P)
    q = rnd(a * y, P)
    for how in (np.rint, np.floor):
        r = rnd(a - b * q, P, how)
        np.testing.assert_array_equal(rnd(q + r * y, P), want)


@pytest.mark.parametrize("P", P_ALL)
def test_root(P):
    n = 0
    for scale in (1.0, 2.0):        # both parities of the exponent
        a = significands(P) * scale
        x = 1.0 / np.sqrt(a)
        u = grid(x, P)
        s = np.sqrt(a)              # never a midpoint of P bits, so RN of RN is RN
        want = rnd(s, P)
        for y in (np.floor(x / u) * u, np.ceil(x / u) * u):
            ok = np.abs(y - x) <= 0.55 * u
            g = rnd(a * y, P)
            got = rnd(g + rnd(a - g * g, P) * (0.5 * y), P)
            np.testing.assert_array_equal(got[ok], want[ok])
            n += ok.sum()
    assert n >= 2 ** P
