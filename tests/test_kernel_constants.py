"""Constants of the CUDA kernel that stand for exact decisions of the
reference's arithmetic."""
import math
import os
import re

import pytest

CUH = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "odevec_b200", "csrc",
                   "bdf_kernel.cuh")


def _tau(order, order2):
    """src/odevec.F90:1034-1054 with IEEE doubles"""
    last = [0.0, 1.0, 1.0 / 3.0, 1.0 / 11.0, 1.0 / 50.0, 1.0 / 274.0, 1.0 / 1764.0]
    fac = 1.0
    for i in range(1, order + 1):
        fac = fac * i
    if order - 1 == order2:
        return (order2 + 1.0) / fac
    return (order2 + 1.0) / (fac * last[order])


@pytest.mark.parametrize("q", [1, 2, 3, 4, 5])
def test_local_error_bound(q):
    """c_lte[q] is the smallest double x for which sqrt(x) / tau(q,q) > 1."""
    text = open(CUH).read()
    vals = re.search(r"c_lte\[6\] = \{([^}]*)\}", text).group(1).split(",")
    x = float.fromhex(vals[q].strip())
    tau = _tau(q, q)
    assert math.sqrt(x) / tau > 1.0
    assert not math.sqrt(math.nextafter(x, 0.0)) / tau > 1.0


@pytest.mark.parametrize("q", [1, 2, 3, 4, 5])
def test_convergence_quotient(q):
    """a / D < 1 for the rounded quotient exactly when a < D, next to D."""
    D = _tau(q, q) / (2.0 * (q + 2.0))
    a = D
    for _ in range(40):
        assert (a / D < 1.0) == (a < D)
        a = math.nextafter(a, 0.0)
    a = D
    for _ in range(40):
        assert (a / D < 1.0) == (a < D)
        a = math.nextafter(a, math.inf)


@pytest.mark.parametrize("mantissa", ["random", "small", "large"])
def test_reciprocal_iteration(mantissa):
    """The kernel's branch-free reciprocal: three Newton steps with exact
    residuals from an estimate good to about 20 bits give the correctly
    rounded 1/x, whichever way the estimate is off, for every significand but
    the all-ones one (which the kernel sends to the IEEE reciprocal)."""
    import random
    from fractions import Fraction as F
    rng = random.Random(7)
    fma = lambda a, b, c: float(F(a) * F(b) + F(c))
    for _ in range(400):
        m = {"random": rng.getrandbits(52), "small": rng.getrandbits(6),
             "large": (1 << 52) - 2 - rng.getrandbits(6)}[mantissa]
        x = math.ldexp(1.0 + m * 2.0 ** -52, rng.randint(-900, 900))
        want = float(1 / F(x))
        for off in (-1.0, -0.3, 0.0, 0.4, 1.0):
            r = want * (1.0 + off * 2.0 ** -20)
            for _ in range(3):
                r = fma(fma(-x, r, 1.0), r, r)
            assert r == want


@pytest.mark.parametrize("kind", ["pivot", "count"])
def test_quotient_iteration(kind):
    """The kernel's branch-free quotients -- by a pivot, and by a species count
    that is no power of two -- are correctly rounded: the product with the
    rounded reciprocal, corrected twice with its exact residual."""
    import random
    from fractions import Fraction as F
    rng = random.Random(11)
    fma = lambda a, b, c: float(F(a) * F(b) + F(c))
    for _ in range(3000):
        if kind == "pivot":
            d = math.ldexp(1.0 + rng.choice([rng.getrandbits(52), rng.getrandbits(4), (1 << 52) - 2 - rng.getrandbits(4)])
                           * 2.0 ** -52, rng.randint(-390, 390)) * rng.choice([-1.0, 1.0])
            e = rng.randint(-490, 490)
        else:
            d, e = float(rng.choice([3, 5, 6, 7, 9, 12])), rng.randint(-890, 990)
        x = math.ldexp(1.0 + rng.choice([rng.getrandbits(52), rng.getrandbits(4), (1 << 52) - 1 - rng.getrandbits(4)])
                       * 2.0 ** -52, e)
        r = 1.0 / d
        q = x * r
        q = fma(fma(-q, d, x), r, q)
        q = fma(fma(-q, d, x), r, q)
        assert q == x / d


def test_no_rule_for_one_chip():
    """The launch rules take the SM count from the device."""
    csrc = os.path.dirname(CUH)
    for name in os.listdir(csrc):
        if name.endswith((".cuh", ".cu", ".h", ".hpp")):
            code = re.sub(r"/\*.*?\*/|//[^\n]*", "", open(os.path.join(csrc, name)).read(), flags=re.S)
            assert not re.search(r"\b148\b", code), name


def _exponents(pattern):
    """[lo, hi) of the binary exponents that a range test of the kernel lets
    through: upper word - (lo << 20) >= (span << 20) is outside"""
    lo, span = map(int, re.search(pattern, open(CUH).read(), re.S).groups())
    return lo - 1023, lo - 1023 + span


RANGE = r"\((\d+)u << 20\) >= \((\d+)u << 20\)"


@pytest.mark.parametrize("kind", ["weight", "pivot", "count"])
def test_branch_free_ranges(kind):
    """At the ends of the ranges that the kernel's own tests let through, the
    branch-free reciprocals and quotients are correctly rounded and nothing
    on the way under- or overflows."""
    from fractions import Fraction as F
    fma = lambda a, b, c: float(F(a) * F(b) + F(c))
    values = lambda lo, hi: [math.ldexp(1.0 + m * 2.0 ** -52, e) for e in (lo, lo + 1, hi - 2, hi - 1)
                             for m in (0, 1, 0x5555555555555, 0xaaaaaaaaaaaab, (1 << 52) - 2)]

    def reciprocal(x):
        want = float(1 / F(x))
        for off in (-1.0, 1.0):
            r = want * (1.0 + off * 2.0 ** -20)
            for _ in range(3):
                r = fma(fma(-x, r, 1.0), r, r)
            assert r == want
        return want

    if kind == "weight":
        for x in values(*_exponents(r"unsigned rcp_odd\(.*?" + RANGE)):
            reciprocal(x)
        return
    if kind == "pivot":
        divisors = values(*_exponents(r"ov_pivot\(const PivotRef& p\).*?" + RANGE))
        xs = values(*_exponents(r"ov_divp\(T x, const PivotRef& p\).*?" + RANGE))
    else:
        divisors = [3.0, 5.0, 6.0, 7.0, 9.0, 12.0]
        xs = values(*_exponents(r"double div_n\(double x\).*?" + RANGE))
    for d in divisors:
        r = reciprocal(d)
        for x in xs:
            q = x * r
            q = fma(fma(-q, d, x), r, q)
            q = fma(fma(-q, d, x), r, q)
            assert q == x / d and abs(q) >= 2.0 ** -1022
