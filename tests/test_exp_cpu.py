"""The exponentials of the cooling kernel (exp_n, exp10_n) from the constants in
the source, every operation rounded once in exact rational arithmetic, against
50-digit values: below 1.5 and 2.5 units in the last place over the range in
which they are taken."""
import pathlib
import re
from decimal import Decimal, getcontext
from fractions import Fraction as F
import math

import numpy as np
import pytest

getcontext().prec = 50
TEXT = (pathlib.Path(__file__).resolve().parent.parent / "walicxe2d_b200" / "csrc" / "w2d_cool.cuh").read_text()


def table(name):
    body = re.search(r"\b%s\[\d+\] = \{(.*?)\};" % name, TEXT, re.S).group(1)
    body = re.sub(r"//[^\n]*", "", body)
    return [float.fromhex(x) if "0x" in x else float(x) for x in re.findall(r"-?0x[0-9a-f.p+-]+|-?\d[\d.e+-]*", body)]


E, E10 = table("kExp"), table("kExp10")


def fma(a, b, c):
    return float(F(a) * F(b) + F(c))


def scale(r, t):
    """exp_scale"""
    p = E[4]
    for k in range(5, 15):
        p = fma(p, r, E[k])
    for _ in range(2):
        p = fma(p, r, E[15])
    return p * 2.0 ** int(t - E[1])


def exp_n(x):
    t = fma(x, E[0], E[1])
    n = t - E[1]
    return scale(fma(-n, E[3], fma(-n, E[2], x)), t)


def exp10_n(x):
    t = fma(x, E10[0], E[1])
    n = t - E[1]
    z = fma(-n, E10[2], fma(-n, E10[1], x))
    return scale(fma(z, E10[3], z * E10[4]), t)


def ulps(got, want):
    return abs(Decimal(got) - want) / Decimal(math.ulp(float(want)))


def points(limit, unit, rng):
    """Random arguments, small ones, the ends, and both sides of where the
    reduction changes its multiple."""
    k = rng.integers(-int(limit / unit) + 1, int(limit / unit), 150) + 0.5
    near = k * unit
    return np.concatenate([rng.uniform(-limit, limit, 600), rng.uniform(-1, 1, 100), 10.0 ** rng.uniform(-20, 0, 50),
                           -10.0 ** rng.uniform(-20, 0, 50), near, np.nextafter(near, np.inf),
                           np.nextafter(near, -np.inf), [0.0, -0.0, np.nextafter(limit, 0), -np.nextafter(limit, 0)]])


# The result 1 + r (1 + r g), |r| <= 0.347: the last operation rounds by half a
# unit, the one before by a quarter at most, the reduced argument's rounding (of
# 0.35 at most) and the fit (2^-61) add less than a half.  10^x carries r through
# three more roundings.
@pytest.mark.parametrize("f,base,limit,unit,bound", [(exp_n, None, 700.0, math.log(2.0), 1.5),
                                                     (exp10_n, Decimal(10), 300.0, math.log10(2.0), 2.5)])
def test_exponential(f, base, limit, unit, bound):
    worst = 0
    for x in points(limit, unit, np.random.default_rng(7)):
        x = float(x)
        want = Decimal(x).exp() if base is None else (Decimal(x) * base.ln()).exp()
        worst = max(worst, ulps(f(x), want))
    assert worst < bound, worst
    print(f.__name__, "worst error in ulp", float(worst))


def test_exponentials_of_zero():
    assert exp_n(0.0) == exp_n(-0.0) == exp10_n(0.0) == 1.0
