"""The two series of the device code's power function, read from its source,
against the functions they stand for in 50-digit arithmetic."""
import math
import os
import re
from decimal import Decimal as D, localcontext
from fractions import Fraction

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                      "wdsgpu_b200", "csrc", "wds_math.cuh")


def _coefficients(name, arg):
    txt = open(SOURCE).read()
    hx = [re.search(r"double %s = (0x[0-9a-fp.+-]+);" % name, txt).group(1)]
    hx += re.findall(r"%s = fma\(%s, %s, (0x[0-9a-fp.+-]+)\);" % (name, name, arg), txt)
    fr = [Fraction(float.fromhex(h)) for h in hx]
    return [D(f.numerator) / D(f.denominator) for f in fr]


def _horner(c, x):
    v = D(0)
    for a in c:
        v = v * x + a
    return v


def _series(term):
    s, k = D(0), 0
    while True:
        a = term(k)
        s, k = s + a, k + 1
        if abs(a) < D(10) ** -45:
            return s


def test_series_of_the_logarithm():
    # log2 m = (2 / ln 2) s (1 + z p(z)), s = (m - 1) / (m + 1), z = s^2, for m in
    # [sqrt(1/2), sqrt(2)]: p(z) = sum z^k / (2 k + 3)
    with localcontext() as ctx:
        ctx.prec = 50
        p = _coefficients("p", "z")
        zmax = ((D(2).sqrt() - 1) / (D(2).sqrt() + 1)) ** 2
        err = max(abs(_horner(p, z) - _series(lambda k: z ** k / (2 * k + 3))) * z
                  for z in (zmax * i / 300 for i in range(1, 301)))
    assert len(p) == 8 and math.log2(err) < -60.5


def test_series_of_the_exponential():
    # e^t = 1 + t + t^2 q(t) for |t| <= ln(2) / 2
    with localcontext() as ctx:
        ctx.prec = 50
        q = _coefficients("q", "t")
        h = D(2).ln() / 2
        err = max(abs(1 + t + t * t * _horner(q, t) - t.exp()) / t.exp()
                  for t in (h * i / 150 for i in range(-150, 151)))
    assert len(q) == 11 and math.log2(err) < -61.2
