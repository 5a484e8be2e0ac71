"""The FP64 form's own steps of a term, restated with the constants of the kernel's
source: sine and cosine by Cody-Waite reduction and polynomials, division by the
bin spacing by residual steps."""
import os
import re
from fractions import Fraction

import numpy as np

SRC = os.path.join(os.path.dirname(__file__), "..", "srg_b200", "csrc", "bp_kernel.cuh")


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def constants():
    body = open(SRC).read().split("void sincos_pos")[1].split("// quarter turns")[0]
    body = re.sub(r"//.*", "", body)
    num = [float(v) for v in re.findall(r"(?<![\w.])-?\d+\.\d+(?:e[-+]\d+)?", body)]
    magic, twoopi, p2, p1 = num[:4]
    return magic, twoopi, p2, p1, num[4:10], num[10:]


def test_sine_and_cosine():
    magic, twoopi, p2, p1, sc, cc = constants()
    assert len(sc) == 6 and len(cc) == 8 and p1 == -np.pi / 2
    rng = np.random.default_rng(3)
    xs = list(rng.uniform(1.0e8, 3.0e8, 400)) + [0.0, 0.5, np.pi / 4, np.pi / 2, 1e3, 2.0 ** 30 - 1]
    pi = Fraction("3.14159265358979323846264338327950288419716939937510582097494459230781640629")
    for x in xs:
        m = fma(x, twoopi, magic)
        n = m - magic
        r = fma(n, p2, fma(n, p1, x))
        # the reduced argument: to 2^-53 of pi / 4
        exact = Fraction(x) - Fraction(int(n)) * pi / 2
        assert abs(Fraction(r) - exact) <= Fraction(1, 2 ** 53)
        z = r * r
        s = fma(z, sc[0], sc[1])
        for c in sc[2:]:
            s = fma(z, s, c)
        s = fma(z * r, s, r)
        c = fma(z, cc[0], cc[1])
        for k in cc[2:]:
            c = fma(z, c, k)
        q = int(n) & 3
        sn = [s, c, -s, -c][q]
        cs = [c, -s, -c, s][q]
        want = np.longdouble(exact.numerator) / np.longdouble(exact.denominator)
        ws, wc = np.sin(want), np.cos(want)
        ws, wc = [(ws, wc), (wc, -ws), (-ws, -wc), (-wc, ws)][q]
        assert abs(np.longdouble(sn) - ws) <= 2.0 ** -53 * 1.2
        assert abs(np.longdouble(cs) - wc) <= 2.0 ** -53 * 1.2


def test_division_by_the_bin_spacing():
    rng = np.random.default_rng(4)
    for d in [2.329562114, 2.329562114 / 2, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52, *rng.uniform(0.3, 20.0, 40)]:
        inv = 1.0 / d
        for x in [0.0, d, *rng.uniform(0.0, 6.0e4, 150)]:
            q = x * inv
            q = fma(fma(-q, d, x), inv, q)
            q = fma(fma(-q, d, x), inv, q)
            assert q == x / d
