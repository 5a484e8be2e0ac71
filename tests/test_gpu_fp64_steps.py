"""The FP64 form's own steps as device code: square root and division bit for bit
the correctly rounded ones, sine and cosine within their stated bound."""
import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

from srg_b200 import _lib

PI = Fraction("3.14159265358979323846264338327950288419716939937510582097494459230781640629")


def steps(x, d):
    import torch
    x, d = (torch.from_numpy(np.ascontiguousarray(v, np.float64)).cuda() for v in (x, d))
    out = [torch.empty_like(x) for _ in range(4)]
    _lib.check(_lib.lib().srg_test_fp64_steps_device(
        *[C.c_void_p(t.data_ptr()) for t in (x, d)], x.numel(), *[C.c_void_p(t.data_ptr()) for t in out],
        C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    return [t.cpu().numpy() for t in out]


def bits(a):
    return np.ascontiguousarray(a).view(np.uint64)


@pytest.mark.gpu
def test_square_root():
    rng = np.random.default_rng(1)
    r = rng.uniform(6e5, 1.3e6, 1 << 20)            # slant ranges
    g = rng.uniform(1.0, 4.0, 1 << 18)
    near = np.concatenate([r, g])
    sq = near * near                                # roots next to a double
    half = sq * (1.0 + np.spacing(near) / near)     # and next to a midpoint of two
    x = np.concatenate([rng.uniform(3e11, 2e12, 1 << 20), sq, np.nextafter(sq, 0), np.nextafter(sq, 9e99),
                        half, np.nextafter(half, 0), np.nextafter(half, 9e99),
                        2.0 ** rng.uniform(-900, 1000, 1 << 18), [1.0, 2.0, 4.0, 2.0 ** -900, 2.0 ** 1000]])
    got = steps(x, np.ones_like(x))[0]
    assert np.array_equal(bits(got), bits(np.sqrt(x)))


@pytest.mark.gpu
def test_division():
    rng = np.random.default_rng(2)
    n = 1 << 20
    d = np.concatenate([rng.uniform(0.3, 20.0, n), -rng.uniform(0.3, 20.0, n),         # bin spacings
                        rng.uniform(-60.0, 60.0, n),                                    # time differences
                        np.repeat([1.0, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52, 2.329562114, 10.0, -10.0, 1e-3], 4096)])
    x = rng.uniform(-6e4, 6e4, d.size)
    q = np.rint(rng.uniform(2.0 ** 52, 2.0 ** 53, d.size))
    mid = (q + 0.5 * rng.integers(0, 2, d.size)) * d * 2.0 ** -40                       # quotients next to a midpoint
    small = x * 2.0 ** rng.uniform(-900, -200, d.size)
    for v in (x, mid, np.nextafter(mid, 9e99), np.nextafter(mid, -9e99), small,
              np.zeros_like(x), np.copysign(np.zeros_like(x), -1.0)):
        got = steps(v, d)[1]
        assert np.array_equal(bits(got), bits(v / d))


def reduced(x):
    """x less the nearest multiple n of pi/2 in 80 bits, and n mod 4."""
    a = Fraction(int(PI / 2 * 2 ** 32), 2 ** 32)          # 33 bits: n a is exact in 64
    b = Fraction(int((PI / 2 - a) * 2 ** 65), 2 ** 65)
    c = PI / 2 - a - b
    n = np.rint(x * 0.63661977236758138)
    xl, nl = x.astype(np.longdouble), n.astype(np.longdouble)
    ld = lambda f: np.longdouble(f.numerator) / np.longdouble(f.denominator)  # noqa: E731
    return ((xl - nl * ld(a)) - nl * ld(b)) - nl * ld(c), n.astype(np.int64) & 3


def test_reduction_of_the_reference():
    x = np.random.default_rng(5).uniform(0, 2.0 ** 30, 500)
    r, q = reduced(x)
    for xi, ri, qi in zip(x, r, q):
        n = int(np.rint(xi * 0.63661977236758138))
        exact = Fraction(xi) - n * PI / 2
        assert abs(Fraction(*map(int, ri.as_integer_ratio())) - exact) < Fraction(1, 2 ** 61) and qi == n & 3


@pytest.mark.gpu
def test_sine_and_cosine():
    rng = np.random.default_rng(3)
    k = rng.integers(0, 683565275, 1 << 16)
    near = k * (np.pi / 2)                                # next to multiples of pi/2
    x = np.concatenate([rng.uniform(0, 2.0 ** 30, 1 << 19), rng.uniform(0, 10.0, 1 << 18), near,
                        np.nextafter(near, 9e99), 10.0 ** rng.uniform(-12, 0, 1 << 14), (k + 0.5) * (np.pi / 2),
                        [0.0, 0.5, np.pi / 4, np.nextafter(2.0 ** 30, 0)]])
    x = x[x < 2.0 ** 30]
    sn, cs = steps(x, np.ones_like(x))[2:]
    r, q = reduced(x)
    s, c = np.sin(r), np.cos(r)
    ws = np.choose(q, [s, c, -s, -c])
    wc = np.choose(q, [c, -s, -c, s])
    bound = np.longdouble(1.2 * 2.0 ** -53)
    assert np.abs(sn - ws).max() <= bound
    assert np.abs(cs - wc).max() <= bound
