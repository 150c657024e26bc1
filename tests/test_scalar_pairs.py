"""The resident solve's recursion scalars as pairs of floats (Sc and Scc in
tg_resident.cu), restated in numpy: quotients of random pairs against FP64.
A pair holds about 2^-47 of a value; a complex quotient is three products, two
sums and two divisions of such pairs, so 2^-42 of its magnitude bounds it."""
import numpy as np

f = np.float32


def fma(a, b, c):  # a b exact in FP64; one rounding more than a fused one at most
    return f(np.float64(a) * np.float64(b) + np.float64(c))


def norm(h, l):
    s = f(h + l)
    return s, f(l - f(s - h))


def add(a, b):
    s = f(a[0] + b[0])
    t = f(s - a[0])
    return norm(s, f(f(a[0] - f(s - t)) + f(b[0] - t)) + f(a[1] + b[1]))


def mul(a, b):
    p = f(a[0] * b[0])
    return norm(p, fma(a[0], b[1], fma(a[1], b[0], fma(a[0], b[0], -p))))


def div(a, b):
    q = f(a[0] / b[0])
    return norm(q, f(fma(-q, b[1], f(fma(-q, b[0], a[0]) + a[1])) / b[0]))


def neg(a):
    return -a[0], -a[1]


def cdiv(ax, ay, bx, by):
    m = np.maximum(abs(bx[0]), abs(by[0]))
    s = np.exp2(-np.floor(np.log2(np.float64(m)))).astype(f)
    ax, ay, bx, by = [(f(v[0] * s), f(v[1] * s)) for v in (ax, ay, bx, by)]
    d = add(mul(bx, bx), mul(by, by))
    return div(add(mul(ax, bx), mul(ay, by)), d), div(add(mul(ay, bx), neg(mul(ax, by))), d)


def pair(x):
    h = x.astype(f)
    return h, (x - h).astype(f)


def val(p):
    return np.float64(p[0]) + np.float64(p[1])


def test_quotients():
    rng = np.random.default_rng(7)
    n = 20000
    mag = lambda: rng.standard_normal(n) * 10.0 ** rng.uniform(-12, 4, n)
    a, b = pair(mag()), pair(mag())
    q = val(a) / val(b)
    assert np.max(abs(val(div(a, b)) - q) / abs(q)) < 2.0 ** -44
    v = [pair(mag()) for _ in range(4)]
    z, w = val(v[0]) + 1j * val(v[1]), val(v[2]) + 1j * val(v[3])
    x, y = cdiv(*v)
    assert np.max(abs(val(x) + 1j * val(y) - z / w) / abs(z / w)) < 2.0 ** -42
