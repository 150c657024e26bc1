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
    r = f(f(1) / b[0])
    q = f(a[0] * r)
    return norm(q, f(fma(-q, b[1], f(fma(-q, b[0], a[0]) + a[1])) * r))


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


def mac(s, a, b):  # ff2_mac, one lane
    p = f(a[0] * b[0])
    e = fma(a[1], b[0], fma(a[0], b[1], fma(a[0], b[0], -p)))
    t = f(s[0] + p)
    q = f(t - s[0])
    return t, f(s[1] + f(f(f(s[0] - f(t - q)) + f(p - q)) + e))


def nms(c, a, b):  # c - a b, complex
    (ar, ai), (br, bi) = a, b
    return (mac(mac(c[0], neg(ar), br), ai, bi), mac(mac(c[1], neg(ar), bi), neg(ai), br))


def test_row_elimination():
    """A row of the approximate inverse's factor (L D L^T of the row's matrix and
    L^T y = e_m) in pairs against FP64, on random complex symmetric matrices with
    dominant diagonals.  m <= 16 steps of products good to 2^-44, of values that
    stay below the diagonal: 2^-38 of the row's largest entry bounds them."""
    rng = np.random.default_rng(3)
    n = 500
    split = lambda z: (pair(np.ascontiguousarray(z.real)), pair(np.ascontiguousarray(z.imag)))
    for m in (1, 2, 5, 16):
        B = rng.uniform(-1, 0, (n, m, m)) + 1j * rng.uniform(0, 0.3, (n, m, m))
        B = (B + B.transpose(0, 2, 1)) / 2
        B[:, range(m), range(m)] = (0.1 + abs(B).sum(2)) * (1 + 0.2j)
        M = [[split(B[:, a, b]) for b in range(m)] for a in range(m)]
        D = B.copy()
        for j in range(m):
            d = norm(*M[j][j][0]), norm(*M[j][j][1])
            lp = {r: cdiv(norm(*M[r][j][0]), norm(*M[r][j][1]), *d) for r in range(j + 1, m)}
            ld = {r: D[:, r, j] / D[:, j, j] for r in lp}
            for r in lp:
                for c in range(j + 1, r + 1):
                    M[r][c] = nms(M[r][c], lp[r], M[c][j])
                    D[:, r, c] = D[:, r, c] - ld[r] * D[:, c, j]
            for r in lp:
                M[r][j], D[:, r, j] = lp[r], ld[r]
        e = np.eye(m)[m - 1]
        t, u = [split(np.full(n, x + 0j)) for x in e], [np.full(n, x + 0j) for x in e]
        for r in range(m - 1, 0, -1):
            for c in range(r):
                t[c], u[c] = nms(t[c], M[r][c], t[r]), u[c] - D[:, r, c] * u[r]
        y = np.array([val(x[0]) + 1j * val(x[1]) for x in t])
        assert np.max(abs(y - np.array(u)) / np.max(abs(np.array(u)), axis=0)) < 2.0 ** -38
        dm = val(M[m - 1][m - 1][0]) + 1j * val(M[m - 1][m - 1][1])
        assert np.max(abs(dm / D[:, m - 1, m - 1] - 1)) < 2.0 ** -38
