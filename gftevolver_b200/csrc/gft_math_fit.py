"""Regenerates the minimax coefficients of gft_math.cuh (run: python gft_math_fit.py).

Remez exchange (E. Ya. Remez, 1934) in 50-digit arithmetic for the polynomial forms
the kernels evaluate (s = r^2):
  sin r = r + r^3 P(s) on |r| <= pi/2, weighted to the relative error of sin;
  cos r = 1 + s Q(s) on |r| <= pi/2, weighted to the absolute error of cos;
  asin x = x + x^3 A(x^2) on |x| <= 1/4 (float), 1/8 (double), relative error;
  sqrt(1 - c) - 1 = -c/2 + c^2 G(c) on 0 <= c <= 1/64, relative error.
Prints each polynomial's maximum error and its coefficients, lowest order first.
"""
from mpmath import lu_solve, matrix, mp, mpf, pi

mp.dps = 50


def remez(f, w, b, deg, iters=25, grid=4000):
    """Coefficients of the polynomial of degree `deg` that minimises max |w (f - p)| on [0, b], and that maximum."""
    n = deg + 2
    xs = [b / 2 * (1 - mp.cos(pi * k / grid)) for k in range(grid + 1)]
    fx, wx = [f(x) for x in xs], [w(x) for x in xs]
    s = [b / 2 * (1 - mp.cos(pi * k / (n - 1))) for k in range(n)]
    last = None
    for _ in range(iters):
        lhs, rhs = matrix(n, n), matrix(n, 1)
        for i in range(n):
            for j in range(deg + 1):
                lhs[i, j] = s[i] ** j
            lhs[i, deg + 1] = (-1) ** i / w(s[i])
            rhs[i] = f(s[i])
        sol = lu_solve(lhs, rhs)
        c = [sol[j] for j in range(deg + 1)]
        err = [wx[k] * (fx[k] - mp.polyval(c[::-1], xs[k])) for k in range(grid + 1)]
        pts = []
        for i in range(grid + 1):
            if i in (0, grid) or (err[i] - err[i - 1]) * (err[i + 1] - err[i]) <= 0:
                if pts and (err[i] > 0) == (err[pts[-1]] > 0):
                    if abs(err[i]) > abs(err[pts[-1]]):
                        pts[-1] = i
                else:
                    pts.append(i)
        while len(pts) > n:
            pts.pop(0 if abs(err[pts[0]]) < abs(err[pts[-1]]) else -1)
        worst = max(abs(e) for e in err)
        if len(pts) < n or (last is not None and abs(worst - last) < worst * mpf(10) ** -6):
            break
        last, s = worst, [xs[k] for k in pts]
    return c, worst


def power(coef):
    return lambda s: mp.polyval(coef[::-1], s)


TINY = mpf(10) ** -30
SIN = power([mpf((-1) ** (k + 1)) / mp.factorial(2 * k + 3) for k in range(30)])
COS = power([mpf((-1) ** (k + 1)) / mp.factorial(2 * k + 2) for k in range(30)])
ASIN = power([mp.binomial(2 * n, n) / (mpf(4) ** n * (2 * n + 1)) for n in range(1, 40)])
SQRT = power([mp.binomial(mpf(1) / 2, k) * (-1) ** k for k in range(2, 45)])
HALF_PI_SQ = (pi / 2) ** 2 * mpf("1.0000001")

if __name__ == "__main__":
    for name, f, w, b, deg in (
            ("sin float", SIN, lambda s: s / (1 + s * SIN(s)), HALF_PI_SQ, 3),
            ("cos float", COS, lambda s: s, HALF_PI_SQ, 4),
            ("asin float", ASIN, lambda s: s / (1 + s * ASIN(s)), mpf(1) / 16, 3),
            ("sqrt1m float", SQRT, lambda c: c / (mpf(1) / 2 - c * SQRT(c)), mpf(1) / 64, 1),
            ("sin double", SIN, lambda s: s / (1 + s * SIN(s)), HALF_PI_SQ, 7),
            ("cos double", COS, lambda s: s, HALF_PI_SQ, 8),
            ("asin double", ASIN, lambda s: s / (1 + s * ASIN(s)), mpf(1) / 64, 5),
            ("sqrt1m double", SQRT, lambda c: c / (mpf(1) / 2 - c * SQRT(c)), mpf(1) / 64, 5)):
        c, e = remez(f, lambda s, w=w: max(w(s), TINY), b, deg)
        print(f"{name}: error {mp.nstr(e, 3)}, coefficients {[mp.nstr(x, 18, min_fixed=0, max_fixed=0) for x in c]}")
