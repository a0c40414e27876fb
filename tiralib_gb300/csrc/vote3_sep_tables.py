"""Makes vote3_sep_tables.inc: |o|^-2k, k = 1, 2, 3, as sums of exponentials
of |o|^2 with shared exponents, for the separable 3D vote (vote3_sep.cu).

    python3 vote3_sep_tables.py > vote3_sep_tables.inc

s = |o|^2 takes the integers 1 .. smax.  For a count T of exponentials, b[0] =
0 and T - 1 free exponents exp(u):

  - weights by linear least squares of the relative residual
    s^k sum_t w_k[t] exp(-b[t] s) - 1, for each k, at 200 values of s at most
    (1 .. 40 and a geometric sequence to smax);
  - the free exponents by nonlinear least squares (trust region) on those
    residuals, started from the T - 1 solution with one exponent more on the
    same curve (T = 4: geometric from 1.2 / smax to 3.2);
  - ten rounds of reweighting: a point's weight times (0.2 + |error| / largest
    error)^0.6, which levels the errors; the round with the smallest largest
    error over every s of 1 .. smax is taken.

Rows: for each half window hw = 2 .. 20, smax = 3 hw^2, the smallest T whose
largest relative error is at most TOL; of the rows of one T the widest.
"""
import numpy as np
from scipy.optimize import least_squares

TOL = 1.5e-7
MAX_HW = 20


def sample(smax):
    near = min(smax, 40)
    return np.unique(np.concatenate([np.arange(1, near + 1), np.round(np.geomspace(near, smax, 160))])).astype(float)


def solve_weights(b, s, level):
    E = np.exp(-np.outer(s, b))
    w, r = [], []
    for k in range(3):
        A = E * (s ** (k + 1) * level[k])[:, None]
        scale = np.abs(A).max(0)
        x = np.linalg.lstsq(A / scale, level[k], rcond=1e-14)[0]
        w.append(x / scale)
        r.append(A @ w[k] - level[k])
    return w, np.concatenate(r)


def largest_error(b, w, smax):
    s = np.arange(1, smax + 1, dtype=float)
    E = np.exp(-np.outer(s, b))
    return max(np.abs(E @ w[k] * s ** (k + 1) - 1).max() for k in range(3))


def fit(u, smax, rounds=10):
    s = sample(smax)
    level = [np.ones_like(s) for _ in range(3)]
    exponents = lambda u: np.concatenate([[0.0], np.exp(u)])
    best = None
    for _ in range(rounds):
        r = least_squares(lambda u: solve_weights(exponents(u), s, level)[1], u, x_scale=0.1, xtol=1e-10, ftol=1e-10,
                          gtol=1e-15, max_nfev=60)
        u = np.sort(r.x)
        b = exponents(u)
        w = solve_weights(b, s, level)[0]
        m = largest_error(b, w, smax)
        if best is None or m < best[0]:
            best = (m, u.copy(), b, w)
        E = np.exp(-np.outer(s, b))
        for k in range(3):
            level[k] = level[k] * (0.2 + np.abs(E @ w[k] * s ** (k + 1) - 1) / m) ** 0.6
        top = max(x.max() for x in level)
        level = [np.maximum(x / top, 1e-4) for x in level]
    return best


def smallest(hw):
    smax = 3 * hw * hw
    u = np.linspace(np.log(1.2 / smax), np.log(3.2), 3)
    while True:
        m, u, b, w = fit(u, smax)
        if m <= TOL:
            return len(b), smax, m, b, w
        n = len(u)
        u = np.interp(np.linspace(0, 1, n + 1), np.linspace(0, 1, n), u) + np.linspace(-0.13, 0.06, n + 1)


def main():
    rows = {}
    for hw in range(2, MAX_HW + 1):
        row = smallest(hw)
        rows[row[0]] = row
    print("// Made by vote3_sep_tables.py, which says how.  {smax, T, {b}, {w1}, {w2}, {w3}}: s^-1, s^-2, s^-3 on")
    print("// s = 1 .. smax, relative error at most %.1e" % max(r[2] for r in rows.values()))
    for T, smax, m, b, w in sorted(rows.values()):
        num = lambda v: "{" + ", ".join("%.17g" % x for x in v) + "}"
        print("    {%d, %d,\n     %s},"  % (smax, T, ",\n     ".join(num(v) for v in (b, *w))))


if __name__ == "__main__":
    main()
