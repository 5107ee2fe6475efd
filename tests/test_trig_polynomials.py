"""The polynomials of the batched FP64 sines and cosines (scp_b200/csrc/trig.cuh)
on the CPU: read from the source, evaluated in 40 digits for their truncation
errors, and fitted again by the same Remez exchange (on the absolute error of the
function, the first term held fixed, coefficients rounded to double)."""
import os
import re

import pytest

mpmath = pytest.importorskip("mpmath")
mp, mpf = mpmath.mp, mpmath.mpf

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "scp_b200", "csrc", "trig.cuh")
HEX = r"-?0x[0-9a-f.]+p[-+]\d+"


def coefficients():
    """Lowest power of s = r^2 first: sine and cosine to pi/4, sine to pi/2."""
    text = open(SOURCE).read()
    pair, sine = text.index("void sincos_batch("), text.index("void sin_batch(")

    def horner(body, name):
        first = re.search(r"double %s = __fma_rn\((%s), s, (%s)\);" % (name, HEX, HEX), body)
        rest = re.findall(r"\b%s = __fma_rn\(%s, s, (-?[0-9a-fx.p+-]+)\);" % (name, name), body)
        c = [first.group(1), first.group(2), *rest]
        return [float.fromhex(v) if "0x" in v else float(v) for v in reversed(c)]

    return horner(text[pair:sine], "p"), horner(text[pair:sine], "c"), horner(text[sine:], "p")


def functions(kind):
    """What the polynomial in s stands for, and the weight of its error:
    sin r = r + r s p(s), cos r = 1 + s q(s)."""
    if kind == "sin":
        return (lambda s: (mp.sin(mp.sqrt(s)) - mp.sqrt(s)) / (mp.sqrt(s) * s)), (lambda s: mp.sqrt(s) * s)
    return (lambda s: (mp.cos(mp.sqrt(s)) - 1) / s), (lambda s: s)


def remez(f, w, n, a, b):
    """Polynomial of degree n with the least maximum of |w (p - f)| on [a, b]."""
    m = n + 2
    xs = [(a + b) / 2 - (b - a) / 2 * mp.cos(mp.pi * mpf(i) / (m - 1)) for i in range(m)]
    grid = [a + (b - a) * mpf(i) / 2000 for i in range(2001)]
    for _ in range(30):
        A, B = mp.matrix(m, m), mp.matrix(m, 1)
        for i, x in enumerate(xs):
            for j in range(n + 1):
                A[i, j] = x ** j
            A[i, n + 1] = (-1) ** i / w(x)
            B[i] = f(x)
        c = [v for v in mp.lu_solve(A, B)][:n + 1]
        err = [w(x) * (mp.polyval(c[::-1], x) - f(x)) for x in grid]
        peaks = []
        for i, e in enumerate(err):
            sign = 1 if e > 0 else -1
            if all(sign * e >= sign * err[k] for k in (i - 1, i + 1) if 0 <= k < len(err)):
                if peaks and (peaks[-1][1] > 0) == (e > 0):
                    if abs(e) > abs(peaks[-1][1]):
                        peaks[-1] = (grid[i], e)
                else:
                    peaks.append((grid[i], e))
        while len(peaks) > m:
            peaks.pop(0 if abs(peaks[0][1]) < abs(peaks[-1][1]) else -1)
        if len(peaks) < m:
            break
        new = [x for x, _ in peaks]
        done = max(abs(p - q) for p, q in zip(new, xs)) < mpf(10) ** -6
        xs = new
        if done:
            break
    return c


# stated in the source: 8e-18, 2e-18, 4e-17
@pytest.mark.parametrize("which,kind,edge,bound", [(0, "sin", 0.25, 8.5e-18), (1, "cos", 0.25, 2.5e-18),
                                                   (2, "sin", 0.5, 4.5e-17)])
def test_truncation_and_fit(which, kind, edge, bound):
    mp.dps = 60
    have = coefficients()[which]
    f, w = functions(kind)
    R = mp.pi * edge
    worst = max(abs(w(x * x) * (mp.polyval([mpf(c) for c in reversed(have)], x * x) - f(x * x)))
                for x in (R * mpf(i) / 1500 for i in range(1, 1501)))
    assert worst <= bound, mp.nstr(worst, 5)
    fit = remez(f, w, len(have) - 1, mpf(10) ** -8, R * R * (1 + mpf(10) ** -6))
    assert [float(c) for c in fit] == have
