"""GPU: the radial solver's own divisions (radial.cu) against the correctly rounded quotient, which is what CUDA's
division and numpy's give.

`quotient` promises the correctly rounded quotient wherever that is 2^-50 units in the last place or more from
the middle of two neighbouring numbers, and one of the two there.  Random operands come that close with odds of
2^-49 each, so they are held to equality; operands made to come close are held to the promise
in exact arithmetic.  The factors, the solution and the counts of a tridiagonal matrix are held to the
recurrences with plain divisions, bit for bit.
"""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 1e-14


def _quotients(engine, a, g):
    out = engine.array(a.size)
    engine.radial_quotients(a.size, engine.upload(a), engine.upload(g), out)
    return out.to_host()


# exponents of a and g: alike; a Sturm count's and a factor's (off^2 or off over pivots from the guard to the
# largest diagonal); the ends of the range
@pytest.mark.parametrize("ea,eg", [((0, 1), (0, 1)), ((20, 40), (-46, 40)), ((-60, 60), (-60, 60)),
                                   ((-100, -98), (97, 99)), ((97, 99), (-100, -98))])
def test_random_quotients(engine, ea, eg):
    rng = np.random.default_rng(ea[0] + 1000)
    m = 1 << 22
    for _ in range(4):
        a, g = [np.ldexp(rng.uniform(1.0, 2.0, m), rng.integers(*e, m)) * rng.choice([-1.0, 1.0], m) for e in (ea, eg)]
        assert np.array_equal(_quotients(engine, a, g), a / g)


def test_exact_quotients(engine):
    """Representable quotients, the middle of two numbers excluded by construction: equality."""
    rng = np.random.default_rng(3)
    q = rng.integers(1 << 25, 1 << 26, 1 << 20).astype(np.float64)
    g = rng.integers(1 << 25, 1 << 26, 1 << 20).astype(np.float64)
    assert np.array_equal(_quotients(engine, q * g, g), q)


def _near_middle(rng, count, r):
    """Pairs (a, g) of 53-bit integers with a 2^54 = M g +- r for an odd 54-bit M: a / g is r / g of half a unit from
    the middle of two neighbouring numbers."""
    a, g = [], []
    while len(a) < count:
        G = int(rng.integers(1 << 52, 1 << 53)) | 1
        s = int(rng.choice([-1, 1])) * r
        M = (-s * pow(G, -1, 1 << 54)) % (1 << 54)
        if M < 1 << 53 or not M & 1:
            continue
        A = (M * G + s) >> 54
        if (M * G + s) != A << 54 or not 1 << 51 <= A < 1 << 53:
            continue
        a.append(A)
        g.append(G)
    return np.array(a, dtype=np.float64), np.array(g, dtype=np.float64)


@pytest.mark.parametrize("r", [1, 3, 5, 7])
def test_quotients_next_to_the_middle_of_two_numbers(engine, r):
    a, g = _near_middle(np.random.default_rng(r), 3000, r)
    q, near = _quotients(engine, a, g), a / g
    off = 0
    for x, y, p, e in zip(a, g, q, near):
        if p == e:
            continue
        off += 1
        # the other neighbour, and no further than half a unit and 2^-50 of one
        assert p in (np.nextafter(e, 0.0), np.nextafter(e, np.inf))
        d = abs(Fraction(float(p)) - Fraction(float(x)) / Fraction(float(y)))
        assert d <= (Fraction(1, 2) + Fraction(1, 1 << 50)) * Fraction(float(np.spacing(e)))
    print(f"r = {r}: {off} of {a.size} are the other neighbour")


def _guard(v):
    return np.where(np.abs(v) < EPS, np.copysign(EPS, np.where(v == 0.0, 1.0, v)), v)


def _counts(diag, oo, E):
    p = diag[0] - E
    c = (p < 0.0).astype(int)
    p = _guard(p)
    for d in diag[1:]:
        p = (d - E) - oo / p
        c += p < 0.0
        p = _guard(p)
    return c


def _thomas(diag, off, shift, u):
    n = diag.size
    f, w, y, x = np.zeros(n), np.empty(n), np.empty(n), np.empty(n)
    d = diag - shift
    w[0] = d[0]
    for i in range(1, n):
        f[i] = off / w[i - 1]
        w[i] = d[i] - f[i] * off
    t = np.float64(0.0)
    for i in range(n):
        t = y[i] = u[i] - f[i] * t
    x[n - 1] = t = y[n - 1] / w[n - 1]
    for i in range(n - 2, -1, -1):
        x[i] = t = (y[i] - off * t) / w[i]
    return f, w, x


@pytest.mark.parametrize("Z,l", [(1, 0), (8, 1), (29, 0), (30, 2)])
@pytest.mark.parametrize("n", [2, 17, 127, 128, 129, 130, 257, 2000])
def test_tridiagonal(engine, Z, l, n):
    """A radial Hamiltonian shifted to just above an eigenvalue, as inverse iteration has it: the second solve is
    for a vector close to the eigenvector, with tails down to the smallest numbers."""
    h = 30.0 / (n + 1)
    r = np.arange(1, n + 1) * h
    off = -0.5 / (h * h)
    diag = 1.0 / (h * h) + 0.5 * l * (l + 1) / (r * r) - Z / r * np.exp(-0.3 * r)
    H = np.diag(diag) + np.diag(np.full(n - 1, off), 1) + np.diag(np.full(n - 1, off), -1)
    ev = np.linalg.eigvalsh(H)
    lo, hi = diag.min() + 2 * off, diag.max() - 2 * off
    # everywhere, at the eigenvalues and next to them, and where the first pivot is exactly zero
    E = np.concatenate([np.linspace(lo, hi, 61), ev[:20], np.nextafter(ev[:10], 0.0), [diag[0]]])
    cnt = engine.array((E.size + 1) // 2)
    f, w, x = engine.array(n), engine.array(n), engine.array(n)
    dd, dE = engine.upload(diag), engine.upload(E)
    for e in ev[:2]:
        shift = e + 1e-10 * max(1.0, abs(e))
        u = np.sin(np.arange(1.0, n + 1))
        for _ in range(3):
            u = u / np.sqrt(np.dot(u, u))
            engine.radial_tridiagonal(n, dd, off, shift, engine.upload(u), f, w, x, E.size, dE, cnt)
            fr, wr, xr = _thomas(diag, off, shift, u)
            assert f.to_host().tobytes() == fr.tobytes() and w.to_host().tobytes() == wr.tobytes()
            got = x.to_host()
            assert got.tobytes() == xr.tobytes(), np.flatnonzero(got != xr)[:5]
            u = xr
    assert np.array_equal(cnt.to_host().view(np.int32)[: E.size], _counts(diag, off * off, E))
