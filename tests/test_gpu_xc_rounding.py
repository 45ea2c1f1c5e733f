"""GPU: PBE96's rounding error on a grid.  The grid kernels rearrange the functional (xc_fast.cuh); their potentials
must be no further from an 80-bit evaluation than those of the functional in the reference's expression order
(xc_evaluate) with differences by division, which is what the grid path computed before the rearrangement.

Tolerance: both errors are 2-norms over 10^4 points or more, whose sampling noise is a few per cent; an
added rounding in the exchange terms or the last sums shows as 15 to 30 per cent.
"""
import numpy as np
import pytest

import dft_b200

pytestmark = pytest.mark.gpu

L = np.longdouble
SLACK = 1.1


def _diff(f, d, h):
    out = np.empty_like(f)
    n = f.shape[d]

    def at(a, b=None):
        s = [slice(None)] * 3
        s[d] = a if b is None else slice(a, b)
        return tuple(s)

    out[at(1, n - 1)] = (f[at(2, n)] - f[at(0, n - 2)]) / (2 * h)
    out[at(0, 1)] = (f[at(1, 2)] - f[at(0, 1)]) / h
    out[at(n - 1, n)] = (f[at(n - 1, n)] - f[at(n - 2, n - 1)]) / h
    return out


def _gradients(f, h):
    g = [_diff(f, 2 - d, h[d]) for d in range(3)]
    return g, np.sqrt(g[0] * g[0] + g[1] * g[1] + g[2] * g[2])


def _divergence(c, g, h):
    return sum(_diff(c * g[d], 2 - d, h[d]) for d in range(3))


def _pbe(a, b, ga, gb):
    """d f / d n_sigma and the gradient coefficients, in the inputs' precision."""
    one = a.dtype.type(1)
    third = one / 3
    n = a + b
    kappa, mu = one * 0.804, one * 0.2195149727645171
    gamma, beta = one * 0.031090690869654895, one * 0.06672455060314922
    delta, fg = beta / gamma, one * 0.51984209978974632953
    fzz, eta = 8 / (9 * fg), one * 1.0e-12
    ax = one * -0.73855876638202240588

    def exchange(r, q):
        r13 = np.cbrt(r)
        s = q / (2 * (one * 3.09366772628014) * r13 * r)
        p0 = 1 + mu / kappa * s * s
        fs = 2 * mu / (p0 * p0)
        return ax * r13 * 4 / 3 * (1 + kappa - kappa / p0 - s * s * fs), ax * (one * 0.161620459673995) * s * fs

    def gcor(q, a1, b1, b2, b3, b4, x):
        q, a1, b1, b2, b3, b4 = (one * v for v in (q, a1, b1, b2, b3, b4))
        q0 = -2 * q * (1 + a1 * x * x)
        q1 = 2 * q * x * (b1 + x * (b2 + x * (b3 + b4 * x)))
        lg = np.log(1 + 1 / q1)
        q3 = q * (b1 / x + 2 * b2 + x * (3 * b3 + 4 * b4 * x))
        return q0 * lg, -2 * q * a1 * lg - q0 * q3 / (q1 * (1 + q1))

    dna, dga = exchange(2 * a, 2 * ga)
    dnb, dgb = exchange(2 * b, 2 * gb)
    # the functional is defined on the rounded polarisation: (1 - z)^(1/3) turns on its last bit
    z = ((a - b) / n).astype(np.float64).astype(a.dtype)
    opz = (1 + z.astype(np.float64)).astype(a.dtype)
    omz = (1 - z.astype(np.float64)).astype(a.dtype)
    pi = a.dtype.type(np.pi)
    gm = ga + gb
    rs = np.cbrt(3 / (4 * pi * n))
    pa, pb = np.cbrt(opz), np.cbrt(omz)
    phi = (pa * pa + pb * pb) / 2
    tkp = 2 * np.sqrt(4 * np.cbrt(3 * pi * pi * n) / pi) * phi
    t = gm / (tkp * n)
    x = np.sqrt(rs)
    eu, eud = gcor(0.0310907, 0.21370, 7.5957, 3.5876, 1.6382, 0.49294, x)
    ep, epd = gcor(0.01554535, 0.20548, 14.1189, 6.1977, 3.3662, 0.62517, x)
    al, ad = gcor(0.0168869, 0.11125, 10.357, 3.6231, 0.88026, 0.49671, x)
    z3, z4 = z ** 3, z ** 4
    f = (opz * pa + omz * pb - 2) / fg
    fz = 4 * third * (pa - pb) / fg
    ec = eu * (1 - f * z4) + ep * f * z4 - al * f * (1 - z4) / fzz
    ecrs = eud * (1 - f * z4) + epd * f * z4 - ad * f * (1 - z4) / fzz
    ecz = 4 * z3 * f * (ep - eu + al / fzz) + fz * (z4 * ep - z4 * eu - (1 - z4) * al / fzz)
    phi3 = phi ** 3
    bb = delta / np.expm1(-ec / (gamma * phi3))
    t2 = t * t
    q4, q5 = 1 + bb * t2, 1 + bb * t2 + bb * bb * t2 * t2
    hh = phi3 * (beta / delta) * np.log(1 + delta * q4 * t2 / q5)
    fac = delta / bb + 1
    bec = bb * bb * fac / (beta * phi3)
    q8 = q5 * q5 + delta * q4 * q5 * t2
    hb = -beta * phi3 * bb * t2 ** 3 * (2 + bb * t2) / q8
    hrs = -(rs / 3) * hb * bec * ecrs
    ht = 2 * beta * phi3 * (1 + 2 * bb * t2) / q8
    comm = hh + hrs - 7 * t2 * ht / 6
    gz = (1 / np.cbrt(opz + eta) - 1 / np.cbrt(omz + eta)) / 3
    bg = -3 * bb * bb * ec * fac / (beta * phi3 * phi)
    hz = 3 * gz * hh / phi + hb * (bg * gz + bec * ecz)
    pref = hz - gz * t2 * ht / phi
    com = ec - rs * ecrs / 3 - z * ecz
    dgc = t * ht / tkp
    return dna + com + ecz + comm + pref * (1 - z), dnb + com - ecz + comm - pref * (1 + z), dga + dgc, dgb + dgc


def _densities(seed, grid, spin):
    """Atomic densities with exponential tails, as SCF densities have; alpha and beta of different extent."""
    rng = np.random.default_rng(seed)
    x, y, z = [np.linspace(grid.bounds[2 * d], grid.bounds[2 * d + 1], grid.shape[d]) for d in range(3)]
    Z, Y, X = np.meshgrid(z, y, x, indexing="ij")
    na, nb = np.zeros_like(X), np.zeros_like(X)
    for q in rng.integers(1, 9, 3):
        c = rng.uniform(-1.2, 1.2, 3)
        r = np.sqrt((X - c[0]) ** 2 + (Y - c[1]) ** 2 + (Z - c[2]) ** 2 + 0.05)
        for out, s, zeta in ((na, 0.55, 0.9), (nb, 0.45, spin)):
            k = zeta * (0.8 + 0.12 * q)
            out += s * q * k ** 3 / np.pi * np.exp(-2.0 * k * r)
    return na, nb


@pytest.mark.parametrize("dims", [(40, 36, 32), (33, 41, 29)])
@pytest.mark.parametrize("spin", [0.9, 0.8])
def test_no_further_from_80_bits_than_the_plain_functional(engine, dims, spin):
    h0 = 0.25
    b = []
    for n in dims:
        b += [-0.5 * h0 * (n - 1), 0.5 * h0 * (n - 1)]
    g = dft_b200.CartesianGrid(*dims, *b)
    h = (g.getDx(), g.getDy(), g.getDz())
    N = g.getSize()
    fast, plain = np.zeros(2), np.zeros(2)
    for seed in (1, 2, 3):
        na, nb = _densities(seed, g, spin)
        # 80 bits
        A, B = na.astype(L), nb.astype(L)
        hl = [L(v) for v in h]
        (vA, mA), (vB, mB) = _gradients(A, hl), _gradients(B, hl)
        d1, d2, c1, c2 = _pbe(A, B, mA, mB)
        want = [d1 - _divergence(c1, vA, hl), d2 - _divergence(c2, vB, hl)]
        # the grid kernels
        da, db = engine.upload(na), engine.upload(nb)
        va, vb = engine.array(N), engine.array(N)
        engine.xc(g, "PBE96", da, db, va, vb)
        got = [va.to_host(na.shape), vb.to_host(na.shape)]
        # the plain functional on the device, differences by division in 64 bits
        (ua, ma), (ub, mb) = _gradients(na, h), _gradients(nb, h)
        out = engine.array(5 * N)
        engine.xc_evaluate("PBE96", N, da, db, engine.upload(ma), engine.upload(mb), out)
        o = out.to_host((N, 5)).reshape(*na.shape, 5)
        ref = [o[..., 1] - _divergence(o[..., 3], ua, h), o[..., 2] - _divergence(o[..., 4], ub, h)]
        for s in range(2):
            norm = np.sqrt(np.sum(want[s] ** 2))
            fast[s] += (np.sqrt(np.sum((got[s] - want[s]) ** 2)) / norm) ** 2
            plain[s] += (np.sqrt(np.sum((ref[s] - want[s]) ** 2)) / norm) ** 2
    print("rms over 3 densities: grid", np.sqrt(fast / 3), "plain", np.sqrt(plain / 3))
    assert np.all(plain < (1e-13) ** 2)
    assert np.all(fast <= SLACK ** 2 * plain)
