"""GPU: the whole-grid functionals (xc_fast.cuh) and the marching divergence against the oracle: every
polarisation from -1 to 1 with both sides of the switch at 1 +- z = 1/4, empty regions, faces, and
boxes smaller and larger than a block.

Tolerance: the formulas are the reference's with rounding errors of a few units per operation; the
potentials and the energy are held to the 1e-12 of their maximum that the plain functional is held to.
"""
import numpy as np
import pytest

import dft_b200

pytestmark = pytest.mark.gpu

RTOL = 1e-12
BOXES = [(5, 4, 6), (32, 8, 4), (33, 9, 35), (64, 17, 5), (31, 40, 12)]


def _densities(n, b, which):
    x, y, z = [np.linspace(b[2 * a], b[2 * a + 1], n[a]) for a in range(3)]
    Z, Y, X = np.meshgrid(z, y, x, indexing="ij")
    r2 = X ** 2 + Y ** 2 + Z ** 2
    total = 3.0 * np.exp(-1.1 * r2) + 0.02 * np.exp(-0.2 * r2)
    if which == "sweep":
        s = np.tanh(1.3 * X + 0.4 * Y) * 0.999
    elif which == "threshold":
        s = np.where(X + Y > 0, 0.75 + 1e-3 * np.sin(5 * Z), -0.75 + 1e-3 * np.sin(4 * X))
    elif which == "polarised":
        s = np.ones_like(X)
    else:
        s = np.zeros_like(X)
    na, nb = 0.5 * total * (1 + s), 0.5 * total * (1 - s)
    if which == "closed":
        na[: n[2] // 3] = 0.0
        nb[: n[2] // 3] = 0.0
    return na.ravel(), nb.ravel()


@pytest.mark.parametrize("n", BOXES)
@pytest.mark.parametrize("which", ["sweep", "threshold", "polarised", "closed"])
@pytest.mark.parametrize("kind", [0, 1])
def test_grid_xc_vs_oracle(engine, port, n, which, kind):
    b = (-3.1, 3.0, -2.7, 2.9, -2.8, 3.2)
    na, nb = _densities(n, b, which)
    g = dft_b200.CartesianGrid(*n, *b)
    N = g.getSize()
    da, db = engine.upload(na), engine.upload(nb)
    va, vb = engine.array(N), engine.array(N)
    e = engine.xc(g, kind, da, db, va, vb)
    for got, s in ((va, 0), (vb, 1)):
        want = port.xc_potential(kind, n, b, na, nb, s)
        assert np.max(np.abs(got.to_host() - want)) <= RTOL * np.max(np.abs(want))
    want = port.xc_energy(kind, n, b, na, nb)
    assert abs(e - want) <= RTOL * abs(want)
