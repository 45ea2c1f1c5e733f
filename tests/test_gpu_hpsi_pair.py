"""GPU: two columns per thread (even rows, 16-byte aligned arrays) and one give the reference's bits at every
row length, band count and chunk edge, aligned or not."""
import numpy as np
import pytest

import dft_b200

pytestmark = pytest.mark.gpu


def _expected(n, h, V, psi):
    """The reference's order of operations (KohnShamHamiltonianMolecule.cpp:59-177), elementwise."""
    i2 = [1.0 / (d * d) for d in h]
    p = psi.reshape(n[2], n[1], n[0])
    lap = (-2.0 * (i2[0] + i2[1] + i2[2])) * p
    for axis, q in ((2, i2[0]), (1, i2[1]), (0, i2[2])):
        lo = [slice(None)] * 3
        hi = [slice(None)] * 3
        lo[axis], hi[axis] = slice(None, -1), slice(1, None)
        lap[tuple(hi)] = lap[tuple(hi)] + p[tuple(lo)] * q
        lap[tuple(lo)] = lap[tuple(lo)] + p[tuple(hi)] * q
    return (-0.5 * lap + V.reshape(p.shape) * p).ravel()


@pytest.mark.parametrize("n", [(2, 3, 4), (30, 9, 5), (32, 8, 7), (33, 8, 7), (34, 17, 9), (64, 16, 33), (66, 5, 70)])
@pytest.mark.parametrize("bands,pad,shift", [(1, 0, 0), (3, 2, 0), (3, 1, 0), (2, 0, 1)])
def test_columns_bit_exact(engine, n, bands, pad, shift):
    g = dft_b200.CartesianGrid(*n, -1.0, 1.3, -0.9, 1.1, -1.2, 0.8)
    N, ld = g.getSize(), g.getSize() + pad
    rng = np.random.default_rng(N + bands)
    V, psi = rng.standard_normal(N), rng.standard_normal(bands * ld + shift)
    dV, dP, dO = engine.upload(V), engine.upload(psi), engine.array(bands * ld + shift)
    off = 8 * shift
    engine.apply_hamiltonian(g, dV, dP.ptr + off, dO.ptr + off, bands, ld)
    got = dO.to_host()[shift:]
    h = (g.getDx(), g.getDy(), g.getDz())
    for b in range(bands):
        row = psi[shift + b * ld: shift + b * ld + N]
        assert np.array_equal(got[b * ld: b * ld + N], _expected(n, h, V, row))
