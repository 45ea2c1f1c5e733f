"""GPU: the tensor-core Gram product at the edges of its tiles, with either operand on the accumulator's rows,
odd leading dimensions, ragged point counts, zeros and numbers below the FP32 range.

Tolerance, per element relative to sum |a| |b|: the split keeps 2 x 11 bits (2^-21 with the dropped
lo*lo), and at these sizes a block adds at most 12 groups of 8 products per 32 points in FP32 (12 x 2^-23
with truncated sums): below 2e-6; 4e-6 is allowed.
"""
import numpy as np
import pytest

import dft_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ka,kb", [(1, 1), (16, 128), (128, 16), (129, 8), (8, 129), (138, 69), (69, 138), (17, 256),
                                   (257, 3), (130, 260)])
@pytest.mark.parametrize("n,pad", [((7, 5, 9), 0), ((16, 16, 16), 1)])
def test_gram_tiles(engine, ka, kb, n, pad):
    g = dft_b200.CartesianGrid(*n, -1.0, 1.0, -1.0, 1.0, -1.0, 1.0)
    N = g.getSize()
    ld = N + pad
    rng = np.random.default_rng(1000 * ka + kb)
    A, B = rng.standard_normal((ka, ld)), rng.standard_normal((kb, ld))
    A[:, ::7] = 0.0
    B[:, 3::11] = 1e-41
    A[:, 5::13] *= 1e-12
    got = np.asarray(engine.gram(g, engine.upload(A), ld, ka, engine.upload(B), ld, kb, precision=1))
    dV = g.getDx() * g.getDy() * g.getDz()
    want = dV * (A[:, :N] @ B[:, :N].T)
    scale = dV * (np.abs(A[:, :N]) @ np.abs(B[:, :N]).T)
    assert np.all(np.abs(got.reshape(ka, kb) - want) <= 4e-6 * scale)
