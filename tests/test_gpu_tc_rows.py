"""GPU: the tensor-core Gram product at the row counts where its kernel changes (80, 144, 224, 304 and 384 rows of
both sides, and one more), over several slices per block.

Tolerance, per element relative to sum |a| |b|: the split keeps 2 x 11 bits (2^-21 with the dropped lo*lo), and a
block adds at most 12 groups of 8 products per 32 points in FP32.  Here a block has at most 512 points, 16
slices: 192 x 2^-23 with truncated sums, below 2.4e-5.
"""
import numpy as np
import pytest

import dft_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ka,kb", [(40, 40), (41, 40), (48, 48), (49, 40), (72, 72), (80, 64), (73, 72), (96, 96), (97, 96),
                                   (112, 112), (113, 112), (128, 128), (160, 112), (176, 128), (177, 128), (200, 128),
                                   (256, 128), (128, 256), (250, 257)])
@pytest.mark.parametrize("n,pad", [((32, 32, 33), 0), ((45, 31, 27), 1)])
def test_gram_rows(engine, ka, kb, n, pad):
    g = dft_b200.CartesianGrid(*n, -1.0, 1.0, -1.0, 1.0, -1.0, 1.0)
    N = g.getSize()
    ld = N + pad
    rng = np.random.default_rng(1000 * ka + kb)
    A, B = rng.standard_normal((ka, ld)), rng.standard_normal((kb, ld))
    A[:, ::7] = 0.0
    got = np.asarray(engine.gram(g, engine.upload(A), ld, ka, engine.upload(B), ld, kb, precision=1))
    dV = g.getDx() * g.getDy() * g.getDz()
    want = dV * (A[:, :N] @ B[:, :N].T)
    scale = dV * (np.abs(A[:, :N]) @ np.abs(B[:, :N]).T)
    assert np.all(np.abs(got.reshape(ka, kb) - want) <= 2.4e-5 * scale)
