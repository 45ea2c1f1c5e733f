"""GPU: H psi on rows of fewer than 16 pairs, whose blocks take one thread per pair: bit-exact at one to fifteen pairs,
at one block and several along y, the last one ragged."""
import numpy as np
import pytest

import dft_b200
from test_gpu_hpsi_pair import _expected

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(2, 300, 3), (4, 129, 5), (10, 57, 4), (14, 37, 6), (20, 20, 33), (26, 40, 7), (30, 18, 9)])
@pytest.mark.parametrize("bands", [1, 5])
def test_short_rows_bit_exact(engine, n, bands):
    g = dft_b200.CartesianGrid(*n, -1.0, 1.3, -0.9, 1.1, -1.2, 0.8)
    N = g.getSize()
    rng = np.random.default_rng(N + bands)
    V, psi = rng.standard_normal(N), rng.standard_normal((bands, N))
    out = engine.array(bands * N)
    engine.apply_hamiltonian(g, engine.upload(V), engine.upload(psi), out, bands, N)
    got = out.to_host((bands, N))
    h = (g.getDx(), g.getDy(), g.getDz())
    for b in range(bands):
        assert np.array_equal(got[b], _expected(n, h, V, psi[b]))
