"""GPU: the screened Poisson solve with its source and solution in the same memory."""
import numpy as np
import pytest

import dft_b200

pytestmark = pytest.mark.gpu


# one level, tile passes on the finest level, streaming passes
@pytest.mark.parametrize("dims", [(9, 8, 7), (31, 30, 33), (97, 96, 90)])
@pytest.mark.parametrize("cycles", [1, 2])
def test_in_place_equals_out_of_place(engine, dims, cycles):
    b = []
    for n in dims:
        half = 0.5 * 0.3 * (n - 1)
        b += [-half, half]
    g = dft_b200.CartesianGrid(*dims, *b)
    N = g.getSize()
    src = np.random.default_rng(3).standard_normal(N)
    x = engine.array(N)
    engine.screened_poisson(g, engine.upload(src), x, 2.0, cycles)
    inplace = engine.upload(src)
    engine.screened_poisson(g, inplace, inplace, 2.0, cycles)
    assert inplace.to_host().tobytes() == x.to_host().tobytes()
