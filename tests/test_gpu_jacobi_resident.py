"""The resident Jacobi solve (jacobi_resident.cu) against one sweep per launch: the same bits, sweep
count and last difference at every stop."""
import numpy as np
import pytest

import dft_b200

pytestmark = pytest.mark.gpu


def _solve(engine, mode, g, rho, tol, cap, guess=None):
    vh = engine.upload(guess) if guess is not None else engine.array(g.getSize())
    engine.set_tuning("jacobi_sweeps_per_launch", mode)
    try:
        f = engine.hartree_from_guess if guess is not None else engine.hartree
        s, d = f(g, engine.upload(rho), vh, tol, cap)
    finally:
        engine.set_tuning("jacobi_sweeps_per_launch", 0)
    return s, d, vh.to_host()


# one interior point, boxes thinner than the halo, rows of one, two and more half warps, the largest boxes that
# fit, one that does not; faces that miss their bound by rounding (Q / |r| on them) in the last
@pytest.mark.parametrize("dims,h", [((3, 3, 3), 0.25), ((4, 3, 9), 0.25), ((17, 5, 6), 0.25), ((18, 33, 20), 0.25),
                                    ((35, 34, 33), 0.25), ((64, 40, 50), 0.25), ((64, 64, 64), 0.25),
                                    ((120, 24, 24), 0.25), ((96, 90, 80), 0.25), ((21, 22, 23), 0.1)])
# stops at every sweep of a round, the cap among them
@pytest.mark.parametrize("cap", [1, 2, 3, 4, 5, 6, 7, 12, 13, 10000])
def test_same_bits(engine, dims, h, cap):
    b = []
    for n in dims:
        half = 0.5 * h * (n - 1)
        b += [-half, half]
    g = dft_b200.CartesianGrid(*dims, *b)
    rng = np.random.default_rng(cap)
    rho = rng.uniform(0.0, 1.0, g.getSize()) ** 8
    tol = 1e-3 if cap == 10000 else 0.0
    ref = _solve(engine, 1, g, rho, tol, cap)
    got = _solve(engine, 0, g, rho, tol, cap)
    assert got[:2] == ref[:2] and got[2].tobytes() == ref[2].tobytes()
    warm = rng.standard_normal(g.getSize())
    ref = _solve(engine, 1, g, rho, tol, cap, warm)
    got = _solve(engine, 0, g, rho, tol, cap, warm)
    assert got[:2] == ref[:2] and got[2].tobytes() == ref[2].tobytes()


@pytest.mark.parametrize("scale", [0.0, -1.0, 1e-300, 1e-310, 1e290])
def test_same_bits_extreme_sources(engine, scale):
    """Zeros, negative, subnormal and huge sources: the division outside its fast range."""
    g = dft_b200.CartesianGrid(20, 21, 22, -2.0, 2.0, -2.0, 2.0, -2.0, 2.0)
    rho = scale * np.random.default_rng(1).uniform(0.0, 1.0, g.getSize())
    ref = _solve(engine, 1, g, rho, 0.0, 50)
    got = _solve(engine, 0, g, rho, 0.0, 50)
    assert got[:2] == ref[:2] and got[2].tobytes() == ref[2].tobytes()
