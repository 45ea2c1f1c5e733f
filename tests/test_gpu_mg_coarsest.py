"""The coarsest multigrid level by itself: grids small enough to be one level, where a Poisson start is this
level's solve of the whole equation (source 4 pi rho) and nothing else."""
import math

import numpy as np
import pytest

import dft_b200

pytestmark = pytest.mark.gpu

H = 0.3
# at most 12288 points and no axis above 9 on one side; odd, even, long
DIMS = [(9, 8, 7), (9, 9, 9), (5, 5, 5), (40, 21, 9), (6, 30, 33)]


def _grid(dims):
    b = []
    for n in dims:
        half = 0.5 * H * (n - 1)
        b += [-half, half]
    return dft_b200.CartesianGrid(*dims, *b)


def _neighbours(v):
    s = np.zeros_like(v)
    s[1:-1, 1:-1, 1:-1] = (v[:-2, 1:-1, 1:-1] + v[2:, 1:-1, 1:-1] + v[1:-1, :-2, 1:-1] + v[1:-1, 2:, 1:-1] +
                           v[1:-1, 1:-1, :-2] + v[1:-1, 1:-1, 2:])
    return s / H ** 2


def _sweeps(src, sor):
    """The level's sweeps from zero: 8 per point of the longest axis by Jacobi, or red-black SOR."""
    nz, ny, nx = src.shape
    den = 6.0 / H ** 2
    inside = np.zeros(src.shape, dtype=bool)
    inside[1:-1, 1:-1, 1:-1] = True
    v = np.zeros_like(src)
    if not sor:
        for _ in range(8 * max(src.shape)):
            v = np.where(inside, (_neighbours(v) + src) / den, 0.0)
        return v
    rj = sum(math.cos(math.pi / (n - 1)) for n in src.shape) / 3.0
    omega = 2.0 / (1.0 + math.sqrt(1.0 - rj * rj))
    need = math.ceil(math.log(1e-4) / math.log(max(omega - 1.0, 1e-3)))
    parity = np.add.outer(np.add.outer(np.arange(nz), np.arange(ny)), np.arange(nx)) & 1
    for _ in range(min(8 * max(src.shape), max(4, need))):
        for colour in (0, 1):
            at = inside & (parity == colour)
            v = np.where(at, v + omega * ((_neighbours(v) + src) / den - v), v)
    return v


def _dirichlet(src):
    """-lap_h v = src inside, zero on the faces, by sine transforms."""
    f = src[1:-1, 1:-1, 1:-1]
    S, lam = [], []
    for m in f.shape:
        k = np.arange(1, m + 1)
        S.append(np.sin(math.pi / (m + 1) * np.outer(k, k)) * math.sqrt(2.0 / (m + 1)))
        lam.append(4.0 / H ** 2 * np.sin(0.5 * math.pi * k / (m + 1)) ** 2)
    den = lam[0][:, None, None] + lam[1][None, :, None] + lam[2][None, None, :]

    def transform(a):
        return np.einsum("ai,bj,ck,ijk->abc", *S, a, optimize=True)

    v = np.zeros_like(src)
    v[1:-1, 1:-1, 1:-1] = transform(transform(f) / den)
    return v


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("sor", [0, 1])
def test_one_level_poisson_start(engine, dims, sor):
    g = _grid(dims)
    rho = np.random.default_rng(11).uniform(0.0, 1.0, g.shape[::-1])
    src = 4.0 * math.pi * rho
    v = engine.array(g.getSize())
    try:
        engine.set_tuning("multigrid_coarsest_sor", sor)
        info = engine.poisson_start(g, None, engine.upload(rho), v, multigrid_cycles=20)
    finally:
        engine.set_tuning("multigrid_coarsest_sor", 1)
    got = v.to_host(src.shape)
    want = _sweeps(src, sor)
    # contracting sweeps of about ten operations each: their rounding does not add up
    assert np.max(np.abs(got - want)) < 1e-12 * np.max(np.abs(want))
    # SOR aims at 1e-4 (the factor of a sweep near its optimum has a linear prefactor: ten sweeps and
    # more); Jacobi's 8 per point leave 4e-3 on 9^3
    assert np.max(np.abs(got - _dirichlet(src))) < 1e-2 * np.max(np.abs(want))
    assert info["multigrid_cycles"] == 1  # from zero: a second one would repeat it
