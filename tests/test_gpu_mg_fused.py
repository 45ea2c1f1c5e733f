"""Fused multigrid passes (mg_fused.cu): the open cycle against a numpy restatement, the Poisson cycles
against the separate passes."""
import numpy as np
import pytest

import dft_b200

pytestmark = pytest.mark.gpu

# odd and even axes (coarse spacings of exactly and just below two fine ones), boxes shorter than a
# tile, one whose flat axis gets finer on the coarse grid, levels on both sides of the size up to
# which a level takes the tile passes
DIMS = [(9, 8, 7), (12, 15, 20), (17, 33, 18), (41, 26, 30), (64, 50, 49), (120, 24, 12), (200, 40, 4),
        (97, 96, 90)]


def _grid(dims, h=0.3):
    b = []
    for n in dims:
        half = 0.5 * h * (n - 1)
        b += [-half, half]
    return dft_b200.CartesianGrid(*dims, *b)


def _coarse(n):
    return max(5, int(np.floor((n - 1) / 2.0 + 0.5)) + 1)


def _transfer(nf, nc, length):
    """Restriction (hat weights times h/H) and linear interpolation along one axis."""
    h, H = length / (nf - 1), length / (nc - 1)
    i, I = np.arange(nf), np.arange(nc)
    R = np.maximum(0.0, 1.0 - np.abs(i[None, :] * h - I[:, None] * H) / H) * (h / H)
    P = np.zeros((nf, nc))
    u = i * h / H
    c = np.clip(np.floor(u).astype(int), 0, nc - 2)
    w = np.clip(u - c, 0.0, 1.0)
    P[i, c] += 1.0 - w
    P[i, c + 1] += w
    return R, P


def _nbsum(v, h):
    s = np.zeros_like(v)
    for ax, d in ((2, h[0]), (1, h[1]), (0, h[2])):
        lo = [slice(None)] * 3
        hi = [slice(None)] * 3
        lo[ax], hi[ax] = slice(0, -1), slice(1, None)
        s[tuple(hi)] += v[tuple(lo)] / d ** 2
        s[tuple(lo)] += v[tuple(hi)] / d ** 2
    return s


def _cycle(src, lengths, shift):
    nz, ny, nx = src.shape
    h = [lengths[0] / (nx - 1), lengths[1] / (ny - 1), lengths[2] / (nz - 1)]
    d = 2.0 * sum(1.0 / q ** 2 for q in h) + shift
    m = (_coarse(nx), _coarse(ny), _coarse(nz))
    if (src.size <= 12288 and min(src.shape) <= 9) or m == (nx, ny, nz):
        v = np.zeros_like(src)
        for _ in range(8 * max(src.shape)):
            v = (_nbsum(v, h) + src) / d
        return v
    T = [_transfer(a, b, l) for a, b, l in zip((nx, ny, nz), m, lengths)]
    v = 0.8 * src / d
    v = v + 0.8 * ((_nbsum(v, h) + src) / d - v)
    r = src - (d * v - _nbsum(v, h))
    r = np.einsum("ai,kji->kja", T[0][0], r)
    r = np.einsum("bj,kja->kba", T[1][0], r)
    r = np.einsum("ck,kba->cba", T[2][0], r)
    e = _cycle(r, lengths, shift)
    e = np.einsum("ia,cba->cbi", T[0][1], e)
    e = np.einsum("jb,cbi->cji", T[1][1], e)
    v = v + np.einsum("kc,cji->kji", T[2][1], e)
    for _ in range(2):
        v = v + 0.8 * ((_nbsum(v, h) + src) / d - v)
    return v


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("q2", [0.01, 2.0, 60.0])
def test_open_cycle(engine, dims, q2):
    g = _grid(dims)
    src = np.random.default_rng(3).standard_normal(g.shape[::-1])
    x = engine.array(g.getSize())
    engine.screened_poisson(g, engine.upload(src), x, q2)
    ref = _cycle(src, [0.3 * (n - 1) for n in dims], q2)
    # some ten passes of about ten operations per level, each a few eps of the values it combines;
    # the coarsest level's sweeps contract, so their rounding does not add up
    assert np.max(np.abs(x.to_host(ref.shape) - ref)) < 1e-12 * np.max(np.abs(ref)) * max(1.0, 1.0 / q2)


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("cycles", [1, 2, 7])
def test_poisson_cycles(engine, dims, cycles):
    g = _grid(dims)
    rho = engine.array(g.getSize())
    engine.synthetic_density(g, 7, rho)
    out = []
    try:
        for fused in (0, 1):
            engine.set_tuning("multigrid_fused_restriction", fused)
            v = engine.array(g.getSize())
            info = engine.poisson_start(g, None, rho, v, multigrid_cycles=cycles)
            out.append((v.to_host(), info["multigrid_cycles"], info["coarse_cycles"]))
    finally:
        engine.set_tuning("multigrid_fused_restriction", 1)
    assert out[0][1:] == out[1][1:]
    # the cycles contract: what is left is the rounding of the last one's few hundred operations
    assert np.max(np.abs(out[0][0] - out[1][0])) < 1e-12 * np.max(np.abs(out[0][0]))


def test_poisson_spacing_is_part_of_the_captured_cycle(engine):
    """The same buffers and points with another spacing: a captured cycle must not be reused."""
    dims = (40, 40, 40)
    N = 40 ** 3
    rho, v = engine.array(N), engine.array(N)
    for h in (0.3, 0.2, 0.3):
        g = _grid(dims, h)
        engine.synthetic_density(g, 5, rho)
        engine.poisson_start(g, None, rho, v, multigrid_cycles=40)
        sweeps, _ = engine.hartree_from_guess(g, rho, v)
        assert sweeps == 1
