"""FP64 Gram, rotation and residual kernels (dense_fp64.cu) at the edges of their tiles, against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


@pytest.fixture(scope="module")
def eng():
    import dft_b200
    e = dft_b200.Engine(0)
    yield e
    e.close()


def _grid(nx, ny, nz):
    import dft_b200
    return dft_b200.CartesianGrid(nx, ny, nz, -1.0, 1.0, -1.5, 1.5, -2.0, 2.0)


# 1, tile edges (8 columns, 16 rows), both reductions (nel <= 1024 and above), several column tiles;
# point counts below one step, ragged (odd leading dimension: 8-byte loads) and even
SHAPES = [(1, 1), (8, 8), (9, 7), (17, 16), (36, 12), (33, 31), (40, 40), (129, 72), (150, 73), (24, 150)]


@pytest.mark.parametrize("dims", [(2, 2, 2), (5, 7, 3), (16, 16, 9), (33, 31, 17)])
@pytest.mark.parametrize("ka,kb", SHAPES)
def test_gram(eng, dims, ka, kb):
    g = _grid(*dims)
    N = g.getSize()
    rng = np.random.default_rng(ka * 1000 + kb)
    A, B = rng.standard_normal((ka, N)), rng.standard_normal((kb, N))
    dV = g.getDx() * g.getDy() * g.getDz()
    C = eng.gram(g, eng.upload(A), N, ka, eng.upload(B), N, kb)
    # any order of N products and sums: |error| <= (N + 2) eps sum |a||b|
    bound = (N + 2) * EPS * dV * (np.abs(A) @ np.abs(B).T)
    assert np.all(np.abs(C - dV * (A @ B.T)) <= 2 * bound)


@pytest.mark.parametrize("dims", [(2, 2, 2), (5, 7, 3), (16, 16, 9), (33, 31, 17)])
@pytest.mark.parametrize("k,m", [(1, 1), (4, 8), (5, 9), (19, 17), (36, 12), (70, 69), (150, 73), (400, 80)])
def test_rotate(eng, dims, k, m):
    g = _grid(*dims)
    N = g.getSize()
    rng = np.random.default_rng(k * 1000 + m)
    V, Y = rng.standard_normal((k, N)), rng.standard_normal((k, m))
    X = eng.upload(np.full((m, N), 7.0))
    eng.rotate(g, eng.upload(V), N, k, Y, X, N)
    bound = (k + 2) * EPS * (np.abs(Y).T @ np.abs(V))
    assert np.all(np.abs(X.to_host((m, N)) - Y.T @ V) <= 2 * bound)


@pytest.mark.parametrize("dims", [(12, 12, 12), (13, 11, 15)])
@pytest.mark.parametrize("nocc,nb", [(1, 2), (3, 9), (9, 17)])
def test_eigensolve_orbitals(eng, dims, nocc, nb):
    """Residuals and orthonormality of the converged block: the residual pass, the in-place
    rotations and the final Ritz vectors."""
    g = _grid(*dims)
    N = g.getSize()
    rng = np.random.default_rng(nb)
    V = rng.uniform(-3.0, 0.0, N)
    psi, out = eng.array(nb * N), eng.array(nb * N)
    dV_, tol = eng.upload(V), 1e-8
    e, _ = eng.solve_orbitals(g, dV_, nocc, nb, psi, N, tol=tol)
    eng.apply_hamiltonian(g, dV_, psi, out, nb, N)
    P, HP = psi.to_host((nb, N)), out.to_host((nb, N))
    dV = g.getDx() * g.getDy() * g.getDz()
    # the solver's own stop, plus the rounding of H psi (|H| eps)
    hmax = 2.0 * (g.getDx() ** -2 + g.getDy() ** -2 + g.getDz() ** -2) + 3.0
    res = np.sqrt(dV * np.sum((HP - e[:, None] * P) ** 2, axis=1))[:nocc]
    assert np.all(res < tol + 64 * hmax * EPS)
    # one projected Cholesky QR pass is accepted below a loss of 1e-12 per basis extension
    assert np.max(np.abs(dV * P @ P.T - np.eye(nb))) < 1e-10
