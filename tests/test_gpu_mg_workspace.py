"""GPU: the Poisson multigrid's workspace, and the start iterate that it keeps in the caller's array."""
import pytest

import dft_b200

pytestmark = pytest.mark.gpu


def _grid(dims, h=0.3):
    b = []
    for n in dims:
        half = 0.5 * h * (n - 1)
        b += [-half, half]
    return dft_b200.CartesianGrid(*dims, *b)


@pytest.mark.parametrize("fused,fields", [(1, 5.0), (0, 6.7)])
def test_workspace(fused, fields):
    """Four fields of the grid, three of each level below and two of each nested level (4 + 3/7 + 2/7); the
    separate passes' restriction temporaries add 3/4 of a field per level and solve.  Grids that fitted the
    memory with 6.7 fields still have to."""
    torch = pytest.importorskip("torch")
    g = _grid((192, 192, 192))
    e = dft_b200.Engine(0)
    try:
        e.set_tuning("multigrid_fused_restriction", fused)
        rho, v = e.array(g.getSize()), e.array(g.getSize())
        e.synthetic_density(g, 3, rho)
        before = torch.cuda.mem_get_info(0)[0]
        e.poisson_start(g, None, rho, v, multigrid_cycles=3)
        used = before - torch.cuda.mem_get_info(0)[0]
        rho.free()
        v.free()
    finally:
        e.close()
    # allocations come in 2 MiB pieces, a handful of them, and captured graphs take some
    assert used < fields * 8 * g.getSize() + (24 << 20)


@pytest.mark.parametrize("dims", [(48, 48, 48), (64, 50, 49), (33, 70, 41), (96, 90, 80), (128, 31, 57)])
def test_cycles_run_together_stop_where_single_ones_do(engine, dims):
    """Cycles are launched in batches; one that meets the tolerance early is repeated from the batch's start.  Limits
    that end the solve at every count give the iterates that the batches must have passed through."""
    g = _grid(dims)
    rho, v, w = [engine.array(g.getSize()) for _ in range(3)]
    for seed in range(1, 7):
        engine.synthetic_density(g, seed, rho)
        info = engine.poisson_start(g, None, rho, v, multigrid_cycles=60)
        used = info["multigrid_cycles"]
        assert used < 60 and info["residual"] < 0.5e-8
        last = engine.poisson_start(g, None, rho, w, multigrid_cycles=used)
        assert last["multigrid_cycles"] == used and last["residual"] == info["residual"]
        assert w.to_host().tobytes() == v.to_host().tobytes()
        short = engine.poisson_start(g, None, rho, w, multigrid_cycles=used - 1)
        assert short["multigrid_cycles"] == used - 1 and short["residual"] >= 0.5e-8
