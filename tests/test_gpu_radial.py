"""GPU: the radial solver's staged chains against the oracle, at the edges of a stage (128 points) and of a
batch of 16, and the same atom in batches of every cluster size.

Tolerance: the solver replays the reference's sequential arithmetic; what differs are the device's
transcendental functions (a few ulp).  The bound is the one of the full batch of 60 atoms: 1e-9 Ha and
one SCF iteration.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [(5, [1, 8]), (16, [1, 8, 11]), (17, [1, 8, 11])] + [
    (n, [1, 8, 11, 30]) for n in (127, 128, 129, 144, 257, 384, 385)]


@pytest.mark.parametrize("points,Zs", CASES)
def test_stage_edges_vs_oracle(engine, port, points, Zs):
    for kind, name in ((0, "PZ81"), (1, "PBE96")):
        res = engine.solve_atoms(Zs, [name] * len(Zs), points, 20.0)
        for Z, r in zip(Zs, res):
            c = port.solve_atom(Z, kind, points, 20.0)
            assert r.status == 0 and r.converged == c["converged"], (Z, name)
            assert abs(r.iterations - c["iterations"]) <= 1, (Z, name)
            assert abs(r.energy.total - c["total"]) < 1e-9, (Z, name)
            assert np.max(np.abs(np.array(r.eigenvalues) - np.array(c["eigenvalues"]))) < 1e-9, (Z, name)


def test_same_bits_in_any_batch(engine):
    """Blocks per atom: 4 in a batch of one, 2 in 40, 1 in 80."""
    sets = []
    for batch in (1, 40, 80):
        Zs = [12] + [1] * (batch - 1)
        r = engine.solve_atoms(Zs, ["PBE96"] * batch, 257, 20.0)[0]
        sets.append((r.status, r.iterations, r.energy.total, r.energy.kinetic, tuple(r.eigenvalues)))
    assert sets[0][0] == 0
    assert sets[0] == sets[1] == sets[2]
