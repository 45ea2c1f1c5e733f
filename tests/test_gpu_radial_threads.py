"""GPU: radial batches of different sizes from two threads with a context each."""
import threading

import pytest

import dft_b200

pytestmark = pytest.mark.gpu


def test_two_contexts_at_once():
    """Every call succeeds and gives what it gives alone, whatever the other thread's point count asks of the
    kernel's shared memory."""
    sizes = (800, 6)
    alone, errors, got = [], [], [[], []]
    engines = [dft_b200.Engine(0) for _ in sizes]
    stop = threading.Event()

    def key(r):
        return (r.status, r.iterations, r.energy.total, tuple(r.eigenvalues))

    def work(t):
        try:
            for _ in range(400):
                if stop.is_set():
                    return
                got[t].append(key(engines[t].solve_atoms([1], ["PZ81"], sizes[t], 10.0)[0]))
        except Exception as e:  # noqa: BLE001
            errors.append((sizes[t], repr(e)))
        finally:
            if t == 0:
                stop.set()

    try:
        for e, n in zip(engines, sizes):
            alone.append(key(e.solve_atoms([1], ["PZ81"], n, 10.0)[0]))
        threads = [threading.Thread(target=work, args=(t,)) for t in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        for e in engines:
            e.close()
    assert not errors
    for t in range(2):
        assert got[t] and set(got[t]) == {alone[t]}
