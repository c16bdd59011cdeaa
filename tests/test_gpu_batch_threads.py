"""Batches used from several host threads: different batches at the same time, and the solutions of
one solved batch.  Every result is compared bit for bit with the same call made alone."""
import threading

import numpy as np
import pytest

from bem3d_elastostatic_b200.mesh import loaded_box

pytestmark = pytest.mark.gpu


def _batch(ks, loads=1):
    from bem3d_elastostatic_b200.api import Batch

    rng = np.random.default_rng(len(ks))
    b = Batch()
    for k in ks:
        b.add(*loaded_box(*rng.uniform(0.7, 1.5, 3), k, 0.3, 1.0, rng.standard_normal((loads, 3))))
    b.assemble()
    return b


def _run(*jobs):
    errors = []

    def guarded(job):
        try:
            job()
        except Exception as exc:  # noqa: BLE001 - reported by the main thread
            errors.append(exc)

    threads = [threading.Thread(target=guarded, args=(job,)) for job in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_small_batches_beside_a_large_system():
    """7,206 unknowns, whose pivot gather needs more shared memory than a launch has by default,
    captured and replayed while another thread captures solves of 78 unknowns."""
    big = _batch([10])
    big.solve("fp64", tol=1e-15)
    ref = big.solution(0)
    stop = threading.Event()

    def small():
        while not stop.is_set():
            b = _batch([1])
            b.solve("fp64")
            b.close()

    def large():
        try:
            for i in range(12):
                big.solve("fp64", tol=1e-15 * (1 + i // 2))  # captured anew, replayed
                assert np.array_equal(big.solution(0), ref)
        finally:
            stop.set()

    _run(small, large)
    big.close()


def test_solutions_fetched_by_several_threads():
    ks = [1, 2, 3, 4] * 4
    b = _batch(ks, loads=2)
    b.solve("fp64")
    ref = [b.solution(i) for i in range(len(ks))]
    for _ in range(5):
        b.solve("fp64")  # nothing fetched yet

        def fetch(first):
            for i in range(first, len(ks), 4):
                assert np.array_equal(b.solution(i), ref[i])

        _run(*(lambda f=f: fetch(f) for f in range(4)))
    b.close()
