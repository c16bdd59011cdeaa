"""Bounded device waits that run out: the call returns BEM_ERR_TIMEOUT, and the context solves
correctly afterwards.  The waits are made to run out by a message that its sender withholds.

Bar of the solves that follow: the backward error ||b - A x|| / (||A|| ||x|| + ||b||) at 1e-14
(FP64 rounding of a residual at these orders)."""
import numpy as np
import pytest

from bem3d_elastostatic_b200 import _lib

pytestmark = pytest.mark.gpu


def _system(n, seed=3):
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((n, n), dtype=np.float32).astype(np.float64) / np.sqrt(n)
    A[np.diag_indices(n)] += 3.0
    return np.asfortranarray(A), rng.standard_normal(n)


def _backward_error(A, x, b):
    return np.abs(b - A @ x).max() / (np.abs(A).sum(1).max() * np.abs(x).max() + np.abs(b).max())


# the first sub-panel, an inner one and the last with two CTAs; of a fresh workspace and a used one
@pytest.mark.parametrize("n,pivots", [(300, [0]), (1500, [0, 700, 1219]), (9000, [40])])
def test_withheld_pivot(n, pivots):
    from bem3d_elastostatic_b200.api import solve_system

    A, b = _system(n)
    ctx = _lib.Context(0)
    for pivot in pivots:
        ctx.set_option(_lib.BEM_OPT_WAIT_LIMIT_MS, 100)
        ctx.set_option(_lib.BEM_OPT_WITHHOLD_PIVOT, pivot)
        with pytest.raises(_lib.BemError) as exc:
            solve_system(A, b, "fp64", ctx=ctx)
        assert exc.value.code == _lib.BEM_ERR_TIMEOUT
    ctx.set_option(_lib.BEM_OPT_WITHHOLD_PIVOT, -1)
    ctx.set_option(_lib.BEM_OPT_WAIT_LIMIT_MS, 2000)
    x, _ = solve_system(A, b, "fp64", ctx=ctx)
    assert _backward_error(A, x, b) <= 1e-14
    ctx.close()


def test_wait_limit_of_a_replayed_factorisation():
    """The limit in force is the one set last, also for a factorisation captured before."""
    import time

    from bem3d_elastostatic_b200.api import solve_system

    A, b = _system(600)
    ctx = _lib.Context(0)
    ctx.set_option(_lib.BEM_OPT_WITHHOLD_PIVOT, 0)
    seconds = []
    for limit in (1500, 50, 1500):
        ctx.set_option(_lib.BEM_OPT_WAIT_LIMIT_MS, limit)
        t = time.perf_counter()
        with pytest.raises(_lib.BemError):
            solve_system(A, b, "fp64", ctx=ctx)
        seconds.append(time.perf_counter() - t)
    assert seconds[0] >= 1.5 and seconds[2] >= 1.5  # one wait runs out per solve
    assert seconds[1] <= 1.0
    ctx.close()


def test_no_result_of_a_failed_solve(cube8_mesh):
    """The FP64 solve factors A in place: after a wait that ran out neither A nor the solution is
    taken for one."""
    from bem3d_elastostatic_b200.api import Quadesth

    q = Quadesth(cube8_mesh)
    q.precompute_element_geometry()
    q.ghmat8()
    x = q.solve_linear_system("fp64-ir")
    q.set_option(_lib.BEM_OPT_WAIT_LIMIT_MS, 50)
    q.set_option(_lib.BEM_OPT_WITHHOLD_PIVOT, 0)
    with pytest.raises(_lib.BemError) as exc:
        q.solve_linear_system("fp64")
    assert exc.value.code == _lib.BEM_ERR_TIMEOUT
    q.set_option(_lib.BEM_OPT_WITHHOLD_PIVOT, -1)
    q.set_option(_lib.BEM_OPT_WAIT_LIMIT_MS, 2000)
    for call in (q.reorganize_solution, lambda: q.solve_linear_system("fp64")):
        with pytest.raises(_lib.BemError) as exc:
            call()
        assert exc.value.code == _lib.BEM_ERR_STATE
    q.ghmat8()
    y = q.solve_linear_system("fp64")
    assert np.abs(y - x).max() <= 1e-10 * np.abs(x).max()
    q.close()


# the first panel of a step and the second; one, two and four rows per thread come with the orders
@pytest.mark.parametrize("precision", ["fp32-ir", "fp64"])
@pytest.mark.parametrize("ks,pivot", [([3, 1, 4], 0), ([6] * 5 + [2], 45), ([6] * 44, 33)])
def test_batch_withheld_pivot(ks, pivot, precision):
    from bem3d_elastostatic_b200.api import Batch
    from bem3d_elastostatic_b200.mesh import loaded_box

    rng = np.random.default_rng(len(ks))
    b = Batch()
    for k in ks:
        b.add(*loaded_box(*rng.uniform(0.7, 1.5, 3), k, rng.uniform(0.1, 0.4), 1.0, rng.standard_normal((2, 3))))
    b.assemble()
    b.set_option(_lib.BEM_OPT_WAIT_LIMIT_MS, 50)
    b.set_option(_lib.BEM_OPT_WITHHOLD_PIVOT, pivot)
    for _ in range(2):  # captured and replayed
        with pytest.raises(_lib.BemError) as exc:
            b.solve(precision)
        assert exc.value.code == _lib.BEM_ERR_TIMEOUT
    b.set_option(_lib.BEM_OPT_WITHHOLD_PIVOT, -1)
    b.set_option(_lib.BEM_OPT_WAIT_LIMIT_MS, 2000)
    assert b.solve(precision)["max_backward_error"] <= 1e-14
    b.close()


# the first, an inner and the last block that is waited for; one owned block a CTA and two (more
# than 148 blocks)
@pytest.mark.parametrize("n,blocks", [(1000, [0, 6]), (4000, [0, 5, 30]), (148 * 128 + 300, [60, 149])])
def test_withheld_sweep_block(n, blocks):
    from bem3d_elastostatic_b200.api import solve_system

    A, b = _system(n)
    ctx = _lib.Context(0)
    for block in blocks:
        ctx.set_option(_lib.BEM_OPT_WAIT_LIMIT_MS, 100)
        ctx.set_option(_lib.BEM_OPT_WITHHOLD_BLOCK, block)
        with pytest.raises(_lib.BemError) as exc:
            solve_system(A, b, "fp32-ir", ctx=ctx)
        assert exc.value.code == _lib.BEM_ERR_TIMEOUT
    ctx.set_option(_lib.BEM_OPT_WITHHOLD_BLOCK, -1)
    ctx.set_option(_lib.BEM_OPT_WAIT_LIMIT_MS, 2000)
    x, _ = solve_system(A, b, "fp32-ir", ctx=ctx)
    assert _backward_error(A, x, b) <= 1e-14
    ctx.close()


def test_no_solution_of_a_failed_batch_solve():
    from bem3d_elastostatic_b200.api import Batch
    from bem3d_elastostatic_b200.mesh import loaded_box

    b = Batch()
    b.add(*loaded_box(1.0, 0.8, 1.2, 4, 0.3))
    b.assemble()
    b.solve("fp64")
    x = b.solution(0)
    b.set_option(_lib.BEM_OPT_WAIT_LIMIT_MS, 50)
    b.set_option(_lib.BEM_OPT_WITHHOLD_PIVOT, 0)
    with pytest.raises(_lib.BemError):
        b.solve("fp64")
    with pytest.raises(_lib.BemError) as exc:  # the vectors hold the failed solve's
        b.solution(0)
    assert exc.value.code == _lib.BEM_ERR_ARG
    b.set_option(_lib.BEM_OPT_WITHHOLD_PIVOT, -1)
    b.solve("fp64")
    assert np.array_equal(b.solution(0), x)
    b.close()
