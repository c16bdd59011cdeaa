"""Systems with NaN entries: every factorisation ends, with an error or a solution that shows them,
and the context solves the next system.  A search for a pivot among NaN alone must still end at one
of its rows: the orders end in a full 32 x 32 window, in a ragged one and in one row, and the
columns of NaN lie in the first and in the last sub-panel of A and of its transpose.
"""
import numpy as np
import pytest

from bem3d_elastostatic_b200 import _lib

pytestmark = pytest.mark.gpu


def _system(n):
    rng = np.random.default_rng(n)
    return rng.standard_normal((n, n)) / np.sqrt(n) + 3.0 * np.eye(n), rng.standard_normal(n)


def _spoiled(A):
    n = A.shape[0]
    for rows, cols in [(slice(None), n - 1), (n - 1, slice(None)), (slice(None), 0), (0, slice(None)),
                       (n // 2, n // 3), (slice(None), slice(None))]:
        B = A.copy()
        B[rows, cols] = np.nan
        yield B


@pytest.mark.parametrize("pivoting", [_lib.BEM_PIVOT_WINDOW, _lib.BEM_PIVOT_PARTIAL])
@pytest.mark.parametrize("precision", ["fp64", "fp64-ir", "fp32-ir", "bf16-ir"])
@pytest.mark.parametrize("n", [96, 129, 700])
def test_nan_entries(n, precision, pivoting):
    from bem3d_elastostatic_b200.api import SolverFailure, solve_system

    A, b = _system(n)
    ctx = _lib.Context(0)
    for B in _spoiled(A):
        try:
            x, _ = solve_system(B, b, precision, ctx=ctx, pivoting=pivoting)
            assert not np.isfinite(x).all()
        except SolverFailure:
            pass
        except _lib.BemError as exc:
            assert exc.code == _lib.BEM_ERR_NOCONV, exc
    x, _ = solve_system(A, b, precision, ctx=ctx, pivoting=pivoting)
    assert np.abs(A @ x - b).max() <= 1e-13 * np.abs(A).sum(1).max() * np.abs(x).max()
    ctx.close()


@pytest.mark.parametrize("n", [96, 129, 700])
def test_nan_entries_dgesv(n):
    from bem3d_elastostatic_b200.api import dgesv

    A, b = _system(n)
    ctx = _lib.Context(0)
    for B in _spoiled(A):
        _, ipiv, X, info = dgesv(B, b, ctx=ctx)
        assert (ipiv >= 1).all() and (ipiv <= n).all()
        assert info != 0 or not np.isfinite(X).all()
    X = dgesv(A, b, ctx=ctx)[2]
    assert np.abs(A @ X[:, 0] - b).max() <= 1e-13 * np.abs(A).sum(1).max() * np.abs(X).max()
    ctx.close()


@pytest.mark.parametrize("precision", ["fp32-ir", "fp64"])
def test_batch_with_a_collapsed_element(precision):
    """A system whose normals are 0 / 0 does not count as converged; the one beside it does."""
    from bem3d_elastostatic_b200.api import Batch, SolverFailure
    from bem3d_elastostatic_b200.mesh import loaded_box

    b = Batch()
    good, bad = loaded_box(1.0, 1.0, 1.0, 3, 0.3), loaded_box(1.0, 1.0, 1.0, 2, 0.3)
    nodes = bad[0].kconec[:, 0] - 1
    for v in (bad[0].x, bad[0].y, bad[0].z):
        v[nodes] = v[nodes[0]]
    b.add(*good)
    b.add(*bad)
    b.assemble()
    try:
        b.solve(precision, tol=1e-13)
        assert b.info["max_backward_error"] == np.inf
    except SolverFailure:  # a zero pivot among the NaN
        assert b.info["singular"] == 1
    assert b.info["converged"] == 1
    b.close()
