"""Calls that share the context's kept buffers, in orders that grow and reuse them, and the
adjoint's regular pairs with full, ragged and few groups of elements.

dgesv: bit for bit what a fresh context returns.  Adjoint: the compliance does not change when the
body is moved, so the shape gradient sums to zero in each direction; an entry's error is below 1e-8
of the largest, so the sum's is below 1e-8 of the sum of magnitudes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_dgesv_orders_on_one_context():
    from bem3d_elastostatic_b200 import _lib
    from bem3d_elastostatic_b200.api import dgesv

    ctx = _lib.Context(0)
    rng = np.random.default_rng(5)
    for n, nrhs in [(200, 1), (1500, 4), (33, 0), (200, 3), (1500, 4), (600, 40)]:
        A, B = rng.standard_normal((n, n)), rng.standard_normal((n, nrhs))
        for got, ref in zip(dgesv(A, B, ctx=ctx), dgesv(A, B)):
            assert np.array_equal(got, ref)


@pytest.mark.parametrize("m", [1, 3, 4])
def test_shape_gradient_sums_to_zero(m):
    from bem3d_elastostatic_b200.adjoint import compliance_gradient
    from bem3d_elastostatic_b200.mesh import hollow_sphere

    mesh = hollow_sphere(m, nu=0.3)
    _, gX, _, _ = compliance_gradient(mesh, range(mesh.ne // 2, mesh.ne))
    assert (np.abs(gX.sum(0)) <= 1e-8 * np.abs(gX).sum(0)).all()


@pytest.mark.parametrize("n", [294, 100, 900])
def test_dgesv_leaves_the_factors_of_a_solve(n):
    """A transposed solve with the factors of an FP64 solve, before and after a dgesv of the same
    order (294), a smaller and a larger one on the same context."""
    from bem3d_elastostatic_b200 import _lib
    from bem3d_elastostatic_b200.api import Quadesth, dgesv
    from bem3d_elastostatic_b200.mesh import uniaxial_cube

    q = Quadesth(uniaxial_cube(2))
    q.precompute_element_geometry()
    q.ghmat8()
    q.solve_linear_system("fp64")
    rng = np.random.default_rng(n)
    g = rng.standard_normal(q.mesh.ndof)

    def transposed():
        y = g.copy()
        q.ctx.check(q.ctx.L.bem_solve_transposed(q.ctx.h, _lib.ptr(y)), "solve_transposed")
        return y

    before = transposed()
    dgesv(rng.standard_normal((n, n)), rng.standard_normal(n), ctx=q.ctx)
    assert np.array_equal(transposed(), before)
    q.close()
