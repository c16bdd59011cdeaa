"""FP64 LU with partial pivoting at the orders where the sub-panel's cluster changes: one
CTA, a remainder of 32 columns, the first order with two CTAs, 16 CTAs at one line per
thread and at two; against LAPACK's dgetrf of A^T.

Bars: the pivots equal (random entries leave no ties that rounding could turn), the factors
within 1e-10 of their largest value (element growth of a few hundred units of rounding at
these orders), the solution's backward error at 1e-13.
"""
import numpy as np
import pytest
from scipy.linalg import lu_factor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 513, 1100, 4130, 8300])
def test_dgesv_factors(n):
    from bem3d_elastostatic_b200.api import dgesv

    rng = np.random.default_rng(n)
    A = np.asfortranarray(rng.standard_normal((n, n)))
    B = np.asfortranarray(rng.standard_normal((n, 2)))
    S, ipiv, X, info = dgesv(A, B)
    ref, piv = lu_factor(A.T)
    assert info == 0
    assert np.array_equal(ipiv - 1, piv)
    assert np.abs(S.T - ref).max() <= 1e-10 * np.abs(ref).max()
    r = np.abs(B - A @ X).max() / (np.abs(A).sum(1).max() * np.abs(X).max())
    assert r <= 1e-13


def test_ties_take_the_first_row():
    """Entries +-1: the first steps' candidates tie exactly, the smallest row wins."""
    from bem3d_elastostatic_b200.api import dgesv

    A = np.asfortranarray(np.sign(np.random.default_rng(0).standard_normal((700, 700))))
    _, ipiv, _, info = dgesv(A, np.ones(700))
    _, piv = lu_factor(A.T)
    assert info == 0 and np.array_equal(ipiv[:4] - 1, piv[:4])


@pytest.mark.parametrize("n,col", [(40, 0), (600, 599), (1300, 77)])
def test_zero_pivot_is_reported(n, col):
    """A^T with a zero column (row `col` of A zero): info is that step, as dgetrf's."""
    from bem3d_elastostatic_b200.api import dgesv

    A = np.asfortranarray(np.random.default_rng(n).standard_normal((n, n)))
    A[col, :] = 0.0
    _, _, _, info = dgesv(A, np.ones(n))
    assert info == col + 1
