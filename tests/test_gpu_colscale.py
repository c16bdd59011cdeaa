"""The scaled FP32 copy of the equilibrated mode at odd and even orders and at the edges of a
thread's pairs and turns.  Rows in units 2^k leave r_i A_ij c_j, the factors and the Krylov
vectors as they are, bit for bit, since the row scales are powers of two: a solve that stops
after its first cycle (tolerance 1e-3) returns the same bits for A x = b and D A x = D b.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# and the last order of four CTAs per SM, the first of two
@pytest.mark.parametrize("n", [14144, 14145])
def test_row_units_change_nothing_where_the_ctas_change(n):
    test_row_units_change_nothing(n)


@pytest.mark.parametrize("n", [2, 33, 1001, 2047, 2048, 2049, 16387])
def test_row_units_change_nothing(n):
    from bem3d_elastostatic_b200.api import solve_system

    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    A /= np.sqrt(n)
    A[np.diag_indices(n)] += 3.0
    b = rng.standard_normal(n)
    x, info = solve_system(A, b, "bf16-ir", tol=1e-3)
    d = 2.0 ** rng.integers(-6, 7, n)
    y, scaled = solve_system(A * d[:, None], b * d, "bf16-ir", tol=1e-3)
    assert info["restarts"] == scaled["restarts"] and info["iterations"] == scaled["iterations"]
    assert np.array_equal(x, y)
    assert np.abs(A @ x - b).max() <= 1e-3 * (np.abs(A).sum(1).max() * np.abs(x).max() + np.abs(b).max())
