"""The sweeps of FP32 factors at orders where the schedule changes: one block, a ragged last block,
one block more than the CTAs of a sweep.  Both mixed modes against
the substitution sweeps (a context created with BEM_SWEEP_INV=0).  Each solution carries the
refinement's own error, below 1e-12 of its largest entry for these well-conditioned systems, so
their difference has the bar 2e-12; the preconditioners differ by FP64 rounding only, so the
refinement takes the same number of steps, or one more.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32-ir", "bf16-ir"])
@pytest.mark.parametrize("n", [100, 128, 129, 1000, 148 * 128 + 3])
def test_ring_sweeps(precision, n, monkeypatch):
    from bem3d_elastostatic_b200.api import solve_system

    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    A /= np.sqrt(n)
    A[np.diag_indices(n)] += 3.0
    b = rng.standard_normal(n)
    x, info = solve_system(A, b, precision)
    monkeypatch.setenv("BEM_SWEEP_INV", "0")
    y, sub = solve_system(A, b, precision)
    assert info["fallbacks"] == sub["fallbacks"]
    assert abs(info["iterations"] - sub["iterations"]) <= 1
    assert np.abs(x - y).max() <= 2e-12 * np.abs(y).max()
