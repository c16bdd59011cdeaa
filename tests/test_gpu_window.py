"""The FP32 window LU where windows need interchanges, meet exact ties and zero pivots: systems
whose 32 x 32 diagonal blocks are permuted, scaled or singular, solved by the mixed modes against
LAPACK.  Bar: 1e-10 of the solution's largest entry (well-conditioned systems).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def system(kind, n, rng):
    A = 0.3 * rng.standard_normal((n, n)) / np.sqrt(n)
    if kind == "diagonal":
        A += 2.0 * np.eye(n)
    elif kind == "permuted":  # large entries off the diagonal, inside each 32-block
        for b in range(0, n, 32):
            k = min(32, n - b)
            A[b + rng.permutation(k), b + np.arange(k)] += 2.0 * rng.choice([-1.0, 1.0], k)
    elif kind == "ties":  # equal magnitudes in a block's rows: Hadamard blocks
        H = np.array([[1.0]])
        while H.shape[0] < 32:
            H = np.block([[H, H], [H, -H]])
        for b in range(0, n - 31, 32):
            A[b:b + 32, b:b + 32] += H / 4.0
        A[n // 32 * 32:, n // 32 * 32:] += 2.0 * np.eye(n % 32)
    return np.asfortranarray(A)


@pytest.mark.parametrize("precision", ["fp32-ir", "bf16-ir"])
@pytest.mark.parametrize("kind,n", [("diagonal", 640), ("permuted", 1500), ("permuted", 2100), ("ties", 1312)])
def test_windows(precision, kind, n):
    from bem3d_elastostatic_b200.api import solve_system

    rng = np.random.default_rng(n)
    A = system(kind, n, rng)
    b = rng.standard_normal(n)
    x, info = solve_system(A, b, precision)
    ref = np.linalg.solve(A, b)
    assert info["fallbacks"] == 0
    assert np.abs(x - ref).max() <= 1e-10 * np.abs(ref).max()
