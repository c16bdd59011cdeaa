"""The batch solve across its step shapes: orders that end inside a panel and inside a block
row, one CTA per panel cluster up to sixteen, one to four rows per thread, few and many systems
at once.  Bar: the backward error of every load case against the assembled FP64 system, 1e-14
(FP64 rounding of a residual at these orders), and both precisions' solutions equal to 1e-9
(condition numbers up to 1e5 on backward errors of 1e-15 to 1e-16).
"""
import numpy as np
import pytest

from bem3d_elastostatic_b200.mesh import loaded_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ks,loads", [([1], 1), ([1, 6, 2], 8), ([3, 5] * 2, 5), ([6] * 12, 2), ([6] * 44 + [1, 4], 3)])
def test_backward_error(ks, loads):
    from bem3d_elastostatic_b200.api import Batch

    rng = np.random.default_rng(len(ks))
    b = Batch()
    for k in ks:
        b.add(*loaded_box(*rng.uniform(0.7, 1.5, 3), k, rng.uniform(0.1, 0.4), 1.0, rng.standard_normal((loads, 3))))
    b.assemble()
    x = {}
    for precision in ("fp32-ir", "fp64"):
        info = b.solve(precision)
        assert info["singular"] == 0 and info["max_backward_error"] <= 1e-14
        x[precision] = [b.solution(i) for i in range(len(ks))]
    for i in range(0, len(ks), max(1, len(ks) // 5)):
        A, F = b.system(i)
        for xs in x.values():
            r = np.abs(F - A @ xs[i]).max(0) / (np.abs(A).sum(1).max() * np.abs(xs[i]).max(0) + np.abs(F).max(0))
            assert r.max() <= 1e-14, (i, r)
        d = np.abs(x["fp64"][i] - x["fp32-ir"][i]).max() / np.abs(x["fp64"][i]).max()
        assert d <= 1e-9, (i, d)
    b.close()


def test_systems_added_after_a_solve():
    """The captured solve belongs to the systems it was captured for."""
    from bem3d_elastostatic_b200.api import Batch

    b = Batch()
    first = loaded_box(1.0, 1.0, 1.0, 2, 0.3)
    b.add(*first)
    b.assemble()
    b.solve("fp64")
    x0 = b.solution(0)
    b.add(*loaded_box(1.2, 0.9, 1.0, 3, 0.2))
    b.assemble()
    assert b.solve("fp64")["systems"] == 2
    assert np.abs(b.solution(0) - x0).max() <= 1e-12 * np.abs(x0).max()
    b.close()


def test_system_above_the_clusters_capacity():
    """8,718 unknowns in FP64, above the 8,192 of a cluster: the LU of one CTA per system, for the
    small system beside it too."""
    from bem3d_elastostatic_b200.api import Batch

    rng = np.random.default_rng(11)
    b = Batch()
    for k in (2, 11):
        b.add(*loaded_box(*rng.uniform(0.7, 1.5, 3), k, 0.3, 1.0, rng.standard_normal((2, 3))))
    b.assemble()
    info = b.solve("fp64")
    assert info["lu_threads"] == 512 and info["singular"] == 0 and info["max_backward_error"] <= 1e-14
    for i in range(2):
        A, F = b.system(i)
        x = b.solution(i)
        r = np.abs(F - A @ x).max(0) / (np.abs(A).sum(1).max() * np.abs(x).max(0) + np.abs(F).max(0))
        assert r.max() <= 1e-14, (i, r)
    assert b.solve("fp32-ir")["lu_threads"] == 256  # within the 16,384 of FP32
    b.close()
