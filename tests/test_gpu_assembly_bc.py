"""Assembly with every mix of prescribed components, on quad9 and tri6 elements, against the
oracle.  Bars of the parity suite: A and H, G within 1e-12 of the row's largest entry, FI
within 1e-12 of its own; the FP32 far field within 2e-6 of the row's largest entry (FP32
products accumulated in FP32).
"""
import numpy as np
import pytest

import oracle as O
from bem3d_elastostatic_b200.mesh import loaded_box
from test_gpu_points import octahedron

pytestmark = pytest.mark.gpu


def mixed_mesh(name, combos):
    """Elements cycle through the given sets of prescribed components, every value non-zero
    (a node's prescribed displacement may differ between its elements: the first one counts)."""
    mesh = octahedron() if name == "tri6" else loaded_box(1.0, 0.7, 1.2, 3 if name == "box3" else 2, 0.23)[0]
    rng = np.random.default_rng(len(combos))
    for e in range(mesh.ne):
        for ld in range(3):
            mesh.kode[3 * e + ld] = 0 if ld in combos[e % len(combos)] else 1
    mesh.bc[:] = rng.standard_normal(mesh.bc.shape)
    mesh.pins = np.zeros(0, np.int32)
    return mesh


def rows_close(got, ref, rel):
    return np.abs(got - ref).max(1) <= rel * np.abs(ref).max(1)


@pytest.mark.parametrize("name", ["box", "box3", "tri6"])
@pytest.mark.parametrize("combos", [[()], [(0,), (), (1,), (2,)], [(0, 2), (1,), ()], [(0, 1, 2), ()],
                                    [(), (0, 1, 2), (2,), (1, 2)]])
def test_system_for_prescribed_components(name, combos):
    from bem3d_elastostatic_b200.api import Quadesth

    mesh = mixed_mesh(name, combos)
    Ar, Fr = O.Oracle(mesh).ghmat8()[:2]
    q = Quadesth(mesh)
    q.precompute_element_geometry()
    A, F = q.ghmat8(return_system=True)
    assert rows_close(A, Ar, 1e-12).all()
    assert np.abs(F - Fr).max() <= 1e-12 * np.abs(Fr).max()
    A, F = q.ghmat8("fp32-far", return_system=True)
    assert rows_close(A, Ar, 2e-6).all()
    assert np.abs(F - Fr).max() <= 2e-6 * np.abs(Fr).max()


def test_unloaded_elements_leave_no_trace():
    """Zero tractions: FI comes from the prescribed displacements alone, and is zero for none."""
    from bem3d_elastostatic_b200.api import Quadesth

    mesh = mixed_mesh("box", [(0, 1, 2), ()])
    mesh.bc[:] = 0.0
    q = Quadesth(mesh)
    q.precompute_element_geometry()
    _, F = q.ghmat8(return_system=True)
    assert np.all(F == 0.0)


def test_hg_tri6():
    from bem3d_elastostatic_b200.api import Quadesth

    mesh = octahedron()
    Hr, Gr = O.Oracle(mesh).hg()
    q = Quadesth(mesh)
    q.precompute_element_geometry()
    H, G = q.hg()
    # columns of the nodes a tri6 element does not have stay as allocated: compare its 18
    cols = (27 * np.arange(mesh.ne)[:, None] + np.arange(18)).reshape(-1)
    assert rows_close(H, Hr, 1e-12).all() and rows_close(G[:, cols], Gr[:, cols], 1e-12).all()
