"""The mixed modes at panel widths of one to eight 128-blocks, on orders with ragged last
panels: the panel's triangle inverses take a different number of block columns each.  Bar: 1e-10
of the FP64 reference solution, the mixed modes' bound, and no fallback to partial pivoting.
"""
import numpy as np
import pytest

from bem3d_elastostatic_b200.mesh import loaded_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32-ir", "bf16-ir"])
@pytest.mark.parametrize("width", [128, 256, 384, 640, 896, 1024])
def test_panel_widths(precision, width):
    from bem3d_elastostatic_b200 import _lib
    from bem3d_elastostatic_b200.api import Quadesth

    q = Quadesth(loaded_box(1.0, 0.9, 1.2, 6, 0.31, top_tractions=np.array([[0.3, -0.5, 1.0]]))[0])  # 2,598 DOF
    q.precompute_element_geometry()
    q.ghmat8()
    ref = q.solve_linear_system("fp64-ir")
    q.set_option(_lib.BEM_OPT_PANEL_WIDTH, width)
    x = q.solve_linear_system(precision)
    assert q.solve_info["fallbacks"] == 0
    assert np.abs(x - ref).max() <= 1e-10 * np.abs(ref).max()
