"""Internal points at the edges of the kernels' tiles and rules, against the oracle.

Bar: 1e-10 of the largest value, the parity suite's bound for internal displacements and
stresses (the sums agree to rounding, ~1e-13; principal stresses are formed from them by the
same closed form and not compared near double eigenvalues).
"""
import numpy as np
import pytest

import oracle as O
from bem3d_elastostatic_b200.mesh import Mesh, loaded_box

pytestmark = pytest.mark.gpu


def octahedron(nu=0.3):
    """Eight tri6 elements, clamped on one face, loaded on another."""
    v = np.array([[1, 0, 0], [-1, 0, 0], [0, 1.2, 0], [0, -1.2, 0], [0, 0, 0.9], [0, 0, -0.9]], float)
    nodes = [tuple(p) for p in v]
    conn = []
    for i in (0, 1):
        for j in (2, 3):
            for k in (4, 5):
                tri = (i, j, k) if np.dot(np.cross(v[j] - v[i], v[k] - v[i]), v[i]) > 0 else (i, k, j)
                el = list(tri)
                for a, b in ((0, 1), (1, 2), (2, 0)):
                    m = tuple(0.5 * (v[tri[a]] + v[tri[b]]))
                    if m not in nodes:
                        nodes.append(m)
                    el.append(nodes.index(m))
                conn.append(el + [0, 0, 0])
    ne = 8
    xyz = np.array(nodes)
    kode = np.ones(3 * ne, dtype=np.int32)
    kode[:3] = 0
    bc = np.zeros((27, ne), order="F")
    bc[:, 7] = np.tile([0.3, -0.7, 1.0], 9)
    return Mesh(xyz[:, 0], xyz[:, 1], xyz[:, 2], np.full(ne, 6), np.array(conn).T + 1, kode, bc,
                1.0 / (2.0 * (1.0 + nu)), nu)


def box(k):
    return loaded_box(1.0, 0.8, 1.3, k, 0.27, top_tractions=np.array([[0.4, -0.2, 1.0]]))[0]


@pytest.mark.parametrize("name,points,kelvin", [
    ("box", 1, False), ("box", 33, True), ("box", 257, False), ("box4", 300, False), ("tri6", 40, False)])
def test_points_at_tile_edges(name, points, kelvin):
    """One point, a remainder of a warp and of a tile, near lists of 1 to 8 slices; tri6
    elements near and far (points outside the body have only a formal value, the same sums)."""
    from bem3d_elastostatic_b200.api import Quadesth

    mesh = octahedron() if name == "tri6" else box(4 if name == "box4" else 2)
    rng = np.random.default_rng(points)
    pts = rng.uniform(0.05, 0.75, (points, 3)) * (1.0 if name != "tri6" else 0.3)
    if name == "tri6":
        pts[::2] += 9.0
    q = Quadesth(mesh)
    q.run()
    u, t = q.reorganize_solution()
    got = q.compute_internal_points(pts, kelvin_consistent=kelvin)
    ref = O.Oracle(mesh.with_points(*pts.T)).internal_points(u, t, kelvin_consistent=kelvin)
    for g, r in zip((got[0], got[1], got[3]), (ref[0], ref[1], ref[3])):
        assert np.abs(g - r).max() <= 1e-10 * np.abs(r).max()


def test_points_in_halves():
    """More (point, near element) pairs than are evaluated at a time: the range is halved,
    and every point keeps its value."""
    from bem3d_elastostatic_b200.api import Quadesth

    mesh = box(2)
    q = Quadesth(mesh)
    q.run()
    pts = np.random.default_rng(3).uniform(0.05, 0.75, (1_100_001, 3))  # 24 elements, all near
    big = q.compute_internal_points(pts)
    for sl in (slice(0, 500), slice(549_800, 550_300), slice(1_099_501, 1_100_001)):
        small = q.compute_internal_points(pts[sl])
        for a, b in zip(big[:2], small[:2]):
            assert np.abs(a[..., sl] - b).max() <= 1e-12 * np.abs(b).max()
