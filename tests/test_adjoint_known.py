"""The prescribed displacements by dof against the incidences one by one: meshes with shared nodes,
mixed conditions and nodes with more than eight elements.  Equal, value for value.
"""
import types

import numpy as np
import pytest

from bem3d_elastostatic_b200.adjoint import _known_values


def one_by_one(mesh):
    uk, vp = np.zeros(mesh.ndof, dtype=bool), np.zeros(mesh.ndof)
    order = [[] for _ in range(mesh.n)]
    for e in range(mesh.ne):
        for k in range(int(mesh.nconec[e])):
            order[mesh.kconec[k, e] - 1].append((e, k))
    for i in range(mesh.n):
        for ld in range(3):
            for e, k in order[i][:8]:
                if mesh.kode[3 * e + ld] == 0:
                    uk[3 * i + ld], vp[3 * i + ld] = True, mesh.bc[3 * k + ld, e]
                    break
    return uk, vp


@pytest.mark.parametrize("ne,n,nodes", [(1, 9, 9), (40, 30, 9), (64, 500, 8), (200, 12, 9)])
def test_known_values(ne, n, nodes):
    rng = np.random.default_rng(ne)
    mesh = types.SimpleNamespace(
        ne=ne, n=n, ndof=3 * n, nconec=rng.integers(1, nodes + 1, ne), kconec=rng.integers(1, n + 1, (9, ne)),
        kode=rng.integers(0, 2, 3 * ne), bc=rng.standard_normal((27, ne)))
    for got, ref in zip(_known_values(mesh), one_by_one(mesh)):
        assert np.array_equal(got, ref)
