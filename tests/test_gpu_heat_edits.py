"""A heat field whose arrays change between two calls: each call's matrices are
those of a fresh field with the arrays as they are then."""
import copy

import numpy as np
import pytest

from emerge_b200.heat import Legrange2, tet_mass_matrix, tet_stiffness_matrix
from emerge_b200.mesh import TetMesh, structured_box

pytestmark = pytest.mark.gpu


def _field():
    return Legrange2(TetMesh(*structured_box(5, 4, 3, jitter=0.1, seed=7)))


def _same_as_fresh(f):
    fresh = copy.copy(f)
    fresh.mesh = copy.copy(f.mesh)
    for o, names in ((fresh, ["tet_to_field"]), (fresh.mesh, ["nodes", "tets"])):
        for name in names:
            setattr(o, name, getattr(o, name).copy())
    n = f.mesh.n_tets
    cond = np.broadcast_to(np.eye(3)[:, :, None], (3, 3, n)) * np.linspace(1.0, 2.0, n)
    for call, coef in ((tet_stiffness_matrix, cond), (tet_mass_matrix, np.linspace(1.0, 3.0, n))):
        got = [cm.to_csc(v) for v, cm in (call(f, coef),)][0]
        want = [cm.to_csc(v) for v, cm in (call(fresh, coef),)][0]
        call(f, coef)  # f is the field that is kept again
        assert np.array_equal(got.indptr, want.indptr) and np.array_equal(got.indices, want.indices)
        assert np.array_equal(got.data, want.data)


def _edit_nodes(f):
    f.mesh.nodes[2] *= 1.25


def _edit_dofs(f):
    p = np.random.default_rng(0).permutation(f.n_field)
    f.tet_to_field[...] = p[f.tet_to_field]


def _edit_tets(f):
    f.mesh.tets[:2] = f.mesh.tets[1::-1].copy()


def _replace_nodes(f):
    f.mesh.nodes = f.mesh.nodes * 0.5


def _replace_dofs(f):
    f.tet_to_field = (f.tet_to_field + 1) % f.n_field


def _renumber(f):
    f.n_field += 3


@pytest.mark.parametrize("edit", [_edit_nodes, _edit_dofs, _edit_tets, _replace_nodes, _replace_dofs, _renumber])
def test_matrices_follow_the_field(edit):
    f = _field()
    _, cmap = tet_stiffness_matrix(f, np.tile(np.eye(3)[:, :, None], (1, 1, f.mesh.n_tets)))
    assert tet_mass_matrix(f, np.ones(f.mesh.n_tets))[1] is cmap
    edit(f)
    _same_as_fresh(f)


def test_arrays_replaced_many_times():
    """A new array may get the address of the one that it replaces."""
    f = _field()
    for k in range(1, 9):
        f.tet_to_field = (f.tet_to_field + k) % f.n_field
        _same_as_fresh(f)
