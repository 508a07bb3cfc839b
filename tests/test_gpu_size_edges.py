"""Sizes at which the plan build and the key sort change kernels: 12 and 13 tets
about an edge (candidates in registers, in shared memory), and one whole
shared-memory tile of 2,048 keys or two."""
import numpy as np
import pytest

from emerge_b200.assembly import GpuCSCMapping, tet_mass_stiffness_matrices
from emerge_b200.mesh import Nedelec2Field, TetMesh, plane_tris, structured_box
from emerge_b200.robin import RobinTerm
from oracle import oracle as O
from tests.test_gpu_block_records import _fan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [12, 13])
def test_tets_about_an_edge(n):
    f = Nedelec2Field(TetMesh(*_fan(n)))
    er = np.zeros((3, 3, n), np.complex128)
    for d in range(3):
        er[d, d] = 1.0
    _, _, om = O.tet_mass_stiffness_matrices(f, er, er, np.zeros(0, np.int64))
    _, _, cm = tet_mass_stiffness_matrices(f, er, er, np.zeros(0, np.int64))
    assert np.array_equal(cm.indptr, om.indptr) and np.array_equal(cm.indices, om.indices)


# 8 keys per triangle, padded to a power of two: 1,024, 2,048, 2,048, 4,096, 4,096, 8,192
@pytest.mark.parametrize("n", [128, 129, 256, 257, 512, 513])
def test_keys_of_a_tile(n):
    f = Nedelec2Field(TetMesh(*structured_box(13, 12, 2, jitter=0.1, seed=1)))
    face = plane_tris(f.mesh, 2, float(f.mesh.nodes[2].min()))
    ids = np.resize(np.random.default_rng(0).permutation(face), n)
    rng = np.random.default_rng(n)
    U = rng.normal(size=(3, 6, n)) + 1j * rng.normal(size=(3, 6, n))
    got = RobinTerm(f, ids, GpuCSCMapping.from_field(f)).force(U).cpu().numpy()
    b = O.force_entries(f, ids, U)
    assert np.linalg.norm(got - b) <= 1e-12 * np.linalg.norm(b)
