"""The pattern of entities with few to many incident tets (where the plan's
candidate sort changes form) against the CPU oracle, and its capacity limit."""
import numpy as np
import pytest

from emerge_b200 import _lib as L
from emerge_b200.assembly import GpuCSCMapping, tet_mass_stiffness_matrices
from emerge_b200.mesh import Nedelec2Field, TetMesh
from oracle import oracle as O
from tests.test_gpu_block_records import _fan

pytestmark = pytest.mark.gpu


# 6 edge candidates per tet: up to 32, 64, 128, 256 and past it; 4 face candidates
@pytest.mark.parametrize("n", [3, 5, 6, 8, 9, 10, 11, 16, 17, 21, 22, 32, 33, 42, 43, 64, 65])
def test_fan_pattern(n):
    f = Nedelec2Field(TetMesh(*_fan(n)))
    er = np.zeros((3, 3, n), np.complex128)
    for d in range(3):
        er[d, d] = 1.0
    _, _, om = O.tet_mass_stiffness_matrices(f, er, er, np.zeros(0, np.int64))
    _, _, cm = tet_mass_stiffness_matrices(f, er, er, np.zeros(0, np.int64))
    assert np.array_equal(cm.indptr, om.indptr) and np.array_equal(cm.indices, om.indices)


@pytest.mark.parametrize("n", [84, 85])
def test_capacity(n):
    """84 tets: the axis and seven spokes, one chunk, have more than 1,024 rows; 85: the axis has 256 adjacent edges."""
    with pytest.raises(L.EmgError):
        GpuCSCMapping.from_field(Nedelec2Field(TetMesh(*_fan(n))))
