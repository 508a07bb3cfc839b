"""The key sort behind the port term and the chunk order, at sizes around its
shared-memory tile: the forcing vector of n boundary triangles (8 n keys padded
to a power of two) against the CPU oracle."""
import numpy as np
import pytest
import torch

from emerge_b200.assembly import GpuCSCMapping
from emerge_b200.mesh import Nedelec2Field, TetMesh, plane_tris, structured_box
from emerge_b200.robin import RobinTerm
from oracle import oracle as O

pytestmark = pytest.mark.gpu


# keys: 8, 1,024, 8,192, 16,384, 32,768, 65,536, 131,072 and 262,144
@pytest.mark.parametrize("n", [1, 100, 1000, 1025, 2049, 4097, 8193, 16385])
def test_force_at_key_counts(n):
    f = Nedelec2Field(TetMesh(*structured_box(13, 12, 2, jitter=0.1, seed=1)))
    face = plane_tris(f.mesh, 2, float(f.mesh.nodes[2].min()))
    ids = np.resize(np.random.default_rng(0).permutation(face), n)  # a triangle may be listed many times
    rng = np.random.default_rng(n)
    U = rng.normal(size=(3, 6, n)) + 1j * rng.normal(size=(3, 6, n))
    term = RobinTerm(f, ids, GpuCSCMapping.from_field(f))
    got = term.force(U).cpu().numpy()
    b = O.force_entries(f, ids, U)
    assert np.linalg.norm(got - b) <= 1e-12 * np.linalg.norm(b)
    again = term.force(U).cpu().numpy()
    assert np.array_equal(got, again)
