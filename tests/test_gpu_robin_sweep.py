"""A boundary term added to many frequencies in one launch equals the term
added to each, bit for bit, around the number of coefficients of a launch."""
import numpy as np
import pytest
import torch

from emerge_b200.assembly import GpuCSCMapping
from emerge_b200.mesh import Nedelec2Field, TetMesh, plane_tris, structured_box
from emerge_b200.robin import RobinTerm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf", [1, 3, 63, 64, 65, 130])
def test_apply_sweep(nf):
    f = Nedelec2Field(TetMesh(*structured_box(3, 2, 3, jitter=0.1, seed=5)))
    c = GpuCSCMapping.from_field(f)
    term = RobinTerm(f, plane_tris(f.mesh, 2, float(f.mesh.nodes[2].max())), c)
    g = torch.Generator(device="cuda").manual_seed(nf)
    A = torch.view_as_complex(torch.randn(nf, c.nnz, 2, generator=g, device="cuda", dtype=torch.float64))
    gamma = np.random.default_rng(nf).normal(size=(nf, 2)) @ np.array([1.0, 1.0j])
    want = A.clone()
    for i in range(nf):
        term.apply(want[i], gamma[i])
    assert torch.equal(term.apply_sweep(A, gamma), want)
