"""Small meshes, whose tets several CTAs share by block rows (five, three or two
parts, or none): A in the block layout equals A in the packed layout, which is
never split, bit for bit."""
import numpy as np
import pytest
import torch

from emerge_b200.assembly import DeviceMaterial, DeviceMesh, GpuCSCMapping, _Job, _prec
from emerge_b200.mesh import Nedelec2Field, TetMesh, structured_box

pytestmark = pytest.mark.gpu


# CTAs of 128 tets on 148 SMs, two per SM in FP64 (five parts up to 59 CTAs, three up
# to 98, two up to 148) and five in the mixed form (148, 246, 370); diagonal
# tensors: CTAs of 64 in FP64
@pytest.mark.parametrize("grid", [(1, 1, 1), (6, 4, 10), (11, 5, 15), (12, 6, 20), (12, 6, 30), (17, 7, 38), (20, 10, 35)])
@pytest.mark.parametrize("kind,precision", [("iso", "fp64"), ("iso", "mixed"), ("iso", "exact"), ("diag", "fp64"),
                                            ("diag", "mixed")])
def test_parts(grid, kind, precision):
    f = Nedelec2Field(TetMesh(*structured_box(*grid, jitter=0.1, seed=grid[2])))
    dm = DeviceMesh(f, np.array([0], np.int64) if grid[0] > 1 else None)
    rng = np.random.default_rng(1)
    e = rng.uniform(1, 5, dm.n_tets) * (1 - 0.01j)
    if kind == "iso":
        mat = DeviceMaterial(e, None, dm.n_tets, dm.device)
    else:
        t = np.zeros((3, 3, dm.n_tets), np.complex128)
        for d in range(3):
            t[d, d] = e * (1 + 0.1 * d)
        mat = DeviceMaterial(t, t, dm.n_tets, dm.device)
    job = _Job(dm, mat, _prec(precision))
    out = []
    for layout in ("packed", "block"):
        c = GpuCSCMapping(dm, value_layout=layout)
        c.workspace(job.precision).fill_(255)  # NaNs: a row that no part writes shows
        out.append(c.assemble_device(job, 1.0, -1234.5)[: c.nnz])
        dm.check_status()
    assert bool(torch.isfinite(torch.view_as_real(out[1])).all()) and torch.equal(out[0], out[1])
