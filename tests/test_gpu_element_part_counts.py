"""Small meshes on both sides of the CTA counts up to which their tets are shared
by five, three or two CTAs (29, 49 and 74 of 148 SMs): A in the block layout equals
A in the packed layout, which is never shared, bit for bit."""
import numpy as np
import pytest
import torch

from emerge_b200.assembly import DeviceMaterial, DeviceMesh, GpuCSCMapping, _Job, _prec
from emerge_b200.mesh import Nedelec2Field, TetMesh, structured_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctas", [29, 30, 49, 50, 74, 75])
@pytest.mark.parametrize("kind,precision,per_cta", [("iso", "fp64", 128), ("iso", "mixed", 128), ("full", "fp64", 64)])
def test_at_cta_counts(ctas, kind, precision, per_cta):
    nodes, tets = structured_box(16, 10, 10, jitter=0.1, seed=6)
    n = (ctas - 1) * per_cta + 1  # the last CTA has one tet
    dm = DeviceMesh(Nedelec2Field(TetMesh(nodes, tets[:, :n])), None)
    rng = np.random.default_rng(ctas)
    if kind == "iso":
        mat = DeviceMaterial(rng.uniform(1, 5, n) * (1 - 0.01j), None, n, dm.device)
    else:
        t = rng.uniform(-0.2, 0.2, (2, 3, 3, n)) * (1 - 0.02j)
        for d in range(3):
            t[:, d, d] = rng.uniform(1, 5, (2, n))
        t[:, :, :, ::2] += t.transpose(0, 2, 1, 3)[:, :, :, ::2].copy()  # every other tet reciprocal
        mat = DeviceMaterial(t[0], t[1], n, dm.device)
    job = _Job(dm, mat, _prec(precision))
    out = []
    for layout in ("packed", "block"):
        c = GpuCSCMapping(dm, value_layout=layout)
        c.workspace(job.precision).fill_(255)  # NaNs: a row that no part writes shows
        out.append(c.assemble_device(job, 1.0, -1234.5)[: c.nnz])
        dm.check_status()
    assert bool(torch.isfinite(torch.view_as_real(out[1])).all()) and torch.equal(out[0], out[1])
