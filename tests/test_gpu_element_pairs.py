"""The two-lanes-per-tet element kernels (diagonal and full complex tensors in
FP64) at the edges of a warp's and a CTA's tets, with reciprocal and other
tensors in one warp: element blocks against the CPU oracle, A in the packed
and block layouts against its sum."""
import numpy as np
import pytest
import torch

from emerge_b200.assembly import DeviceMaterial, DeviceMesh, ElemValues, GpuCSCMapping, LinComb, _Job, _prec
from emerge_b200.mesh import Nedelec2Field, TetMesh, structured_box
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _case(n, kind, which):
    nodes, tets = structured_box(4, 3, 2, jitter=0.12, seed=9)
    f = Nedelec2Field(TetMesh(nodes, tets[:, :n]))
    rng = np.random.default_rng(n)
    t = np.zeros((2, 3, 3, n), np.complex128)
    for d in range(3):
        t[:, d, d] = rng.uniform(1, 6, (2, n)) * (1 - 0.01j * rng.uniform(0, 1, (2, n)))
    if kind == "full":
        off = rng.uniform(-0.3, 0.3, (2, 3, 3, n)) * (1 + 0.2j)
        sym = off + off.transpose(0, 2, 1, 3)
        other = {"none": np.zeros(n, bool), "one": np.arange(n) == n - 1, "odd": np.arange(n) % 2 == 1}[which]
        off = np.where(other, off, sym)
        for d in range(3):
            off[:, d, d] = 0
        t += off
    return f, t[0], t[1]


@pytest.mark.parametrize("kind,which", [("diag", "none"), ("full", "none"), ("full", "one"), ("full", "odd")])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 63, 64, 65, 129])
def test_element_pairs(n, kind, which):
    f, er, ur = _case(n, kind, which)
    dE, dB, ocmap = O.tet_mass_stiffness_matrices(f, er, ur, np.zeros(0, np.int64))
    dm = DeviceMesh(f, None)
    job = _Job(dm, DeviceMaterial(er, ur, dm.n_tets, dm.device), _prec("fp64"))
    for name, ref in (("K", dE), ("M", dB)):
        got, ref = np.asarray(ElemValues(job, name)).reshape(n, 400), np.asarray(ref).reshape(n, 400)
        # per tet, relative to its largest entry: the bound of the FP64 form's element blocks
        assert (np.abs(got - ref).max(axis=1) <= 1e-13 * np.abs(ref).max(axis=1)).all()
    a, b = 1.0 + 0.5j, -3000.0 + 70.0j
    ref = ocmap.values_lincomb(dE, dB, a, b)
    out = []
    for layout in ("packed", "block"):
        c = GpuCSCMapping(dm, value_layout=layout)
        out.append(c.to_device(LinComb(job, {"K": a, "M": b})))
        assert np.linalg.norm(out[-1].cpu().numpy() - ref) <= 1e-12 * np.linalg.norm(ref)
    assert torch.equal(out[0], out[1])
