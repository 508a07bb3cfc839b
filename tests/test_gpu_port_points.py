"""Port overlap integrals for every length of the triangle rule and triangle
counts around a CTA's, and the solution at points of every vertex order,
against the CPU oracle (1e-12 relative, the bound of the reference's own
output)."""
import numpy as np
import pytest

from emerge_b200.mesh import Nedelec2Field, TetMesh, plane_tris, structured_box
from emerge_b200.postprocess import FieldOnDevice, PortOverlap
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _field(seed):
    nodes, tets = structured_box(4, 3, 2, jitter=0.12, seed=seed)
    rng = np.random.default_rng(seed)
    p = rng.permutation(nodes.shape[1])  # new numbers for the vertices: all vertex orders occur
    new = np.empty_like(p)
    new[p] = np.arange(p.size)
    f = Nedelec2Field(TetMesh(nodes[:, p], new[tets]))
    return f, rng.normal(size=f.n_field) + 1j * rng.normal(size=f.n_field)


@pytest.mark.parametrize("nq,nb", [(1, 1), (2, 7), (6, 8), (7, 9), (15, 16), (16, 17), (16, 24)])
def test_rule_lengths(nq, nb):
    f, x = _field(nq)
    rng = np.random.default_rng(nb)
    L = rng.dirichlet(np.ones(3), nq).T
    rule = np.concatenate([rng.uniform(0.1, 1, (1, nq)), L])
    fod = FieldOnDevice(f)
    po = PortOverlap(fod, plane_tris(f.mesh, 2, float(f.mesh.nodes[2].min()))[:nb], rule)
    U = rng.normal(size=(3, nq, nb)) + 1j * rng.normal(size=(3, nq, nb))
    tot, per = po(x, U, 0.7)
    rtot, rper = O.port_overlap(f, x, po.ids, po.tri_tets, rule, U, 0.7)
    scale = np.abs(rper).max()
    assert np.abs(per.cpu().numpy() - rper).max() <= 1e-12 * scale
    assert abs(tot - rtot) <= 1e-12 * scale * nb


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000])
def test_points(n):
    f, x = _field(n)
    rng = np.random.default_rng(n)
    tet = rng.integers(0, f.ntets, n)
    pts = np.einsum("dvn,vn->dn", f.mesh.nodes[:, f.mesh.tets[:, tet]], rng.dirichlet(np.ones(4), n).T)
    ref = O.ned2_interp(f, x, pts, tet)
    for p in (np.ascontiguousarray(pts), np.asfortranarray(pts)):  # either layout of the caller's array
        got = FieldOnDevice(f).interpolate(x, p, tet).cpu().numpy()
        assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
