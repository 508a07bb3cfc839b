"""Full tensors: a tet's element values do not depend on the tets beside it. A
reciprocal tet has the same bits whether its neighbours are reciprocal or not,
and column shards, which group the tets in other ways, merge into the unsharded
matrix bit for bit."""
import numpy as np
import pytest

from emerge_b200.assembly import DeviceMaterial, DeviceMesh, ElemValues, _Job, _prec, tet_mass_stiffness_matrices
from emerge_b200.mesh import Nedelec2Field, TetMesh, structured_box
from emerge_b200.partition import ShardedAssembly, merge_blocks, partition

pytestmark = pytest.mark.gpu


def _tensors(n, other, seed=4):
    """eps and mu of n tets, complex and full: symmetric, except where `other`."""
    rng = np.random.default_rng(seed)
    t = rng.uniform(-0.3, 0.3, (2, 3, 3, n)) * (1 + 0.2j * rng.uniform(-1, 1, (2, 3, 3, n)))
    sym = t + t.transpose(0, 2, 1, 3)
    t = np.where(other, t, sym)
    for d in range(3):
        t[:, d, d] = rng.uniform(1, 6, (2, n)) * (1 - 0.01j * rng.uniform(0, 1, (2, n)))
    return t[0], t[1]


@pytest.mark.parametrize("precision", ["fp64", "exact"])
@pytest.mark.parametrize("step", [2, 16])
def test_reciprocal_tets_keep_their_values(precision, step):
    f = Nedelec2Field(TetMesh(*structured_box(5, 4, 6, jitter=0.12, seed=9)))
    dm = DeviceMesh(f, None)
    n = dm.n_tets
    other = np.arange(n) % step == step - 1
    values = []
    for o in (np.zeros(n, bool), other):
        er, ur = _tensors(n, o)
        job = _Job(dm, DeviceMaterial(er, ur, n, dm.device), _prec(precision))
        values.append([np.asarray(ElemValues(job, k)).reshape(n, 400) for k in ("K", "M")])
    for alone, beside in zip(*values):
        assert np.array_equal(alone[~other], beside[~other])
        assert not np.array_equal(alone[other], beside[other])


@pytest.mark.parametrize("precision", ["fp64", "exact"])
def test_shards_of_full_tensors_merge_to_full(precision):
    f = Nedelec2Field(TetMesh(*structured_box(9, 5, 14, jitter=0.12, seed=2)))
    n = f.ntets
    er, ur = _tensors(n, np.arange(n) % 7 == 3)
    cond = np.arange(5, n, 67)
    E, B, cmap = tet_mass_stiffness_matrices(f, er, ur, cond, precision=precision)
    ref = cmap.to_csc(E - B * 250.0 ** 2)
    for world in (2, 3):
        blocks = [ShardedAssembly(f, er, ur, s, precision).block(1.0 + 0j, complex(-250.0 ** 2))
                  for s in partition(f.mesh, world, cond)]
        ip, ix, vv = merge_blocks(blocks, f.n_field)
        assert np.array_equal(ip, ref.indptr) and np.array_equal(ix, ref.indices), world
        assert np.array_equal(vv, ref.data), world
