"""Submatrices of few solve DoFs (sorted) and of many (through the mask): the ids
ascending and distinct, the pattern and values those of scipy's slicing."""
import numpy as np
import pytest

from emerge_b200.assembly import tet_mass_stiffness_matrices
from emerge_b200.mesh import Nedelec2Field, TetMesh, structured_box
from emerge_b200.solve_dofs import SolveSubmatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("part", [0, 1, 2, 63, 64, 65, 10_000])
def test_ids(part):
    f = Nedelec2Field(TetMesh(*structured_box(5, 4, 3, jitter=0.1, seed=3)))
    er = np.zeros((3, 3, f.ntets), np.complex128)
    for d in range(3):
        er[d, d] = 2.0 - 0.1j
    E, B, cmap = tet_mass_stiffness_matrices(f, er, np.ones((3, 3, 1)) * np.eye(3)[:, :, None] * np.ones(f.ntets),
                                             np.zeros(0, np.int64))
    N = f.n_field
    n = min(part * N // (64 * 64) if part < 10_000 else N, N)  # from none to N / 64 and past it, and all
    rng = np.random.default_rng(part)
    ids = rng.permutation(N)[:n]
    ids = rng.permutation(np.r_[ids, ids[: n // 3]])  # any order, some twice
    sub = SolveSubmatrix(cmap, ids)
    want = np.unique(ids)
    assert sub.solve_ids.dtype == np.int64 and np.array_equal(sub.solve_ids, want)
    assert np.array_equal(sub.d_ids.cpu().numpy(), want)
    A = cmap.to_csc(E - B * 2.0)
    ref = A[:, want][want, :].tocsc()
    ref.sort_indices()
    assert sub.M == want.size and sub.nnz == ref.nnz
    assert np.array_equal(sub.d_indptr[: sub.M + 1].cpu().numpy(), ref.indptr)
    assert np.array_equal(sub.d_indices[: sub.nnz].cpu().numpy(), ref.indices)
    assert np.array_equal(sub.values(cmap.to_device(E - B * 2.0)).cpu().numpy(), ref.data)
