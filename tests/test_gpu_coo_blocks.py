"""The COO -> CSC mapping of element blocks against that of the same slots as
lists: pattern, slot order and runs are the same."""
import numpy as np
import pytest
import torch

from emerge_b200.heat import GpuCOOMapping

pytestmark = pytest.mark.gpu


# DoFs per tet of their own and of the field's size (0: all DoFs of a tet the same), with one
# column shared by every tet: lists on both sides of the register sort's 512 slots
@pytest.mark.parametrize("D,nT,N", [(10, 1, 40), (10, 7, 30), (10, 52, 300), (10, 51, 12), (10, 300, 900), (10, 5, 1),
                                    (1, 33, 5), (3, 200, 50), (4, 0, 7), (20, 40, 100)])
def test_blocks(D, nT, N):
    rng = np.random.default_rng(D * 1000 + nT)
    t2f = rng.integers(0, N, (D, nT))
    t2f[rng.integers(0, D), :] = N - 1
    got = GpuCOOMapping.from_tet_to_field(t2f, N)
    rows = np.repeat(t2f.T, D, axis=1).ravel()
    cols = np.tile(t2f.T, (1, D)).ravel()
    want = GpuCOOMapping.from_rowcol(rows, cols, N)
    assert got.nnz == want.nnz and got.S == want.S and got.block_dofs == D
    assert torch.equal(got.d_indptr, want.d_indptr)
    assert torch.equal(got.d_indices[: got.nnz], want.d_indices[: got.nnz])
    assert torch.equal(got.d_perm[: got.S], want.d_perm[: got.S])
    assert torch.equal(got.d_run, want.d_run)
