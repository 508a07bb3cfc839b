"""The COO -> CSC mapping where columns hold few slots: a lane sorts a column of up
to 8, its warp the longer ones, from 10 slots per column on a warp each; against a
host sort."""
import numpy as np
import pytest

from emerge_b200 import _lib as L
from emerge_b200.heat import GpuCOOMapping

pytestmark = pytest.mark.gpu


def _check(got, rows, cols, N):
    order = np.lexsort((rows, cols))
    key = cols[order].astype(np.int64) * N + rows[order]
    first = np.flatnonzero(np.r_[True, key[1:] != key[:-1]]) if key.size else np.zeros(0, np.int64)
    assert got.nnz == first.size
    assert np.array_equal(got.indices, rows[order][first])
    assert np.array_equal(got.indptr, np.r_[0, np.cumsum(np.bincount(cols[order][first], minlength=N))])
    assert np.array_equal(got.d_perm[: got.S].cpu().numpy(), order)
    assert np.array_equal(got.d_run.cpu().numpy(), np.r_[first, rows.size])


@pytest.mark.parametrize("lengths", [[0], [1], [7], [8], [9], [0, 8, 9], [7, 8, 9, 31, 32, 33], [0] * 60 + [513, 64, 2]])
@pytest.mark.parametrize("N", [1, 31, 33, 256, 1000])
def test_lengths(lengths, N):
    n = np.resize(lengths, N)
    cols = np.repeat(np.arange(N), n)
    rng = np.random.default_rng(N + sum(lengths))
    rows = rng.integers(0, min(N, 9), cols.size)
    p = rng.permutation(cols.size)
    _check(GpuCOOMapping.from_rowcol(rows[p], cols[p], N), rows[p], cols[p], N)


@pytest.mark.parametrize("D,nT,N", [(1, 500, 300), (2, 50, 300), (3, 200, 400), (10, 4, 100)])
def test_blocks(D, nT, N):
    t2f = np.random.default_rng(D).integers(0, N, (D, nT))
    rows, cols = np.repeat(t2f.T, D, axis=1).ravel(), np.tile(t2f.T, (1, D)).ravel()
    _check(GpuCOOMapping.from_tet_to_field(t2f, N), rows, cols, N)


def test_row_out_of_range():
    import torch

    cols = torch.arange(100, dtype=torch.int32, device="cuda")
    rows = torch.zeros_like(cols)
    rows[57] = 100
    with pytest.raises(L.EmgError):
        GpuCOOMapping(rows, cols, 100)
