"""The COO -> CSC mapping at the column lengths where its sort changes: slots
per column around each power of two and past the register sort, with
duplicate rows, against a host sort."""
import numpy as np
import pytest

from emerge_b200.heat import GpuCOOMapping

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [[0, 1, 2, 31, 32, 33], [63, 64, 65, 127, 128, 129], [255, 256, 257, 0, 511, 512],
                                     [513, 3], [1024, 1500, 5000]])
@pytest.mark.parametrize("rows_of", ["few", "many"])
def test_column_lengths(lengths, rows_of):
    rng = np.random.default_rng(sum(lengths))
    N = max(len(lengths), 6000)
    cols = np.repeat(np.arange(len(lengths)), lengths)
    rows = rng.integers(0, 7 if rows_of == "few" else N, cols.size)
    p = rng.permutation(cols.size)
    rows, cols = rows[p], cols[p]
    vals = rng.integers(-1000, 1000, cols.size).astype(np.float64)  # sums are exact
    A = GpuCOOMapping.from_rowcol(rows, cols, N).to_csc(vals)
    order = np.lexsort((rows, cols))
    key = cols[order] * N + rows[order]
    first = np.flatnonzero(np.r_[True, key[1:] != key[:-1]])
    assert np.array_equal(A.indices, rows[order][first])
    assert np.array_equal(A.indptr, np.r_[0, np.cumsum(np.bincount(cols[order][first], minlength=N))])
    assert np.array_equal(A.data, np.add.reduceat(vals[order], first))
