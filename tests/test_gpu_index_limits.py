"""Patterns whose last entry lies at the end of the int32 range: the kernels'
strided walks end at the last entry and the result is right up to it."""
import numpy as np
import pytest
import torch

from emerge_b200 import _lib as L
from emerge_b200.heat import GpuCOOMapping

pytestmark = pytest.mark.gpu
LAST = 2 ** 31 - 1


def _needs(gib):
    if torch.cuda.mem_get_info()[0] < gib << 30:
        pytest.skip(f"needs {gib} GiB of free device memory")


@pytest.mark.parametrize("end", [LAST, LAST - 1, LAST - 7, LAST - 8])
def test_submatrix_at_the_last_nonzero(end):
    """Only the last four columns are kept, so only their rows are read."""
    _needs(12)
    dev = torch.device("cuda", torch.cuda.current_device())
    N = 64
    lengths = [3, 33, 64, 17]
    keep = np.zeros(N, np.uint8)
    keep[60:] = 1
    starts = end - sum(lengths) + np.r_[0, np.cumsum(lengths)]
    indptr = np.r_[np.linspace(0, starts[0], 61).astype(np.int64)[:60], starts].astype(np.int32)
    rng = np.random.default_rng(end % 100)
    rows = [np.sort(rng.permutation(N)[:n]) for n in lengths]
    d_indices = torch.empty(end, dtype=torch.int32, device=dev)
    d_indices[int(starts[0]):] = torch.from_numpy(np.concatenate(rows).astype(np.int32)).to(dev)
    d_indptr, d_keep = torch.from_numpy(indptr).to(dev), torch.from_numpy(keep).to(dev)
    lib, st, sel = L.lib(), L.stream_handle(dev), L.Select()
    L.check(lib.emg_select_init(N, L.ctypes.byref(sel)))
    ws = torch.empty(sel.workspace_bytes, dtype=torch.uint8, device=dev)
    ip = torch.empty(N + 1, dtype=torch.int32, device=dev)
    status = torch.zeros(2, dtype=torch.int64, device=dev)
    L.check(lib.emg_select_build(L.ctypes.byref(sel), L.ptr(d_indptr), L.ptr(d_indices), L.ptr(d_keep), L.ptr(ws),
                                 L.ptr(ip), L.ptr(status), st))
    want = [(r[r >= 60] - 60, starts[j] + np.flatnonzero(r >= 60)) for j, r in enumerate(rows)]
    assert sel.M == 4 and sel.nnz_sel == sum(r.size for r, _ in want)
    ix = torch.empty(max(sel.nnz_sel, 1), dtype=torch.int32, device=dev)
    take = torch.empty(max(sel.nnz_sel, 1), dtype=torch.int32, device=dev)
    L.check(lib.emg_select_finish(L.ctypes.byref(sel), L.ptr(d_indptr), L.ptr(d_indices), L.ptr(d_keep), L.ptr(ws),
                                  L.ptr(ip), L.ptr(ix), L.ptr(take), st))
    assert np.array_equal(ip[:5].cpu().numpy(), np.r_[0, np.cumsum([r.size for r, _ in want])])
    assert np.array_equal(ix[: sel.nnz_sel].cpu().numpy(), np.concatenate([r for r, _ in want]))
    assert np.array_equal(take[: sel.nnz_sel].cpu().numpy(), np.concatenate([t for _, t in want]))


def test_coo_mapping_of_the_most_slots():
    """2^31 - 2 slots, 512 to a column, rows 0 and 1 in turn."""
    _needs(80)
    dev = torch.device("cuda", torch.cuda.current_device())
    S, per = LAST - 1, 512
    N = -(-S // per)
    cols = torch.arange(S, dtype=torch.int32, device=dev)
    rows = cols & 1
    cols >>= 9
    cm = GpuCOOMapping(rows, cols, N)
    del rows, cols
    assert cm.nnz == 2 * N
    d = torch.arange(N + 1, dtype=torch.int32, device=dev)
    assert torch.equal(cm.d_indptr, 2 * d)
    assert torch.equal(cm.d_indices, (torch.arange(2 * N, dtype=torch.int32, device=dev) & 1))
    last = S - (N - 1) * per
    run = torch.arange(2 * N + 1, dtype=torch.int64, device=dev) * (per // 2)
    run[-2:] = torch.tensor([S - last // 2, S])
    assert torch.equal(cm.d_run.to(torch.int64), run)
    tail = np.arange(S - last, S)
    assert np.array_equal(cm.d_perm[S - last: S].cpu().numpy(), np.r_[tail[::2], tail[1::2]])
    A = cm.to_device(torch.ones(S, dtype=torch.float64, device=dev))
    assert bool((A[:-2] == per // 2).all()) and A[-2:].tolist() == [last // 2, last // 2]
