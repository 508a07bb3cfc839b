"""Element values in the block layout at any address: stored 32 bytes at a time
where the array allows it and one by one elsewhere, the same values either way,
nothing beside them touched."""
import numpy as np
import pytest
import torch

from emerge_b200 import _lib as L
from emerge_b200.assembly import DeviceMaterial, DeviceMesh, _prec
from emerge_b200.mesh import Nedelec2Field, TetMesh, structured_box

pytestmark = pytest.mark.gpu


def _material(kind, nT):
    rng = np.random.default_rng(3)
    t = np.zeros((3, 3, nT), np.complex128)
    for d in range(3):
        t[d, d] = rng.uniform(1, 4, nT) * (1 - 0.02j)
    if kind == "iso":
        return t[0, 0]
    if kind == "full":  # not symmetric: the second pass adds to the first one's values
        t += rng.uniform(-0.2, 0.2, (3, 3, nT)) * (1 - 0.1j)
    return t


# grids of 6, 18 and 126 tets: a part of a warp, ragged warps and, at 16, 32, 64 or 128 tets per
# warp and CTA, whole ones with a remainder
@pytest.mark.parametrize("grid", [(1, 1, 1), (3, 1, 1), (7, 3, 1)])
@pytest.mark.parametrize("kind", ["iso", "diag", "full"])
@pytest.mark.parametrize("precision,off", [("fp64", 16), ("fp64", 32), ("exact", 48), ("mixed", 8), ("mixed", 16),
                                           ("mixed", 64)])
def test_values_at_any_address(grid, kind, precision, off):
    dm = DeviceMesh(Nedelec2Field(TetMesh(*structured_box(*grid, jitter=0.1, seed=5))), None)
    er = _material(kind, dm.n_tets)
    mat = DeviceMaterial(er, None if kind == "iso" else er, dm.n_tets, dm.device)
    prec = _prec(precision)
    size = 8 if precision == "mixed" else 16

    def values(layout, n, at):
        buf = torch.full((at + n * size + 256,), 0xA5, dtype=torch.uint8, device=dm.device)
        ms = mat.struct()
        L.check(L.lib().emg_element_values(L.ptr(dm.nodes), dm.n_nodes, L.ptr(dm.tets), dm.n_tets, L.ptr(dm.tetids),
                                           dm.n_assy, L.ctypes.byref(ms), prec, L.EMG_OUT_LINCOMB, layout, 1.0, 0.25,
                                           -30.0, 0.5, L.ctypes.c_void_p(buf.data_ptr() + at), L.ptr(dm.status),
                                           L.stream_handle(dm.device)))
        dm.check_status()
        assert bool((buf[:at] == 0xA5).all()) and bool((buf[at + n * size:] == 0xA5).all())
        return buf[at: at + n * size].cpu().numpy().view(np.complex64 if size == 8 else np.complex128)

    got = values(L.EMG_LAYOUT_BLOCK, dm.n_assy * 220, off)
    assert np.array_equal(got, values(L.EMG_LAYOUT_BLOCK, dm.n_assy * 220, 0))
    # and the packed layout's values: block (i, j), value k is its entry (min, max) of the pair's DoFs
    packed = values(L.EMG_LAYOUT_PACKED, dm.n_assy * 210, 0).reshape(-1, 210)
    first = lambda i: i if i < 6 else i + 6
    second = lambda i: i + 6 if i < 6 else i + 10
    at = []
    for i in range(10):
        for j in range(i, 10):
            for x, y in ((first(i), first(j)), (first(i), second(j)), (second(i), first(j)), (second(i), second(j))):
                x, y = min(x, y), max(x, y)
                at.append(x * (41 - x) // 2 + (y - x))
    assert np.array_equal(got.reshape(-1, 220), packed[:, at])
