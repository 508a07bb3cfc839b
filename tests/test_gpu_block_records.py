"""The block gather's records: long lists (many tets around an edge, meshes
that are not conforming, blocks stored different ways round) and value arrays
that only allow narrow loads, each against the packed gather or the aligned
array, bit for bit."""
import numpy as np
import pytest
import torch

from emerge_b200 import _lib as L
from emerge_b200.assembly import DeviceMaterial, DeviceMesh, GpuCSCMapping, _Job, _prec
from emerge_b200.mesh import Nedelec2Field, TetMesh, orient_positive, structured_box

pytestmark = pytest.mark.gpu


def _both(field, precision):
    dm = DeviceMesh(field, None)
    rng = np.random.default_rng(5)
    er = rng.uniform(1, 8, dm.n_tets) * (1 - 1j * rng.uniform(1e-3, 1e-2, dm.n_tets))
    job = _Job(dm, DeviceMaterial(er, None, dm.n_tets, dm.device), _prec(precision))
    out = []
    for layout in ("packed", "block"):
        c = GpuCSCMapping(dm, value_layout=layout)
        out.append(c.assemble_device(job, 1.0 + 0.25j, -2345.5 + 1.25j)[: c.nnz])
        dm.check_status()
    return out


def _fan(n):
    """n tets around one edge: a closed ring of vertices about the axis (0, 1)."""
    a = 2 * np.pi * np.arange(n) / n
    ring = np.stack([np.cos(a), np.sin(a), 0.1 * np.cos(3 * a)])
    nodes = np.concatenate([np.array([[0.0, 0.0], [0.0, 0.0], [-1.0, 1.0]]), ring], axis=1)
    k = np.arange(n)
    tets = np.stack([0 * k, 0 * k + 1, 2 + k, 2 + (k + 1) % n])
    return nodes, orient_positive(nodes, tets)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [3, 7, 8, 9, 16, 17, 33])
def test_self_list_lengths(n, precision):
    p, b = _both(Nedelec2Field(TetMesh(*_fan(n))), precision)
    assert torch.equal(p, b) and torch.count_nonzero(b) > 0


@pytest.mark.parametrize("n", [3, 5])
def test_face_shared_by_more_than_two_tets(n):
    """Not conforming: n tets on one face, so pairs of its entities share n."""
    apex = np.stack([np.linspace(0.2, 0.5, n), np.linspace(0.4, 0.1, n), np.linspace(0.5, 2.0, n)])
    nodes = np.concatenate([np.array([[0.0, 1.0, 0.0], [0.0, 0.0, 1.0], [0.0, 0.0, 0.0]]), apex], axis=1)
    k = np.arange(n)
    tets = orient_positive(nodes, np.stack([0 * k, 0 * k + 1, 0 * k + 2, 3 + k]))
    p, b = _both(Nedelec2Field(TetMesh(nodes, tets)), "fp64")
    assert torch.equal(p, b) and torch.count_nonzero(b) > 0


def test_blocks_stored_different_ways_round():
    """Two tets whose edge numbers disagree about two shared edges' vertices."""
    nodes = np.array([[0.0, 1.0, 0.0, 0.1, 0.2], [0.0, 0.0, 1.0, 0.2, 0.1], [0.0, 0.0, 0.0, 1.0, -1.0]])
    m = TetMesh(nodes, orient_positive(nodes, np.array([[0, 1, 2, 3], [0, 1, 2, 4]]).T))
    t2e = m.tet_to_edge.copy()
    shared = np.intersect1d(t2e[:, 0], t2e[:, 1])
    s0, s1 = (int(np.flatnonzero(t2e[:, 1] == e)[0]) for e in shared[:2])
    t2e[[s0, s1], 1] = t2e[[s1, s0], 1]
    m.tet_to_edge = t2e
    p, b = _both(Nedelec2Field(m), "fp64")
    assert torch.equal(p, b)


@pytest.mark.parametrize("precision,off", [("fp64", 16), ("fp64", 32), ("mixed", 8), ("mixed", 16)])
def test_values_at_any_alignment(precision, off):
    """A value array `off` bytes past a 256-byte boundary."""
    f = Nedelec2Field(TetMesh(*structured_box(5, 3, 4, jitter=0.1, seed=2)))
    dm = DeviceMesh(f, None)
    job = _Job(dm, DeviceMaterial(np.full(dm.n_tets, 2.0 - 0.1j), None, dm.n_tets, dm.device), _prec(precision))
    c = GpuCSCMapping(dm)
    want = c.assemble_device(job, 1.0, -2.0).clone()
    n = c.workspace(job.precision).numel()
    ws = torch.zeros(n + 256, dtype=torch.uint8, device=dm.device)
    ws[off: off + n] = c.workspace(job.precision)[:n]
    got = torch.zeros_like(want)
    L.check(L.lib().emg_gather(L.ctypes.byref(c.plan), L.ptr(c.d_plan), L.ptr(c.d_indptr),
                               L.ctypes.c_void_p(ws.data_ptr() + off), None, job.precision, L.EMG_LAYOUT_BLOCK, 1.0, 0.0,
                               0.0, 0.0, L.ptr(got), None, L.stream_handle(dm.device)))
    assert torch.equal(want, got)
