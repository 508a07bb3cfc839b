"""Topology arrays that list an edge several times in a tet: the block gather's
records of a chunk stay within the chunk's words and apart from each other."""
import numpy as np
import pytest

from emerge_b200.assembly import DeviceMesh, GpuCSCMapping
from emerge_b200.mesh import Nedelec2Field, TetMesh, orient_positive

pytestmark = pytest.mark.gpu
PAIR_WORDS, LONG = 22, 0xFFFFFFFE


def _repeated_edges(n):
    """n tets on one face. Edge e[j] takes all slots of tet j that the edges
    before it leave (at least one), and one slot of every later tet: the lists of
    the face's pairs with them are as long and their first tets as often repeated
    as six slots allow."""
    t = np.linspace(0.0, 1.0, n)
    nodes = np.concatenate([np.array([[0.0, 1.0, 0.0], [0.0, 0.0, 1.0], [0.0, 0.0, 0.0]]),
                            np.stack([0.2 + 0.3 * t, 0.4 - 0.3 * t, 0.5 + t])], axis=1)
    k = np.arange(n)
    m = TetMesh(nodes, orient_positive(nodes, np.stack([0 * k, 0 * k + 1, 0 * k + 2, 3 + k])))
    e = np.linspace(0, m.n_edges - 1, 6).astype(np.int64)
    m.tet_to_edge = np.stack([e[np.minimum(np.arange(6), j)] for j in range(n)], axis=1)
    return Nedelec2Field(m)


@pytest.mark.parametrize("n", [1, 2, 3, 6, 20, 24])
def test_records_of_repeated_edges(n):
    f = _repeated_edges(n)
    c = GpuCSCMapping(DeviceMesh(f, None), value_layout="block")
    blob, p = c.d_plan.cpu().numpy(), c.plan
    n_chunks = -(-f.mesh.n_edges // 8) + -(-f.mesh.n_tris // 8)
    desc = blob[p.off_hoff: p.off_hoff + 64 * n_chunks].reshape(n_chunks, 64)
    words = blob[p.off_pidx: p.off_pidx + 4 * PAIR_WORDS * p.n_items].view(np.uint32)
    longest = 0
    for d in desc:
        I0 = int(d[:4].view(np.int32)[0])
        H, nI = (int(x) for x in d[12:16].view(np.uint16))
        own = words[PAIR_WORDS * I0: PAIR_WORDS * (I0 + nI)]
        assert 2 * H + nI <= own.size
        pairs = own[: 2 * H].reshape(H, 2)
        lists = pairs[(pairs[:, 1] == LONG) & (pairs[:, 0] != 0), 0]
        at, size = (lists & 0xFFFF).astype(int), (lists >> 16).astype(int)
        taken = np.concatenate([np.arange(a, a + s) for a, s in zip(at, size)] + [np.arange(2 * H + nI)])
        assert np.unique(taken).size == taken.size and (taken.size == 0 or taken.max() < own.size)
        for a, s in zip(at, size):
            assert ((own[a: a + s] & 0x7FFFFFFF) < 55 * n).all()
        longest = max([longest, *size])
    assert n <= 2 or longest >= n
