"""The frequency-sweep form with outputs that allow 32-byte accesses and with
outputs that do not (an odd 16-byte offset, an odd nonzero count): the same
values bit for bit, and those of the formula."""
import ctypes

import numpy as np
import pytest
import torch

from emerge_b200 import _lib as L

pytestmark = pytest.mark.gpu


def _form(K, M, P, coef, out, stride):
    c = np.ascontiguousarray(coef)
    L.check(L.lib().emg_form_sweep(L.ptr(K), L.ptr(M), L.ptr(P), K.numel(), c.ctypes.data_as(ctypes.POINTER(ctypes.c_double)),
                                   c.shape[0], L.ptr(out), stride, L.stream_handle(K.device)))


@pytest.mark.parametrize("nnz", [1, 2, 511, 512, 513, 100_001, 100_002])
@pytest.mark.parametrize("nf,with_p", [(1, False), (5, True), (33, False)])
def test_alignments(nnz, nf, with_p):
    g = torch.Generator(device="cuda").manual_seed(nnz)
    K, M, P = (torch.view_as_complex(torch.randn(nnz, 2, generator=g, device="cuda", dtype=torch.float64)) for _ in range(3))
    P = P if with_p else None
    coef = np.random.default_rng(nf).normal(size=(nf, 6))
    outs = []
    for off, stride in ((0, nnz + nnz % 2), (1, nnz + nnz % 2), (0, nnz + 1 - nnz % 2)):
        buf = torch.zeros(nf * stride + 4, dtype=torch.complex128, device="cuda")
        _form(K, M, P, coef, buf[off:], stride)
        outs.append(torch.stack([buf[off + f * stride: off + f * stride + nnz] for f in range(nf)]))
        assert torch.count_nonzero(buf) == nf * nnz  # nothing beside the rows
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    c = torch.from_numpy(coef).cuda()
    c = torch.complex(c[:, 0::2].contiguous(), c[:, 1::2].contiguous())
    ref = c[:, :1] * K + c[:, 1:2] * M + (c[:, 2:] * P if with_p else 0)
    # four (six) products of N(0, 1) values summed in FP64: a few ulps of their sum of magnitudes
    assert float((outs[0] - ref).abs().max()) <= 1e-14 * 40
