"""Host arrays of either memory order reach the device whole before the upload
returns, so that any stream may read them."""
import warnings

import numpy as np
import pytest
import torch

from emerge_b200.assembly import _to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["C", "F"])
@pytest.mark.parametrize("host,dtype", [(np.float64, torch.float64), (np.int64, torch.int32)])
def test_upload_is_complete(order, host, dtype):
    """12M values: the device still turns them over when the copy is done."""
    dev = torch.device("cuda", torch.cuda.current_device())
    a = np.asarray(np.arange(12_000_000).reshape(3, -1).astype(host), order=order)
    _to_dev(a, dtype, dev)  # memory and kernels are there
    stream = torch.cuda.Stream(dev)
    with torch.cuda.stream(stream):
        t = _to_dev(a, dtype, dev)
        done = stream.query()
    assert done
    assert t.is_contiguous() and torch.equal(t.cpu(), torch.from_numpy(np.ascontiguousarray(a)).to(dtype))


def test_read_only_array():
    a = np.asfortranarray(np.arange(120_000.0).reshape(3, -1))
    a.setflags(write=False)
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        t = _to_dev(a, torch.float64, torch.device("cuda", torch.cuda.current_device()))
    assert torch.equal(t.cpu(), torch.from_numpy(a.copy()))


@pytest.mark.parametrize("n", [1, 2, 21845, 21846])
def test_either_side_turns_it(n):
    """65,536 values and more are turned over on the device."""
    a = np.asfortranarray(np.arange(3 * n).reshape(3, n))
    t = _to_dev(a, torch.int32, torch.device("cuda", torch.cuda.current_device()))
    assert t.is_contiguous() and torch.equal(t.cpu(), torch.from_numpy(a.copy()).to(torch.int32))
