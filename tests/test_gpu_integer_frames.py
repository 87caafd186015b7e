"""Camera integers through the host-buffer path: every pixel type that travels
as it is, types and layouts that do not, and conversion lengths around the
vector width.  The conversion is exact, so results equal those of the float32
stack bit for bit.
"""
import numpy as np
import pytest
import torch

import nanopyx_gb300 as nx
from nanopyx_gb300 import _device, _native as N

pytestmark = pytest.mark.gpu


def _stack(dtype, T=23, H=20, W=37):
    rng = np.random.default_rng(3)
    hi = 120 if np.dtype(dtype).itemsize == 1 else 30000
    x = rng.integers(0, hi, (T, H, W))
    if np.issubdtype(np.dtype(dtype), np.signedinteger):
        x -= hi // 2
    return x.astype(dtype)


@pytest.mark.parametrize("dtype", ["u1", "i1", "u2", "i2", ">u2", "i4", "f8"])
@pytest.mark.parametrize("layout", ["c", "strided", "one_frame"])
def test_same_as_float32(dtype, layout):
    x = _stack(dtype)
    if layout == "strided":
        x = x[::2, 1:, ::-1]
    elif layout == "one_frame":
        x = x[0]
    kw = dict(frames_per_timepoint=10, temporal_correlation="AVG")
    got = nx.eSRRF(x, **kw)
    assert np.array_equal(got, nx.eSRRF(np.ascontiguousarray(x.astype(np.float32)), **kw))


def test_wrong_rank_is_refused():
    with pytest.raises(ValueError):
        nx.eSRRF(np.zeros((2, 3, 4, 5), np.uint16))


@pytest.mark.parametrize("dtype", [np.uint8, np.int8, np.uint16, np.int16])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 2047, 4104])
@pytest.mark.parametrize("offset", [0, 1])
def test_conversion_lengths_and_alignment(dtype, n, offset):
    info = np.iinfo(dtype)
    h = np.random.default_rng(n).integers(info.min, info.max + 1, n + offset).astype(dtype)
    d = torch.from_numpy(h.view(np.int8)).cuda()
    out = torch.full((n + 1,), -1.0, device="cuda")
    N.check(N.lib().nx_to_float32(d.data_ptr() + offset * h.itemsize,
                                  N.PIXEL_TYPES[h.dtype.char], n, out.data_ptr(),
                                  _device.stream_ptr()))
    assert np.array_equal(out[:n].cpu().numpy(), h[offset:].astype(np.float32))
    assert out[n].item() == -1.0
