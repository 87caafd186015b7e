"""Macro-pixel correction at the edges of its column vectors and row blocks:
rows that do and do not start on 16-byte boundaries, sizes that are no multiple
of the magnification, more partial sums than the staged map takes, and a base
pointer that only allows scalar access.

The map is a compensated float32 sum (relative error 2^-23), divided once and
applied by one IEEE division: 4e-7 of the value bounds it.
"""
import numpy as np
import pytest
import torch

import nanopyx_gb300 as nx

pytestmark = pytest.mark.gpu


def _expect(x, m):
    out = x.astype(np.float64)
    rows, cols = x.shape[1] // m, x.shape[2] // m
    for s in range(x.shape[0]):
        for py in range(m):
            for px in range(m):
                mean = out[s, py:rows * m:m, px:cols * m:m].mean()
                if mean != 0:
                    out[s, py::m, px::m] /= mean
    return out


@pytest.mark.parametrize("shape,m", [((1, 4, 4), 2), ((3, 15, 20), 5), ((2, 64, 132), 4),
                                     ((2, 66, 131), 3), ((1, 321, 515), 5), ((5, 130, 260), 2),
                                     ((1, 832, 96), 16), ((2, 300, 1036), 5)])
def test_columns_and_rows(shape, m):
    rng = np.random.default_rng(m)
    x = (rng.random(shape) + 0.5).astype(np.float32)
    x[:, ::m, ::m] = 0  # a phase whose mean is 0 is left as it is
    ref = _expect(x, m)
    got = nx.macro_pixel_corrector(torch.from_numpy(x).cuda(), m).cpu().numpy()
    assert np.abs(got - ref).max() <= 4e-7 * np.abs(ref).max()


def test_unaligned_base():
    from nanopyx_gb300 import _device, _native as N

    m, S, H, W = 5, 2, 40, 80
    rng = np.random.default_rng(1)
    x = (rng.random((S, H, W)) + 0.5).astype(np.float32)
    buf = torch.zeros(S * H * W + 1, device="cuda")
    buf[1:] = torch.from_numpy(x).reshape(-1).cuda()
    L = N.lib()
    ws = _device.workspace(L.nx_macro_pixel_workspace_bytes(S, m))
    N.check(L.nx_macro_pixel_correct(buf.data_ptr() + 4, S, H, W, m, ws.data_ptr(), ws.numel(),
                                     _device.stream_ptr()))
    ref = _expect(x, m)
    got = buf[1:].cpu().numpy().reshape(S, H, W)
    assert np.abs(got - ref).max() <= 4e-7 * np.abs(ref).max()
    assert buf[0].item() == 0.0
