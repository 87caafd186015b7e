"""eSRRF-3D in little memory: the least workspace is no larger than one frame's
gradients and values need, a call with it (one frame at a time) gives the bits of frame
pairs, and so does a run whose larger workspace cannot be had.
"""
import ctypes as C

import numpy as np
import pytest
import torch

import nanopyx_gb300 as nx
from nanopyx_gb300 import _device, _native as N, transform

pytestmark = pytest.mark.gpu


def _range(S, H, W, mxy, mz, mode):
    least, pairs = C.c_size_t(), C.c_size_t()
    N.lib().nx_esrrf3d_workspace_range(S, H, W, mxy, mz, mode, C.byref(least), C.byref(pairs))
    return least.value, pairs.value


@pytest.mark.parametrize("mode", [0, 1])
def test_large_volumes_ask_for_the_least(mode):
    S, H, W, mxy, mz = 256, 2048, 1024, 2, 2
    voxels = S * H * W * mxy * mxy
    need = N.lib().nx_esrrf3d_workspace_bytes(S, H, W, mxy, mz, mode)
    before = 16 * voxels + 12 * S * H * W + (4 * voxels * mz if mode else 0)
    assert need <= before
    assert need == _range(S, H, W, mxy, mz, mode)[0]


@pytest.mark.parametrize("radius", [1.5, 2.0])
@pytest.mark.parametrize("mode", ["average", "std"])
@pytest.mark.parametrize("T", [1, 2, 5])
def test_one_frame_at_a_time(radius, mode, T, monkeypatch):
    x = np.random.default_rng(T).poisson(100, (T, 7, 21, 45)).astype(np.float32)
    kw = dict(magnification_xy=2, magnification_z=2, radius=radius, sensitivity=2, mode=mode)
    ref = nx.eSRRF3D_ST(verbose=False).run(x, **kw)
    least, pairs = _range(7, 21, 45, 2, 2, mode == "std")
    asked = []

    def short(nbytes, device=None, **k):
        asked.append(nbytes)
        if nbytes >= pairs:
            raise torch.cuda.OutOfMemoryError("no memory for frame pairs")
        return _device.workspace(nbytes, device, **k)

    monkeypatch.setattr(transform, "workspace", short)
    assert np.array_equal(nx.eSRRF3D_ST(verbose=False).run(x, **kw), ref)
    assert asked == [pairs, least] and least < pairs
