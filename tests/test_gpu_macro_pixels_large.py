"""Macro-pixel correction at magnifications whose map and partial sums together
exceed 48 KB of shared memory, on images of one macro-pixel row (one partial a
phase) and of more, around the sizes where the partials stop being staged.

The map is a compensated float32 sum (relative error 2^-23), divided once and
applied by one IEEE division: 4e-7 of the value bounds it.
"""
import numpy as np
import pytest
import torch

import nanopyx_gb300 as nx
from nanopyx_gb300 import _device, _native as N
from oracle import esrrf_np as O

pytestmark = pytest.mark.gpu
SHAPES = [((1, 78, 156), 78), ((1, 79, 100), 79), ((1, 100, 100), 80), ((2, 100, 163), 80),
          ((1, 90, 180), 90), ((1, 91, 95), 91), ((1, 170, 85), 85)]


@pytest.mark.parametrize("shape,m", SHAPES)
@pytest.mark.parametrize("static", [False, True])
def test_large_maps(shape, m, static):
    x = (np.random.default_rng(m).random(shape) + 0.5).astype(np.float32)
    ref = O.macro_pixel_correct(x, m)
    t = torch.from_numpy(x).cuda()
    if static:
        N.check(N.lib().nx_macro_pixel_correct_static(t.data_ptr(), *shape, m,
                                                      _device.stream_ptr()))
        got = t.cpu().numpy()
    else:
        got = nx.macro_pixel_corrector(t, m).cpu().numpy()
    assert np.abs(got - ref).max() <= 4e-7 * np.abs(ref).max()
