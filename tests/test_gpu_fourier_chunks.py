"""The Fourier interpolation in chunks of frames whose number follows the size of the
interpolated square: every frame of a stack longer than the longest chunk (64), or
than the shortest (8, large squares), equals the frame interpolated alone, bit for
bit -- a frame's arithmetic does not depend on its chunk.
"""
import numpy as np
import pytest

import nanopyx_gb300 as nx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,m", [((67, 20, 24), 2), ((65, 1, 3), 2), ((10, 130, 100), 8),
                                     ((18, 250, 256), 4)])
def test_frames_alone(shape, m):
    x = np.random.default_rng(m).poisson(50, shape).astype(np.float32)
    got = nx.fht_space_interpolation(x, m)
    for t in (0, 7, 8, 9, shape[0] - 2, shape[0] - 1):
        np.testing.assert_array_equal(got[t], nx.fht_space_interpolation(x[t], m))
