"""The Fourier interpolation's matrix products at the edges of their tiles (the
smallest size the 128 x 128 tiles take, partly filled tiles, frames stacked
into one product, more than one chunk of frames) and the tabulated RGC over
phases and windows.

The products are float32 sums of up to 256 terms (error ~ 16 x 2^-24 of the
amplitude) and the rescale adds a few roundings: 1e-5 of the range.  The RGC
test's gradients are exact; its weights and directions are good to 2^-22, the
mean of up to 169 terms keeps that: 1e-5.
"""
import numpy as np
import pytest

import nanopyx_gb300 as nx
from conftest import rel_err
from oracle import esrrf_np as O

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("shape,m", [((1, 9, 16), 2), ((3, 30, 32), 3), ((2, 48, 48), 2),
                                     ((9, 20, 33), 3), ((2, 70, 40), 5), ((2, 130, 257), 2)])
def test_interpolation_tiles(shape, m):
    x = np.random.default_rng(m).poisson(50, shape).astype(np.float32)
    assert rel_err(nx.fht_space_interpolation(x, m), O.fht_space_interpolation(x, m)) <= TOL


@pytest.mark.parametrize("m,radius", [(1, 1.5), (2, 3.0), (3, 0.5), (5, 1.5), (5, 3.0), (8, 1.0)])
@pytest.mark.parametrize("pad", [False, True])
def test_rgc_phases_and_windows(m, radius, pad):
    rng = np.random.default_rng(m)
    T, H, W = 2, 5 * m, 43 * m
    gx, gy = (rng.integers(-20, 21, (T, 2 * H, 2 * W)).astype(np.float32) for _ in range(2))
    img = rng.integers(50, 150, (T, H, W)).astype(np.float32)
    got = nx.RadialGradientConvergence(verbose=False).run(gx, gy, img, m, radius, 2,
                                                          pad_edges=pad)
    ref = O.radial_gradient_convergence(gx, gy, img, m, radius, 2, pad_edges=pad)
    if ref.max() > ref.min():
        assert rel_err(got, ref) <= TOL
    else:
        assert not got.any()
