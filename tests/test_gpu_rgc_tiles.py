"""The tabulated RGC over its tiles of 32 x 8 input pixels (several and partly
filled ones both ways, windows up to the largest table) and at the ends of the
gradients' range, where their squares leave float32.

Oracle: weights and directions are good to 2^-22 and the mean of up to 625 terms
keeps that: 1e-5 of the range.  A gradient's scale changes nothing: its direction
is good to 4 x 2^-24 either way, so the scaled results differ by < 2e-6.
"""
import numpy as np
import pytest

import nanopyx_gb300 as nx
from conftest import rel_err
from oracle import esrrf_np as O

pytestmark = pytest.mark.gpu


def inputs(m, T, h, w):
    rng = np.random.default_rng(10 * m + w)
    gx, gy = (rng.integers(-20, 21, (T, 2 * h * m, 2 * w * m)).astype(np.float32)
              for _ in range(2))
    return gx, gy, rng.integers(50, 150, (T, h * m, w * m)).astype(np.float32)


@pytest.mark.parametrize("m,radius,h,w", [(1, 2.0, 17, 70), (2, 1.5, 8, 32), (2, 1.5, 9, 33),
                                          (2, 6.0, 20, 40), (3, 2.0, 16, 31), (3, 2.5, 9, 33),
                                          (4, 1.0, 10, 65),
                                          (5, 2.0, 9, 35), (8, 1.0, 9, 33)])
@pytest.mark.parametrize("pad", [False, True])
def test_rgc_tiles(m, radius, h, w, pad):
    gx, gy, img = inputs(m, 2, h, w)
    got = nx.RadialGradientConvergence(verbose=False).run(gx, gy, img, m, radius, 2,
                                                          pad_edges=pad)
    ref = O.radial_gradient_convergence(gx, gy, img, m, radius, 2, pad_edges=pad)
    assert rel_err(got, ref) <= 1e-5


@pytest.mark.parametrize("power", [-100, -70, 60, 100])
def test_gradient_scale(power):
    gx, gy, img = inputs(2, 1, 12, 20)
    run = nx.RadialGradientConvergence(verbose=False).run
    ref = run(gx, gy, img, 2, 1.5, 1)
    k = np.float32(2.0 ** power)
    assert rel_err(run(gx * k, gy * k, img, 2, 1.5, 1), ref) <= 2e-6
